"""State transfers between pageable host memory and the device around the sizes where they go through
the staging slots (2 MB and up, in chunks of 2 MB): every byte arrives, from several threads at once
too (GPU)."""
import threading

import numpy as np
import pytest

import flowpro_v2_b200 as fg
from tests import cases

pytestmark = pytest.mark.gpu


def _mesh(nx, ny):
    m, tt = cases.channel(nx, ny, seed=3)
    return fg.GpuMesh(cases.euler_props(3), m.vertices, m.elements, tt, m.wall_distance)


def _roundtrip(g, seed, wide=True):
    rng = np.random.default_rng(seed)
    for which in (0, 1, 2):
        W = rng.standard_normal((g.n_elem, g.nb))
        if not wide:  # an array that does not start at a page
            W = np.concatenate([np.zeros(7), W.ravel()])[7:].reshape(g.n_elem, g.nb)
        g.set_state(W, which)
        assert np.array_equal(g.get_state(which), W)


# 24 unknowns, 192 bytes an element: 2 MB are 10,923 elements; one below, one above, several ragged
# chunks, more chunks than slots
@pytest.mark.parametrize("nx,ny", [(73, 74), (74, 74), (110, 109), (150, 190), (301, 211)])
def test_roundtrip(nx, ny):
    g = _mesh(nx, ny)
    _roundtrip(g, nx)
    _roundtrip(g, ny, wide=False)
    g.close()


def test_roundtrip_from_several_threads():
    gs = [_mesh(120, 100) for _ in range(3)]
    bad = []

    def work(i):
        try:
            for k in range(4):
                _roundtrip(gs[i], 10 * i + k)
        except Exception as e:  # noqa: BLE001
            bad.append(e)

    ts = [threading.Thread(target=work, args=(i,)) for i in range(3)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad
    for g in gs:
        g.close()
