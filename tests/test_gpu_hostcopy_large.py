"""State transfers between pageable host memory and the device around the sizes from which they go through
the staging slots (20 MB down, 32 MB up, chunks of 2 MB): every byte arrives, from several threads at
once too (GPU)."""
import threading

import pytest

from tests.test_gpu_hostcopy import _mesh, _roundtrip

pytestmark = pytest.mark.gpu


# 24 unknowns, 192 bytes an element: 20 MB are 109,227 elements, 32 MB 174,763; below, at and above each, and
# a ragged number of chunks
@pytest.mark.parametrize("nx,ny", [(300, 182), (234, 234), (257, 256), (295, 296), (296, 296), (421, 371)])
def test_roundtrip(nx, ny):
    g = _mesh(nx, ny)
    _roundtrip(g, nx)
    _roundtrip(g, ny, wide=False)
    g.close()


def test_roundtrip_from_several_threads():
    gs = [_mesh(310, 300) for _ in range(3)]
    bad = []

    def work(i):
        try:
            for k in range(2):
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
