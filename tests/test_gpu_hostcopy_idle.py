"""A download behind long work on the stream: the copying threads start when the data is about to come, so
the wait costs one core at most, not one for each of them (GPU)."""
import time

import numpy as np
import pytest

import flowpro_v2_b200 as fg
from flowpro_v2_b200 import meshgen
from tests import cases

pytestmark = pytest.mark.gpu


def test_threads_do_not_wait_for_earlier_work():
    m = meshgen.bump_channel(nx=548, ny=183, seed=1, wall=meshgen.WALL)
    tt = fg.create_neighbor_matrix(2, m.elements, m.boundary)
    g = fg.GpuMesh(cases.ns_props(3), m.vertices, m.elements, tt, m.wall_distance)
    g.limiter()
    want = g.get_state()
    g._check(fg.lib().fp_residual_repeat(g.ctx, 3000))  # about a thousand launches are still queued when it returns
    wall, cpu = time.perf_counter(), time.process_time()
    got = g.get_state()
    wall, cpu = time.perf_counter() - wall, time.process_time() - cpu
    assert np.array_equal(got, want)
    assert wall > 0.03  # there was something to wait for
    # the waiting core, and eight threads for the 38 MB (under 5 ms each)
    assert cpu < 1.5 * wall + 0.04, (cpu, wall)
    g.close()
