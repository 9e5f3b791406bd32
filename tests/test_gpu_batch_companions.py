"""A merged case does not depend on the cases it is merged with: the same two cases beside a small and beside
a large third one give the same states and solver records, bit for bit (GPU)."""
import numpy as np
import pytest

import flowpro_v2_b200 as fg
from flowpro_v2_b200 import meshgen
from tests import cases

pytestmark = pytest.mark.gpu


def _case(nx, ny, p_out, order, seed):
    m = meshgen.bump_channel(nx=nx, ny=ny, height=0.08, seed=seed, wall=meshgen.INVISCID_WALL)
    props = dict(cases.euler_props(order), pOut=p_out, dampTol=3)
    return props, m.vertices, m.elements, fg.create_neighbor_matrix(2, m.elements, m.boundary), None


@pytest.mark.parametrize("order,large", [(2, (360, 120)), (3, (360, 120))])
def test_values_do_not_depend_on_companions(order, large):
    got = []
    for third in ((20, 8), large):
        b = fg.GpuBatch([_case(60, 21, 0.84, order, 1), _case(*third, 0.9, order, 2), _case(90, 31, 0.87, order, 3)])
        out, status = b.solve(steps=5, cfl=4.0, vary_cfl=1, max_cfl=1e5, linear_tol=1e-2, preconditioner="blockilu0",
                              jacobian=fg.JAC_MATRIXFREE, precision=fg.FP32, jac_lag=3, restart=40, max_restarts=5)
        assert np.all(status == 0)
        got.append([(out[i], b.case_state(i)) for i in (0, 2)])
        b.close()
    for (o0, w0), (o1, w1) in zip(*got):
        assert np.array_equal(o0, o1)
        assert np.array_equal(w0, w1)
