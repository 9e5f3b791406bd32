"""Block-Jacobi inverses and transposed products at every number of unknowns (GPU).

The inverses are seen through GMRES with block Jacobi against the block ILU(0) solution (another
inversion code); the transposed product through the identity <A^T y, x> = <y, A x>, which the solves of
both systems give: <x1, b2> = <A^-1 b1, b2> = <b1, A^-T b2> = <b1, x2>.  Solutions converged to 1e-12 (times
the condition of the preconditioned operator) give both to 1e-8."""
import numpy as np
import pytest

import flowpro_v2_b200 as fg
from tests.test_gpu_ilu_factor import KINDS, _assembled

pytestmark = pytest.mark.gpu


def _dims(kind, k):
    # one element range below, at and above the elements a thread block inverts
    return [(1, 1), (3, 3), (17, 9)][k] if KINDS[kind][1] == "channel" else [(1, 1, 1), (2, 1, 1), (5, 4, 3)][k]


@pytest.mark.parametrize("precision", [fg.FP64, fg.FP32])
@pytest.mark.parametrize("size", [0, 1, 2])
@pytest.mark.parametrize("kind", sorted(KINDS))
def test_block_jacobi_and_transposed_solve(kind, size, precision):
    g, b1 = _assembled(kind, _dims(kind, size))
    b2 = np.random.default_rng(99).standard_normal(b1.shape)
    opts = dict(restart=150, max_restarts=4, tol=1e-12)
    ok1, x1, _ = g.block_solve(b1, preconditioner="blockjacobi", precision=precision, **opts)
    ok2, x2, _ = g.block_solve(b2, transpose=True, preconditioner="blockjacobi", precision=precision, **opts)
    ok3, x3, _ = g.block_solve(b1, preconditioner="blockilu0", precision=fg.FP64, **opts)
    assert ok1 and ok2 and ok3
    assert np.max(np.abs(x1 - x3)) <= 1e-8 * np.max(np.abs(x3))
    scale = np.linalg.norm(x1) * np.linalg.norm(b2)
    assert abs(np.vdot(x1, b2) - np.vdot(b1, x2)) <= 1e-8 * scale
    g.close()
