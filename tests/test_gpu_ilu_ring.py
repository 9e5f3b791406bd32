"""The streamed block ILU(0) application at every number of unknowns it is compiled for, against the
register kernel (GPU).

Both apply the same factors; they add a row's products in different orders.  GMRES is left with a
preconditioner that is equal to rounding, so the solutions of the same system, each converged to a
preconditioned residual of 1e-12, agree to a small multiple of that times the condition of the
preconditioned operator: 1e-9 of the largest entry is taken.  The elements in flight per thread
block (fp_set_ilu_sweep 2 .. 6) must not change a bit."""
import numpy as np
import pytest

import flowpro_v2_b200 as fg
from flowpro_v2_b200 import meshgen
from tests import cases

pytestmark = pytest.mark.gpu

# unknowns per element: props, mesh (channel or box)
KINDS = {
    4: (lambda: cases.euler_props(1), "channel"),
    6: (lambda: cases.scalar_props(3), "channel"),
    10: (lambda: cases.scalar_props(4), "channel"),
    12: (lambda: cases.euler_props(2), "channel"),
    16: (lambda: cases.adiabatic_props(2, 3), "box"),
    18: (lambda: cases.adiabatic_props(3), "channel"),
    20: (lambda: cases.euler3_props(2), "box"),
    24: (lambda: cases.ns_props(3, reynolds=500.0), "channel"),
    30: (lambda: cases.adiabatic_props(4), "channel"),
    40: (lambda: cases.euler_props(4), "channel"),
    50: (lambda: cases.euler3_props(3), "box"),
}


def _solve(kind, mesh, size, precision, variant):
    props = KINDS[kind][0]()
    wall = meshgen.WALL if str(props.get("isFlowViscous")) == "true" else meshgen.INVISCID_WALL
    m, tt = cases.channel(*size, seed=4, wall=wall) if mesh == "channel" else cases.box(*size, seed=4)
    g = fg.GpuMesh(props, m.vertices, m.elements, tt, m.wall_distance)
    assert g.nb == kind
    g.set_ilu_sweep(variant)
    rng = np.random.default_rng(kind)
    w0 = g.get_state(0)
    W = cases.perturbed(w0, g.n_basis, g.n_eqs, rng, 0.02) if np.any(w0) else 0.1 * rng.standard_normal(w0.shape)
    for which in (0, 1, 2):
        g.set_state(W, which)
    g.limiter()
    dt = 3.0 * g.time_step_bound() if np.any(w0) else 1e-2
    fg.JacobiAssembler(g).assemble_exact(dt, -1)
    rhs = rng.standard_normal(W.shape)
    ok, x, its = g.block_solve(rhs, preconditioner="blockilu0", precision=precision, restart=40, max_restarts=5, tol=1e-12)
    g.close()
    return ok, x, its


# fewer elements than thread blocks, a ragged number, and (3D) several positions per block
SIZES = {"channel": [(2, 2), (13, 7), (41, 23)], "box": [(2, 1, 1), (5, 3, 3), (9, 7, 5)]}


@pytest.mark.parametrize("precision", [fg.FP64, fg.FP32])
@pytest.mark.parametrize("size", [0, 1, 2])
@pytest.mark.parametrize("kind", sorted(KINDS))
def test_streamed_sweep_matches_register_sweep(kind, size, precision):
    mesh = KINDS[kind][1]
    dims = SIZES[mesh][size]
    ok0, x0, it0 = _solve(kind, mesh, dims, precision, 0)
    ok1, x1, it1 = _solve(kind, mesh, dims, precision, 1)
    assert ok0 and ok1
    assert abs(it0 - it1) <= 1
    assert np.max(np.abs(x0 - x1)) <= 1e-9 * np.max(np.abs(x1))
    ok2, x2, it2 = _solve(kind, mesh, dims, precision, 2)  # one element in flight per thread block
    assert ok2 and it2 == it0 and np.array_equal(x2, x0)
