"""The block ILU(0) factorisation at every number of unknowns it is compiled for (GPU).

The factors are not exported; they are seen through a solve.  On a chain of elements without a cycle
(a strip of two triangles, a tetrahedron) block ILU(0) has no fill to drop, so it is the exact block LU
of the matrix and GMRES preconditioned with it converges in two iterations: the second one is there
because a computed inverse is off by the block's condition times the precision.  On general meshes
the solution preconditioned with it equals the block-Jacobi one (another factorisation code) to the
GMRES tolerance times the condition of the operator: 1e-8 of the largest entry at 1e-12."""
import numpy as np
import pytest

import flowpro_v2_b200 as fg
from flowpro_v2_b200 import meshgen
from tests import cases

pytestmark = pytest.mark.gpu

# unknowns per element: props, mesh
KINDS = {
    1: (lambda: cases.scalar_props(1), "channel"),
    3: (lambda: cases.scalar_props(2), "channel"),
    4: (lambda: cases.euler_props(1), "channel"),
    5: (lambda: cases.euler3_props(1), "box"),
    6: (lambda: cases.scalar_props(3), "channel"),
    9: (lambda: cases.adiabatic_props(2), "channel"),
    10: (lambda: cases.scalar_props(4), "channel"),
    12: (lambda: cases.euler_props(2), "channel"),
    15: (lambda: cases.sa_props(2), "channel"),
    16: (lambda: cases.adiabatic_props(2, 3), "box"),
    18: (lambda: cases.adiabatic_props(3), "channel"),
    20: (lambda: cases.euler3_props(2), "box"),
    24: (lambda: cases.euler_props(3), "channel"),
    30: (lambda: cases.sa_props(3), "channel"),
    40: (lambda: cases.euler_props(4), "channel"),
    50: (lambda: cases.euler3_props(3), "box"),
}


def _assembled(kind, dims):
    props = KINDS[kind][0]()
    sa = props["model"] == "SpalartAllmaras"
    wall = meshgen.WALL if sa else meshgen.INVISCID_WALL
    m, tt = cases.channel(*dims, seed=6, wall=wall) if KINDS[kind][1] == "channel" else cases.box(*dims, seed=6)
    if sa:
        m.wall_distance[:] = np.maximum(m.wall_distance, 1e-3)
    g = fg.GpuMesh(props, m.vertices, m.elements, tt, m.wall_distance)
    assert g.nb == kind
    rng = np.random.default_rng(kind)
    w0 = g.get_state(0)
    W = cases.perturbed(w0, g.n_basis, g.n_eqs, rng, 0.01) if np.any(w0) else 0.1 * rng.standard_normal(w0.shape)
    for which in (0, 1, 2):
        g.set_state(W, which)
    g.limiter()
    dt = 2.0 * g.time_step_bound() if np.any(w0) else 1e-2
    fg.JacobiAssembler(g).assemble_exact(dt, -1)
    return g, rng.standard_normal(W.shape)


@pytest.mark.parametrize("kind", sorted(k for k in KINDS if KINDS[k][1] == "channel"))
def test_exact_on_a_chain(kind):
    g, rhs = _assembled(kind, (1, 1))  # two triangles
    ok, x, its = g.block_solve(rhs, preconditioner="blockilu0", precision=fg.FP64, restart=10, max_restarts=1, tol=1e-10)
    assert ok and its <= 2
    g.close()


@pytest.mark.parametrize("precision", [fg.FP64, fg.FP32])
@pytest.mark.parametrize("kind", sorted(KINDS))
def test_solution_equals_block_jacobi(kind, precision):
    # ragged numbers of elements, several rows per thread block at the largest sizes
    dims = (23, 11) if KINDS[kind][1] == "channel" else (9, 6, 5)
    g, rhs = _assembled(kind, dims)
    ok0, x0, _ = g.block_solve(rhs, preconditioner="blockjacobi", precision=fg.FP64, restart=100, max_restarts=5, tol=1e-12)
    ok1, x1, _ = g.block_solve(rhs, preconditioner="blockilu0", precision=precision, restart=100, max_restarts=5, tol=1e-12)
    assert ok0 and ok1
    assert np.max(np.abs(x0 - x1)) <= 1e-8 * np.max(np.abs(x0))
    g.close()
