"""A linear solve that meets a non-finite value fails and leaves no trace: the next solve on the same context
gives what it gave before, bit for bit (GPU).  The numbers of elements are not multiples of 128, so the
vectors have padding."""
import numpy as np
import pytest

import flowpro_v2_b200 as fg
from tests import cases

pytestmark = pytest.mark.gpu


def _case():
    m, tt = cases.channel(10, 5, seed=5)
    g = fg.GpuMesh(cases.euler_props(2), m.vertices, m.elements, tt, m.wall_distance)
    W = cases.perturbed(g.get_state(0), g.n_basis, g.n_eqs, np.random.default_rng(5), 0.01)
    for which in (0, 1, 2):
        g.set_state(W, which)
    g.limiter()
    bad = W.copy()
    bad[7, 0] = np.nan
    return g, W, bad


@pytest.mark.parametrize("prec", ["blockjacobi", "blockilu0"])
def test_matrix_free_solve_after_a_non_finite_state(prec):
    g, W, bad = _case()
    dt = 5.0 * g.time_step_bound()
    fg.JacobiAssembler(g).assemble_preconditioner(dt, -1, prec, fg.FP32)
    ls = fg.LinearSolver(g, prec, precision=fg.FP32, jacobian=fg.JAC_MATRIXFREE, restart=30, max_restarts=5, tol=1e-8)
    ok, want = ls.solve()
    assert ok
    g.set_state(bad)
    ok, _ = ls.solve()  # the preconditioner is kept, the tangent is not a number
    assert not ok
    g.set_state(W)
    ok, x = ls.solve()
    assert ok and np.array_equal(x, want)
    g.close()


def test_assembled_solve_after_non_finite_blocks():
    g, W, bad = _case()
    dt = 0.5 * g.time_step_bound()
    asm = fg.JacobiAssembler(g)
    ls = fg.LinearSolver(g, "none", restart=60, max_restarts=10, tol=1e-8)
    asm.assemble(dt, -1)
    ok, want = ls.solve()
    assert ok
    g.set_state(bad)
    asm.assemble(dt, -1)
    ok, _ = ls.solve()
    assert not ok
    g.set_state(W)
    asm.assemble(dt, -1)
    ok, x = ls.solve()
    assert ok and np.array_equal(x, want)
    g.close()
