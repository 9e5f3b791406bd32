"""The streamed block ILU(0) application on meshes on which a thread block takes more positions than its
ring has slots (64), for every number of elements in flight and for defaults that do not divide 64
(GPU).

The values must not depend on the elements in flight by a bit, and equal the register kernel's to
rounding: both precondition the same system, solved to a preconditioned residual of 1e-12, so the
solutions agree to 1e-9 of the largest entry, as on the small meshes of test_gpu_ilu_ring.py.  In a
batch the positions of finished cases pass through the ring without blocks of their own."""
import numpy as np
import pytest

import flowpro_v2_b200 as fg
from flowpro_v2_b200 import meshgen
from tests import cases

pytestmark = pytest.mark.gpu

# props, mesh: 265 positions a thread block (2 elements in flight by default), 68 (3), 327 (3), 118 (4)
KINDS = {
    12: (lambda: cases.euler_props(2), lambda: cases.channel(140, 140, seed=4)),
    20: (lambda: cases.euler3_props(2), lambda: cases.box(14, 12, 10, seed=4)),
    40: (lambda: cases.euler_props(4), lambda: cases.channel(110, 110, seed=4)),
    50: (lambda: cases.euler3_props(3), lambda: cases.box(12, 11, 11, seed=4)),
}


@pytest.mark.parametrize("precision", [fg.FP64, fg.FP32])
@pytest.mark.parametrize("kind", sorted(KINDS))
def test_more_positions_than_slots(kind, precision):
    m, tt = KINDS[kind][1]()
    g = fg.GpuMesh(KINDS[kind][0](), m.vertices, m.elements, tt, m.wall_distance)
    assert g.nb == kind
    rng = np.random.default_rng(kind)
    W = cases.perturbed(g.get_state(0), g.n_basis, g.n_eqs, rng, 0.02)
    for which in (0, 1, 2):
        g.set_state(W, which)
    g.limiter()
    fg.JacobiAssembler(g).assemble_exact(3.0 * g.time_step_bound(), -1)
    rhs = rng.standard_normal(W.shape)
    opts = dict(preconditioner="blockilu0", precision=precision, restart=40, max_restarts=5, tol=1e-12)
    ok, x0, it0 = g.block_solve(rhs, **opts)
    assert ok
    tried = 0
    for variant in (2, 3, 4, 5, 6):
        g.set_ilu_sweep(variant)
        try:
            ok, x, its = g.block_solve(rhs, **opts)
        except fg.FlowGpuError:  # more than the block size allows
            continue
        assert ok and its == it0 and np.array_equal(x, x0), variant
        tried += 1
    assert tried >= 2
    g.set_ilu_sweep(1)
    ok, x1, it1 = g.block_solve(rhs, **opts)
    assert ok and abs(it1 - it0) <= 1
    assert np.max(np.abs(x0 - x1)) <= 1e-9 * np.max(np.abs(x1))
    g.close()


@pytest.mark.parametrize("order,n,most", [(2, 8, 9000), (4, 4, 7000)])
def test_batch_with_finished_cases(order, n, most):
    """cases of uneven size and Mach number: their linear solves end at different iterations, and the
    target stops some of them early"""
    built = []
    for c in meshgen.serving_cases(n, seed=11, min_elements=3000, max_elements=most):
        m = meshgen.bump_channel(nx=c["nx"], ny=c["ny"], height=c["height"], seed=c["seed"], wall=meshgen.INVISCID_WALL)
        props = dict(cases.euler_props(order), pOut=c["pOut"])
        built.append((props, m.vertices, m.elements, fg.create_neighbor_matrix(2, m.elements, m.boundary), None))
    got = []
    for variant in (0, 2, 3, 4):
        b = fg.GpuBatch(built)
        b._check(fg.lib().fp_set_ilu_sweep(b.ctx, variant))
        out, status = b.solve(steps=6, cfl=4.0, vary_cfl=1, max_cfl=1e5, linear_tol=1e-6, preconditioner="blockilu0",
                              jacobian=fg.JAC_MATRIXFREE, precision=fg.FP32, jac_lag=3, restart=40, max_restarts=5,
                              target_residuum=0.3)
        got.append((out, status, [b.case_state(i) for i in range(n)]))
        b.close()
    assert np.all(got[0][1] == 0)
    assert len(set(got[0][0][:, 6])) > 1  # iterations differ from case to case
    for out, status, W in got[1:]:
        assert np.array_equal(out, got[0][0]) and np.array_equal(status, got[0][1])
        assert all(np.array_equal(a, c) for a, c in zip(W, got[0][2]))
