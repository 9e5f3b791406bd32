"""Exact element blocks and the adjoint product, formed from the flux Jacobians at the quadrature points,
against the tangent operator (another kernel: forward mode through the face and element passes), for every
compiled model and order, with and without artificial viscosity, and numbers of elements that leave a
thread block's last elements empty (GPU).

Both are sums of at most a few thousand FP64 products per entry, in different orders: they agree to the
rounding of such a sum, 1e-11 of the largest entry."""
import numpy as np
import pytest

import flowpro_v2_b200 as fg
from flowpro_v2_b200 import meshgen
from tests import cases

pytestmark = pytest.mark.gpu

MODELS = {
    "euler": (lambda o: cases.euler_props(o), "channel", (1, 2, 3, 4)),
    "vanleer": (lambda o: cases.euler_props(o, flux="vanLeer"), "channel", (3,)),
    "ns": (lambda o: cases.ns_props(o, reynolds=500.0), "channel", (1, 2, 3, 4)),
    "sa": (lambda o: cases.sa_props(o), "channel", (2, 3, 4)),
    "adiabatic": (lambda o: cases.adiabatic_props(o), "channel", (1, 2, 3, 4)),
    "scalar": (lambda o: cases.scalar_props(o), "channel", (1, 2, 3, 4)),
    "scalar_diff": (lambda o: cases.scalar_props(o, 0.1), "channel", (2, 3)),
    "euler3": (lambda o: cases.euler3_props(o), "box", (1, 2, 3)),
    "ns3": (lambda o: cases.ns3_props(o), "box", (1, 2, 3)),
    "adiabatic3": (lambda o: cases.adiabatic_props(o, 3), "box", (2, 3)),
}
CASES = [(k, o, d) for k, v in MODELS.items() for o in v[2] for d in (False, True) if not (d and (o == 1 or "scalar" in k))]


@pytest.mark.parametrize("kind,order,damp", CASES)
def test_blocks_and_adjoint_product_match_the_tangent(kind, order, damp):
    props = MODELS[kind][0](order)
    viscous = kind in ("ns", "sa", "ns3")
    wall = meshgen.WALL if viscous else meshgen.INVISCID_WALL
    if damp:
        props["dampTol"] = 3.0
    m, tt = cases.channel(7, 5, seed=order, wall=wall) if MODELS[kind][1] == "channel" else cases.box(3, 2, 2, seed=2, wall=wall)
    if kind == "sa":
        m.wall_distance[:] = np.maximum(m.wall_distance, 1e-3)
    g = fg.GpuMesh(props, m.vertices, m.elements, tt, m.wall_distance)
    rng = np.random.default_rng(order)
    w0 = g.get_state(0)
    W = cases.perturbed(w0, g.n_basis, g.n_eqs, rng, 0.1 if damp else 0.02) if np.any(w0) else 0.1 * rng.standard_normal(w0.shape)
    for which in (0, 1, 2):
        g.set_state(W, which)
    g.limiter()
    if damp:
        assert np.max(g.limiter_values()[0]) > 0
    v, lam = rng.standard_normal(W.shape), rng.standard_normal(W.shape)
    jv, jl = g.jvp(v), g.vjp(lam)
    scale = np.linalg.norm(jv) * np.linalg.norm(lam)
    assert abs(np.vdot(lam, jv) - np.vdot(jl, v)) <= 1e-11 * scale
    asm = fg.JacobiAssembler(g)
    asm.assemble_exact(0.0, -1)  # the steady operator -dR/dW
    diag, neigh, _ = asm.blocks()
    Av = np.einsum("eij,ei->ej", diag, v)
    At = np.einsum("eij,ej->ei", diag, lam)
    for k in range(tt.shape[1]):
        e = np.nonzero(tt[:, k] >= 0)[0]
        Av[e] += np.einsum("eij,ei->ej", neigh[e, k], v[tt[e, k]])
        np.add.at(At, tt[e, k], np.einsum("eij,ej->ei", neigh[e, k], lam[e]))
    assert np.max(np.abs(Av + jv)) <= 1e-11 * np.max(np.abs(jv))
    assert np.max(np.abs(At + jl)) <= 1e-11 * np.max(np.abs(jl))
    g.close()


@pytest.mark.parametrize("kind,order,damp", CASES)
def test_finite_difference_blocks_match_differences_of_the_residual(kind, order, damp):
    """A column of the finite-difference blocks against the difference of two residuals of the whole mesh
    (the face and element passes).  Both round sums of a few dozen terms of the size |A| |W|, and the
    difference is divided by h: 64 x 2^-52 / h = 1.4e-6 of that size."""
    props = MODELS[kind][0](order)
    wall = meshgen.WALL if kind in ("ns", "sa", "ns3") else meshgen.INVISCID_WALL
    if damp:
        props["dampTol"] = 3.0
    m, tt = cases.channel(7, 5, seed=order, wall=wall) if MODELS[kind][1] == "channel" else cases.box(3, 2, 2, seed=2, wall=wall)
    if kind == "sa":
        m.wall_distance[:] = np.maximum(m.wall_distance, 1e-3)
    g = fg.GpuMesh(props, m.vertices, m.elements, tt, m.wall_distance)
    rng = np.random.default_rng(order)
    w0 = g.get_state(0)
    W = cases.perturbed(w0, g.n_basis, g.n_eqs, rng, 0.1 if damp else 0.02) if np.any(w0) else 0.1 * rng.standard_normal(w0.shape)
    for which in (0, 1, 2):
        g.set_state(W, which)
    g.limiter()
    asm = fg.JacobiAssembler(g, bdf_order=1)
    asm.assemble(0.0, -1)  # no mass term
    diag, neigh, _ = asm.blocks()
    h = 1e-8
    tol = 64 * 2.0 ** -52 / h * max(np.max(np.abs(diag)), np.max(np.abs(neigh))) * max(1.0, np.max(np.abs(W)))
    R = g.residuum(W)
    last = len(tt) - 1  # the last element: its block is partly empty
    for e, i in [(0, 0), (last, W.shape[1] - 1)] + [(int(rng.integers(len(tt))), int(rng.integers(W.shape[1]))) for _ in range(4)]:
        Wp = W.copy()
        Wp[e, i] += h
        d = (g.residuum(Wp) - R) / h
        want = np.zeros_like(d)
        want[e] = -diag[e, i]
        for k in range(tt.shape[1]):  # neighbours whose face k is e's
            for f in np.nonzero(tt[:, k] == e)[0]:
                want[f] -= neigh[f, k, i]
        assert np.max(np.abs(d - want)) <= tol
    g.close()
