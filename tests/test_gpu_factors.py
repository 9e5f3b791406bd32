"""The preconditioners' values, at every compiled number of unknowns: one application against numpy's inverses
and block ILU(0) of the exported blocks (GPU).

One iteration of GMRES from zero gives a multiple of M^-1 b, so the solution's direction is the
application.  Tolerances: the same algorithm in numpy at single precision, blocks rounded to it, is off by
e32 from the double one; both are first-order rounding errors of the same recurrences (other pivot
scaling, other order of sums), so the device may be off by 20 e32 in FP32 and by 20 e32 2^-29 + 1e-13 in
FP64.  One row's update dropped from the factorisation shows at 1e-3 (one unknown) to 3e-1.

The updates of a row's off-diagonal blocks exist only where two neighbours of an element are neighbours
themselves: in the stars, elements around one inner vertex that all touch one another."""
import numpy as np
import pytest

import flowpro_v2_b200 as fg
from flowpro_v2_b200 import meshgen
from tests import cases
from tests.test_gpu_ilu_factor import KINDS, _assembled

pytestmark = pytest.mark.gpu


def _blocks(g, asm, dtype):
    diag, neigh, _ = asm.blocks()
    return np.swapaxes(diag, 1, 2).astype(dtype), np.swapaxes(neigh, 2, 3).astype(dtype)


def _jacobi(D, b):
    return np.einsum("erc,ec->er", np.linalg.inv(D).astype(np.float64), b)


def _ilu0(D, N, tt, rank, b):
    """y = U^-1 L^-1 b, factors in the dtype of the blocks, the application in double"""
    D, N = D.copy(), N.copy()
    ne, nf = tt.shape
    order = np.argsort(rank)
    face = [{int(j): f for f, j in enumerate(tt[i]) if j > -1} for i in range(ne)]
    for i in order:
        for k in sorted((j for j in face[i] if rank[j] < rank[i]), key=lambda j: rank[j]):
            L = N[i, face[i][k]] @ D[k]  # D[k]: inverse of the finished row
            N[i, face[i][k]] = L
            D[i] -= L @ N[k, face[k][i]]
            for j in face[i]:
                if rank[j] > rank[k] and j in face[k]:
                    N[i, face[i][j]] -= L @ N[k, face[k][j]]
        D[i] = np.linalg.inv(D[i])
    D, N = D.astype(np.float64), N.astype(np.float64)
    y = b.copy()
    for i in order:
        for j, f in face[i].items():
            if rank[j] < rank[i]:
                y[i] -= N[i, f] @ y[j]
    x = np.zeros_like(y)
    for i in order[::-1]:
        s = y[i].copy()
        for j, f in face[i].items():
            if rank[j] > rank[i]:
                s -= N[i, f] @ x[j]
        x[i] = D[i] @ s
    return x


def _star(kind):
    """a triangle (tetrahedron) cut into three (four) elements at an inner point"""
    props = KINDS[kind][0]()
    if KINDS[kind][1] == "channel":
        v = np.array([(0, 0), (1, 0), (0.3, 0.9), (0.45, 0.3)])
        el, faces = [(0, 1, 3), (1, 2, 3), (2, 0, 3)], [(0, 1), (1, 2), (2, 0)]
    else:
        v = np.array([(0, 0, 0), (1, 0, 0), (0.2, 1, 0), (0.3, 0.2, 0.9), (0.35, 0.3, 0.25)])
        el = [(4, 1, 2, 3), (0, 4, 2, 3), (0, 1, 4, 3), (0, 1, 2, 4)]
        faces = [(1, 2, 3), (0, 2, 3), (0, 1, 3), (0, 1, 2)]
    kinds = [meshgen.INLET, meshgen.OUTLET] + [meshgen.INVISCID_WALL] * (len(faces) - 2)
    bnd = np.array([(t,) + f for t, f in zip(kinds, faces)], dtype=np.int32)
    el = np.array(el, dtype=np.int32)
    tt = fg.create_neighbor_matrix(v.shape[1], el, bnd)
    g = fg.GpuMesh(props, v.astype(np.float64), el, tt, np.full(len(v), 0.1))
    rng = np.random.default_rng(kind)
    w0 = g.get_state(0)
    W = cases.perturbed(w0, g.n_basis, g.n_eqs, rng, 0.01) if np.any(w0) else 0.1 * rng.standard_normal(w0.shape)
    for which in (0, 1, 2):
        g.set_state(W, which)
    g.limiter()
    fg.JacobiAssembler(g).assemble_exact(2.0 * g.time_step_bound() if np.any(w0) else 1e-2, -1)
    return g, rng.standard_normal(W.shape)


@pytest.mark.parametrize("prec,mesh", [("blockjacobi", "general"), ("blockilu0", "general"), ("blockilu0", "star")])
@pytest.mark.parametrize("kind", sorted(KINDS))
def test_application_equals_numpy(kind, prec, mesh):
    g, b = _star(kind) if mesh == "star" else _assembled(kind, (9, 7) if KINDS[kind][1] == "channel" else (4, 3, 2))
    asm = fg.JacobiAssembler(g)
    tt, rank = g.neighbors, g.dof_order()
    if mesh == "star":
        assert np.sum(tt > -1) == len(tt) * (len(tt) - 1)  # every element touches every other

    def apply(dtype):
        D, N = _blocks(g, asm, dtype)
        return _jacobi(D, b) if prec == "blockjacobi" else _ilu0(D, N, tt, rank, b)

    want = apply(np.float64)
    e32 = np.max(np.abs(apply(np.float32) - want)) / np.max(np.abs(want))
    assert e32 < 1e-3  # the comparison means something
    for precision, tol in ((fg.FP64, 20 * e32 * 2.0**-29 + 1e-13), (fg.FP32, 20 * e32)):
        for variant in (0, 1):
            g.set_ilu_sweep(variant)
            _, x, its = g.block_solve(b, preconditioner=prec, precision=precision, restart=1, max_restarts=1, tol=1e-300)
            assert its == 1
            scale = np.vdot(x, want) / np.vdot(x, x)
            err = np.max(np.abs(scale * x - want)) / np.max(np.abs(want))
            assert err <= tol, (precision, variant, err, e32)
    g.close()
