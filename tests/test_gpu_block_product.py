"""The operator's and the block-Jacobi product at every compiled number of unknowns (below, at and beside
multiples of eight, the columns a thread loads together): GMRES to 1e-12 against a dense solve of the same
blocks, and the transposed system against the transposed dense solve, 1e-8 as LinearSolverTest (GPU)."""
import numpy as np
import pytest

import flowpro_v2_b200 as fg
from flowpro_v2_b200 import meshgen
from tests import cases
from tests.test_gpu_jacobian import CASES, MODELS
from tests.test_gpu_parity import _dense_from_blocks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [fg.FP64, fg.FP32])
@pytest.mark.parametrize("kind,order", sorted({(k, o) for k, o, _ in CASES}))
def test_block_products_against_dense_solve(kind, order, precision):
    wall = meshgen.WALL if kind in ("ns", "sa", "ns3") else meshgen.INVISCID_WALL
    m, tt = cases.channel(5, 4, seed=order, wall=wall) if MODELS[kind][1] == "channel" else cases.box(2, 2, 1, seed=2, wall=wall)
    if kind == "sa":
        m.wall_distance[:] = np.maximum(m.wall_distance, 1e-3)
    g = fg.GpuMesh(MODELS[kind][0](order), m.vertices, m.elements, tt, m.wall_distance)
    g.limiter()
    asm = fg.JacobiAssembler(g, bdf_order=1)
    asm.assemble(g.time_step_bound() if "scalar" not in kind else 0.05, -1)
    diag, neigh, _ = asm.blocks()
    A = _dense_from_blocks(diag, neigh, tt)
    b = np.random.default_rng(order).standard_normal((g.n_elem, g.nb))
    for transpose in (False, True):
        want = np.linalg.solve(A.T if transpose else A, b.reshape(-1)).reshape(-1, g.nb)
        ok, x, _ = g.block_solve(b, transpose=transpose, preconditioner="blockjacobi", precision=precision, restart=150,
                                 max_restarts=4, tol=1e-12)
        assert ok
        assert np.max(np.abs(x - want)) <= 1e-8 * np.max(np.abs(want))
    g.close()
