"""Changing the kernel of the block ILU(0) application after a sweep that timed out (GPU).

Both kernels publish through the same words, one as bare values, the other with an epoch in the high
half.  A value between 2.2e-314 and 4.2e-314 reads as a word of epoch 1: the interrupted sweep of the streamed
kernel publishes those everywhere, and the register kernel must not take them for its own."""
import numpy as np
import pytest

import flowpro_v2_b200 as fg
from tests import cases

pytestmark = pytest.mark.gpu


def _assembled():
    m, tt = cases.channel(40, 30, seed=5)
    g = fg.GpuMesh(cases.euler_props(1), m.vertices, m.elements, tt, m.wall_distance)
    asm = fg.JacobiAssembler(g)
    asm.assemble_exact(1e-3 * g.time_step_bound(), -1)  # so short that the matrix is its diagonal to 1e-3
    return g, asm


@pytest.mark.parametrize("precision", [fg.FP64, fg.FP32])
def test_register_kernel_after_a_timed_out_streamed_sweep(precision):
    opts = dict(preconditioner="blockilu0", precision=precision, restart=20, max_restarts=2, tol=1e-10)
    g, _ = _assembled()
    b = np.random.default_rng(1).standard_normal((g.n_elem, g.nb))
    g.set_ilu_sweep(1)
    ok, want, _ = g.block_solve(b, **opts)
    assert ok
    g.close()
    g, asm = _assembled()
    ok, _, _ = g.block_solve(b, **opts)  # factorised, with the normal limit
    assert ok
    tiny = 3e-314 * np.einsum("eii->ei", asm.blocks()[0])  # inv(A) of it: 3e-314 everywhere
    g.set_wait_limit(0)
    with pytest.raises(fg.FlowGpuError) as ei:
        g.block_solve(tiny, **opts)
    assert "flowgpu error 8" in str(ei.value)  # FP_ERR_TIMEOUT
    g.set_wait_limit(1 << 19)
    g.set_ilu_sweep(1)
    ok, x, _ = g.block_solve(b, **opts)
    assert ok and np.array_equal(x, want)
    g.close()
