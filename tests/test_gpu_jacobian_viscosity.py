"""Element blocks and the adjoint product where the artificial viscosity acts on some elements and not on others:
the blocks times a vector against the tangent operator (another code, which forms every gradient), finite
differences against the exact blocks, and the adjoint product against the transposed blocks (GPU).

The exact ones are sums of some thousand products: 1e-12 of the largest entry.  The finite differences have the step
1e-8: 1e-6 as everywhere."""
import numpy as np
import pytest

import flowpro_v2_b200 as fg
from tests import cases

pytestmark = pytest.mark.gpu

MODELS = {
    "euler": (cases.euler_props, "channel"),
    "adiabatic": (cases.adiabatic_props, "channel"),
    "euler3": (cases.euler3_props, "box"),
}
CASES = [("euler", 2), ("euler", 3), ("euler", 4), ("adiabatic", 2), ("adiabatic", 3), ("euler3", 2), ("euler3", 3)]


@pytest.mark.parametrize("const", [0.0, 1e-3])
@pytest.mark.parametrize("kind,order", CASES)
def test_blocks_with_artificial_viscosity(kind, order, const):
    m, tt = cases.channel(17, 9, seed=order) if MODELS[kind][1] == "channel" else cases.box(5, 4, 3, seed=order)
    props = dict(MODELS[kind][0](order), dampTol=3.0, dampConst=const)
    g = fg.GpuMesh(props, m.vertices, m.elements, tt, m.wall_distance)
    rng = np.random.default_rng(order)
    W = g.get_state(0)
    # noise where the sensor answers in one half of the domain, smooth in the other
    left = np.mean(m.vertices[m.elements][:, :, 0], axis=1) < np.median(m.vertices[:, 0])
    amp = np.where(left, 0.2, 1e-6)[:, None]
    W = W * (1 + amp * (2 * rng.random(W.shape) - 1))
    for which in (0, 1, 2):
        g.set_state(W, which)
    g.limiter()
    eps = g.limiter_values()[0]
    assert 0 < np.count_nonzero(eps) < eps.size
    asm = fg.JacobiAssembler(g)
    asm.assemble_exact(0.0, -1.0)
    D, N, _ = asm.blocks()
    asm.assemble(0.0, -1.0)
    Df, Nf, _ = asm.blocks()
    D, N, Df, Nf = (np.swapaxes(a, -1, -2) for a in (D, N, Df, Nf))
    scale = max(np.max(np.abs(D)), np.max(np.abs(N)))
    assert np.max(np.abs(D - Df)) <= 1e-6 * scale and np.max(np.abs(N - Nf)) <= 1e-6 * scale
    v = rng.standard_normal(W.shape)
    y, yt = np.einsum("erc,ec->er", D, v), np.einsum("erc,er->ec", D, v)
    for f in range(tt.shape[1]):
        on = tt[:, f] > -1
        y[on] += np.einsum("erc,ec->er", N[on, f], v[tt[on, f]])
        np.add.at(yt, tt[on, f], np.einsum("erc,er->ec", N[on, f], v[on]))
    jv, vj = g.jvp(v), g.vjp(v)
    assert np.max(np.abs(y + jv)) <= 1e-12 * np.max(np.abs(jv))
    assert np.max(np.abs(yt + vj)) <= 1e-12 * np.max(np.abs(vj))
    g.close()
