"""The work that users of this library have it do, as measurable cases.

Each case is one call sequence of a flow computation through the public entry points: explicit
time stepping, the residual of a host's state, implicit steps with every preconditioner in
earnest use, the batched solve of many small cases, and the derivatives of an adjoint study.
The meshes are the seeded ones of flowpro_v2_b200.meshgen (bump channel, bump box, NACA 0012
O-grid); a case's seed gives the state it starts from (the free stream with noise on every
coefficient) and, for the batched cases, the geometries and Mach numbers.

exact() is an independent restatement of the discretisation for the Euler and Navier-Stokes
models in torch, float64: traces by evaluating the Lagrange basis at the physical face points,
derivatives by autograd.
"""
import functools
import math

import numpy as np
import torch

import flowpro_v2_b200 as fg
from flowpro_v2_b200 import meshgen

KAPPA = 1.4


# ---------------------------------------------------------------------------- the cases
def listed():
    return [
        # explicit run on a mesh of the size of FlowPro's shipped GAMM example (627 triangles),
        # with the shock sensor on as that example has it: launches and latency count
        dict(name="explicit-p1-624", kind="explicit", mesh="channel", nx=24, ny=13, nz=0, order=2, viscous=False, damp=True,
             steps=25),
        # 2D Euler p = 1, 15,000 triangles, SSP-RK3: the explicit configuration
        dict(name="explicit-p1-15k", kind="explicit", mesh="channel", nx=150, ny=50, nz=0, order=2, viscous=False, damp=False,
             steps=20),
        # 2D Navier-Stokes p = 2, 200,568 triangles: the benchmark's mesh, stepped explicitly
        dict(name="explicit-ns-p2-200k", kind="explicit", mesh="channel", nx=548, ny=183, nz=0, order=3, viscous=True,
             damp=False, steps=10),
        # 3D Euler p = 2 on tetrahedra
        dict(name="explicit-3d-p2-144k", kind="explicit", mesh="box", nx=60, ny=20, nz=20, order=3, viscous=False, damp=False,
             steps=10),
        # one residual of a host's state (pinned buffers both ways), the benchmark's workload
        dict(name="residual-ns-p2-200k", kind="residual", mesh="channel", nx=548, ny=183, nz=0, order=3, viscous=True,
             damp=False),
        # BDF2 with the reference's finite-difference blocks and block Jacobi: FlowPro's defaults
        dict(name="implicit-ns-bj-50k", kind="implicit", mesh="channel", nx=274, ny=92, nz=0, order=3, model="ns",
             jacobian="fd", preconditioner="blockjacobi", precision="fp64", bdf=2, restart=30, steps=3, lag=1, cfl=10.0),
        # finite-difference blocks, FP64 block ILU(0), GMRES(40): the reference's 3D solve
        dict(name="implicit-3d-ilu64-18k", kind="implicit", mesh="box", nx=30, ny=10, nz=10, order=3, model="euler",
             jacobian="fd", preconditioner="blockilu0", precision="fp64", bdf=1, restart=40, steps=3, lag=1, cfl=5.0),
        # the mixed path: exact tangent as operator, FP32 block ILU(0) of the exact blocks
        dict(name="implicit-3d-mixed-87k", kind="implicit", mesh="box", nx=50, ny=17, nz=17, order=3, model="euler",
             jacobian="tangent", preconditioner="blockilu0", precision="fp32", bdf=1, restart=40, steps=4, lag=10, cfl=20.0),
        # RANS (Spalart-Allmaras) on a coarsened O-grid about the aerofoil, the mixed path
        dict(name="implicit-rans-sa", kind="implicit", mesh="naca", nx=96, ny=0, nz=0, order=3, model="sa",
             jacobian="tangent", preconditioner="blockilu0", precision="fp32", bdf=1, restart=40, steps=4, lag=2, cfl=1.0),
        # many small cases solved together: one order group each of the serving set
        dict(name="serving-p1-12", kind="serving", cases=12, most=12000, order=2, steps=5),
        dict(name="serving-p3-4", kind="serving", cases=4, most=8000, order=4, steps=4),
        # an adjoint study: functional and gradient, tangent and adjoint products, adjoint solve
        dict(name="adjoint-ns-p2-10k", kind="adjoint", mesh="channel", nx=122, ny=41, nz=0, order=3, viscous=True, restart=40),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _channel(rng, lo, hi):
    ny = max(5, int(round(math.sqrt(_log(rng, lo, hi) / 6.0))))
    return dict(mesh="channel", nx=3 * ny - rng.randint(0, 2), ny=ny, nz=0)


def _box(rng, lo, hi):
    n = max(3, int(round((_log(rng, lo, hi) / 18.0) ** (1 / 3))))
    return dict(mesh="box", nx=3 * n - rng.randint(0, 2), ny=n, nz=max(3, n - rng.randint(0, 1)))


def draw(rng):
    kind = rng.choice(["explicit", "explicit", "residual", "implicit", "implicit", "serving", "adjoint"])
    if kind == "explicit":
        d3 = rng.random() < 0.35
        order = rng.choice([2, 3])
        m = _box(rng, 2000, 100000) if d3 else _channel(rng, 600, 180000)
        damp = rng.random() < 0.3
        return dict(kind=kind, order=order, viscous=rng.random() < 0.4 and not damp, damp=damp, steps=rng.randint(5, 10), **m)
    if kind == "residual":
        d3 = rng.random() < 0.3
        return dict(kind=kind, order=rng.choice([2, 3]), viscous=rng.random() < 0.6, damp=False,
                    **(_box(rng, 3000, 80000) if d3 else _channel(rng, 3000, 180000)))
    if kind == "implicit":
        model = rng.choice(["euler", "ns", "sa"])
        prec = rng.choice(["blockjacobi", "blockilu0"])
        mixed = prec == "blockilu0" and rng.random() < 0.5
        if model == "sa":
            m = dict(mesh="naca", nx=2 * rng.randint(24, 56), ny=0, nz=0)
        elif model == "euler" and rng.random() < 0.5:
            m = _box(rng, 2000, 16000)
        else:
            m = _channel(rng, 2000, 40000)
        return dict(kind=kind, order=rng.choice([2, 3]), model=model, jacobian="tangent" if mixed else "fd",
                    preconditioner=prec, precision="fp32" if mixed else "fp64", bdf=rng.choice([1, 2]),
                    restart=rng.choice([30, 40]), steps=rng.randint(2, 3), lag=rng.choice([2, 10]) if mixed else 1,
                    cfl=1.0 if model == "sa" else float(rng.choice([3, 5, 10])), **m)
    if kind == "serving":
        order = rng.choice([2, 3, 4])
        return dict(kind=kind, cases=rng.randint(2, 10), most=rng.randint(2500, 12000 if order == 2 else 6000), order=order,
                    steps=rng.randint(3, 4))
    return dict(kind=kind, order=rng.choice([2, 3]), viscous=True, restart=rng.choice([30, 40]), **_channel(rng, 1500, 9000))


# ---------------------------------------------------------------------------- inputs
def _props(case):
    model = case.get("model") or ("ns" if case["viscous"] else "euler")
    dim = 3 if case["mesh"] == "box" else 2
    p = dict(model="NavierStokes", dimension=dim, kappa=KAPPA, cv=1, isFlowViscous="false", pIn0=1, rhoIn0=1,
             pOut=0.7840 if dim == 3 else 0.8430, order=case["order"], penalty=0, dampTol=3 if case.get("damp") else 0,
             dampConst=0, positivityLimiter="false")
    if model == "ns":
        p.update(isFlowViscous="true", reynolds=500 if dim == 3 else 5000, prandtl=0.72, penalty=1)
    if model == "sa":
        p = dict(model="SpalartAllmaras", dimension=2, kappa=KAPPA, cv=1, pIn0=1, rhoIn0=1, pOut=0.9395, reynolds=3e6,
                 prandtl=0.72, attackAngle=0.0698131700797732, vtIn=3, sigma=0.6667, cb1=0.1355, cb2=0.622, ka=0.41, cw2=0.3,
                 cw3=2, cv1=7.1, Prt=0.9, order=case["order"], penalty=1, dampTol=0, dampConst=0, positivityLimiter="true")
    if case["kind"] == "explicit":
        p["timeMethod"] = "RK"
        p["positivityLimiter"] = "true" if case["damp"] else "false"
    return p


@functools.lru_cache(maxsize=2)
def _mesh(mesh, nx, ny, nz, wall):
    if mesh == "channel":
        m = meshgen.bump_channel(nx=nx, ny=ny, seed=1, wall=wall)
    elif mesh == "box":
        m = meshgen.bump_box(nx=nx, ny=ny, nz=nz, seed=2, wall=wall)
    else:
        m = meshgen.naca0012_o_mesh(n_around=nx, first_height=1e-4, growth=1.3)
    return m, fg.create_neighbor_matrix(m.dim, m.elements, m.boundary)


def _wall(case):
    viscous = case.get("viscous") or case.get("model") == "ns"
    return meshgen.WALL if viscous else meshgen.INVISCID_WALL


def _noise(w0, n_elem, nb, seed, amp):
    """free stream w0 with seeded relative noise of amp on every coefficient, [n_elem, n_eqs * nb]"""
    rng = np.random.default_rng(seed)
    w = np.repeat(np.asarray(w0, dtype=np.float64), nb)[None, :]
    return np.ascontiguousarray(w * (1 + amp * (2 * rng.random((n_elem, w.shape[1])) - 1)))


def _free_stream(props):
    """the free stream of the stagnation state 1, 1 expanded to the outlet pressure"""
    k, p = KAPPA, props["pOut"]
    dim = props["dimension"]
    mach = math.sqrt(2 / (k - 1) * ((1 / p) ** ((k - 1) / k) - 1))
    rho = (1 + (k - 1) / 2 * mach * mach) ** (1 / (1 - k))
    v = mach * math.sqrt(k * p / rho)
    a = props.get("attackAngle", 0.0)
    w = [rho, rho * v * math.cos(a), rho * v * math.sin(a)] + [0.0] * (dim - 2)
    w.append(p / (k - 1) + 0.5 * rho * v * v)
    if props["model"] == "SpalartAllmaras":
        w.append(rho * props["vtIn"])
    return w


def _state(case, seed, n_elem):
    dim = 3 if case["mesh"] == "box" else 2
    o = case["order"]
    nb = o * (o + 1) // 2 if dim == 2 else (4 if o == 2 else 10)
    # with the shock sensor on, noise that it answers to; implicit runs start near the free stream
    amp = 0.1 if case.get("damp") else 0.001 if case["kind"] == "implicit" else 0.01
    return _noise(_free_stream(_props(case)), n_elem, nb, seed, amp)


def _serving(case, seed):
    # the sizes belong to the case, the geometries and Mach numbers to the seed
    sizes, rng = np.random.default_rng([case["cases"], case["most"]]), np.random.default_rng(seed)
    out = []
    for _ in range(case["cases"]):
        n = math.exp(sizes.uniform(math.log(2000), math.log(case["most"])))
        ny = max(5, int(round(math.sqrt(n / 6.0))))
        mach = rng.uniform(0.3, 0.6)
        p_out = (1 + (KAPPA - 1) / 2 * mach * mach) ** (-KAPPA / (KAPPA - 1))
        m = meshgen.bump_channel(nx=3 * ny, ny=ny, height=float(rng.uniform(0.05, 0.12)), seed=int(rng.integers(1, 2**31 - 1)))
        props = dict(model="NavierStokes", dimension=2, kappa=KAPPA, cv=1, isFlowViscous="false", pIn0=1, rhoIn0=1,
                     pOut=p_out, order=case["order"], penalty=0, dampTol=3, dampConst=0)
        out.append((props, m.vertices, m.elements, fg.create_neighbor_matrix(2, m.elements, m.boundary), m.wall_distance))
    return out


def prepare(case, seed):
    s = dict(case=case)
    if case["kind"] == "serving":
        s["batch"] = b = fg.GpuBatch(_serving(case, seed))
        s["W"] = np.zeros(b.n_elem * b.nb)
        b._check(fg.lib().fp_state_get(b.ctx, 0, fg._dp(s["W"])))
        return s
    m, tt = _mesh(case["mesh"], case["nx"], case["ny"], case["nz"], _wall(case))
    s["mesh"] = g = fg.GpuMesh(_props(case), m.vertices, m.elements, tt, wall_distance=m.wall_distance)
    W = _state(case, seed, g.n_elem)
    s["W"] = torch.from_numpy(W).pin_memory().numpy()
    if case["kind"] == "residual":
        g.limiter()
        s["R"] = torch.empty(W.shape, dtype=torch.float64).pin_memory().numpy()
    if case["kind"] == "adjoint":
        g.set_state(W)
        g.limiter()
        s["v"] = np.random.default_rng([seed, 1]).standard_normal(W.shape)
    return s


# ---------------------------------------------------------------------------- one pass
def run(s):
    case = s["case"]
    if case["kind"] == "serving":
        b = s["batch"]
        for which in (0, 1, 2):
            b._check(fg.lib().fp_state_set(b.ctx, which, fg._dp(s["W"])))
        out, status = b.solve(steps=case["steps"], cfl=4.0, vary_cfl=1, max_cfl=1e5, linear_tol=1e-2,
                              preconditioner="blockilu0", precision=fg.FP32, jacobian=fg.JAC_MATRIXFREE, restart=40,
                              max_restarts=5, jac_lag=10)
        W = np.empty(b.n_elem * b.nb)
        b._check(fg.lib().fp_state_get(b.ctx, 0, fg._dp(W)))
        return dict(W=W, dt=out[:, 3].copy(), status=status)
    g = s["mesh"]
    if case["kind"] == "residual":
        g._check(fg.lib().fp_residual(g.ctx, fg._dp(s["W"]), fg._dp(s["R"])))
        return s["R"]
    if case["kind"] == "explicit":
        g.set_state(s["W"])
        g.copy_w2wo()
        out = fg.GpuExplicitSolver(g, case["steps"], cfl=0.2).solve()
        return dict(W=g.get_state(), t=float(out[0]), residuum=float(out[1]))
    if case["kind"] == "implicit":
        for which in (0, 1, 2):
            g.set_state(s["W"], which)
        g_out = fg.GpuImplicitSolver(
            g, bdf_order=case["bdf"], steps=case["steps"], cfl=case["cfl"], vary_cfl=1, max_cfl=1e5, linear_tol=1e-2, restart=case["restart"],
            max_restarts=5, preconditioner=case["preconditioner"], jac_lag=case["lag"],
            jacobian=fg.JAC_MATRIXFREE if case["jacobian"] == "tangent" else fg.JAC_ASSEMBLED,
            precision=fg.FP32 if case["precision"] == "fp32" else fg.FP64).solve()
        return dict(W=g.get_state(), t=float(g_out[0]))
    value, grad = g.functional(fg.FUNCTIONAL_DRAG)
    jv = g.jvp(s["v"])
    vj = g.vjp(s["v"])
    fg.JacobiAssembler(g).assemble_exact(0.0, -1.0)
    _, psi, _ = g.adjoint_solve(grad, preconditioner="blockjacobi", restart=case["restart"], max_restarts=1, tol=1e-12)
    return dict(value=value, grad=grad, jvp=jv, vjp=vj, psi=psi)


# ---------------------------------------------------------------------------- work
def _sizes(case):
    if case["kind"] == "serving":
        lo, hi = math.log(2000), math.log(case["most"])
        n = case["cases"] * (math.exp(hi) - math.exp(lo)) / max(hi - lo, 1e-9)
        return 2, n, 4
    if case["mesh"] == "naca":
        m, _ = _mesh("naca", case["nx"], 0, 0, _wall(case))
        return 2, m.n_elem, 5
    if case["mesh"] == "box":
        return 3, 6 * case["nx"] * case["ny"] * case["nz"], 5
    return 2, 2 * case["nx"] * case["ny"], 4


def work(case):
    """Bytes and FP64 operations of one pass.  Residual: each trace once per face and side, each
    flux once per point (Euler ~25 + 12 dim operations, viscous ~40 dim more), the two
    projections.  A residual reads and writes the state once, with geometry and connectivity.
    Implicit: the blocks' products per quadrature point, the factorisation's block operations,
    and a nominal 15 GMRES iterations a step (each streams the factors, the operator's blocks
    where stored, and the basis four times)."""
    dim, n, ne = _sizes(case)
    o = case["order"]
    nb = o * (o + 1) // 2 if dim == 2 else (4 if o == 2 else 10)
    nq = (6, 7, 16)[o - 2] if dim == 2 else (6, 14)[o - 2]
    nqf = o if dim == 2 else (6, 7)[o - 2]
    nc, nf = ne * nb, dim + 1
    viscous = case.get("viscous") or case.get("model") in ("ns", "sa")
    tr = 1 + (dim if viscous else 0)
    flux = 25 + 12 * dim + (40 * dim if viscous else 0)
    res = n * (nq * (2 * nc * (tr + dim) + dim * flux) + nf / 2 * nqf * (4 * nc * tr + 2 * flux + 4 * nc))
    state = 8.0 * n * nc
    mesh = n * (8.0 * (dim * dim + 1 + nf * (dim + 2)) + 8 * nf)
    if case["kind"] == "residual":
        return dict(bytes=2 * state + mesh, flops=res)
    if case["kind"] == "explicit":
        k = 3 * case["steps"]
        return dict(bytes=k * (3 * state + mesh), flops=k * (res + 2 * n * nc * (nb + 2)))
    blocks = n * (1 + nf) * nc * nc
    jac = n * (nq * 2 * nc * nc * (1 + dim) / 2 + nf * nqf * 4 * nc * nc / 2)
    if case["kind"] == "adjoint":
        its = case["restart"]
        return dict(bytes=8.0 * blocks * (its + 1) + 4 * its * its / 2 * state + 10 * state,
                    flops=2 * blocks * its + jac + 6 * res + n * 2.0 * nc**3)
    steps = case["steps"]
    stored = case["kind"] == "implicit" and case["jacobian"] == "fd"
    ilu = case["kind"] == "serving" or case["preconditioner"] == "blockilu0"
    prec = (4.0 if not stored else 8.0) * (blocks if ilu else n * nc * nc)
    built = steps if case.get("lag", 10) == 1 else max(1, steps // case.get("lag", 10))
    its = 15 * steps
    by = built * 2 * prec + its * (prec + (8.0 * blocks if stored else 2 * state + mesh) + 4 * 8 * state)
    fl = built * (jac + n * 2.0 * nc**3 * (1 + (2 * nf / 2 if ilu else 0))) + its * (2 * blocks * (2 if stored else 1) + 2 * res)
    return dict(bytes=by, flops=fl)


# ---------------------------------------------------------------------------- independent float64 values
# quadrature rules of FlowPro: triangles of degree 4, 5 (weights sum to 1), tetrahedra of degree
# 3, 5 (weights sum to 1/6), lines of 2, 3 points on [-1, 1]
_TRI4 = ([0.10810301816807, 0.445948490915965, 0.816847572980459, 0.091576213509771, 0.445948490915965, 0.445948490915965,
          0.091576213509771, 0.09157621350977, 0.445948490915965, 0.10810301816807, 0.09157621350977, 0.816847572980459],
         [0.223381589678012, 0.109951743655322] * 3)
_TRI5 = ([0.333333333333333, 0.333333333333334, 0.05971587178977, 0.470142064105115, 0.797426985353087, 0.101286507323456,
          0.470142064105115, 0.470142064105115, 0.101286507323456, 0.101286507323457, 0.470142064105115, 0.05971587178977,
          0.101286507323457, 0.797426985353087],
         [0.225] + [0.132394152788506, 0.125939180544827] * 3)
_LINE = {2: ([-0.577350269189626, 0.577350269189626], [1.0, 1.0]),
         3: ([-0.774596669241483, 0.0, 0.774596669241483], [0.555555555555556, 0.888888888888889, 0.555555555555555])}
_TET3 = ([0.190117002439, 0.0114033294446, 0.358620720467, 0.158685163227, 0.585662805655, 0.130847168952, 0.0109052122112,
          0.281523802124, 0.362126829946, 0.571226052149, 0.146918390087, 0.140372805794, 0.170816925165, 0.152818143091,
          0.638493299962, 0.162001491699, 0.183850350492, 0.0127183663137],
         [0.0220946711907, 0.0374025278196, 0.0213444021185, 0.0420006634683, 0.0234374016101, 0.0203870004596])
_TET5 = ([0.0927352503109, 0.721794249067, 0.0927352503109, 0.454496295874, 0.454496295874, 0.0455037041256,
          0.0455037041256, 0.454496295874, 0.0455037041256, 0.0455037041256, 0.454496295874, 0.454496295874,
          0.310885919263, 0.0673422422101, 0.310885919263, 0.0673422422101, 0.310885919263, 0.310885919263,
          0.310885919263, 0.310885919263, 0.310885919263, 0.310885919263, 0.310885919263, 0.0673422422101,
          0.721794249067, 0.0927352503109, 0.0927352503109, 0.0927352503109, 0.0927352503109, 0.721794249067,
          0.0927352503109, 0.0927352503109, 0.0927352503109, 0.454496295874, 0.0455037041256, 0.0455037041256,
          0.454496295874, 0.0455037041256, 0.454496295874, 0.0455037041256, 0.0455037041256, 0.454496295874],
         [0.0122488405194, 0.00709100346285, 0.00709100346285, 0.00709100346285, 0.018781320953, 0.018781320953,
          0.018781320953, 0.018781320953, 0.0122488405194, 0.0122488405194, 0.0122488405194, 0.00709100346285,
          0.00709100346285, 0.00709100346285])


class _Plain:
    """The discretisation on one mesh in torch float64 (order 2 or 3)."""

    def __init__(self, case, device):
        m, _ = _mesh(case["mesh"], case["nx"], case["ny"], case["nz"], _wall(case))
        self.o, self.dim, self.visc = case["order"], m.dim, bool(case["viscous"])
        self.damp = 3.0 if case.get("damp") else 0.0
        p = _props(case)
        self.p_out, self.ne = p["pOut"], m.dim + 2
        t = lambda a, k=torch.float64: torch.as_tensor(np.array(a), dtype=k, device=device)  # noqa: E731
        dim, o = self.dim, self.o
        if self.visc:
            mach = math.sqrt(2 / (KAPPA - 1) * ((1 / self.p_out) ** ((KAPPA - 1) / KAPPA) - 1))
            rho = (1 + (KAPPA - 1) / 2 * mach**2) ** (-1 / (KAPPA - 1))
            pin = (1 + (KAPPA - 1) / 2 * mach**2) ** (-KAPPA / (KAPPA - 1))
            self.re, self.pr = p["reynolds"] / (rho * mach * math.sqrt(KAPPA * pin / rho)), p["prandtl"]
        # monomials and nodal coefficients
        self.ex = [e for k in range(o) for e in np.ndindex(*([k + 1] * dim)) if sum(e) == k]
        if dim == 2:
            nodes = []
            for i in range(o):
                x = i / (o - 1)
                for j in range(i + 1):
                    y = x / 2 if i == 0 else j / i * x
                    nodes.append((y, x - y))
        else:
            v = [(0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1)]
            nodes = v + ([tuple((np.array(v[a]) + np.array(v[b])) / 2) for a in range(4) for b in range(a + 1, 4)] if o == 3 else [])
        nodes = np.array(nodes, dtype=np.float64)
        V = np.stack([np.prod(nodes ** np.array(e), axis=1) for e in self.ex], 1)
        self.C = t(np.linalg.inv(V))
        self.nb = len(self.ex)
        # geometry
        X, el = t(m.vertices), t(m.elements, torch.int64)
        self.n = el.shape[0]
        self.x0 = X[el[:, 0]]
        J = torch.stack([X[el[:, i + 1]] - self.x0 for i in range(dim)], 2)
        self.Ji = torch.linalg.inv(J)
        det = torch.linalg.det(J).abs()
        q, w = (_TRI4, _TRI5)[o - 2] if dim == 2 else (_TET3, _TET5)[o - 2]
        self.xq, self.wq = t(q).reshape(-1, dim), t(w)
        self.jac = det / 2 if dim == 2 else det
        area = self.jac * self.wq.sum()
        centre = X[el].mean(1)
        # faces: the vertex sets of element sides, paired
        fv = [[k for k in f] for f in ([(0, 1), (1, 2), (2, 0)] if dim == 2 else [(0, 2, 1), (0, 1, 3), (1, 2, 3), (2, 0, 3)])]
        nf = dim + 1
        sides = torch.stack([el[:, f] for f in fv], 1).reshape(-1, dim)  # [n * nf, dim]
        key = torch.sort(sides, 1)[0].cpu().numpy()
        code = key[:, 0].astype(np.int64)
        for d in range(1, dim):
            code = code * X.shape[0] + key[:, d]
        order = np.argsort(code, kind="stable")
        same = code[order][1:] == code[order][:-1]
        first, second = order[:-1][same], order[1:][same]
        alone = np.setdiff1d(np.arange(code.size), np.concatenate([first, second]))
        bkey = np.sort(m.boundary[:, 1:], 1).astype(np.int64)
        bcode = bkey[:, 0]
        for d in range(1, dim):
            bcode = bcode * X.shape[0] + bkey[:, d]
        bo = np.argsort(bcode)
        self.bc = t(m.boundary[bo[np.searchsorted(bcode[bo], code[alone])], 0], torch.int64)
        if dim == 2:
            s = t(_LINE[o][0])
            lam, self.wf = torch.stack([(1 - s) / 2, (1 + s) / 2], 1), t(_LINE[o][1])
        else:
            s = t((_TRI4, _TRI5)[o - 2][0]).reshape(-1, 2)
            lam, self.wf = torch.stack([1 - s.sum(1), s[:, 0], s[:, 1]], 1), t((_TRI4, _TRI5)[o - 2][1])

        def face(idx):
            idx = t(idx, torch.int64)
            P = X[sides[idx]]  # [F, dim, dim]
            if dim == 2:
                d = P[:, 1] - P[:, 0]
                n = torch.stack([d[:, 1], -d[:, 0]], 1)
            else:
                n = torch.linalg.cross(P[:, 1] - P[:, 0], P[:, 2] - P[:, 0])
            e = idx // nf
            n = n * torch.sign(((P.mean(1) - centre[e]) * n).sum(1))[:, None]
            L = n.norm(dim=1)
            return e, n / L[:, None], L / 2, torch.einsum("pv,fvd->fpd", lam, P), P.mean(1)

        self.l, self.nrm, self.jf, xf, _ = face(first)
        self.r = t(second, torch.int64) // nf
        self.dl = ((centre[self.l] - centre[self.r]) * self.nrm).sum(1).abs()
        self.bl, self.bn, self.bj, xb, cb = face(alone)
        self.bdl = ((centre[self.bl] - cb) * self.bn).sum(1).abs()
        self.L, self.R, self.B = self._tab(self.l, xf), self._tab(self.r, xf), self._tab(self.bl, xb)
        self.phi, dphi = self._basis(self.xq)
        self.dphi = torch.einsum("qjr,erd->eqjd", dphi, self.Ji)
        M = torch.einsum("q,qi,qj->ij", self.wq, self.phi, self.phi)
        self.Mi = torch.linalg.inv(M)
        self.mean = (self.wq @ self.phi) / self.wq.sum()
        side = torch.zeros(self.n, dtype=torch.float64, device=device)
        wsum = self.wf.sum()
        for e, j in ((self.l, self.jf), (self.r, self.jf), (self.bl, self.bj)):
            side.index_add_(0, e, j * wsum)
        self.size = nf * area / side
        lin = torch.cat([torch.ones_like(self.xq[:, :1]), self.xq], 1)
        T = torch.einsum("q,qi,qj->ij", self.wq, lin, self.phi)
        self.trun = self.Mi @ T.T @ torch.linalg.inv(torch.einsum("q,qi,qj->ij", self.wq, lin, lin)) @ T

    def _basis(self, xi):
        """values [.., nb] and reference gradients [.., nb, dim] at reference points xi [.., dim]"""
        f, g = [], []
        for e in self.ex:
            f.append(torch.stack([xi[..., d] ** k for d, k in enumerate(e)], -1).prod(-1))
            g.append(torch.stack([(0 * xi[..., 0] if e[d] == 0 else
                                   e[d] * torch.stack([xi[..., c] ** (k - (c == d)) for c, k in enumerate(e)], -1).prod(-1))
                                  for d in range(self.dim)], -1))
        return torch.stack(f, -1) @ self.C, torch.einsum("...id,ij->...jd", torch.stack(g, -2), self.C)

    def _tab(self, e, x):
        phi, d = self._basis(torch.einsum("fij,fpj->fpi", self.Ji[e], x - self.x0[e][:, None]))
        return phi, torch.einsum("fpjr,frd->fpjd", d, self.Ji[e]) if self.visc or self.damp else None

    def pressure(self, w):
        return (KAPPA - 1) * (w[..., -1] - (w[..., 1:-1] ** 2).sum(-1) / (2 * w[..., 0]))

    def flux(self, w, n):
        v = (w[..., 1:-1] * n).sum(-1) / w[..., 0]
        p = self.pressure(w)
        return torch.cat([(w[..., 0] * v)[..., None], w[..., 1:-1] * v[..., None] + p[..., None] * n,
                          ((w[..., -1] + p) * v)[..., None]], -1)

    def speed(self, w):
        return (w[..., 1:-1] / w[..., :1]).norm(dim=-1) + torch.sqrt(KAPPA * self.pressure(w) / w[..., 0])

    def stress(self, w, dw):
        """viscous flux [.., m, d] of the state w [.., m] with gradients dw [.., m, d]"""
        rho = w[..., 0, None, None]
        vel = w[..., 1:-1, None] / rho
        vj = (dw[..., 1:-1, :] - dw[..., :1, :] * vel) / rho
        p = self.pressure(w)[..., None]
        dp = (KAPPA - 1) * (dw[..., -1, :] - dw[..., 0, :] * (vel**2).sum(-2) / 2 - rho[..., 0] * (vel * vj).sum(-2))
        heat = (rho[..., 0] * dp - p * dw[..., 0, :]) / rho[..., 0] ** 2
        tau = vj + vj.transpose(-1, -2) - 2 / 3 * torch.diag_embed(vj.diagonal(dim1=-2, dim2=-1).sum(-1)[..., None].expand(*vj.shape[:-1]))
        en = (vel * tau).sum(-2) + KAPPA / (KAPPA - 1) / self.pr * heat
        return torch.cat([0 * en[..., None, :], tau, en[..., None, :]], -2) / self.re

    def boundary(self, w, n):
        rho, mom, p = w[..., 0], w[..., 1:-1], self.pressure(w)
        cat = lambda r, m, e: torch.cat([r[..., None], m, e[..., None]], -1)  # noqa: E731
        slip = cat(rho, mom - (mom * n).sum(-1, keepdim=True) * n, w[..., -1])
        stick = cat(rho, 0 * mom, p / (KAPPA - 1))
        mach = torch.sqrt((2 / (KAPPA - 1) * ((1 / p) ** ((KAPPA - 1) / KAPPA) - 1)).clamp(min=0))
        ri = (1 + (KAPPA - 1) / 2 * mach**2) ** (1 / (1 - KAPPA))
        vi = mach * torch.sqrt(KAPPA * p / ri)
        inlet = cat(ri, -(ri * vi)[..., None] * n, p / (KAPPA - 1) + 0.5 * ri * vi**2)
        v2 = (mom**2).sum(-1) / rho**2
        outlet = cat(rho, mom, self.p_out / (KAPPA - 1) + rho * v2 / 2)
        outlet = torch.where((v2 < KAPPA * p / rho)[..., None], outlet, w)
        b = self.bc[:, None, None]
        wall = torch.where(b == meshgen.WALL, stick if self.visc else slip, slip)
        return torch.where(b == meshgen.INLET, inlet, torch.where(b == meshgen.OUTLET, outlet, wall))

    def limiter(self, W):
        """artificial viscosity per element from the shock sensor of the density"""
        eps = torch.zeros(self.n, dtype=W.dtype, device=W.device)
        if not self.damp:
            return eps
        w = W.reshape(self.n, self.ne, self.nb)
        rho = w[:, 0]
        tr = rho @ self.trun.T if self.o > 2 else (rho @ self.mean)[:, None].expand(-1, self.nb)
        num = (((rho - tr) @ self.phi.T) ** 2 * self.wq).sum(1)
        se = torch.log10((num / ((rho @ self.phi.T) ** 2 * self.wq).sum(1)).abs())
        s0 = math.log10(1 / (self.o - 1) ** 4)
        s = 0.5 * (1 + torch.sin(math.pi * (se - s0) / (2 * self.damp)))
        s = torch.where(se < s0 - self.damp, 0 * s, torch.where(se > s0 + self.damp, 0 * s + 1, s))
        return self.speed(w @ self.mean) * self.size / self.o * torch.nan_to_num(s)

    def residual(self, W, eps):
        w = W.reshape(self.n, self.ne, self.nb)
        K = torch.zeros_like(w)
        full = self.visc or self.damp
        val = lambda t, e: torch.einsum("fpj,fmj->fpm", t[0], w[e])  # noqa: E731
        der = lambda t, e: torch.einsum("fpjd,fmj->fpmd", t[1], w[e])  # noqa: E731
        a, b, n = val(self.L, self.l), val(self.R, self.r), self.nrm[:, None]
        lam = torch.maximum(self.speed(a), self.speed(b))[..., None]
        g = -(self.flux(a, n) + self.flux(b, n) - lam * (b - a)) / 2
        ip = 0.0
        if full:
            dn = (der(self.L, self.l) + der(self.R, self.r)) / 2 + 2.0 * ((b - a) / self.dl[:, None, None])[..., None] * n[:, :, None]
            if self.visc:
                g = g + (self.stress((a + b) / 2, dn) * n[:, :, None]).sum(-1)
                ip = a - b
            g = g + (0.5 * (eps[self.l] + eps[self.r]))[:, None, None] * (dn * n[:, :, None]).sum(-1)
        jw = (self.jf[:, None] * self.wf)[..., None]
        K = K.index_add(0, self.l, torch.einsum("fpm,fpj->fmj", jw * (g - ip), self.L[0]))
        K = K.index_add(0, self.r, torch.einsum("fpm,fpj->fmj", jw * (ip - g), self.R[0]))
        a, n = val(self.B, self.bl), self.bn[:, None]
        b = self.boundary(a, n)
        wall = ((self.bc == meshgen.WALL) | (self.bc == meshgen.INVISCID_WALL))[:, None, None]
        p = self.pressure(a)[..., None]
        g = -torch.where(wall, torch.cat([0 * p, p * n, 0 * p], -1), self.flux(b, n))
        if self.visc:
            dn = der(self.B, self.bl) + 2.0 * ((b - a) / self.bdl[:, None, None])[..., None] * n[:, :, None]
            f = (self.stress(b, dn) * n[:, :, None]).sum(-1)
            f = torch.cat([f[..., :-1], 0 * f[..., -1:]], -1) - (a - b)
            g = g + torch.where((self.bc == meshgen.WALL)[:, None, None], f, 0 * f)
        K = K.index_add(0, self.bl, torch.einsum("fpm,fpj->fmj", (self.bj[:, None] * self.wf)[..., None] * g, self.B[0]))
        a = torch.einsum("qj,emj->eqm", self.phi, w)
        I = torch.eye(self.dim, dtype=W.dtype, device=W.device)
        F = torch.stack([self.flux(a, I[d]) for d in range(self.dim)], -1)
        if full:
            dw = torch.einsum("eqjd,emj->eqmd", self.dphi, w)
            F = F - eps[:, None, None, None] * dw
            if self.visc:
                F = F - self.stress(a, dw)
        jw = (self.jac[:, None] * self.wq)[..., None, None]
        return (K + torch.einsum("eqmd,eqjd->emj", jw * F, self.dphi)).reshape(self.n, -1)

    def drag(self, W):
        w = W.reshape(self.n, self.ne, self.nb)
        k = self.bc == meshgen.WALL
        a = torch.einsum("fpj,fmj->fpm", self.B[0][k], w[self.bl[k]])
        return (self.bj[k][:, None] * self.wf * self.bn[k][:, :1] * self.pressure(a)).sum()


def _explicit(P, W, steps):
    t, norms = 0.0, None
    mass = lambda r: torch.einsum("ij,emj->emi", P.Mi, r.reshape(P.n, P.ne, P.nb)).reshape(P.n, -1) / P.jac[:, None]  # noqa: E731
    worst = 0.0
    cfl = 0.0
    for k in range(steps):
        cfl = min(cfl + 0.2 / 20, 0.2)
        mean = W.reshape(P.n, P.ne, P.nb) @ P.mean
        dt = cfl * float((P.size / P.speed(mean) / (2 * (P.o - 1) + 1)).min())
        R = P.residual(W, P.limiter(W))
        n = torch.sqrt((R * mass(R)).reshape(P.n, P.ne, P.nb).sum((0, 2)))
        norms = n if norms is None else torch.maximum(norms, n) if k < 5 else norms
        worst = float((n / norms).max())
        W1 = W + dt * mass(R)
        W2 = 0.75 * W + 0.25 * (W1 + dt * mass(P.residual(W1, P.limiter(W1))))
        W = W / 3 + 2 / 3 * (W2 + dt * mass(P.residual(W2, P.limiter(W2))))
        t += dt
    return W, t, worst


def exact(case, seed):
    if case["kind"] in ("implicit", "serving"):
        return None  # truncated Krylov solves: no value of their own
    device = "cuda" if torch.cuda.is_available() else "cpu"
    P = _Plain(case, device)
    W = torch.as_tensor(_state(case, seed, P.n), device=device)
    if case["kind"] == "explicit":
        W, t, r = _explicit(P, W, case["steps"])
        return dict(W=W.cpu().numpy(), t=t, residuum=r)
    eps = P.limiter(W)
    if case["kind"] == "residual":
        return P.residual(W, eps).cpu().numpy()
    v = torch.as_tensor(np.random.default_rng([seed, 1]).standard_normal(tuple(W.shape)), device=device)
    W.requires_grad_(True)
    value = P.drag(W)
    grad, = torch.autograd.grad(value, W)
    R = P.residual(W, eps)
    u = torch.zeros_like(R, requires_grad=True)
    vu, = torch.autograd.grad(R, W, u, create_graph=True)  # linear in u: its derivative along v is the tangent
    jv, = torch.autograd.grad(vu, u, v, retain_graph=True)
    vj, = torch.autograd.grad(R, W, v)
    return dict(value=float(value.detach()), grad=grad.cpu().numpy(), jvp=jv.cpu().numpy(), vjp=vj.cpu().numpy(), psi=None)
