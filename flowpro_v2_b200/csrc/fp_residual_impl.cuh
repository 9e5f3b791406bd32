// Residual-side kernel templates (instantiated per model in fp_res_*.cu): residual, SSP-RK3 stages, limiter (artificial viscosity),
// positivity limiter, residual norms, time-step bound, finite-difference element
// Jacobian, tangent (JVP).  One element per thread; per-element data in the
// field-major SoA layout of fp_kernels.cuh.
#pragma once
#include <atomic>
#include <cstdio>
#include <type_traits>

#include "fp_ctx.h"
#include "fp_dispatch.cuh"
#include "fp_launch.h"

namespace fp {

constexpr int kBlock = 128;

// Minimum resident CTAs per SM requested from ptxas for the face and element kernels
// (caps registers at 65536 / (128 * MINB)).  Four CTAs (128 registers) pay off for the
// face kernel up to ~24 unknowns per element; the element kernels (residual, RK stage,
// BDF right-hand side) of 13-24 unknowns run faster with three (168 registers, fewer
// spills: 2D Navier-Stokes p = 2, 0.078 -> 0.070 ms on 200,568 triangles); larger
// elements spill too much under either cap.
template <class Mdl, int DIM, int ORDER>
struct MinBlocks {
    static constexpr int NC = Mdl::NE * nbasis_of(DIM, ORDER);
#ifdef FP_MINB_FACE
    static constexpr int face = FP_MINB_FACE;
#else
    static constexpr int face = NC <= 24 ? 4 : Mdl::kViscous ? 2 : 3;
#endif
#ifdef FP_MINB_ELEM
    static constexpr int elem = FP_MINB_ELEM;
#else
    static constexpr int elem = NC <= 12 ? 4 : NC <= 24 ? 3 : 2;
#endif
};

template <class Mdl, int DIM, int ORDER>
using E = Element<Mdl, DIM, ORDER>;

// coefficient c of the face's neighbour, staged by the calling thread in a shared array laid
// out [c][thread] (BLOCK threads); the neighbour index is the face's own
template <int BLOCK>
struct NbShared {
    const double* p;
    __device__ double operator()(int c, int) const { return p[c * BLOCK]; }
};

// coefficient c of the calling thread in a shared array laid out [c][thread] (BLOCK threads)
template <int BLOCK>
struct OwnShared {
    const double* p;
    __device__ double operator[](int c) const { return p[c * BLOCK]; }
};

// The element's own coefficients in the face and element kernels stay in shared memory,
// one column per thread ([c][thread]), instead of NC registers: that keeps the kernels'
// per-point state in registers instead of spilling it.  Up to kShNC unknowns the array is
// static; larger elements take it from the dynamic shared memory of the launch
// (own_smem_bytes, set up by the launchers).
constexpr int kShNC = 24;
extern __shared__ __align__(16) double fp_dyn_smem[];
template <int NC>
constexpr size_t own_smem_bytes() {
    return NC > kShNC ? (size_t)NC * kBlock * sizeof(double) : 0;
}
template <class Mdl, int DIM, int ORDER>
__device__ __forceinline__ OwnShared<kBlock> own_coeffs(const double* __restrict__ W, int ld, int e, double* wsh) {
    constexpr int NC = Element<Mdl, DIM, ORDER>::NC;
#pragma unroll
    for (int c = 0; c < NC; c++) wsh[c * kBlock + threadIdx.x] = ldg(W + (size_t)c * ld + e);
    return OwnShared<kBlock>{wsh + threadIdx.x};
}
// the tangent kernel's coefficients and direction, [c][thread] each, in dynamic shared
// memory when two CTAs of it fit an SM (up to 53 unknowns), else registers
template <int NC>
constexpr size_t matfree_smem_bytes() {
    return 2 * (size_t)NC * kBlock * sizeof(double) <= 106 * 1024 ? 2 * (size_t)NC * kBlock * sizeof(double) : 0;
}
template <int BLOCK>
struct OwnDualShared {
    const double* v;
    const double* d;
    __device__ Dual<1> operator[](int c) const {
        Dual<1> x;
        x.v = v[c * BLOCK];
        x.d[0] = d[c * BLOCK];
        return x;
    }
};
#define FP_OWN_COEFFS(NC_)                                                   \
    __shared__ double own_wsh_static[(NC_) <= kShNC ? (NC_) * kBlock : 1]; \
    double* own_wsh = (NC_) <= kShNC ? own_wsh_static : fp_dyn_smem

template <class Mdl, int DIM, int ORDER>
__device__ __forceinline__ void load_w(const double* __restrict__ W, int ld, int e, double* w) {
#pragma unroll
    for (int c = 0; c < E<Mdl, DIM, ORDER>::NC; c++) w[c] = ldg(W + (size_t)c * ld + e);
}

// ---------------------------------------------------------------------------- residual
// Face pass of the face-based residual: one thread per face computes the integrand of
// DGpure.residuumWall (DGpure.java:204-353) once and stores both sides' weighted
// contributions, G[0][p] = jw (C - cIP_e Jmp) for the owner and G[1][q] = jw (-C + cIP_nb Jmp)
// for the neighbour at its own quadrature point q = qmap[perm][p] (every term of the face
// integrand is odd in the normal, and the neighbour's normal is the negated one).
//
// Inviscid models need no gradients of the traces where the face's artificial viscosity is zero
// (Element::needs_gradients).  Such a face then reads each coefficient of its two elements once,
// adds it to the traces of all NQF points (face_traces), keeps those in shared memory and runs the
// points over them: a point-by-point pass reads the neighbour's coefficients, a scattered gather,
// once per point.  3D Euler p = 2, 144,000 tetrahedra: 277 -> 146 us; with the volume integral
// without gradients an SSP-RK3 step of ten 34.4 -> 28.0 ms with the copies of the state.
template <int NC, int NTR, bool VISC>
constexpr size_t face_smem_bytes() {  // [c][thread] coefficients of both sides (to kShNC) or the owner's; traces of both
    const int coeffs = NC <= kShNC ? 2 * NC : NC, traces = VISC ? 0 : 2 * NTR;
    return (size_t)(coeffs > traces ? coeffs : traces) * kBlock * sizeof(double);
}

// the traces of one side of a face at the points p0 .. p0 + NQ - 1: coef(c) the element's coefficients,
// phi(q, j) the basis at point p0 + q; out[(q * NE + m) * stride]
template <class Mdl, int DIM, int ORDER, int NQ, class T, class Coef, class Phi, class Out>
__device__ __forceinline__ void face_traces(const Coef& coef, const Phi& phi, const Out& out) {
    using El = E<Mdl, DIM, ORDER>;
    constexpr int NB = El::NB, NE = El::NE;
    T acc[NQ][NE];
#pragma unroll
    for (int q = 0; q < NQ; q++)
#pragma unroll
        for (int m = 0; m < NE; m++) acc[q][m] = 0.0;
#pragma unroll
    for (int j = 0; j < NB; j++) {
        T c[NE];
#pragma unroll
        for (int m = 0; m < NE; m++) c[m] = coef(m * NB + j);
#pragma unroll
        for (int q = 0; q < NQ; q++) {
            const double ph = phi(q, j);
#pragma unroll
            for (int m = 0; m < NE; m++) acc[q][m] += c[m] * ph;
        }
    }
#pragma unroll
    for (int q = 0; q < NQ; q++)
#pragma unroll
        for (int m = 0; m < NE; m++) out(q, m, acc[q][m]);
}

template <class Mdl, int DIM, int ORDER>
__global__ void __launch_bounds__(kBlock, (MinBlocks<Mdl, DIM, ORDER>::face))
    k_face(DevMesh M, const double* __restrict__ W, int f0, int f1) {
    using El = E<Mdl, DIM, ORDER>;
    using GL = GeoLayout<DIM>;
    using TB = Tab<DIM, ORDER>;
    constexpr int NC = El::NC, NE = El::NE, NQF = El::NQF, NP = El::NP, NB = El::NB;
    const int f = f0 + blockIdx.x * blockDim.x + threadIdx.x;  // faces f0 .. f1 - 1
    const DevFaces& F = M.F;
    if (f >= f1) return;
    const int ld = M.ld, ldf = F.ldf;
    const int e = F.fl[f], k = F.fk[f], TT = F.fr[f];
    double n[DIM], Jac, dL;
    El::face_geo(M, e, k, n, Jac, dL);
    const bool interior = TT > -1;
    int kr_face = 0, pm = 0;
    double eps_nb = 0, cip_nb = 0;
    if (interior) {
        const int fc = F.fc[f];
        kr_face = fc / NP;
        pm = fc - kr_face * NP;
        eps_nb = ldg(M.eps + TT);
        cip_nb = ldg(M.cip + TT);
    }
    const double eps_e = ldg(M.eps + e);
    const double cip_e = ldg(M.cip + e);
    const bool ip = Mdl::kViscous && (interior || Mdl::isIPFace(TT));
    double* G0 = F.G + f;
    double* G1 = F.G + (size_t)NQF * NE * ldf + f;
    double* sh = fp_dyn_smem + threadIdx.x;
    if constexpr (!Mdl::kViscous) {
        if (!El::needs_gradients(M, interior, eps_e, eps_nb)) {
            face_traces<Mdl, DIM, ORDER, NQF, double>(
                [&](int c) { return ldg(W + (size_t)c * ld + e); },
                [&](int q, int j) { return ldg(M.tab + TB::o_phiL + (k * NQF + q) * NB + j); },
                [&](int q, int m, double v) { sh[(q * NE + m) * kBlock] = v; });
            if (interior)
                face_traces<Mdl, DIM, ORDER, NQF, double>(
                    [&](int c) { return ldg(W + (size_t)c * ld + TT); },
                    [&](int q, int j) { return ldg(M.tab + TB::o_phiR + ((kr_face * NP + pm) * NQF + q) * NB + j); },
                    [&](int q, int m, double v) { sh[((NQF + q) * NE + m) * kBlock] = v; });
#pragma unroll 1
            for (int p = 0; p < NQF; p++) {
                double WL[NE], WR[NE], C[NE], Jm[NE];
#pragma unroll
                for (int m = 0; m < NE; m++) WL[m] = sh[(p * NE + m) * kBlock];
                if (interior) {
#pragma unroll
                    for (int m = 0; m < NE; m++) WR[m] = sh[((NQF + p) * NE + m) * kBlock];
                }
                El::template point_flux<false>(M, e, k, p, TT, n, dL, eps_e, eps_nb, WL, WR, (double*)nullptr, (double*)nullptr,
                                               C, Jm);
                const double jw = Jac * ldg(M.tab + TB::o_wf + p);
                const int q = interior ? F.qmap[pm * NQF + p] : 0;
#pragma unroll
                for (int m = 0; m < NE; m++) {
                    G0[(size_t)(p * NE + m) * ldf] = jw * C[m];
                    if (interior) G1[(size_t)(q * NE + m) * ldf] = jw * -C[m];
                }
            }
            return;
        }
    }
    const auto w = own_coeffs<Mdl, DIM, ORDER>(W, ld, e, fp_dyn_smem);
    double Jinv[DIM * DIM], JinvR[DIM * DIM];
#pragma unroll
    for (int i = 0; i < DIM * DIM; i++) Jinv[i] = ldg(M.geo + (size_t)(GL::JINV + i) * ld + e);
    if (interior) {
#pragma unroll
        for (int i = 0; i < DIM * DIM; i++) JinvR[i] = ldg(M.geo + (size_t)(GL::JINV + i) * ld + TT);
    }
    // the neighbour's coefficients, read at every quadrature point: up to kShNC unknowns
    // they are staged once per face in shared memory beside the owner's (48 KB per CTA)
    constexpr bool kShNb = NC <= kShNC;
    if constexpr (kShNb) {
        if (interior) {
#pragma unroll
            for (int c = 0; c < NC; c++) sh[(NC + c) * kBlock] = ldg(W + (size_t)c * ld + TT);
        }
    }
    using NbA = std::conditional_t<kShNb, NbShared<kBlock>, NbPlain>;
    NbA nbl;
    if constexpr (kShNb)
        nbl = NbShared<kBlock>{sh + NC * kBlock};
    else
        nbl = NbPlain{W, ld};
#pragma unroll 1
    for (int p = 0; p < NQF; p++) {
        double C[NE], Jm[NE];
        El::template face_point<true>(M, e, k, p, TT, n, dL, Jinv, JinvR, kr_face, pm, eps_e, eps_nb, w, nbl, C, Jm);
        const double jw = Jac * ldg(M.tab + TB::o_wf + p);
        const int q = interior ? F.qmap[pm * NQF + p] : 0;
#pragma unroll
        for (int m = 0; m < NE; m++) {
            G0[(size_t)(p * NE + m) * ldf] = jw * (ip ? C[m] - cip_e * Jm[m] : C[m]);
            if (interior) G1[(size_t)(q * NE + m) * ldf] = jw * (ip ? -C[m] + cip_nb * Jm[m] : -C[m]);
        }
    }
}

// The face pass of a mesh too small to fill the GPU with faces: one thread per face and quadrature
// point (blockIdx.y), NQF times the threads, each of which reads the coefficients itself.  Up to
// kFewFaces faces, two thread blocks of the other kernel per SM, a pass is bound by the length of one
// thread's chain: 15,000 triangles p = 1 (22,700 faces) 13.0 -> 7.6 us.
constexpr int kFewFaces = 2 * 148 * kBlock;
struct OwnPlain {
    const double* W;
    size_t ld;
    int e;
    __device__ double operator[](int c) const { return ldg(W + c * ld + e); }
};
template <class Mdl, int DIM, int ORDER>
__global__ void __launch_bounds__(kBlock) k_face_points(DevMesh M, const double* __restrict__ W) {
    using El = E<Mdl, DIM, ORDER>;
    using GL = GeoLayout<DIM>;
    constexpr int NE = El::NE, NQF = El::NQF, NP = El::NP;
    const int f = blockIdx.x * blockDim.x + threadIdx.x, p = blockIdx.y;
    const DevFaces& F = M.F;
    if (f >= F.nFaces) return;
    const int ld = M.ld, ldf = F.ldf;
    const int e = F.fl[f], k = F.fk[f], TT = F.fr[f];
    double n[DIM], Jac, dL;
    El::face_geo(M, e, k, n, Jac, dL);
    const bool interior = TT > -1;
    int kr_face = 0, pm = 0;
    double eps_nb = 0, cip_nb = 0;
    if (interior) {
        const int fc = F.fc[f];
        kr_face = fc / NP;
        pm = fc - kr_face * NP;
        eps_nb = ldg(M.eps + TT);
        cip_nb = ldg(M.cip + TT);
    }
    const double eps_e = ldg(M.eps + e), cip_e = ldg(M.cip + e);
    const bool ip = Mdl::kViscous && (interior || Mdl::isIPFace(TT));
    const OwnPlain w{W, (size_t)ld, e};
    const NbPlain nbl{W, ld};
    double Jinv[DIM * DIM], JinvR[DIM * DIM], C[NE], Jm[NE];
    if (El::needs_gradients(M, interior, eps_e, eps_nb)) {
#pragma unroll
        for (int i = 0; i < DIM * DIM; i++) Jinv[i] = ldg(M.geo + (size_t)(GL::JINV + i) * ld + e);
        if (interior) {
#pragma unroll
            for (int i = 0; i < DIM * DIM; i++) JinvR[i] = ldg(M.geo + (size_t)(GL::JINV + i) * ld + TT);
        }
        El::template face_point<true>(M, e, k, p, TT, n, dL, Jinv, JinvR, kr_face, pm, eps_e, eps_nb, w, nbl, C, Jm);
    } else if constexpr (!Mdl::kViscous) {
        El::template face_point<false>(M, e, k, p, TT, n, dL, Jinv, JinvR, kr_face, pm, eps_e, eps_nb, w, nbl, C, Jm);
    }
    const double jw = Jac * ldg(M.tab + Tab<DIM, ORDER>::o_wf + p);
    const int q = interior ? F.qmap[pm * NQF + p] : 0;
    double* G0 = F.G + f;
    double* G1 = F.G + (size_t)NQF * NE * ldf + f;
#pragma unroll
    for (int m = 0; m < NE; m++) {
        G0[(size_t)(p * NE + m) * ldf] = jw * (ip ? C[m] - cip_e * Jm[m] : C[m]);
        if (interior) G1[(size_t)(q * NE + m) * ldf] = jw * (ip ? -C[m] + cip_nb * Jm[m] : -C[m]);
    }
}

template <class Mdl, int DIM, int ORDER>
__global__ void __launch_bounds__(kBlock, (MinBlocks<Mdl, DIM, ORDER>::elem))
    k_residual(DevMesh M, const double* __restrict__ W, double* __restrict__ R, int e0, int e1) {
    using El = E<Mdl, DIM, ORDER>;
    const int e = e0 + blockIdx.x * blockDim.x + threadIdx.x;  // elements e0 .. e1 - 1
    if (e >= e1) return;
    FP_OWN_COEFFS(El::NC);
    const auto w = own_coeffs<Mdl, DIM, ORDER>(W, M.ld, e, own_wsh);
    double K[El::NC];
    El::residual_from_faces(M, M.F, e, w, K);
#pragma unroll
    for (int c = 0; c < El::NC; c++) R[(size_t)c * M.ld + e] = K[c];
}

// SSP-RK3 stage (RK3.computeExplicitStep, RK3.java:44-86):
// Wout = alpha Wo + beta (Wb + dt M^-1 R(W)); Rsave (optional) = R(W)
template <class Mdl, int DIM, int ORDER>
__global__ void __launch_bounds__(kBlock, (MinBlocks<Mdl, DIM, ORDER>::elem))
    k_rk_stage(DevMesh M, const double* __restrict__ W, const double* __restrict__ Wo, const double* __restrict__ Wb,
               double alpha, double beta, double dt, double* __restrict__ Wout, double* __restrict__ Rsave) {
    using El = E<Mdl, DIM, ORDER>;
    using TB = Tab<DIM, ORDER>;
    constexpr int NB = El::NB, NE = El::NE, NC = El::NC;
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= M.nElem) return;
    const int ld = M.ld;
    FP_OWN_COEFFS(NC);
    const auto w = own_coeffs<Mdl, DIM, ORDER>(W, ld, e, own_wsh);
    double K[NC];
    El::residual_from_faces(M, M.F, e, w, K);
    if (Rsave) {
#pragma unroll
        for (int c = 0; c < NC; c++) Rsave[(size_t)c * ld + e] = K[c];
    }
    const double ijac = 1.0 / ldg(M.geo + (size_t)GeoLayout<DIM>::JAC * ld + e);
#pragma unroll
    for (int m = 0; m < NE; m++)
#pragma unroll
        for (int i = 0; i < NB; i++) {
            double s = 0;
#pragma unroll
            for (int j = 0; j < NB; j++) s += ldg(M.tab + TB::o_MinvRef + i * NB + j) * K[m * NB + j];
            const size_t c = (size_t)(m * NB + i) * ld + e;
            const double wo = alpha != 0.0 ? ldg(Wo + c) : 0.0;
            Wout[c] = alpha * wo + beta * (ldg(Wb + c) + dt * (s * ijac));
        }
}

// Matrix-free Newton operator y = a1 M v - (dR/dW) v (the FD-assembled block matrix
// a1 M - dR/dW of BDF2.assembleJacobiMatrix, applied through the tangent of the residual)
template <class Mdl, int DIM, int ORDER>
__global__ void __launch_bounds__(kBlock)
    k_matfree(DevMesh M, const double* __restrict__ W, const double* __restrict__ V, double a1, double* __restrict__ Y) {
    using El = E<Mdl, DIM, ORDER>;
    using TB = Tab<DIM, ORDER>;
    constexpr int NC = El::NC, NB = El::NB, NE = El::NE;
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= M.nElem) return;
    case_coefficients(M, e, a1);
    const int ld = M.ld;
    // the element's coefficients and tangent in dynamic shared memory ([c][thread] each)
    // when two CTAs' worth fit an SM, else in registers
    constexpr bool kSh = matfree_smem_bytes<NC>() > 0;
    Dual<1> wr[kSh ? 1 : NC];
    double* shv = fp_dyn_smem;
    double* shd = fp_dyn_smem + NC * kBlock;
    if constexpr (kSh) {
#pragma unroll
        for (int c = 0; c < NC; c++) {
            shv[c * kBlock + threadIdx.x] = ldg(W + (size_t)c * ld + e);
            shd[c * kBlock + threadIdx.x] = ldg(V + (size_t)c * ld + e);
        }
    } else {
#pragma unroll
        for (int c = 0; c < NC; c++) {
            wr[c].v = ldg(W + (size_t)c * ld + e);
            wr[c].d[0] = ldg(V + (size_t)c * ld + e);
        }
    }
    using Own = std::conditional_t<kSh, OwnDualShared<kBlock>, const Dual<1>*>;
    Own w;
    if constexpr (kSh)
        w = OwnDualShared<kBlock>{shv + threadIdx.x, shd + threadIdx.x};
    else
        w = wr;
    Dual<1> K[NC];
    El::residual(M, e, w, NbDual<1>{W, V, ld}, K);
    const double jac = ldg(M.geo + (size_t)GeoLayout<DIM>::JAC * ld + e);
#pragma unroll
    for (int m = 0; m < NE; m++)
#pragma unroll
        for (int i = 0; i < NB; i++) {
            double s = 0;
#pragma unroll
            for (int j = 0; j < NB; j++) s += mass_entry<DIM, ORDER>(M, e, 0, i, j, jac) * w[m * NB + j].d[0];
            Y[(size_t)(m * NB + i) * ld + e] = a1 * s - K[m * NB + i].d[0];
        }
}

// Two-pass form of the same operator: the tangent of each face integrand once per face
// (k_face_tan, both sides' weighted contributions into the face buffer G, as k_face does for
// the residual), then per element the gathered face tangents plus the tangent of the volume
// integral (k_matfree_elem).  The element-gather form above evaluates every interior face
// twice, once from each side.  The limiter's eps and c_IP are constants of the step here as
// there (BDF2.assembleJacobiMatrix differentiates the residual at fixed limiter values).
template <class Mdl, int DIM, int ORDER>
__global__ void __launch_bounds__(kBlock, 2) k_face_tan(DevMesh M, const double* __restrict__ W, const double* __restrict__ V) {
    using El = E<Mdl, DIM, ORDER>;
    using GL = GeoLayout<DIM>;
    constexpr int NC = El::NC, NE = El::NE, NQF = El::NQF, NP = El::NP;
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    const DevFaces& F = M.F;
    if (f >= F.nFaces) return;
    const int ld = M.ld, ldf = F.ldf;
    const int e = F.fl[f], k = F.fk[f], TT = F.fr[f];
    if (M.case_live && !__ldg(M.case_live + M.case_of[e])) return;
    // the owner's coefficients and tangent in dynamic shared memory ([c][thread] each) when two
    // CTAs' worth fit an SM, else in registers
    constexpr bool kSh = matfree_smem_bytes<NC>() > 0;
    Dual<1> wr[kSh ? 1 : NC];
    double* shv = fp_dyn_smem;
    double* shd = fp_dyn_smem + NC * kBlock;
    if constexpr (kSh) {
#pragma unroll
        for (int c = 0; c < NC; c++) {
            shv[c * kBlock + threadIdx.x] = ldg(W + (size_t)c * ld + e);
            shd[c * kBlock + threadIdx.x] = ldg(V + (size_t)c * ld + e);
        }
    } else {
#pragma unroll
        for (int c = 0; c < NC; c++) {
            wr[c].v = ldg(W + (size_t)c * ld + e);
            wr[c].d[0] = ldg(V + (size_t)c * ld + e);
        }
    }
    using Own = std::conditional_t<kSh, OwnDualShared<kBlock>, const Dual<1>*>;
    Own w;
    if constexpr (kSh)
        w = OwnDualShared<kBlock>{shv + threadIdx.x, shd + threadIdx.x};
    else
        w = wr;
    double Jinv[DIM * DIM];
#pragma unroll
    for (int i = 0; i < DIM * DIM; i++) Jinv[i] = ldg(M.geo + (size_t)(GL::JINV + i) * ld + e);
    double n[DIM], Jac, dL;
    El::face_geo(M, e, k, n, Jac, dL);
    const bool interior = TT > -1;
    int kr_face = 0, pm = 0;
    double JinvR[DIM * DIM];
    double eps_nb = 0, cip_nb = 0;
    if (interior) {
        const int fc = F.fc[f];
        kr_face = fc / NP;
        pm = fc - kr_face * NP;
#pragma unroll
        for (int i = 0; i < DIM * DIM; i++) JinvR[i] = ldg(M.geo + (size_t)(GL::JINV + i) * ld + TT);
        eps_nb = ldg(M.eps + TT);
        cip_nb = ldg(M.cip + TT);
    }
    const double eps_e = ldg(M.eps + e);
    const double cip_e = ldg(M.cip + e);
    const bool ip = Mdl::kViscous && (interior || Mdl::isIPFace(TT));
    double* G0 = F.G + f;
    double* G1 = F.G + (size_t)NQF * NE * ldf + f;
    const NbDual<1> nbl{W, V, ld};
#pragma unroll 1
    for (int p = 0; p < NQF; p++) {
        Dual<1> C[NE], Jm[NE];
        El::template face_point<true>(M, e, k, p, TT, n, dL, Jinv, JinvR, kr_face, pm, eps_e, eps_nb, w, nbl, C, Jm);
        const double jw = Jac * ldg(M.tab + Tab<DIM, ORDER>::o_wf + p);
        const int q = interior ? F.qmap[pm * NQF + p] : 0;
#pragma unroll
        for (int m = 0; m < NE; m++) {
            const double c = C[m].d[0], j = Jm[m].d[0];
            G0[(size_t)(p * NE + m) * ldf] = jw * (ip ? c - cip_e * j : c);
            if (interior) G1[(size_t)(q * NE + m) * ldf] = jw * (ip ? -c + cip_nb * j : -c);
        }
    }
}

template <class Mdl, int DIM, int ORDER>
__global__ void __launch_bounds__(kBlock, 2)
    k_matfree_elem(DevMesh M, const double* __restrict__ W, const double* __restrict__ V, double a1, double* __restrict__ Y) {
    using El = E<Mdl, DIM, ORDER>;
    using TB = Tab<DIM, ORDER>;
    using GL = GeoLayout<DIM>;
    constexpr int NC = El::NC, NB = El::NB, NE = El::NE, NQF = El::NQF, NF = El::NF;
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= M.nElem) return;
    if (M.case_live && !__ldg(M.case_live + M.case_of[e])) return;
    case_coefficients(M, e, a1);
    const int ld = M.ld;
    constexpr bool kSh = matfree_smem_bytes<NC>() > 0;
    Dual<1> wr[kSh ? 1 : NC];
    double* shv = fp_dyn_smem;
    double* shd = fp_dyn_smem + NC * kBlock;
    if constexpr (kSh) {
#pragma unroll
        for (int c = 0; c < NC; c++) {
            shv[c * kBlock + threadIdx.x] = ldg(W + (size_t)c * ld + e);
            shd[c * kBlock + threadIdx.x] = ldg(V + (size_t)c * ld + e);
        }
    } else {
#pragma unroll
        for (int c = 0; c < NC; c++) {
            wr[c].v = ldg(W + (size_t)c * ld + e);
            wr[c].d[0] = ldg(V + (size_t)c * ld + e);
        }
    }
    using Own = std::conditional_t<kSh, OwnDualShared<kBlock>, const Dual<1>*>;
    Own w;
    if constexpr (kSh)
        w = OwnDualShared<kBlock>{shv + threadIdx.x, shd + threadIdx.x};
    else
        w = wr;
    Dual<1> K[NC];
    // gathered face tangents (their values are not needed: only K.d is used)
    const DevFaces& F = M.F;
#pragma unroll 1
    for (int k = 0; k < NF; k++) {
        const int code = F.efc[(size_t)k * ld + e];
        const int f = code >> 1, side = code & 1;
        const double* G = F.G + (size_t)side * NQF * NE * F.ldf + f;
#pragma unroll
        for (int q = 0; q < NQF; q++) {
            const double* phi = M.tab + TB::o_phiL + (k * NQF + q) * NB;
#pragma unroll
            for (int m = 0; m < NE; m++) {
                const double g = ldg(G + (size_t)(q * NE + m) * F.ldf);
#pragma unroll
                for (int j = 0; j < NB; j++) K[m * NB + j].d[0] += g * ldg(phi + j);
            }
        }
    }
    double Jinv[DIM * DIM];
#pragma unroll
    for (int i = 0; i < DIM * DIM; i++) Jinv[i] = ldg(M.geo + (size_t)(GL::JINV + i) * ld + e);
    El::volume(M, e, w, Jinv, ldg(M.eps + e), K);
    const double jac = ldg(M.geo + (size_t)GL::JAC * ld + e);
#pragma unroll
    for (int m = 0; m < NE; m++)
#pragma unroll
        for (int i = 0; i < NB; i++) {
            double s = 0;
#pragma unroll
            for (int j = 0; j < NB; j++) s += mass_entry<DIM, ORDER>(M, e, 0, i, j, jac) * w[m * NB + j].d[0];
            Y[(size_t)(m * NB + i) * ld + e] = a1 * s - K[m * NB + i].d[0];
        }
}

// ---------------------------------------------------------------------------- limiter
// integral means of the element's coefficients w (an array or an accessor)
template <class Mdl, int DIM, int ORDER, class WA>
__device__ __forceinline__ void element_means(const DevMesh& M, const WA& w, double* Ws) {
    using TB = Tab<DIM, ORDER>;
#pragma unroll
    for (int m = 0; m < Mdl::NE; m++) {
        double s = 0;
#pragma unroll
        for (int j = 0; j < TB::NB; j++) s = s + w[m * TB::NB + j] * ldg(M.tab + TB::o_Is + j);
        Ws[m] = s;
    }
}

// DGpure.limiter + shock_senzor (DGpure.java:358-452): eps = lambda h / order * sensor,
// c_IP = penalty for diffusive models; both zero for piecewise constants.
template <class Mdl, int DIM, int ORDER, class WA>
__device__ __forceinline__ void limiter_values(const DevMesh& M, int e, const WA& w, double dampTol, double penalty,
                                               const double* __restrict__ trun, double& ep, double& ci) {
    using TB = Tab<DIM, ORDER>;
    constexpr int NB = TB::NB, NE = Mdl::NE, NQV = TB::NQV;
    const int ld = M.ld;
    ep = 0;
    ci = 0;
    if (ORDER > 1) {
        if (dampTol > 0) {
            double Ws[NE];
            element_means<Mdl, DIM, ORDER>(M, w, Ws);
            double u[DIM];
#pragma unroll
            for (int d = 0; d < DIM; d++) u[d] = 0;
            const double lam = val(Mdl::maxEigenvalue(Ws, u, M.P));
            double rho[NB], tr[NB];
#pragma unroll
            for (int j = 0; j < NB; j++) rho[j] = w[j];
            if (ORDER > 2) {
#pragma unroll
                for (int i = 0; i < NB; i++) {
                    double s = 0;
#pragma unroll
                    for (int j = 0; j < NB; j++) s += ldg(trun + i * NB + j) * rho[j];
                    tr[i] = s;
                }
            } else {
                double avg = 0;
#pragma unroll
                for (int j = 0; j < NB; j++) avg = avg + rho[j] * ldg(M.tab + TB::o_Is + j);
#pragma unroll
                for (int i = 0; i < NB; i++) tr[i] = avg;
            }
            const double jac = ldg(M.geo + (size_t)GeoLayout<DIM>::JAC * ld + e);
            double Se = 0, pod = 0;
#pragma unroll 1
            for (int q = 0; q < NQV; q++) {
                double ri = 0, rt = 0;
#pragma unroll
                for (int j = 0; j < NB; j++) {
                    const double ph = ldg(M.tab + TB::o_phi + q * NB + j);
                    ri += rho[j] * ph;
                    rt += tr[j] * ph;
                }
                const double jw = jac * ldg(M.tab + TB::o_w + q);
                Se += jw * (ri - rt) * (ri - rt);
                pod += jw * ri * ri;
            }
            Se = log10(fabs(Se / pod));
            const double S0 = log10(1. / pow((double)(ORDER - 1), 4.0));
            double shock = 0.5 * (1 + sin(M_PI * (Se - S0) / (2 * dampTol)));
            if (Se < S0 - dampTol) shock = 0;
            if (Se > S0 + dampTol) shock = 1;
            if (isnan(shock)) shock = 0;
            ep = lam * ldg(M.geo + (size_t)GeoLayout<DIM>::SIZE * ld + e) / ORDER * shock;
        }
        if (Mdl::kViscous) ci = penalty;
    }
}

template <class Mdl, int DIM, int ORDER>
__global__ void __launch_bounds__(kBlock)
    k_limiter(DevMesh M, const double* __restrict__ W, double dampTol, double penalty, const double* __restrict__ trun,
              double* __restrict__ eps, double* __restrict__ cip) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= M.nElem) return;
    double ep, ci;
    limiter_values<Mdl, DIM, ORDER>(M, e, OwnPlain{W, (size_t)M.ld, e}, dampTol, penalty, trun, ep, ci);
    eps[e] = ep;
    cip[e] = ci;
}

// ---------------------------------------------------------------------------- positivity limiter
// Element.positivityLimiter (Element.java:385-476): largest theta in [0,1] (30 bisection
// steps per point) that makes Wavg + theta (W(x) - Wavg) admissible in all volume and
// face quadrature points; W = mean + theta (W - mean).
template <class Mdl, int DIM, int ORDER>
__device__ double admissible_theta(const double* w, const double* Wavg, const double* phi) {
    constexpr int NB = nbasis_of(DIM, ORDER), NE = Mdl::NE;
    double Wx[NE];
#pragma unroll
    for (int m = 0; m < NE; m++) {
        double s = 0;
#pragma unroll
        for (int j = 0; j < NB; j++) s += w[m * NB + j] * ldg(phi + j);
        Wx[m] = s;
    }
    if (Mdl::isAdmissible(Wx)) return 1;
    double lo = 0, hi = 1, Wt[NE];
    for (int it = 0; it < 30; it++) {
        double mid = 0.5 * (lo + hi);
#pragma unroll
        for (int m = 0; m < NE; m++) Wt[m] = Wavg[m] + mid * (Wx[m] - Wavg[m]);
        if (Mdl::isAdmissible(Wt))
            lo = mid;
        else
            hi = mid;
    }
    return lo;
}

// limits the coefficients w in place; true where it changed them
template <class Mdl, int DIM, int ORDER>
__device__ __forceinline__ bool limit_positivity(const DevMesh& M, double* w) {
    using TB = Tab<DIM, ORDER>;
    constexpr int NB = TB::NB, NE = Mdl::NE;
    if (NB == 1) return false;
    double Wavg[NE];
    element_means<Mdl, DIM, ORDER>(M, w, Wavg);
    if (!Mdl::isAdmissible(Wavg)) return false;
    double theta = 1;
    for (int q = 0; q < TB::NQV; q++) theta = fmin(theta, admissible_theta<Mdl, DIM, ORDER>(w, Wavg, M.tab + TB::o_phi + q * NB));
    for (int k = 0; k < TB::NF; k++)
        for (int p = 0; p < TB::NQF; p++)
            theta = fmin(theta, admissible_theta<Mdl, DIM, ORDER>(w, Wavg, M.tab + TB::o_phiL + (k * TB::NQF + p) * NB));
    if (theta >= 1) return false;
#pragma unroll
    for (int m = 0; m < NE; m++)
#pragma unroll
        for (int i = 0; i < NB; i++) {
            const double mean = ldg(M.tab + TB::o_one + i) * Wavg[m];
            w[m * NB + i] = mean + theta * (w[m * NB + i] - mean);
        }
    return true;
}

template <class Mdl, int DIM, int ORDER>
__global__ void __launch_bounds__(kBlock) k_positivity(DevMesh M, double* __restrict__ W, int* __restrict__ count) {
    constexpr int NB = Tab<DIM, ORDER>::NB, NC = Mdl::NE * NB;
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= M.nElem || NB == 1) return;
    double w[NC];
    load_w<Mdl, DIM, ORDER>(W, M.ld, e, w);
    if (!limit_positivity<Mdl, DIM, ORDER>(M, w)) return;
#pragma unroll
    for (int c = 0; c < NC; c++) W[(size_t)c * M.ld + e] = w[c];
    atomicAdd(count, 1);
}

// ---------------------------------------------------------------------------- reductions
// element norms R_m^T M^-1 R_m (Element.l2NormsSquared)
template <class Mdl, int DIM, int ORDER>
__device__ __forceinline__ void element_norms(const DevMesh& M, int e, const double* __restrict__ R, double* nrm) {
    using TB = Tab<DIM, ORDER>;
    constexpr int NB = TB::NB, NE = Mdl::NE;
    const int ld = M.ld;
    const double ijac = 1.0 / ldg(M.geo + (size_t)GeoLayout<DIM>::JAC * ld + e);
#pragma unroll
    for (int m = 0; m < NE; m++) {
        double r[NB];
#pragma unroll
        for (int j = 0; j < NB; j++) r[j] = ldg(R + (size_t)(m * NB + j) * ld + e);
        double sum = 0;
#pragma unroll
        for (int i = 0; i < NB; i++) {
            double t = 0;
#pragma unroll
            for (int j = 0; j < NB; j++) t += ldg(M.tab + TB::o_MinvRef + i * NB + j) * ijac * r[j];
            sum += r[i] * t;
        }
        nrm[m] = sum;
    }
}
// elemSize / lambda / factor (State.getTimeStep, Element.delta_t) of the element's mean state
template <class Mdl, int DIM, int ORDER, class WA>
__device__ __forceinline__ double element_dt(const DevMesh& M, int e, const WA& w, double factor) {
    constexpr int NE = Mdl::NE;
    const int ld = M.ld;
    double Ws[NE];
    element_means<Mdl, DIM, ORDER>(M, w, Ws);
    double u[DIM];
#pragma unroll
    for (int d = 0; d < DIM; d++) {
        u[d] = 0;
        if (M.vu)
            for (int v2 = 0; v2 < DIM + 1; v2++) u[d] += ldg(M.vu + (size_t)(v2 * DIM + d) * ld + e) / (DIM + 1);
    }
    const double lam = val(Mdl::maxEigenvalue(Ws, u, M.P));
    return lam > 0 ? ldg(M.geo + (size_t)GeoLayout<DIM>::SIZE * ld + e) / lam / factor : 1.0e300;
}
// the block's sums of nrm[0 .. NE - 1] into part[block * NE + m], the same tree for any caller
template <int NE>
__device__ __forceinline__ void block_sums(const double* nrm, double* part) {
    __shared__ double sh[kBlock][NE];
#pragma unroll
    for (int m = 0; m < NE; m++) sh[threadIdx.x][m] = nrm[m];
    __syncthreads();
    for (int s = kBlock / 2; s > 0; s >>= 1) {
        if ((int)threadIdx.x < s)
#pragma unroll
            for (int m = 0; m < NE; m++) sh[threadIdx.x][m] += sh[threadIdx.x + s][m];
        __syncthreads();
    }
    if (threadIdx.x == 0)
#pragma unroll
        for (int m = 0; m < NE; m++) part[(size_t)blockIdx.x * NE + m] = sh[0][m];
}
__device__ __forceinline__ void block_min(double v, double* part) {
    __shared__ double sh[kBlock];
    sh[threadIdx.x] = v;
    __syncthreads();
    for (int s = kBlock / 2; s > 0; s >>= 1) {
        if ((int)threadIdx.x < s) sh[threadIdx.x] = fmin(sh[threadIdx.x], sh[threadIdx.x + s]);
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = sh[0];
}

// per-block partial sums of the element norms
template <class Mdl, int DIM, int ORDER>
__global__ void __launch_bounds__(kBlock) k_norms(DevMesh M, const double* __restrict__ R, double* __restrict__ part) {
    constexpr int NE = Mdl::NE;
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    double nrm[NE];
#pragma unroll
    for (int m = 0; m < NE; m++) nrm[m] = 0;
    if (e < M.nElem) element_norms<Mdl, DIM, ORDER>(M, e, R, nrm);
    block_sums<NE>(nrm, part);
}

// per-block minimum of elemSize / lambda
template <class Mdl, int DIM, int ORDER>
__global__ void __launch_bounds__(kBlock) k_dtbound(DevMesh M, const double* __restrict__ W, double factor, double* __restrict__ part) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    block_min(e < M.nElem ? element_dt<Mdl, DIM, ORDER>(M, e, OwnPlain{W, (size_t)M.ld, e}, factor) : 1.0e300, part);
}

// What follows an SSP-RK3 stage, in one pass over the elements instead of a kernel or a copy each:
// the positivity limiter (A.pos: Win -> Wout, the same array or another one), the artificial viscosity
// of the state (A.eps), a copy of it (A.copy), and at the end of a step the partial norms of the
// spatial residual R and the partial time-step bounds of the new state.
template <class Mdl, int DIM, int ORDER>
__global__ void __launch_bounds__(kBlock) k_after_stage(DevMesh M, AfterStage A) {
    using TB = Tab<DIM, ORDER>;
    constexpr int NE = Mdl::NE, NC = NE * TB::NB;
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    double nrm[NE], dt = 1.0e300;
#pragma unroll
    for (int m = 0; m < NE; m++) nrm[m] = 0;
    if (e < M.nElem) {
        const int ld = M.ld;
        if (A.pos || A.copy || A.eps || A.dtPart) {
            double w[NC];
#pragma unroll
            for (int c = 0; c < NC; c++) w[c] = A.Win[(size_t)c * ld + e];
            if (A.pos) {
                limit_positivity<Mdl, DIM, ORDER>(M, w);
#pragma unroll
                for (int c = 0; c < NC; c++) A.Wout[(size_t)c * ld + e] = w[c];
            }
            if (A.copy) {
#pragma unroll
                for (int c = 0; c < NC; c++) A.copy[(size_t)c * ld + e] = w[c];
            }
            if (A.eps) {
                double ep, ci;
                limiter_values<Mdl, DIM, ORDER>(M, e, w, A.dampTol, A.penalty, A.trun, ep, ci);
                A.eps[e] = ep;
                A.cip[e] = ci;
            }
            if (A.dtPart) dt = element_dt<Mdl, DIM, ORDER>(M, e, w, A.factor);
        }
        if (A.normPart) element_norms<Mdl, DIM, ORDER>(M, e, A.R, nrm);
    }
    if (A.normPart) block_sums<NE>(nrm, A.normPart);
    if (A.dtPart) block_min(dt, A.dtPart);
}

// per-element forms of the two reductions above, for a batch of cases (summed or minimised
// per case afterwards): out[m][e] = R_m^T M^-1 R_m of element e, out[e] = elemSize / lambda / factor
template <class Mdl, int DIM, int ORDER>
__global__ void __launch_bounds__(kBlock) k_norms_elem(DevMesh M, const double* __restrict__ R, double* __restrict__ out) {
    constexpr int NE = Mdl::NE;
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= M.nElem) return;
    double nrm[NE];
    element_norms<Mdl, DIM, ORDER>(M, e, R, nrm);
#pragma unroll
    for (int m = 0; m < NE; m++) out[(size_t)m * M.ld + e] = nrm[m];
}

template <class Mdl, int DIM, int ORDER>
__global__ void __launch_bounds__(kBlock)
    k_dtbound_elem(DevMesh M, const double* __restrict__ W, double factor, double* __restrict__ out) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e < M.nElem) out[e] = element_dt<Mdl, DIM, ORDER>(M, e, OwnPlain{W, (size_t)M.ld, e}, factor);
}

// ---------------------------------------------------------------------------- implicit RHS
// Implicit.assembleResiduum (BDF2.java:279-317): R(W), RHS = R - M (a1 W + a2 Wo + a3 Wo2),
// per-block partial sums of |RHS|^2.
template <class Mdl, int DIM, int ORDER>
__global__ void __launch_bounds__(kBlock, (MinBlocks<Mdl, DIM, ORDER>::elem))
    k_rhs(DevMesh M, const double* __restrict__ W, const double* __restrict__ Wo, const double* __restrict__ Wo2, double a1,
          double a2, double a3, double* __restrict__ R, double* __restrict__ rhs, double* __restrict__ part) {
    using El = E<Mdl, DIM, ORDER>;
    using TB = Tab<DIM, ORDER>;
    constexpr int NB = El::NB, NE = El::NE, NC = El::NC;
    __shared__ double sh[kBlock];
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    double loc = 0;
    FP_OWN_COEFFS(NC);
    if (e < M.nElem) {
        case_coefficients(M, e, a1, a2, a3);
        const int ld = M.ld;
        const auto w = own_coeffs<Mdl, DIM, ORDER>(W, ld, e, own_wsh);
        double K[NC];
        El::residual_from_faces(M, M.F, e, w, K);
        const double jac = ldg(M.geo + (size_t)GeoLayout<DIM>::JAC * ld + e);
#pragma unroll
        for (int m = 0; m < NE; m++) {
            double y[NB], yo[NB], yo2[NB];
#pragma unroll
            for (int j = 0; j < NB; j++) {
                const size_t c = (size_t)(m * NB + j) * ld + e;
                y[j] = a1 * w[m * NB + j] + a2 * ldg(Wo + c) + (a3 != 0.0 ? a3 * ldg(Wo2 + c) : 0.0);
                if (M.mass) {  // moving mesh: M a1 W + Mo a2 Wo + Mo2 a3 Wo2 (BDF2.assembleRHS)
                    y[j] = a1 * w[m * NB + j];
                    yo[j] = a2 * ldg(Wo + c);
                    yo2[j] = a3 * ldg(Wo2 + c);
                }
            }
#pragma unroll
            for (int i = 0; i < NB; i++) {
                double s = 0;
                if (M.mass) {
#pragma unroll
                    for (int j = 0; j < NB; j++)
                        s += mass_entry<DIM, ORDER>(M, e, 0, i, j, jac) * y[j] + mass_entry<DIM, ORDER>(M, e, 1, i, j, jac) * yo[j] +
                             mass_entry<DIM, ORDER>(M, e, 2, i, j, jac) * yo2[j];
                } else {
#pragma unroll
                    for (int j = 0; j < NB; j++) s += ldg(M.tab + TB::o_Mref + i * NB + j) * jac * y[j];
                }
                const double v = K[m * NB + i] - s;
                rhs[(size_t)(m * NB + i) * ld + e] = v;
                R[(size_t)(m * NB + i) * ld + e] = K[m * NB + i];
                loc += v * v;
            }
        }
    }
    sh[threadIdx.x] = loc;
    __syncthreads();
    for (int s = kBlock / 2; s > 0; s >>= 1) {
        if ((int)threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = sh[0];
}

// ---------------------------------------------------------------------------- moving mesh
// Mass matrix of time level lev from the current geometry (DGpure.recalculateMassMatrix,
// DGpure.java:575-593): M_ij = sum_p jac w_p phi_i(p) phi_j(p), in the reference's order.
template <int DIM, int ORDER>
__global__ void __launch_bounds__(kBlock) k_mass_geo(DevMesh M, int lev, double* __restrict__ mass) {
    using TB = Tab<DIM, ORDER>;
    constexpr int NB = TB::NB, NQV = TB::NQV;
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= M.nElem) return;
    const int ld = M.ld;
    const double jac = ldg(M.geo + (size_t)GeoLayout<DIM>::JAC * ld + e);
    for (int i = 0; i < NB; i++)
        for (int j = 0; j < NB; j++) {
            double m = 0;
            for (int q = 0; q < NQV; q++)
                m = m + jac * ldg(M.tab + TB::o_w + q) * ldg(M.tab + TB::o_phi + q * NB + i) * ldg(M.tab + TB::o_phi + q * NB + j);
            mass[((size_t)(lev * NB + i) * NB + j) * ld + e] = m;
        }
}

// Discrete geometric conservation law (Element.applyGCLMassMatrix, Element.java:568-630): the
// current level's mass matrix becomes M = (B - a2 Mo - a3 Mo2) / a1 with
// B_ij = sum_faces int (u.n) phi_i phi_j ds - int u . grad(phi_i phi_j) dx, u the mesh velocity
// interpolated from the element's vertices, so that a uniform state satisfies the BDF update
// exactly on the moving mesh.
template <int DIM, int ORDER>
__global__ void __launch_bounds__(kBlock) k_gcl_mass(DevMesh M, double a1, double a2, double a3, double* __restrict__ mass) {
    using TB = Tab<DIM, ORDER>;
    using GL = GeoLayout<DIM>;
    constexpr int NB = TB::NB, NQV = TB::NQV, NQF = TB::NQF, NF = TB::NF, NV = TB::NV, NVF = TB::NVF;
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= M.nElem || !M.vu) return;
    const int ld = M.ld;
    double B[NB][NB];
#pragma unroll
    for (int i = 0; i < NB; i++)
#pragma unroll
        for (int j = 0; j < NB; j++) B[i][j] = 0;
    for (int k = 0; k < NF; k++) {
        double n[DIM];
#pragma unroll
        for (int d = 0; d < DIM; d++) n[d] = ldg(M.geo + (size_t)(GL::NRM + k * DIM + d) * ld + e);
        const double jf = ldg(M.geo + (size_t)(GL::JF + k) * ld + e);
        for (int p = 0; p < NQF; p++) {
            double un = 0;
#pragma unroll
            for (int d = 0; d < DIM; d++) {
                double ud = 0;
#pragma unroll
                for (int v = 0; v < NVF; v++)
                    ud += ldg(M.tab + TB::o_finterp + p * NVF + v) * ldg(M.vu + (size_t)(face_vertex<DIM>(k, v) * DIM + d) * ld + e);
                un += ud * n[d];
            }
            const double* base = M.tab + TB::o_phiL + (k * NQF + p) * NB;
            const double jw = jf * ldg(M.tab + TB::o_wf + p) * un;
#pragma unroll
            for (int i = 0; i < NB; i++)
#pragma unroll
                for (int j = 0; j < NB; j++) B[i][j] += jw * ldg(base + i) * ldg(base + j);
        }
    }
    double Jinv[DIM * DIM];
#pragma unroll
    for (int i = 0; i < DIM * DIM; i++) Jinv[i] = ldg(M.geo + (size_t)(GL::JINV + i) * ld + e);
    const double jac = ldg(M.geo + (size_t)GL::JAC * ld + e);
    for (int q = 0; q < NQV; q++) {
        double u[DIM];
#pragma unroll
        for (int d = 0; d < DIM; d++) u[d] = 0;
#pragma unroll
        for (int v = 0; v < NV; v++)
#pragma unroll
            for (int d = 0; d < DIM; d++) u[d] += ldg(M.tab + TB::o_interp + q * NV + v) * ldg(M.vu + (size_t)(v * DIM + d) * ld + e);
        const double* base = M.tab + TB::o_phi + q * NB;
        const double* dphi = M.tab + TB::o_dphi + q * NB * DIM;
        const double jw = jac * ldg(M.tab + TB::o_w + q);
        double ug[NB];  // u . grad phi_i (physical gradients J^-T grad_xi phi_i)
#pragma unroll
        for (int i = 0; i < NB; i++) {
            double s = 0;
#pragma unroll
            for (int d = 0; d < DIM; d++) {
                double gd = 0;
#pragma unroll
                for (int qq = 0; qq < DIM; qq++) gd += Jinv[qq * DIM + d] * ldg(dphi + i * DIM + qq);
                s += u[d] * gd;
            }
            ug[i] = s;
        }
#pragma unroll
        for (int i = 0; i < NB; i++)
#pragma unroll
            for (int j = 0; j < NB; j++) B[i][j] -= jw * (ug[i] * ldg(base + j) + ldg(base + i) * ug[j]);
    }
#pragma unroll
    for (int i = 0; i < NB; i++)
#pragma unroll
        for (int j = 0; j < NB; j++) {
            const size_t o = (size_t)(i * NB + j) * ld + e, lv = (size_t)NB * NB * ld;
            mass[o] = (B[i][j] - a2 * mass[o + lv] - a3 * mass[o + 2 * lv]) / a1;
        }
}

// a contiguous column of NC values, two at a time where their address allows it
template <int NC, class T>
__device__ __forceinline__ void store_column(T* dst, const double* v) {
    if constexpr (NC % 2 == 0) {
        using T2 = std::conditional_t<sizeof(T) == 8, double2, float2>;
#pragma unroll
        for (int r = 0; r < NC; r += 2) {
            T2 x;
            x.x = (T)v[r];
            x.y = (T)v[r + 1];
            reinterpret_cast<T2*>(dst)[r / 2] = x;
        }
    } else {
#pragma unroll
        for (int r = 0; r < NC; r++) dst[r] = (T)v[r];
    }
}

}  // namespace fp
#include "fp_jacobian.cuh"
namespace fp {

// ---------------------------------------------------------------------------- surface integrals
// kind 0: force on the faces of boundary type bc, F = -sum int stressVector ds
//         (Deformation2DRigid.calculateForces, Deformation2DRigid.java:81-105);
// kind 1 / 2: lift / drag coefficient functional, int p n_y (n_x) ds on faces of type bc
//         (LiftCoefficient.java:31-49, DragCoefficient.java:30-48, summed as
//         Element.computeFunctional, Element.java:789-862), and optionally its exact
//         gradient dI/dW (forward mode over the trace state, state layout).
// Per-block partial sums part[block * 4 + v] (deterministic order on the host).
template <class Mdl, int DIM, int ORDER>
__global__ void __launch_bounds__(kBlock)
    k_surface(DevMesh M, const double* __restrict__ W, int kind, int bc, double* __restrict__ part, double* __restrict__ dIdW) {
    using El = E<Mdl, DIM, ORDER>;
    using TB = Tab<DIM, ORDER>;
    using GL = GeoLayout<DIM>;
    constexpr int NB = El::NB, NE = El::NE, NQF = El::NQF, NF = El::NF, NC = El::NC;
    __shared__ double sh[kBlock][4];
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    if (e < M.nElem) {
        const int ld = M.ld;
        bool any = false;
#pragma unroll
        for (int k = 0; k < NF; k++) any = any || M.tt[(size_t)k * ld + e] == bc;
        const bool grad = dIdW != nullptr && kind > 0;
        double g[NC];
#pragma unroll
        for (int c = 0; c < NC; c++) g[c] = 0.0;
        if (any) {
            double w[NC];
            load_w<Mdl, DIM, ORDER>(W, ld, e, w);
            double Jinv[DIM * DIM];
#pragma unroll
            for (int q = 0; q < DIM * DIM; q++) Jinv[q] = ldg(M.geo + (size_t)(GL::JINV + q) * ld + e);
#pragma unroll 1
            for (int k = 0; k < NF; k++) {
                if (M.tt[(size_t)k * ld + e] != bc) continue;
                double n[DIM], Jac, dL;
                El::face_geo(M, e, k, n, Jac, dL);
#pragma unroll 1
                for (int p = 0; p < NQF; p++) {
                    const double* phi = M.tab + TB::o_phiL + (k * NQF + p) * NB;
                    const double* dphi = M.tab + TB::o_dphiL + (k * NQF + p) * NB * DIM;
                    double WL[NE], dWL[DIM * NE], gr[DIM * NE];
#pragma unroll
                    for (int m = 0; m < NE; m++) {
                        WL[m] = 0.0;
#pragma unroll
                        for (int d = 0; d < DIM; d++) gr[d * NE + m] = 0.0;
#pragma unroll
                        for (int j = 0; j < NB; j++) {
                            WL[m] += w[m * NB + j] * ldg(phi + j);
#pragma unroll
                            for (int d = 0; d < DIM; d++) gr[d * NE + m] += w[m * NB + j] * ldg(dphi + j * DIM + d);
                        }
                    }
#pragma unroll
                    for (int m = 0; m < NE; m++)
#pragma unroll
                        for (int d = 0; d < DIM; d++) {
                            double s = 0.0;
#pragma unroll
                            for (int q = 0; q < DIM; q++) s += Jinv[q * DIM + d] * gr[q * NE + m];
                            dWL[d * NE + m] = s;
                        }
                    const double jw = Jac * ldg(M.tab + TB::o_wf + p);
                    if (kind == 0) {
                        double sv[DIM];
                        Mdl::stressVector(WL, dWL, n, sv, M.P);
#pragma unroll
                        for (int d = 0; d < DIM; d++) acc[d] -= jw * sv[d];
                    } else {
                        Dual<NE> Wd[NE];
#pragma unroll
                        for (int m = 0; m < NE; m++) {
                            Wd[m] = Dual<NE>(WL[m]);
                            Wd[m].d[m] = 1.0;
                        }
                        const Dual<NE> val = Mdl::functionalPressure(Wd, M.P) * n[kind == 1 ? 1 : 0];
                        acc[0] += jw * val.v;
                        if (grad) {
#pragma unroll
                            for (int m = 0; m < NE; m++) {
                                const double gm = jw * val.d[m];
#pragma unroll
                                for (int j = 0; j < NB; j++) g[m * NB + j] += gm * ldg(phi + j);
                            }
                        }
                    }
                }
            }
        }
        if (grad) {
#pragma unroll
            for (int c = 0; c < NC; c++) dIdW[(size_t)c * ld + e] = g[c];
        }
    }
#pragma unroll
    for (int v = 0; v < 4; v++) sh[threadIdx.x][v] = acc[v];
    __syncthreads();
    for (int s2 = kBlock / 2; s2 > 0; s2 >>= 1) {
        if ((int)threadIdx.x < s2)
#pragma unroll
            for (int v = 0; v < 4; v++) sh[threadIdx.x][v] += sh[threadIdx.x + s2][v];
        __syncthreads();
    }
    if (threadIdx.x == 0)
#pragma unroll
        for (int v = 0; v < 4; v++) part[(size_t)blockIdx.x * 4 + v] = sh[0][v];
}

// ---------------------------------------------------------------------------- launch table
inline unsigned grid_of(int n) { return (unsigned)((n + kBlock - 1) / kBlock); }

template <class Mdl, int DIM, int ORDER>
struct Launch {
    // dynamic shared memory of the face and element kernels (the element's coefficients when
    // they do not fit the static array), allowed once per kernel before its first launch
    static constexpr size_t kDyn = own_smem_bytes<Element<Mdl, DIM, ORDER>::NC>();
    static constexpr size_t kDynFace = face_smem_bytes<Element<Mdl, DIM, ORDER>::NC,
                                                       Element<Mdl, DIM, ORDER>::NQF * Element<Mdl, DIM, ORDER>::NE, Mdl::kViscous>();
    template <class K>
    static void allow_dyn(K* kernel, size_t bytes = kDyn) {
        if (bytes > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    }
    // the attribute belongs to the current device: set once per device (the first 64 devices
    // are remembered; beyond them it is set on every call, which is harmless)
    static void prepare() {
        static std::atomic<unsigned long long> done{0};
        int dev = 0;
        cudaGetDevice(&dev);
        const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
        if (bit && (done.load(std::memory_order_acquire) & bit)) return;
        allow_dyn(k_face<Mdl, DIM, ORDER>, kDynFace);
        allow_dyn(k_residual<Mdl, DIM, ORDER>);
        allow_dyn(k_rk_stage<Mdl, DIM, ORDER>);
        allow_dyn(k_rhs<Mdl, DIM, ORDER>);
        constexpr size_t mf = matfree_smem_bytes<Element<Mdl, DIM, ORDER>::NC>();
        if (mf > 48 * 1024) {
            cudaFuncSetAttribute(k_matfree<Mdl, DIM, ORDER>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mf);
            cudaFuncSetAttribute(k_face_tan<Mdl, DIM, ORDER>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mf);
            cudaFuncSetAttribute(k_matfree_elem<Mdl, DIM, ORDER>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mf);
        }
        done.fetch_or(bit, std::memory_order_release);
    }
    static void faces(const DevMesh& M, cudaStream_t s, const double* W) {
        prepare();
        if (M.F.nFaces <= kFewFaces && Element<Mdl, DIM, ORDER>::NQF > 1)
            k_face_points<Mdl, DIM, ORDER><<<dim3(grid_of(M.F.nFaces), Element<Mdl, DIM, ORDER>::NQF), kBlock, 0, s>>>(M, W);
        else
            k_face<Mdl, DIM, ORDER><<<grid_of(M.F.nFaces), kBlock, kDynFace, s>>>(M, W, 0, M.F.nFaces);
    }
    static void elements(const DevMesh& M, cudaStream_t s, const double* W, double* R) {
        prepare();
        k_residual<Mdl, DIM, ORDER><<<grid_of(M.nElem), kBlock, kDyn, s>>>(M, W, R, 0, M.nElem);
    }
    static void faces_range(const DevMesh& M, cudaStream_t s, const double* W, int f0, int f1) {
        prepare();
        if (f1 > f0) k_face<Mdl, DIM, ORDER><<<grid_of(f1 - f0), kBlock, kDynFace, s>>>(M, W, f0, f1);
    }
    static void elements_range(const DevMesh& M, cudaStream_t s, const double* W, double* R, int e0, int e1) {
        prepare();
        if (e1 > e0) k_residual<Mdl, DIM, ORDER><<<grid_of(e1 - e0), kBlock, kDyn, s>>>(M, W, R, e0, e1);
    }
    static void residual(const DevMesh& M, cudaStream_t s, const double* W, double* R) {
        faces(M, s, W);
        elements(M, s, W, R);
    }
    static void rk_stage(const DevMesh& M, cudaStream_t s, const double* W, const double* Wo, const double* Wb, double a,
                         double b, double dt, double* Wout, double* Rsave) {
        faces(M, s, W);
        k_rk_stage<Mdl, DIM, ORDER><<<grid_of(M.nElem), kBlock, kDyn, s>>>(M, W, Wo, Wb, a, b, dt, Wout, Rsave);
    }
    // the matrix-free operator: tangent face pass (face buffer G as scratch) + element pass
    static void matfree(const DevMesh& M, cudaStream_t s, const double* W, const double* V, double a1, double* Y) {
        prepare();
        constexpr size_t sm = matfree_smem_bytes<Element<Mdl, DIM, ORDER>::NC>();
        k_face_tan<Mdl, DIM, ORDER><<<grid_of(M.F.nFaces), kBlock, sm, s>>>(M, W, V);
        k_matfree_elem<Mdl, DIM, ORDER><<<grid_of(M.nElem), kBlock, sm, s>>>(M, W, V, a1, Y);
    }
    // the element-gather form (both sides of every face), kept for comparison
    static void matfree_gather(const DevMesh& M, cudaStream_t s, const double* W, const double* V, double a1, double* Y) {
        prepare();
        k_matfree<Mdl, DIM, ORDER><<<grid_of(M.nElem), kBlock, matfree_smem_bytes<Element<Mdl, DIM, ORDER>::NC>(), s>>>(
            M, W, V, a1, Y);
    }
    static void limiter(const DevMesh& M, cudaStream_t s, const double* W, double dampTol, double penalty, const double* trun,
                        double* eps, double* cip) {
        k_limiter<Mdl, DIM, ORDER><<<grid_of(M.nElem), kBlock, 0, s>>>(M, W, dampTol, penalty, trun, eps, cip);
    }
    static void positivity(const DevMesh& M, cudaStream_t s, double* W, int* count) {
        k_positivity<Mdl, DIM, ORDER><<<grid_of(M.nElem), kBlock, 0, s>>>(M, W, count);
    }
    static void after_stage(const DevMesh& M, cudaStream_t s, const AfterStage& A) {
        k_after_stage<Mdl, DIM, ORDER><<<grid_of(M.nElem), kBlock, 0, s>>>(M, A);
    }
    static void norms(const DevMesh& M, cudaStream_t s, const double* R, double* part) {
        k_norms<Mdl, DIM, ORDER><<<grid_of(M.nElem), kBlock, 0, s>>>(M, R, part);
    }
    static void dtbound(const DevMesh& M, cudaStream_t s, const double* W, double factor, double* part) {
        k_dtbound<Mdl, DIM, ORDER><<<grid_of(M.nElem), kBlock, 0, s>>>(M, W, factor, part);
    }
    static void rhs(const DevMesh& M, cudaStream_t s, const double* W, const double* Wo, const double* Wo2, double a1,
                    double a2, double a3, double* R, double* rhs, double* part) {
        faces(M, s, W);
        k_rhs<Mdl, DIM, ORDER><<<grid_of(M.nElem), kBlock, kDyn, s>>>(M, W, Wo, Wo2, a1, a2, a3, R, rhs, part);
    }
    // finite-difference blocks, with the traces' gradients where they are read, as below
    template <bool GRAD>
    static void fd_as(const DevMesh& M, cudaStream_t s, const double* W, double h, double a1, double* Adiag, double* Aneigh) {
        using C = FdCfg<Mdl, DIM, ORDER, GRAD>;
        cudaFuncSetAttribute(k_fd<Mdl, DIM, ORDER, GRAD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
        k_fd<Mdl, DIM, ORDER, GRAD>
            <<<(unsigned)((M.nElem + C::E - 1) / C::E), C::THREADS, C::SMEM, s>>>(M, W, h, a1, Adiag, Aneigh);
    }
    static void fd(const DevMesh& M, cudaStream_t s, const double* W, double h, double a1, double* Adiag, double* Aneigh) {
        if (Mdl::kViscous || Mdl::kSource || M.artificial)
            fd_as<true>(M, s, W, h, a1, Adiag, Aneigh);
        else if constexpr (!Mdl::kViscous && !Mdl::kSource)
            fd_as<false>(M, s, W, h, a1, Adiag, Aneigh);
    }
    // exact blocks and adjoint product: with the gradients' matrices where a model or the artificial
    // viscosity reads gradients (the limiter leaves none without dampTol)
    template <bool GRAD, int MODE, class T>
    static void jacobian_as(const DevMesh& M, cudaStream_t s, const double* W, double a1, double* Ad, double* An, T* F,
                            const double* lam, double* g) {
        using C = JacCfg<Mdl, DIM, ORDER, GRAD>;
        cudaFuncSetAttribute(k_jacobian<Mdl, DIM, ORDER, GRAD, MODE, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
        k_jacobian<Mdl, DIM, ORDER, GRAD, MODE, T>
            <<<(unsigned)((M.nElem + C::E - 1) / C::E), C::THREADS, C::SMEM, s>>>(M, W, a1, Ad, An, F, lam, g);
    }
    template <int MODE, class T>
    static void jacobian(const DevMesh& M, cudaStream_t s, const double* W, double a1, double* Ad, double* An, T* F,
                         const double* lam, double* g) {
        if (Mdl::kViscous || Mdl::kSource || M.artificial)
            jacobian_as<true, MODE, T>(M, s, W, a1, Ad, An, F, lam, g);
        else if constexpr (!Mdl::kViscous && !Mdl::kSource)
            jacobian_as<false, MODE, T>(M, s, W, a1, Ad, An, F, lam, g);
    }
    static void jac_exact(const DevMesh& M, cudaStream_t s, const double* W, double a1, double* Adiag, double* Aneigh) {
        jacobian<JAC_BLOCKS, double>(M, s, W, a1, Adiag, Aneigh, nullptr, nullptr, nullptr);
    }
    static void jac_exact_factor(const DevMesh& M, cudaStream_t s, const double* W, double a1, void* F, int fp32) {
        if (fp32)
            jacobian<JAC_FACTOR, float>(M, s, W, a1, nullptr, nullptr, (float*)F, nullptr, nullptr);
        else
            jacobian<JAC_FACTOR, double>(M, s, W, a1, nullptr, nullptr, (double*)F, nullptr, nullptr);
    }
    static void norms_elem(const DevMesh& M, cudaStream_t s, const double* R, double* out) {
        k_norms_elem<Mdl, DIM, ORDER><<<grid_of(M.nElem), kBlock, 0, s>>>(M, R, out);
    }
    static void dtbound_elem(const DevMesh& M, cudaStream_t s, const double* W, double factor, double* out) {
        k_dtbound_elem<Mdl, DIM, ORDER><<<grid_of(M.nElem), kBlock, 0, s>>>(M, W, factor, out);
    }
    static void mass_geo(const DevMesh& M, cudaStream_t s, int lev, double* mass) {
        k_mass_geo<DIM, ORDER><<<grid_of(M.nElem), kBlock, 0, s>>>(M, lev, mass);
    }
    static void gcl_mass(const DevMesh& M, cudaStream_t s, double a1, double a2, double a3, double* mass) {
        k_gcl_mass<DIM, ORDER><<<grid_of(M.nElem), kBlock, 0, s>>>(M, a1, a2, a3, mass);
    }
    static void vjp(const DevMesh& M, cudaStream_t s, const double* W, const double* lam, double* g) {
        jacobian<JAC_VJP, double>(M, s, W, 0.0, nullptr, nullptr, nullptr, lam, g);
    }
    static void surface(const DevMesh& M, cudaStream_t s, const double* W, int kind, int bc, double* part, double* dIdW) {
        k_surface<Mdl, DIM, ORDER><<<grid_of(M.nElem), kBlock, 0, s>>>(M, W, kind, bc, part, dIdW);
    }
    static Launchers table() {
        Launchers t;
        t.nc = Element<Mdl, DIM, ORDER>::NC;
        t.ntrun = Tab<DIM, ORDER>::NB * Tab<DIM, ORDER>::NB;
        t.residual = residual;
        t.faces = faces;
        t.elements = elements;
        t.faces_range = faces_range;
        t.elements_range = elements_range;
        t.rk_stage = rk_stage;
        t.matfree = matfree;
        t.matfree_gather = matfree_gather;
        t.limiter = limiter;
        t.positivity = positivity;
        t.after_stage = after_stage;
        t.norms = norms;
        t.dtbound = dtbound;
        t.rhs = rhs;
        t.fd = fd;
        t.jac_exact = jac_exact;
        t.jac_exact_factor = jac_exact_factor;
        t.vjp = vjp;
        t.mass_geo = mass_geo;
        t.norms_elem = norms_elem;
        t.dtbound_elem = dtbound_elem;
        t.gcl_mass = gcl_mass;
        t.surface = surface;
        return t;
    }
};

}  // namespace fp
