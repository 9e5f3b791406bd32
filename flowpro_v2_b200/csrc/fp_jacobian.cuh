// Element Jacobian blocks: exact ones and the adjoint product here, finite differences below.
//
// Exact blocks come from the flux Jacobians at the quadrature points.  Column i = (mi, bi) of an element's blocks is the derivative of the element residual, and of the
// element's face contributions to its neighbours, along the coefficient of basis function bi in equation
// mi.  The integrand at a point depends on that coefficient through the state phi_bi and, where gradients
// are read, the reference gradients dphi_bi, so the NE x NE matrices of the integrand with respect to the
// state and each reference gradient hold all there is to know about the point: one tangent of the
// integrand per equation and set (S = 1, or 1 + DIM with gradients), instead of one of the whole element
// residual, traces included, per column.
//
// A thread block takes E elements.  Faces first: the traces of all their points, the matrices (a thread
// per element, point and seed direction) into shared memory, then a thread per element and column
// multiplies them with the basis.  Then the volume points the same way.
//
// What bounds it: the products with the basis, about NC multiply-adds a point and column, each
// shared-memory load feeding NB of them.  Measured, ms: 86,700 tetrahedra p = 2 (50 unknowns, FP32 factor
// storage) 38.7 -> 8.4; 8,832 triangles Spalart-Allmaras p = 2 1.24 -> 0.55; the adjoint product of 10,004
// triangles Navier-Stokes p = 2 0.63 -> 0.16.  Where gradients are read only through the artificial viscosity,
// their matrices exist only at the points that have any: 106,400 triangles Euler p = 1 with the shock sensor on,
// none active 1.07 -> 0.82, 17 % of the elements active 1.08 -> 0.97 (0.84 before these kernels); 61,440
// tetrahedra 4.2 -> 3.0 and 4.3 -> 3.5 (3.3).
#pragma once

namespace fp {

enum JacMode { JAC_BLOCKS, JAC_FACTOR, JAC_VJP };

template <class Mdl, int DIM, int ORDER, bool GRAD>
struct JacCfg {
    using El = Element<Mdl, DIM, ORDER>;
    static constexpr int NC = El::NC, NE = El::NE, NB = El::NB;
    static constexpr int S = GRAD ? 1 + DIM : 1;               // what a column enters a point through
    static constexpr int PF = El::NF * El::NQF, PV = El::NQV;  // points of an element
    static constexpr int OUT = DIM + (Mdl::kSource ? 1 : 0);   // volume integrand: reference gradients, source
    static constexpr int TRF = 2 * NE * S, TRV = NE * S;       // trace values of a point
    static constexpr int MATF = S * NE * NE, MATV = S * OUT * NE * NE;
    static constexpr int LAM = OUT * NE;                       // adjoint weights of a point (faces: NE)
    static constexpr int cmax(int a, int b) { return a > b ? a : b; }
    // doubles of shared memory per element: traces, matrices, adjoint weights, each as many as the faces or
    // the volume take
    static constexpr int TR = cmax(PF * TRF, PV * TRV), MAT = cmax(PF * MATF, PV * MATV), LM = cmax(PF * NE, PV * LAM);
    static constexpr int PER = TR + MAT + LM;
    static constexpr int THREADS = 256;
    static constexpr int cmin(int a, int b) { return a < b ? a : b; }
    static constexpr int E = cmax(1, cmin(cmin(32, THREADS / NC), (108 * 1024 / 8) / PER));
    static constexpr size_t SMEM = (size_t)E * PER * sizeof(double);
    static constexpr int CTAS = SMEM <= 112 * 1024 ? 2 : 1;
    // task t of points * S * NE: point, seed set s and equation m.  Where gradients are read only through the
    // artificial viscosity, the sets s > 0 of most points have nothing to do: they come last, so that whole
    // warps skip them.
    static __device__ __forceinline__ void task(int t, int points, int& point, int& s, int& m) {
        if (Mdl::kViscous || Mdl::kSource) {
            point = t / (S * NE);
            const int seed = t - point * S * NE;
            s = seed / NE;
            m = seed - s * NE;
        } else {
            s = t / (points * NE);
            t -= s * points * NE;
            point = t / NE;
            m = t - point * NE;
        }
    }
};

// MODE JAC_BLOCKS: Adiag = a1 M - dR/dW and Aneigh in the field-major storage of the operator; JAC_FACTOR:
// the same values in the block ILU(0) storage F[e][s][c][r] (T); JAC_VJP: g = (dR/dW)^T lam.
template <class Mdl, int DIM, int ORDER, bool GRAD, int MODE, class T>
__global__ void __launch_bounds__(JacCfg<Mdl, DIM, ORDER, GRAD>::THREADS, (JacCfg<Mdl, DIM, ORDER, GRAD>::CTAS))
    k_jacobian(DevMesh M, const double* __restrict__ W, double a1, double* __restrict__ Adiag, double* __restrict__ Aneigh,
               T* __restrict__ F, const double* __restrict__ lam, double* __restrict__ g) {
    using C = JacCfg<Mdl, DIM, ORDER, GRAD>;
    using El = Element<Mdl, DIM, ORDER>;
    using TB = Tab<DIM, ORDER>;
    using GL = GeoLayout<DIM>;
    constexpr int NC = C::NC, NE = C::NE, NB = C::NB, NF = El::NF, NQF = El::NQF, NQV = El::NQV, NP = El::NP, S = C::S, E = C::E;
    extern __shared__ __align__(16) double fp_dyn_smem[];
    double* trc = fp_dyn_smem;                                   // traces
    double* mat = trc + E * C::TR;
    double* lm = mat + E * C::MAT;
    const int e0 = blockIdx.x * E, n = min(E, M.nElem - e0);
    const int ld = M.ld;
    const int el = threadIdx.x / NC, i = threadIdx.x - el * NC;  // this thread's column
    const bool act = el < n;
    const int mi = i / NB, bi = i - mi * NB;
    const int e = e0 + (act ? el : 0);

    // ------------------------------------------------------------------ faces: traces
    for (int t = threadIdx.x; t < n * C::PF; t += C::THREADS) {
        const int x = t / C::PF, pt = t - x * C::PF, k = pt / NQF, p = pt - k * NQF, ee = e0 + x;
        const int TT = M.tt[(size_t)k * ld + ee];
        double* o = trc + (size_t)t * C::TRF;
        double Ji[DIM * DIM], v[NE], dv[GRAD ? DIM * NE : 1];
        const double* phiL = M.tab + TB::o_phiL + (k * NQF + p) * NB;
        if constexpr (GRAD) {
#pragma unroll
            for (int c = 0; c < DIM * DIM; c++) Ji[c] = ldg(M.geo + (size_t)(GL::JINV + c) * ld + ee);
        }
        El::template trace<GRAD>(phiL, M.tab + TB::o_dphiL + (k * NQF + p) * NB * DIM, Ji,
                                 [&](int c) { return ldg(W + (size_t)c * ld + ee); }, v, dv);
#pragma unroll
        for (int m = 0; m < NE; m++) o[m] = v[m];
        if constexpr (GRAD) {
#pragma unroll
            for (int c = 0; c < DIM * NE; c++) o[NE + c] = dv[c];
        }
        const int fc = TT > -1 ? M.fcode[(size_t)k * ld + ee] : 0;
        const double* phiR = M.tab + TB::o_phiR + (fc * NQF + p) * NB;
        if (TT > -1) {
            if constexpr (GRAD) {
#pragma unroll
                for (int c = 0; c < DIM * DIM; c++) Ji[c] = ldg(M.geo + (size_t)(GL::JINV + c) * ld + TT);
            }
            El::template trace<GRAD>(phiR, M.tab + TB::o_dphiR + (fc * NQF + p) * NB * DIM, Ji,
                                     [&](int c) { return ldg(W + (size_t)c * ld + TT); }, v, dv);
#pragma unroll
            for (int m = 0; m < NE; m++) o[NE * S + m] = v[m];
            if constexpr (GRAD) {
#pragma unroll
                for (int c = 0; c < DIM * NE; c++) o[NE * S + NE + c] = dv[c];
            }
        }
        if constexpr (MODE == JAC_VJP) {  // the rows that the point's integrand feeds: the element's and the neighbour's
            for (int m = 0; m < NE; m++) {
                double s = 0;
                for (int j = 0; j < NB; j++) {
                    s += ldg(lam + (size_t)(m * NB + j) * ld + ee) * ldg(phiL + j);
                    if (TT > -1) s -= ldg(lam + (size_t)(m * NB + j) * ld + TT) * ldg(phiR + j);
                }
                lm[t * NE + m] = s;
            }
        }
    }
    __syncthreads();
    // ------------------------------------------------------------------ faces: matrices
    for (int t = threadIdx.x; t < n * C::PF * S * NE; t += C::THREADS) {
        int xp, s, mj;
        C::task(t, n * C::PF, xp, s, mj);
        const int x = xp / C::PF, pt = xp - x * C::PF, k = pt / NQF, p = pt - k * NQF, ee = e0 + x;
        const int TT = M.tt[(size_t)k * ld + ee];
        const bool interior = TT > -1;
        const double eps_e = ldg(M.eps + ee), eps_nb = interior ? ldg(M.eps + TT) : 0.0;
        if (s > 0 && !El::needs_gradients(M, interior, eps_e, eps_nb)) continue;  // nothing reads this matrix
        const double* o = trc + (size_t)xp * C::TRF;
        constexpr int NG = GRAD ? DIM * NE : 1;
        Dual<1> WL[NE], WR[NE], dWL[NG], dWR[NG], Cc[NE], Jm[NE];
#pragma unroll
        for (int m = 0; m < NE; m++) {
            WL[m] = Dual<1>(o[m]);
            if (s == 0 && m == mj) WL[m].d[0] = 1.0;
            if (interior) WR[m] = Dual<1>(o[NE * S + m]);
        }
        if constexpr (GRAD) {
#pragma unroll
            for (int d = 0; d < DIM; d++) {
                // seed s > 0: the reference gradient s - 1 of equation mj
                const double jd = s > 0 ? ldg(M.geo + (size_t)(GL::JINV + (s - 1) * DIM + d) * ld + ee) : 0.0;
#pragma unroll
                for (int m = 0; m < NE; m++) {
                    dWL[d * NE + m] = Dual<1>(o[NE + d * NE + m]);
                    if (m == mj) dWL[d * NE + m].d[0] = jd;
                    if (interior) dWR[d * NE + m] = Dual<1>(o[NE * S + NE + d * NE + m]);
                }
            }
        }
        double nrm[DIM], Jac, dL;
        El::face_geo(M, ee, k, nrm, Jac, dL);
        El::template point_flux<GRAD>(M, ee, k, p, TT, nrm, dL, eps_e, eps_nb, WL, WR, dWL, dWR, Cc, Jm);
        const double jw = Jac * ldg(M.tab + TB::o_wf + p);
        const double cip = Mdl::kViscous && (interior || Mdl::isIPFace(TT)) ? ldg(M.cip + ee) : 0.0;
        double* q = mat + (size_t)xp * C::MATF + s * NE * NE + mj;
#pragma unroll
        for (int m = 0; m < NE; m++) q[m * NE] = jw * (Cc[m].d[0] - cip * Jm[m].d[0]);
    }
    __syncthreads();
    // ------------------------------------------------------------------ faces: products with the basis
    double K[MODE == JAC_VJP ? 1 : NC];
    double gi = 0.0;
    // the faces whose gradients' matrices exist (one bit each)
    unsigned gradFaces = 0u;
    if constexpr (GRAD) {
#pragma unroll
        for (int k = 0; k < NF; k++) {
            const int TT = M.tt[(size_t)k * ld + e];
            if (El::needs_gradients(M, TT > -1, ldg(M.eps + e), TT > -1 ? ldg(M.eps + TT) : 0.0)) gradFaces |= 1u << k;
        }
    }
    // row m of the point's matrix times what the column enters through
    auto entry = [&](const double* q, int k, int m, double ph, const double* dph) {
        double a = q[m * NE + mi] * ph;
        if constexpr (GRAD) {
            if (Mdl::kViscous || (gradFaces >> k & 1u)) {
#pragma unroll
                for (int d = 0; d < DIM; d++) a += q[((1 + d) * NE + m) * NE + mi] * dph[d];
            }
        }
        return a;
    };
    auto column = [&](const double* phi, const double* dphi, double& ph, double* dph) {
        ph = ldg(phi + bi);
        if constexpr (GRAD) {
#pragma unroll
            for (int d = 0; d < DIM; d++) dph[d] = ldg(dphi + bi * DIM + d);
        }
    };
    if (act) {
        if constexpr (MODE == JAC_VJP) {
#pragma unroll 1
            for (int pt = 0; pt < C::PF; pt++) {
                double ph, dph[DIM];
                column(M.tab + TB::o_phiL + pt * NB, M.tab + TB::o_dphiL + pt * NB * DIM, ph, dph);
                const double* q = mat + (size_t)(el * C::PF + pt) * C::MATF;
#pragma unroll
                for (int m = 0; m < NE; m++) gi += entry(q, pt / NQF, m, ph, dph) * lm[(el * C::PF + pt) * NE + m];
            }
        } else {
            // what the element's faces add to its neighbours' rows
#pragma unroll 1
            for (int k = 0; k < NF; k++) {
                const int nb = M.tt[(size_t)k * ld + e];
                if (nb < 0) continue;
                const int fc = M.fcode[(size_t)k * ld + e], kr = fc / NP;
#pragma unroll
                for (int c = 0; c < NC; c++) K[c] = 0.0;
#pragma unroll 1
                for (int p = 0; p < NQF; p++) {
                    const int pt = k * NQF + p;
                    double ph, dph[DIM];
                    column(M.tab + TB::o_phiL + pt * NB, M.tab + TB::o_dphiL + pt * NB * DIM, ph, dph);
                    const double* q = mat + (size_t)(el * C::PF + pt) * C::MATF;
                    const double* phiR = M.tab + TB::o_phiR + (fc * NQF + p) * NB;
                    double a[NE];
#pragma unroll
                    for (int m = 0; m < NE; m++) a[m] = entry(q, k, m, ph, dph);
#pragma unroll
                    for (int j = 0; j < NB; j++) {
                        const double pr = ldg(phiR + j);
#pragma unroll
                        for (int m = 0; m < NE; m++) K[m * NB + j] += a[m] * pr;
                    }
                }
                if constexpr (MODE == JAC_BLOCKS) {
                    double* A = Aneigh + (size_t)kr * NC * NC * ld;
#pragma unroll
                    for (int r = 0; r < NC; r++) A[((size_t)r * NC + i) * ld + nb] = K[r];
                } else {
                    store_column<NC>(F + (((size_t)nb * (1 + NF) + 1 + kr) * NC + i) * NC, K);
                }
            }
#pragma unroll
            for (int c = 0; c < NC; c++) K[c] = 0.0;
#pragma unroll 1
            for (int pt = 0; pt < C::PF; pt++) {
                double ph, dph[DIM];
                const double* phi = M.tab + TB::o_phiL + pt * NB;
                column(phi, M.tab + TB::o_dphiL + pt * NB * DIM, ph, dph);
                const double* q = mat + (size_t)(el * C::PF + pt) * C::MATF;
                double a[NE];
#pragma unroll
                for (int m = 0; m < NE; m++) a[m] = entry(q, pt / NQF, m, ph, dph);
#pragma unroll
                for (int j = 0; j < NB; j++) {
                    const double pj = ldg(phi + j);
#pragma unroll
                    for (int m = 0; m < NE; m++) K[m * NB + j] += a[m] * pj;
                }
            }
        }
    }
    // ------------------------------------------------------------------ volume
    if constexpr (ORDER > 1 || Mdl::kSource) {
        __syncthreads();  // the faces' matrices have been read
        for (int t = threadIdx.x; t < n * NQV; t += C::THREADS) {
            const int x = t / NQV, q = t - x * NQV, ee = e0 + x;
            double* o = trc + (size_t)t * C::TRV;
            const double *phi = M.tab + TB::o_phi + q * NB, *dphi = M.tab + TB::o_dphi + q * NB * DIM;
            double Ji[DIM * DIM], v[NE], dv[GRAD ? DIM * NE : 1];
            if constexpr (GRAD) {
#pragma unroll
                for (int c = 0; c < DIM * DIM; c++) Ji[c] = ldg(M.geo + (size_t)(GL::JINV + c) * ld + ee);
            }
            El::template trace<GRAD>(phi, dphi, Ji, [&](int c) { return ldg(W + (size_t)c * ld + ee); }, v, dv);
#pragma unroll
            for (int m = 0; m < NE; m++) o[m] = v[m];
            if constexpr (GRAD) {
#pragma unroll
                for (int c = 0; c < DIM * NE; c++) o[NE + c] = dv[c];
            }
            if constexpr (MODE == JAC_VJP) {
                for (int m = 0; m < NE; m++) {
                    double s[C::OUT] = {0.0};
                    for (int j = 0; j < NB; j++) {
                        const double l = ldg(lam + (size_t)(m * NB + j) * ld + ee);
#pragma unroll
                        for (int d = 0; d < C::OUT; d++) s[d] += l * (d < DIM ? ldg(dphi + j * DIM + d) : ldg(phi + j));
                    }
#pragma unroll
                    for (int d = 0; d < C::OUT; d++) lm[t * C::LAM + d * NE + m] = s[d];
                }
            }
        }
        __syncthreads();
        for (int t = threadIdx.x; t < n * NQV * S * NE; t += C::THREADS) {
            int xq, s, mj;
            C::task(t, n * NQV, xq, s, mj);
            const int x = xq / NQV, q = xq - x * NQV, ee = e0 + x;
            if (s > 0 && !Mdl::kViscous && !Mdl::kSource && ldg(M.eps + ee) + M.dampConst == 0.0) continue;
            const double* o = trc + (size_t)xq * C::TRV;
            double Ji[DIM * DIM];
#pragma unroll
            for (int c = 0; c < DIM * DIM; c++) Ji[c] = ldg(M.geo + (size_t)(GL::JINV + c) * ld + ee);
            Dual<1> WI[NE], dWI[DIM * NE], Gr[DIM * NE], sw[NE];
#pragma unroll
            for (int m = 0; m < NE; m++) {
                WI[m] = Dual<1>(o[m]);
                if (s == 0 && m == mj) WI[m].d[0] = 1.0;
#pragma unroll
                for (int d = 0; d < DIM; d++) {
                    if constexpr (GRAD) {
                        dWI[d * NE + m] = Dual<1>(o[NE + d * NE + m]);
                        if (s > 0 && m == mj) dWI[d * NE + m].d[0] = ldg(M.geo + (size_t)(GL::JINV + (s - 1) * DIM + d) * ld + ee);
                    } else {
                        dWI[d * NE + m] = Dual<1>(0.0);
                    }
                }
            }
            const double jac = ldg(M.geo + (size_t)GL::JAC * ld + ee);
            El::volume_point(M, ee, q, Ji, jac * ldg(M.tab + TB::o_w + q), ldg(M.eps + ee) + M.dampConst, WI, dWI, Gr, sw);
            double* w = mat + (size_t)xq * C::MATV + s * C::OUT * NE * NE + mj;
#pragma unroll
            for (int d = 0; d < DIM; d++)
#pragma unroll
                for (int m = 0; m < NE; m++) w[(d * NE + m) * NE] = ORDER > 1 ? Gr[d * NE + m].d[0] : 0.0;
            if constexpr (Mdl::kSource) {
#pragma unroll
                for (int m = 0; m < NE; m++) w[(DIM * NE + m) * NE] = sw[m].d[0];
            }
        }
        __syncthreads();
        if (act) {
            const bool gradVol = GRAD && (Mdl::kViscous || Mdl::kSource || ldg(M.eps + e) + M.dampConst != 0.0);
#pragma unroll 1
            for (int q = 0; q < NQV; q++) {
                const double *phi = M.tab + TB::o_phi + q * NB, *dphi = M.tab + TB::o_dphi + q * NB * DIM;
                double ph, dph[DIM];
                column(phi, dphi, ph, dph);
                const double* w = mat + (size_t)(el * NQV + q) * C::MATV + mi;
                auto volume_entry = [&](int d, int m) {
                    double a = w[(d * NE + m) * NE] * ph;
                    if constexpr (GRAD) {
                        if (gradVol) {
#pragma unroll
                            for (int s = 1; s < S; s++) a += w[((s * C::OUT + d) * NE + m) * NE] * dph[s - 1];
                        }
                    }
                    return a;
                };
                if constexpr (MODE == JAC_VJP) {
#pragma unroll
                    for (int d = 0; d < C::OUT; d++)
#pragma unroll
                        for (int m = 0; m < NE; m++) gi += volume_entry(d, m) * lm[(el * NQV + q) * C::LAM + d * NE + m];
                } else {
#pragma unroll
                    for (int d = 0; d < C::OUT; d++) {
                        double a[NE];
#pragma unroll
                        for (int m = 0; m < NE; m++) a[m] = volume_entry(d, m);
#pragma unroll
                        for (int j = 0; j < NB; j++) {
                            const double pj = d < DIM ? ldg(dphi + j * DIM + d) : ldg(phi + j);
#pragma unroll
                            for (int m = 0; m < NE; m++) K[m * NB + j] += a[m] * pj;
                        }
                    }
                }
            }
        }
    }
    if (!act) return;
    if constexpr (MODE == JAC_VJP) {
        g[(size_t)i * ld + e] = gi;
    } else {
        case_coefficients(M, e, a1);
        const double jac = ldg(M.geo + (size_t)GL::JAC * ld + e);
#pragma unroll
        for (int r = 0; r < NC; r++) {
            double a = -K[r];
            const int mr = r / NB, br = r - mr * NB;
            if (mr == mi) a += a1 * mass_entry<DIM, ORDER>(M, e, 0, br, bi, jac);
            K[r] = a;
        }
        if constexpr (MODE == JAC_BLOCKS) {
#pragma unroll
            for (int r = 0; r < NC; r++) Adiag[((size_t)r * NC + i) * ld + e] = K[r];
        } else {
            store_column<NC>(F + ((size_t)e * (1 + NF) * NC + i) * NC, K);
        }
    }
}

// ---------------------------------------------------------------------------- finite differences
// BDF2.assembleJacobiMatrix finite differences (BDF2.java:349-378): per element, the residual with
// W + h e_i for every own unknown i; the diagonal block column A[r][i] = -(R_i[r] - R[r]) / h + a1 M, and
// the block of each face neighbour A_nb[r][i] = (KR_i[r] - KR[r]) / h from this element's face integrals.
//
// Unlike the exact blocks every column needs the integrand itself at every point, and its digits: a rounding
// of 1e-16 shows as 1e-8 in the difference, so every sum keeps the order of the element residual.
//
// A thread block takes E elements and all their columns together, the unperturbed one as column NC.  The
// traces of all points are formed once (a thread per point, side and equation) and kept in shared memory;
// a column replaces one equation's trace.  Per face, and per VCH volume points: a thread per element, point
// and column evaluates the integrand into shared memory, then a thread per element, column and equation
// (ITEMS of them, the NB sums in registers) adds it to its rows.
//
// What bounds it: the NC + 1 evaluations of the flux at each point.  A thread per element and column that
// forms all traces itself, with 2 NC sums in local memory, measured, ms: 18,000 tetrahedra Euler p = 2
// 8.4 -> 3.9; 50,416 triangles Navier-Stokes p = 2 3.1 -> 2.5.  The artificial viscosity of an inviscid model is
// added behind the flux, where there is any (in one evaluation the gradients of both sides stay in registers
// across the flux): 106,400 triangles Euler p = 1 with the shock sensor on, none active 1.29 -> 1.09, 17 %
// active 1.31 -> 1.21 (1.08 by the thread per column); 61,440 tetrahedra 4.7 -> 3.0 and 4.8 -> 3.5 (3.2).
// Viscous tetrahedra keep one thread block per SM: with two they spill 5 KB a thread (61,440 of 20 unknowns
// 6.95 -> 6.5, 18,000 of 50 7.8 -> 6.4).
template <class Mdl, int DIM, int ORDER, bool GRAD>
struct FdCfg {
    using El = Element<Mdl, DIM, ORDER>;
    static constexpr int NC = El::NC, NE = El::NE, NB = El::NB, COLS = NC + 1;
    static constexpr int S = GRAD ? 1 + DIM : 1;
    static constexpr bool VOLUME = ORDER > 1 || Mdl::kSource;
    static constexpr int PF = El::NF * El::NQF, PV = VOLUME ? El::NQV : 0;
    static constexpr int OUT = DIM + (Mdl::kSource ? 1 : 0);
    static constexpr int cmax(int a, int b) { return a > b ? a : b; }
    static constexpr int cmin(int a, int b) { return a < b ? a : b; }
    static constexpr int VCH = cmin(El::NQV, cmax(2, El::NQF / OUT));  // volume points at a time
    static constexpr int TRC = (2 * PF + PV) * NE * S;                 // traces: left and right of the faces, volume
    static constexpr int INT = cmax(El::NQF * NE, VOLUME ? VCH * OUT * NE : 0) * COLS;
    static constexpr int PER = NC + TRC + INT + NC;                    // coefficients, traces, integrands, base rows
    static constexpr int THREADS = 256;
    static constexpr int ITEMS_MAX = cmax(1, cmin(3, 24 / NB));
    static constexpr int E = cmax(1, cmin(32, cmin(THREADS * ITEMS_MAX / (COLS * NE), (100 * 1024 / 8) / PER)));
    static constexpr int ITEMS = (E * COLS * NE + THREADS - 1) / THREADS;
    static constexpr size_t SMEM = (size_t)E * PER * sizeof(double);
    static constexpr int CTAS = SMEM <= 112 * 1024 && !(Mdl::kViscous && DIM == 3) ? 2 : 1;
};

template <class Mdl, int DIM, int ORDER, bool GRAD>
__global__ void __launch_bounds__(FdCfg<Mdl, DIM, ORDER, GRAD>::THREADS, (FdCfg<Mdl, DIM, ORDER, GRAD>::CTAS))
    k_fd(DevMesh M, const double* __restrict__ W, double h, double a1, double* __restrict__ Adiag, double* __restrict__ Aneigh) {
    using C = FdCfg<Mdl, DIM, ORDER, GRAD>;
    using El = Element<Mdl, DIM, ORDER>;
    using TB = Tab<DIM, ORDER>;
    using GL = GeoLayout<DIM>;
    constexpr int NC = C::NC, NE = C::NE, NB = C::NB, NF = El::NF, NQF = El::NQF, NQV = El::NQV, NP = El::NP, S = C::S, E = C::E;
    constexpr int COLS = C::COLS, SLOT = E * COLS;
    extern __shared__ __align__(16) double fp_dyn_smem[];
    double* coef = fp_dyn_smem;           // [c][element]
    double* trc = coef + E * NC;          // [point and side][equation][value, gradient][element]
    double* gw = trc + E * C::TRC;        // [point][component][column][element]
    double* base = gw + E * C::INT;       // [row][element] of the unperturbed column
    const int e0 = blockIdx.x * E, n = min(E, M.nElem - e0);
    const int ld = M.ld;

    for (int t = threadIdx.x; t < NC * E; t += C::THREADS) {
        const int x = t % E;
        coef[t] = x < n ? ldg(W + (size_t)(t / E) * ld + e0 + x) : 0.0;
    }
    __syncthreads();
    // ------------------------------------------------------------------ traces
    for (int t = threadIdx.x; t < (2 * C::PF + C::PV) * NE * E; t += C::THREADS) {
        const int x = t % E, y = t / E, m = y % NE, pt = y / NE, e = e0 + x;
        if (x >= n) continue;
        const double *phi, *dphi;
        int eo = e;  // the element the trace is of
        bool own = true;
        if (pt < C::PF) {
            phi = M.tab + TB::o_phiL + pt * NB;
            dphi = M.tab + TB::o_dphiL + pt * NB * DIM;
        } else if (pt < 2 * C::PF) {
            const int q = pt - C::PF, k = q / NQF, p = q - k * NQF;
            eo = M.tt[(size_t)k * ld + e];
            if (eo < 0) continue;
            own = false;
            const int fc = M.fcode[(size_t)k * ld + e];
            phi = M.tab + TB::o_phiR + (fc * NQF + p) * NB;
            dphi = M.tab + TB::o_dphiR + (fc * NQF + p) * NB * DIM;
        } else {
            phi = M.tab + TB::o_phi + (pt - 2 * C::PF) * NB;
            dphi = M.tab + TB::o_dphi + (pt - 2 * C::PF) * NB * DIM;
        }
        double v, gr[DIM], dv[DIM];
        El::template trace_sums<GRAD>(
            phi, dphi, [&](int j) { return own ? coef[(m * NB + j) * E + x] : ldg(W + (size_t)(m * NB + j) * ld + eo); }, v, gr, 1);
        double* o = trc + (size_t)(y * S) * E + x;
        o[0] = v;
        if constexpr (GRAD) {
            double Ji[DIM * DIM];
#pragma unroll
            for (int c = 0; c < DIM * DIM; c++) Ji[c] = ldg(M.geo + (size_t)(GL::JINV + c) * ld + eo);
            El::physical_gradient(Ji, gr, dv, 1);
#pragma unroll
            for (int d = 0; d < DIM; d++) o[(1 + d) * E] = dv[d];
        }
    }
    // the traces of a point with column i's perturbation: equation mi's is formed again
    auto perturbed = [&](auto grad, int pt, int x, int i, const double* phi, const double* dphi, const double* Ji, double* v, double* dv) {
        constexpr bool G = decltype(grad)::value;
        const int mi = i / NB, bi = i - mi * NB;
        double pv = 0.0, pg[DIM], pd[DIM];
        if (i < NC) {
            El::template trace_sums<G>(
                phi, dphi,
                [&](int j) {
                    const double c = coef[(mi * NB + j) * E + x];
                    return j == bi ? c + h : c;
                },
                pv, pg, 1);
            if constexpr (G) El::physical_gradient(Ji, pg, pd, 1);
        }
        const double* o = trc + (size_t)(pt * NE * S) * E + x;
#pragma unroll
        for (int m = 0; m < NE; m++) {
            v[m] = m == mi ? pv : o[m * S * E];
            if constexpr (G) {
#pragma unroll
                for (int d = 0; d < DIM; d++) dv[d * NE + m] = m == mi ? pd[d] : o[(m * S + 1 + d) * E];
            }
        }
    };
    // the gradient of the perturbed equation alone
    auto perturbed_gradient = [&](int x, int i, const double* phi, const double* dphi, const double* Ji, double* pd) {
        const int mi = i / NB, bi = i - mi * NB;
        double pv, pg[DIM];
        El::template trace_sums<true>(
            phi, dphi,
            [&](int j) {
                const double c = coef[(mi * NB + j) * E + x];
                return j == bi ? c + h : c;
            },
            pv, pg, 1);
        El::physical_gradient(Ji, pg, pd, 1);
    };
    double K[C::ITEMS][NB];
#pragma unroll
    for (int u = 0; u < C::ITEMS; u++)
#pragma unroll
        for (int j = 0; j < NB; j++) K[u][j] = 0.0;
    const double invh = 1.0 / h;
    // ------------------------------------------------------------------ faces
#pragma unroll 1
    for (int k = 0; k < NF; k++) {
        __syncthreads();  // traces; integrands of the last face read
        for (int t = threadIdx.x; t < NQF * SLOT; t += C::THREADS) {
            const int x = t % E, y = t / E, i = y % COLS, p = y / COLS, pt = k * NQF + p, e = e0 + x;
            if (x >= n) continue;
            const int TT = M.tt[(size_t)k * ld + e];
            const bool interior = TT > -1;
            const double eps_e = ldg(M.eps + e), eps_nb = interior ? ldg(M.eps + TT) : 0.0;
            double nrm[DIM], Jac, dL, Cc[NE], Jm[NE];
            El::face_geo(M, e, k, nrm, Jac, dL);
            // gradients in the flux itself only where it reads them; the artificial viscosity's are added
            // behind it, in the order of the element residual, on the faces that have any: kept in registers
            // across the flux they spill
            constexpr bool G = Mdl::kViscous;
            constexpr int NG = G ? DIM * NE : 1;
            const double *phiL = M.tab + TB::o_phiL + pt * NB, *dphiL = M.tab + TB::o_dphiL + pt * NB * DIM;
            const double *oL = trc + (size_t)(pt * NE * S) * E + x, *oR = trc + (size_t)((C::PF + pt) * NE * S) * E + x;
            double Ji[GRAD ? DIM * DIM : 1], WL[NE], WR[NE], dWL[NG], dWR[NG];
            auto geometry = [&] {
#pragma unroll
                for (int c = 0; c < DIM * DIM; c++) Ji[c] = ldg(M.geo + (size_t)(GL::JINV + c) * ld + e);
            };
            if constexpr (G) geometry();
            perturbed(std::bool_constant<G>{}, pt, x, i, phiL, dphiL, Ji, WL, dWL);
            if (interior) {
#pragma unroll
                for (int m = 0; m < NE; m++) {
                    WR[m] = oR[m * S * E];
                    if constexpr (G) {
#pragma unroll
                        for (int d = 0; d < DIM; d++) dWR[d * NE + m] = oR[(m * S + 1 + d) * E];
                    }
                }
            }
            El::template point_flux<G>(M, e, k, p, TT, nrm, dL, eps_e, eps_nb, WL, WR, dWL, dWR, Cc, Jm);
            if constexpr (GRAD && !G) {
                if (El::needs_gradients(M, interior, eps_e, eps_nb)) {
                    const int mi = i / NB;
                    double pd[DIM];
                    if (i < NC) {
                        geometry();
                        perturbed_gradient(x, i, phiL, dphiL, Ji, pd);
                    }
#pragma unroll
                    for (int m = 0; m < NE; m++) {
                        double dWsum = 0.0;
#pragma unroll
                        for (int d = 0; d < DIM; d++)
                            dWsum += ((i < NC && m == mi ? pd[d] : oL[(m * S + 1 + d) * E]) + oR[(m * S + 1 + d) * E]) / 2.0 * nrm[d];
                        Cc[m] += El::artificial_flux(M, dL, eps_e, eps_nb, dWsum, WL[m], WR[m]);
                    }
                }
            }
            const double jw = Jac * ldg(M.tab + TB::o_wf + p);
            const bool ip = Mdl::kViscous && (interior || Mdl::isIPFace(TT));
            const double cip = ip ? ldg(M.cip + e) : 0.0;
            double* o = gw + (size_t)p * NE * SLOT + i * E + x;
#pragma unroll
            for (int m = 0; m < NE; m++) {
                double g = Cc[m];
                if (ip) g -= cip * Jm[m];
                o[m * SLOT] = jw * g;
            }
        }
        __syncthreads();
        double acc[C::ITEMS][NB];
#pragma unroll
        for (int u = 0; u < C::ITEMS; u++) {
            const int t = threadIdx.x + u * C::THREADS, s = t % SLOT, m = t / SLOT, x = s % E;
            if (m >= NE || x >= n) continue;
            const int nb = M.tt[(size_t)k * ld + e0 + x];
            const int fc = nb > -1 ? M.fcode[(size_t)k * ld + e0 + x] : 0;
            const double* phiL = M.tab + TB::o_phiL + k * NQF * NB;
            const double* phiR = M.tab + TB::o_phiR + fc * NQF * NB;
#pragma unroll
            for (int j = 0; j < NB; j++) acc[u][j] = 0.0;
#pragma unroll 1
            for (int p = 0; p < NQF; p++) {
                const double g = gw[(p * NE + m) * SLOT + s];
#pragma unroll
                for (int j = 0; j < NB; j++) {
                    K[u][j] += g * ldg(phiL + p * NB + j);
                    acc[u][j] += g * ldg(phiR + p * NB + j);
                }
            }
            if (s / E == NC) {
#pragma unroll
                for (int j = 0; j < NB; j++) base[(m * NB + j) * E + x] = acc[u][j];
            }
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < C::ITEMS; u++) {
            const int t = threadIdx.x + u * C::THREADS, s = t % SLOT, m = t / SLOT, x = s % E, i = s / E;
            if (m >= NE || x >= n || i == NC) continue;
            const int nb = M.tt[(size_t)k * ld + e0 + x];
            if (nb < 0) continue;
            // block of element nb for its face kr, column i (this element's unknown i)
            const int kr = M.fcode[(size_t)k * ld + e0 + x] / NP;
            double* A = Aneigh + (size_t)kr * NC * NC * ld;
#pragma unroll
            for (int j = 0; j < NB; j++)
                A[((size_t)(m * NB + j) * NC + i) * ld + nb] = (acc[u][j] - base[(m * NB + j) * E + x]) * invh;
        }
    }
    // ------------------------------------------------------------------ volume
    if constexpr (C::VOLUME) {
#pragma unroll 1
        for (int q0 = 0; q0 < NQV; q0 += C::VCH) {
            const int nq = min(C::VCH, NQV - q0);
            __syncthreads();  // integrands of the last points read
            for (int t = threadIdx.x; t < nq * SLOT; t += C::THREADS) {
                const int x = t % E, y = t / E, i = y % COLS, r = y / COLS, q = q0 + r, e = e0 + x;
                if (x >= n) continue;
                double Ji[DIM * DIM], WI[NE], dWI[DIM * NE], Gr[DIM * NE], sw[NE];
#pragma unroll
                for (int c = 0; c < DIM * DIM; c++) Ji[c] = ldg(M.geo + (size_t)(GL::JINV + c) * ld + e);
                const double avc = ldg(M.eps + e) + M.dampConst;
                const double *phi = M.tab + TB::o_phi + q * NB, *dphi = M.tab + TB::o_dphi + q * NB * DIM;
                constexpr bool G = Mdl::kViscous || Mdl::kSource;
                perturbed(std::bool_constant<G>{}, 2 * C::PF + q, x, i, phi, dphi, Ji, WI, dWI);
                if constexpr (!G) {  // read by the artificial viscosity alone
#pragma unroll
                    for (int c = 0; c < DIM * NE; c++) dWI[c] = 0.0;
                    if (GRAD && avc != 0.0) {
                        const double* oV = trc + (size_t)((2 * C::PF + q) * NE * S) * E + x;
                        const int mi = i / NB;
                        double pd[DIM];
                        if (i < NC) perturbed_gradient(x, i, phi, dphi, Ji, pd);
#pragma unroll
                        for (int m = 0; m < NE; m++)
#pragma unroll
                            for (int d = 0; d < DIM; d++) dWI[d * NE + m] = i < NC && m == mi ? pd[d] : oV[(m * S + 1 + d) * E];
                    }
                }
                const double jac = ldg(M.geo + (size_t)GL::JAC * ld + e);
                El::volume_point(M, e, q, Ji, jac * ldg(M.tab + TB::o_w + q), avc, WI, dWI, Gr, sw);
                double* o = gw + (size_t)r * C::OUT * NE * SLOT + i * E + x;
                if constexpr (ORDER > 1) {
#pragma unroll
                    for (int c = 0; c < DIM * NE; c++) o[c * SLOT] = Gr[c];
                }
                if constexpr (Mdl::kSource) {
#pragma unroll
                    for (int m = 0; m < NE; m++) o[(DIM * NE + m) * SLOT] = sw[m];
                }
            }
            __syncthreads();
#pragma unroll
            for (int u = 0; u < C::ITEMS; u++) {
                const int t = threadIdx.x + u * C::THREADS, s = t % SLOT, m = t / SLOT;
                if (m >= NE || s % E >= n) continue;
#pragma unroll 1
                for (int r = 0; r < nq; r++) {
                    const double *phi = M.tab + TB::o_phi + (q0 + r) * NB, *dphi = M.tab + TB::o_dphi + (q0 + r) * NB * DIM;
                    const double* o = gw + (size_t)(r * C::OUT * NE + m) * SLOT + s;
                    if constexpr (ORDER > 1) {
                        double gd[DIM];
#pragma unroll
                        for (int d = 0; d < DIM; d++) gd[d] = o[d * NE * SLOT];
#pragma unroll
                        for (int j = 0; j < NB; j++)
#pragma unroll
                            for (int d = 0; d < DIM; d++) K[u][j] += gd[d] * ldg(dphi + j * DIM + d);
                    }
                    if constexpr (Mdl::kSource) {
                        const double sm = o[DIM * NE * SLOT];
#pragma unroll
                        for (int j = 0; j < NB; j++) K[u][j] += sm * ldg(phi + j);
                    }
                }
            }
        }
    }
    // ------------------------------------------------------------------ diagonal block
    __syncthreads();  // the last face's base rows have been read
#pragma unroll
    for (int u = 0; u < C::ITEMS; u++) {
        const int t = threadIdx.x + u * C::THREADS, s = t % SLOT, m = t / SLOT, x = s % E;
        if (m >= NE || x >= n || s / E != NC) continue;
#pragma unroll
        for (int j = 0; j < NB; j++) base[(m * NB + j) * E + x] = K[u][j];
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < C::ITEMS; u++) {
        const int t = threadIdx.x + u * C::THREADS, s = t % SLOT, m = t / SLOT, x = s % E, i = s / E;
        if (m >= NE || x >= n || i == NC) continue;
        const int e = e0 + x, mi = i / NB, bi = i - mi * NB;
        double c1 = a1;
        case_coefficients(M, e, c1);
        const double jac = ldg(M.geo + (size_t)GL::JAC * ld + e);
#pragma unroll
        for (int j = 0; j < NB; j++) {
            double a = (K[u][j] - base[(m * NB + j) * E + x]) / (-h);
            if (m == mi) a += c1 * mass_entry<DIM, ORDER>(M, e, 0, j, bi, jac);
            Adiag[((size_t)(m * NB + j) * NC + i) * ld + e] = a;
        }
    }
}

}  // namespace fp
