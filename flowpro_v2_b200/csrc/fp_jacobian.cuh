// Exact element Jacobian blocks and the adjoint product, from the flux Jacobians at the quadrature
// points.  Column i = (mi, bi) of an element's blocks is the derivative of the element residual, and of the
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
// triangles Navier-Stokes p = 2 0.63 -> 0.16.
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
        const int seed = t % (S * NE), xp = t / (S * NE), x = xp / C::PF, pt = xp - x * C::PF, k = pt / NQF, p = pt - k * NQF;
        const int s = seed / NE, mj = seed - s * NE, ee = e0 + x;
        const int TT = M.tt[(size_t)k * ld + ee];
        const bool interior = TT > -1;
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
        El::template point_flux<GRAD>(M, ee, k, p, TT, nrm, dL, ldg(M.eps + ee), interior ? ldg(M.eps + TT) : 0.0, WL, WR, dWL,
                                      dWR, Cc, Jm);
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
    // row m of the point's matrix times what the column enters through
    auto entry = [&](const double* q, int m, double ph, const double* dph) {
        double a = q[m * NE + mi] * ph;
        if constexpr (GRAD) {
#pragma unroll
            for (int d = 0; d < DIM; d++) a += q[((1 + d) * NE + m) * NE + mi] * dph[d];
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
                for (int m = 0; m < NE; m++) gi += entry(q, m, ph, dph) * lm[(el * C::PF + pt) * NE + m];
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
                    for (int m = 0; m < NE; m++) a[m] = entry(q, m, ph, dph);
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
                for (int m = 0; m < NE; m++) a[m] = entry(q, m, ph, dph);
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
            const int seed = t % (S * NE), xq = t / (S * NE), x = xq / NQV, q = xq - x * NQV;
            const int s = seed / NE, mj = seed - s * NE, ee = e0 + x;
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
#pragma unroll 1
            for (int q = 0; q < NQV; q++) {
                const double *phi = M.tab + TB::o_phi + q * NB, *dphi = M.tab + TB::o_dphi + q * NB * DIM;
                double ph, dph[DIM];
                column(phi, dphi, ph, dph);
                const double* w = mat + (size_t)(el * NQV + q) * C::MATV + mi;
                auto volume_entry = [&](int d, int m) {
                    double a = w[(d * NE + m) * NE] * ph;
                    if constexpr (GRAD) {
#pragma unroll
                        for (int s = 1; s < S; s++) a += w[((s * C::OUT + d) * NE + m) * NE] * dph[s - 1];
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

}  // namespace fp
