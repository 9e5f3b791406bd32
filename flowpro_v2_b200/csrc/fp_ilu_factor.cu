// Block ILU(0) factorisation (BlockILU0.factor, BlockILU0.java:98-185) of the blocks already in the
// factor storage F[e][s][c][r], in place and in the precision of the factors: one persistent
// cooperative launch, one thread block per row in forward-level order, rows of later levels waiting
// (bounded) for the completion flags of their lower neighbours.
//
// What bounds it.  The dependency chain: 127 levels of 142 rows on 18,000 tetrahedra, and a row of
// 50 unknowns is 0.7 M multiply-adds (11,000 cycles of one SM's FP64 pipe at best), so a level takes
// what one row takes from its last neighbour's flag to its own.  Therefore:
//   * a row keeps only its diagonal block, the lower block in work, L and two blocks of the lower
//     neighbour in shared memory (100 KB at 50 unknowns in FP64, two rows per SM), takes its lower
//     neighbours one by one as they finish, and does not touch its upper blocks unless the pattern
//     updates them (a common neighbour; those go to device memory directly);
//   * the products have compile-time sizes, two columns of the contraction per 16-byte shared load and
//     tiles that give most threads one;
//   * the diagonal block is inverted with one barrier a pivot: a warp holds whole columns, so the
//     owner of the pivot column finds the pivot alone;
//   * dependents read only inv(U_ii) and the upper blocks, so the flag follows the inverse.
// Every value is computed by the same operations in the same order as one thread per entry would:
// sums over m ascending, then subtracted; a_rc -= (a_rp (1 / a_pp)) a_pc for ascending pivots.
//
// Measured per factorisation, ms, before (one 512-thread block per row, all blocks staged, two
// barriers a pivot): 18,000 tetrahedra of 50 unknowns FP64 13.6 -> 6.8,
// 86,700 FP32 46.5 -> 12.5, 8,832 triangles of 30 FP32 6.1 -> 2.2, 53,400 of 12 in 12 merged cases 8.9 ->
// 2.1, 16,600 of 40 in 4 merged cases 13.2 -> 6.1.
#include <cuda_pipeline.h>

#include <algorithm>
#include <type_traits>

#include "fp_ctx.h"

namespace fp {

namespace {

constexpr int kSpin = 1 << 12;  // polls back to back before the sleeping ones

__device__ __forceinline__ unsigned flag_load(const unsigned* f) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(f) : "memory");
    return v;
}
__device__ __forceinline__ void flag_store(unsigned* f, unsigned v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(f), "r"(v) : "memory");
}
// Bounded wait until *f == epoch.  A wait that runs out sets FP_DEV_TIMEOUT and the abort word, which
// ends every other wait of the launch at once; the results are then garbage and the host reports it.
__device__ __forceinline__ void flag_wait(const unsigned* f, unsigned epoch, unsigned* abortw, unsigned* status, int maxPolls) {
    for (int it = 0; it < maxPolls; it++) {
        if (flag_load(f) == epoch) return;
        if ((it & 31) == 31 && *(volatile unsigned*)abortw) return;
        if (it >= kSpin) __nanosleep(64);
    }
    atomicOr(status, (unsigned)FP_DEV_TIMEOUT);
    atomicExch(abortw, 1u);
}

template <class T, int NC>
struct FCfg {
    static constexpr int NT = NC <= 16 ? 128 : 256;     // threads of a row
    static constexpr int W = NT / 32;
    static constexpr int NC2 = NC * NC;
    // tile of the products: rows x columns of a thread
    static constexpr int TM = NC <= 16 ? 1 : NC <= 40 ? 2 : 4;
    static constexpr int TN = NC < 4 ? 1 : NC <= 30 ? 2 : 4;
    static constexpr int GM = (NC + TM - 1) / TM, GN = (NC + TN - 1) / TN;
    static_assert(GM * GN <= NT, "one tile per thread");
    static constexpr int BLOCKS = 5;                    // D, A, L, Y0, Y1
    static constexpr size_t SMEM = (size_t)BLOCKS * NC2 * sizeof(T);
    static constexpr bool VEC = (NC2 * sizeof(T)) % 16 == 0;
    static constexpr int CTAS = SMEM <= 55 * 1024 ? 4 : SMEM <= 75 * 1024 ? 3 : 2;
};

// global -> shared copy of a block by the whole thread block; completes at the next
// __pipeline_wait_prior
template <class T, int NC>
__device__ __forceinline__ void stage(T* dst, const T* src) {
    using C = FCfg<T, NC>;
    if constexpr (C::VEC) {
        constexpr int N = C::NC2 * (int)sizeof(T) / 16;
#pragma unroll
        for (int u = 0; u < (N + C::NT - 1) / C::NT; u++) {
            const int q = u * C::NT + (int)threadIdx.x;
            if (q < N) __pipeline_memcpy_async(reinterpret_cast<int4*>(dst) + q, reinterpret_cast<const int4*>(src) + q, 16);
        }
    } else {
        for (int q = threadIdx.x; q < C::NC2; q += C::NT) __pipeline_memcpy_async(dst + q, src + q, sizeof(T));
    }
}

// acc = X * Y of column-major NC x NC blocks (this thread's tile), summed over ascending columns of X
template <class T, int NC>
struct Tile {
    using C = FCfg<T, NC>;
    T acc[C::TM][C::TN];
    int r0, c0;   // first row and column this thread stores
    // first ones it computes: the last tiles of a ragged block start earlier.  Tiles of four rows are
    // two pairs, r0 and rb, so that the lanes of a warp read 16-byte pieces side by side
    int rb, cb;
    bool on;
    __device__ __forceinline__ Tile() {
        const int t = threadIdx.x;
        r0 = C::TM * (t % C::GM);
        c0 = C::TN * (t / C::GM);
        on = t < C::GM * C::GN;
        if constexpr (C::TM == 4) {  // two pairs, 2 GM rows apart
            r0 = 2 * (t % C::GM);
            rb = r0 + 2 * C::GM < NC - 2 ? r0 + 2 * C::GM : NC - 2;
        } else {
            rb = r0 < NC - C::TM ? r0 : NC - C::TM;
        }
        cb = c0 < NC - C::TN ? c0 : NC - C::TN;
    }
    __device__ __forceinline__ void mul(const T* X, const T* Y) {
#pragma unroll
        for (int a = 0; a < C::TM; a++)
#pragma unroll
            for (int b = 0; b < C::TN; b++) acc[a][b] = T(0);
        if (!on) return;
        constexpr bool pairs = NC % 2 == 0;
        using T2 = std::conditional_t<sizeof(T) == 8, double2, float2>;
        const T* X0 = C::TM == 4 ? X + r0 : X + rb;
        const T* X1 = X + rb - 2;
        Y += cb * NC;
#pragma unroll 5
        for (int m = 0; m < NC - NC % 2; m += 2) {
            T x[2][C::TM], y[C::TN][2];
#pragma unroll
            for (int q = 0; q < 2; q++) {
                if constexpr (pairs && C::TM % 2 == 0) {
#pragma unroll
                    for (int a = 0; a < C::TM; a += 2) {
                        const T2 v = *reinterpret_cast<const T2*>((a == 2 ? X1 : X0) + (m + q) * NC + a);
                        x[q][a] = v.x;
                        x[q][a + 1] = v.y;
                    }
                } else {
#pragma unroll
                    for (int a = 0; a < C::TM; a++) x[q][a] = X0[(m + q) * NC + a];
                }
            }
#pragma unroll
            for (int b = 0; b < C::TN; b++) {
                if constexpr (pairs) {
                    const T2 v = *reinterpret_cast<const T2*>(Y + b * NC + m);
                    y[b][0] = v.x;
                    y[b][1] = v.y;
                } else {
                    y[b][0] = Y[b * NC + m];
                    y[b][1] = Y[b * NC + m + 1];
                }
            }
#pragma unroll
            for (int q = 0; q < 2; q++)
#pragma unroll
                for (int a = 0; a < C::TM; a++)
#pragma unroll
                    for (int b = 0; b < C::TN; b++) acc[a][b] += x[q][a] * y[b][q];
        }
        if constexpr (!pairs) {
#pragma unroll
            for (int a = 0; a < C::TM; a++)
#pragma unroll
                for (int b = 0; b < C::TN; b++) acc[a][b] += X0[(NC - 1) * NC + a] * Y[b * NC + NC - 1];
        }
    }
    template <class Fn>
    __device__ __forceinline__ void each(Fn fn) const {
        if (!on) return;
#pragma unroll
        for (int b = 0; b < C::TN; b++)
#pragma unroll
            for (int a = 0; a < C::TM; a++) {
                const int r = C::TM == 4 ? (a < 2 ? r0 + a : rb + a - 2) : rb + a;
                const int from = C::TM == 4 && a >= 2 ? r0 + 2 * C::GM : r0;
                if ((NC % C::TM == 0 || r >= from) && (NC % C::TN == 0 || cb + b >= c0)) fn((cb + b) * NC + r, acc[a][b]);
            }
    }
};

// Inverse of the NC x NC column-major block D (shared memory) into D, by Gauss-Jordan on [D | I] with
// implicit partial pivoting (unscaled pivot rows).  Warp w holds the columns w, w + W, ... of [D | I],
// lane l the rows l, l + 32 of them.  The owner of column p finds the pivot row br (the unused row with
// the largest |a_rp|, compared in single precision, ties in the leading 18 bits to the lowest row) with
// one key a lane and publishes the multipliers a_rp / a_br,p; after the barrier every warp updates its
// columns c > p, a_rc -= (a_rp / a_br,p) a_br,c, and the owner of column p + 1 does that one first and
// finds the next pivot meanwhile.  A step is a chain of 650 to 1,100 cycles: the barrier, the
// comparison, a division, three shared-memory round trips.  (Measured and dropped: whole rows in a
// warp, 350 instructions a warp and step, 2,300 cycles at two rows of 50 per SM; a flag per step
// instead of the barrier, no gain.)  Columns <= p of the left half are left stale.  At the end the right
// half of row br(p) holds d_p times row p of the inverse, d_p its pivot.  Returns false (the same in
// every thread) for a singular block.
template <class T, int NC>
struct Pivots {
    T mult[2][(NC + 31) / 32 * 32];  // multipliers of a step, two buffers
    T value[NC];     // pivot of a row
    int step[NC];    // and its step
    int row[2];      // pivot row of a step, -1: singular
    // each warp's entries of the pivot row
    alignas(16) T entry[FCfg<T, NC>::W][((2 * NC + FCfg<T, NC>::W - 1) / FCfg<T, NC>::W + 1) & ~1];
};
template <class T, int NC>
__device__ __forceinline__ bool invert(T* D, Pivots<T, NC>& P) {
    using C = FCfg<T, NC>;
    constexpr int W = C::W, RS = (NC + 31) / 32, KS = (2 * NC + W - 1) / W;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    T a[RS][KS];
#pragma unroll
    for (int k = 0; k < KS; k++) {
        const int c = w + W * k;
#pragma unroll
        for (int s = 0; s < RS; s++) {
            const int r = lane + 32 * s;
            a[s][k] = T(0);
            if (r < NC && c < NC) a[s][k] = D[c * NC + r];
            if (c >= NC && c - NC == r) a[s][k] = T(1);
        }
    }
    unsigned used[RS];
#pragma unroll
    for (int s = 0; s < RS; s++) used[s] = 0u;
    // the pivot of step p from column p, given by its owner's registers
    auto find = [&](int p, const T (&col)[RS]) {
        unsigned key = 0u;
#pragma unroll
        for (int s = 0; s < RS; s++) {
            const T v = fabs(col[s]);
            unsigned k = __float_as_uint((float)v) & ~63u;
            if (k == 0u && v > T(0)) k = 64u;  // below float range: still a candidate
            if (!isfinite(v)) k = 0xffffffc0u;
            k |= (unsigned)(63 - (lane + 32 * s));
            if (lane + 32 * s >= NC || ((used[s] >> lane) & 1u)) k = 0u;
            key = max(key, k);
        }
        key = __reduce_max_sync(~0u, key);
        const int br = 63 - (int)(key & 63u);
        T x = col[0];
        if constexpr (RS == 2) x = br >= 32 ? col[1] : x;
        const T pv = __shfl_sync(~0u, x, br & 31);
        const bool bad = key < 64u || !(fabs(pv) > T(0)) || !isfinite(pv);
        const T inv = T(1) / pv;
#pragma unroll
        for (int s = 0; s < RS; s++) P.mult[p & 1][lane + 32 * s] = lane + 32 * s == br ? T(0) : col[s] * inv;
        if (lane == 0) {
            P.row[p & 1] = bad ? -1 : br;
            if (!bad) {
                P.value[br] = pv;
                P.step[br] = p;
            }
        }
    };
    auto column = [&](int k, T (&col)[RS]) {
#pragma unroll
        for (int s = 0; s < RS; s++) col[s] = a[s][k];
    };
    if (w == 0) {
        T col[RS];
        column(0, col);
        find(0, col);
    }
    bool singular = false;
#pragma unroll
    for (int k0 = 0; k0 < (NC + W - 1) / W; k0++) {
#pragma unroll 1
        for (int pw = 0; pw < W; pw++) {
            const int p = W * k0 + pw;
            if (p >= NC || singular) break;
            __syncthreads();
            const int br = P.row[p & 1];
            if (br < 0) {
                singular = true;
                break;
            }
            T m[RS];  // the pivot row keeps its values: its multiplier is zero
#pragma unroll
            for (int s = 0; s < RS; s++) {
                m[s] = P.mult[p & 1][lane + 32 * s];
                used[s] |= br >> 5 == s ? 1u << (br & 31) : 0u;
            }
            auto update = [&](int k, T row) {
#pragma unroll
                for (int s = 0; s < RS; s++) a[s][k] -= m[s] * row;
            };
            auto entry = [&](int k) {
                T x = a[0][k];
                if constexpr (RS == 2) x = br >= 32 ? a[1][k] : x;
                return __shfl_sync(~0u, x, br & 31);
            };
            // the next column first: its owner finds the next pivot while the others update
            const int kn = k0 + 1 < KS ? k0 + 1 : k0;
            const bool next0 = pw + 1 < W && w == pw + 1, next1 = pw + 1 == W && w == 0 && k0 + 1 < KS;
            if (next0 || next1) {
                T col[RS];
                if (next0) {
                    update(k0, entry(k0));
                    column(k0, col);
                } else {
                    update(kn, entry(kn));
                    column(kn, col);
                }
                if (p + 1 < NC) find(p + 1, col);
            }
            // the pivot row's entries of this warp's columns through its own shared memory: half the
            // traffic of a shuffle per column (1,320 -> 1,120 cycles a step at two rows of 50 per SM)
            T* ent = P.entry[w];
            if (lane == (br & 31)) {
#pragma unroll
                for (int k = k0; k < KS; k++) {
                    T x = a[0][k];
                    if constexpr (RS == 2) x = br >= 32 ? a[1][k] : x;
                    ent[k] = x;
                }
            }
            __syncwarp();
#pragma unroll
            for (int k = k0; k < KS; k++) {
                const T row = ent[k];
                if (k == k0) {
                    if (w > pw && !next0) update(k, row);  // columns <= p of this slot, or done
                } else if (k == k0 + 1) {
                    if (!next1) update(k, row);
                } else {
                    update(k, row);
                }
            }
        }
    }
    if (singular) return false;
    __syncthreads();  // every pivot is published
#pragma unroll
    for (int s = 0; s < RS; s++) {
        const int r = lane + 32 * s;
        if (r < NC) {
            const int st = P.step[r];
            const T d = P.value[r];
#pragma unroll
            for (int k = 0; k < KS; k++) {
                const int c = w + W * k;
                if (c >= NC && c < 2 * NC) D[(c - NC) * NC + st] = a[s][k] / d;
            }
        }
    }
    __syncthreads();
    return true;
}

struct FactorArgs {
    int nf, nE;
    const int* lvl;      // rows in forward-level order
    const int* opPtr;    // [nE + 1] program of each row
    const int4* ops;     // (0, f, k, -): L = A_ik inv(U_kk), k over face f; (1, slot, k, h): A_slot -= L U_k,h
    unsigned* done;      // [nE] row flags
    unsigned epoch;
    unsigned *abortw, *status, *sing;
    int maxPolls;
};

// Thread block g takes the rows g, g + gridDim.x, ... in forward-level order.  Every dependency lies in
// an earlier level, every block walks its rows in level order and all blocks are co-resident
// (cooperative launch), so each wait ends.  A singular diagonal block sets FP_DEV_SINGULAR and still
// completes its row, so no dependent waits for it.
template <class T, int NC>
__global__ void __launch_bounds__(FCfg<T, NC>::NT, FCfg<T, NC>::CTAS) k_ilu_rows(FactorArgs A, T* F) {
    using C = FCfg<T, NC>;
    constexpr int NC2 = C::NC2;
    extern __shared__ __align__(16) unsigned char factor_smem[];
    __shared__ Pivots<T, NC> piv;
    T* D = reinterpret_cast<T*>(factor_smem);
    T* Ab = D + NC2;
    T* L = Ab + NC2;
    T* Y0 = L + NC2;
    T* Y1 = Y0 + NC2;
    const int t = threadIdx.x, ns = 1 + A.nf;
    Tile<T, NC> tile;
    for (int q0 = blockIdx.x; q0 < A.nE; q0 += gridDim.x) {
        const int i = A.lvl[q0];
        T* Fi = F + (size_t)i * ns * NC2;
        stage<T, NC>(D, Fi);
        __pipeline_commit();
        const int qEnd = A.opPtr[i + 1];
        for (int q = A.opPtr[i]; q < qEnd;) {
            const int4 op = A.ops[q];  // an L step
            if (t == 0) flag_wait(A.done + op.z, A.epoch, A.abortw, A.status, A.maxPolls);
            __syncthreads();  // the neighbour's row is complete, the buffers are free
            T* Aik = Fi + (size_t)(1 + op.y) * NC2;
            const T* Fk = F + (size_t)op.z * ns * NC2;
            int u = q + 1;  // the updates that follow
            while (u < qEnd && A.ops[u].x == 1) u++;
            stage<T, NC>(Ab, Aik);
            stage<T, NC>(Y0, Fk);
            __pipeline_commit();
            if (u > q + 1) stage<T, NC>(Y1, Fk + (size_t)(1 + A.ops[q + 1].w) * NC2);
            __pipeline_commit();
            __pipeline_wait_prior(1);
            __syncthreads();
            tile.mul(Ab, Y0);
            tile.each([&](int o, T v) {
                L[o] = v;
                Aik[o] = v;
            });
            for (int v = q + 1; v < u; v++) {
                const int slot = A.ops[v].y;
                __pipeline_wait_prior(0);
                __syncthreads();  // L and the neighbour's block are there
                T* Y = (v - q) & 1 ? Y1 : Y0;
                if (v + 1 < u) stage<T, NC>((v - q) & 1 ? Y0 : Y1, Fk + (size_t)(1 + A.ops[v + 1].w) * NC2);
                __pipeline_commit();
                tile.mul(L, Y);
                if (slot == 0)
                    tile.each([&](int o, T x) { D[o] -= x; });
                else
                    tile.each([&](int o, T x) { Fi[(size_t)slot * NC2 + o] -= x; });
            }
            q = u;
        }
        __pipeline_wait_prior(0);
        __syncthreads();
        if (invert<T, NC>(D, piv)) {
            if constexpr (C::VEC) {
                constexpr int N = NC2 * (int)sizeof(T) / 16;
                for (int o = t; o < N; o += C::NT) reinterpret_cast<int4*>(Fi)[o] = reinterpret_cast<const int4*>(D)[o];
            } else {
                for (int o = t; o < NC2; o += C::NT) Fi[o] = D[o];
            }
        } else if (t == 0) {
            atomicOr(A.status, (unsigned)FP_DEV_SINGULAR);
            A.sing[i] = 1u;  // the row's mark
        }
        __syncthreads();  // the row is written, the shared buffers are free again
        if (t == 0) flag_store(A.done + i, A.epoch);
    }
}

template <class T, int NC>
int launch(fp_ctx* c, FactorArgs& a, T* F) {
    using C = FCfg<T, NC>;
    int rc, dev = 0, nsm = 0, perSm = 0;
    if (C::SMEM > 48 * 1024 &&
        (rc = cuda_check(c, cudaFuncSetAttribute(k_ilu_rows<T, NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM),
                         "smem")))
        return rc;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    if ((rc = cuda_check(c, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, k_ilu_rows<T, NC>, C::NT, C::SMEM), "occupancy")))
        return rc;
    if (perSm < 1) return set_err(c, FP_ERR_UNSUPPORTED, "block ILU(0): factorisation block does not fit an SM");
    const int grid = std::max(1, std::min(a.nE, nsm * perSm));
    void* args[] = {&a, (void*)&F};
    return cuda_check(
        c, cudaLaunchCooperativeKernel((const void*)k_ilu_rows<T, NC>, dim3(grid), dim3(C::NT), args, C::SMEM, c->stream),
        "ILU factor");
}

template <class T>
int run(fp_ctx* c, FactorArgs& a, T* F) {
#define FP_ROWS(N) \
    case N:        \
        return launch<T, N>(c, a, F);
    switch (c->nc) {  // the numbers of unknowns of the compiled models and orders
        FP_ROWS(1) FP_ROWS(3) FP_ROWS(4) FP_ROWS(5) FP_ROWS(6) FP_ROWS(9) FP_ROWS(10) FP_ROWS(12) FP_ROWS(15) FP_ROWS(16)
        FP_ROWS(18) FP_ROWS(20) FP_ROWS(24) FP_ROWS(30) FP_ROWS(40) FP_ROWS(50)
    }
#undef FP_ROWS
    return set_err(c, FP_ERR_UNSUPPORTED, "block ILU(0): no factorisation for this number of unknowns");
}

}  // namespace

int ilu_rows(fp_ctx* c, void* F, bool fp32, unsigned epoch) {
    FactorArgs a{};
    a.nf = c->hm.nf;
    a.nE = c->hm.nElem;
    a.lvl = c->d_lvlF;
    a.opPtr = c->d_opPtr;
    a.ops = c->d_ops;
    a.done = c->d_iluFlags + 2;
    a.epoch = epoch;
    a.abortw = c->d_iluFlags;
    a.status = c->d_status;
    a.sing = c->d_ilu_sing;
    a.maxPolls = c->ilu_max_polls;
    return fp32 ? run<float>(c, a, (float*)F) : run<double>(c, a, (double*)F);
}

}  // namespace fp
