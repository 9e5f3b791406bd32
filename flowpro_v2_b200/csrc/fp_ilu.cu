// Block ILU(0) preconditioner on the element-block matrix (BlockILU0.factor / apply,
// flowpro/core/LinearSolvers/preconditioners/BlockILU0.java:22-243).
//
// Rows are taken in the DOF (RCM) order.  Row i of the factor is
//   for each lower neighbour k (rank[k] < rank[i]) in rank order:
//       L_ik = A_ik * inv(U_kk);  A_ij -= L_ik * U_kj  for every column j > k of row i that row k has
//   inv(U_ii) = inverse of the updated A_ii
// which is BlockILU0's loop; the only fill-in-free columns a row k can share with row
// i are i itself and (around a vertex or an edge of valence 3) a common neighbour, both
// handled by the per-element program built on the host.
//
// Device side:
//   * factor values in element-major storage, F[e][s][c][r] (column-major blocks):
//     s = 0 holds inv(U_ee), s = 1 + k the block coupling e with its neighbour over face
//     k (L or U);
//   * rows whose lower neighbours are all finished form a level.  The factorisation is ONE
//     persistent cooperative kernel (fp_ilu_factor.cu), one thread block per row in shared
//     memory; thread blocks take the rows in level order and each row waits (bounded) only for
//     the completion flags of its lower neighbours;
//   * an application (forward L sweep, backward U sweep) is ONE persistent cooperative
//     kernel: thread blocks take the elements in level order, and each element waits
//     (bounded) only for the values of the neighbours it multiplies, so levels overlap and no
//     flag or fence stands between a value and its consumer.  Even numbers of unknowns take
//     fp_ilu_ring.cu, which streams the factor blocks through shared memory; the kernel here
//     (odd numbers, or on request) loads each element's factor entries into registers before
//     the values they multiply arrive, and its words carry the epoch of the application;
//   * the factorisation runs in the precision of the factors: FP64, or FP32 for the
//     mixed-precision GMRES, where the blocks are either gathered from the assembled
//     operator (rounded) or written straight into the FP32 factor storage by the exact
//     Jacobian kernel (no FP64 copy of the blocks exists then), and factorised in place.
#include <algorithm>
#include <cmath>
#include <vector>

#include "fp_ctx.h"

namespace fp {

namespace {

constexpr int kSweepThreads = 512;
constexpr int kMaxNc = 64;   // unknowns per element
constexpr int kMaxF = 4;     // faces per element
constexpr int kMaxJ = 8;     // columns per thread and block in the sweeps: ceil(nc / sweep_group(nc)) <= 8 for nc <= 64

template <class T>
int ialloc(fp_ctx* c, T** p, size_t n) {
    void* q = nullptr;
    cudaError_t e = cudaMalloc(&q, std::max<size_t>(n, 1) * sizeof(T));
    if (e != cudaSuccess) return cuda_check(c, e, "cudaMalloc (ILU)");
    c->allocs.push_back((double*)q);
    *p = (T*)q;
    return FP_OK;
}

// F[e][s] <- A_s(e) transposed into column-major blocks; tiles of 32 elements x 32
// block entries through shared memory so both the field-major read and the
// element-major write are coalesced.  Boundary faces get zero blocks.
template <class T>
__global__ void __launch_bounds__(256) k_ilu_gather(int nElem, int ld, int nc, int nf, const double* __restrict__ Ad,
                                                    const double* __restrict__ An, const int* __restrict__ tt,
                                                    T* __restrict__ F) {
    __shared__ double tile[32][33];
    const int nc2 = nc * nc;
    const int s = blockIdx.y;  // 0 diagonal, 1 + k face k
    const int e0 = blockIdx.x * 32;
    const int lane = threadIdx.x & 31, wy = threadIdx.x >> 5;  // 8 warps
    const double* A = s == 0 ? Ad : An + (size_t)(s - 1) * nc2 * ld;
    for (int o0 = 0; o0 < nc2; o0 += 32) {
        // load: warp row = output entry o, lanes along elements
        for (int j = wy; j < 32; j += 8) {
            const int o = o0 + j, e = e0 + lane;
            double v = 0.0;
            if (o < nc2 && e < nElem) {
                const int cc = o / nc, r = o - cc * nc;  // output (r, cc) column-major
                const bool interior = s == 0 || tt[(size_t)(s - 1) * ld + e] > -1;
                if (interior) v = A[(size_t)(r * nc + cc) * ld + e];
            }
            tile[j][lane] = v;
        }
        __syncthreads();
        // store: warp row = element, lanes along output entries
        for (int j = wy; j < 32; j += 8) {
            const int e = e0 + j, o = o0 + lane;
            if (e < nElem && o < nc2) F[((size_t)e * (1 + nf) + s) * nc2 + o] = (T)tile[lane][j];
        }
        __syncthreads();
    }
}

constexpr int kSpinPolls = 1 << 12;  // polled back to back first (a dependency is usually microseconds away)
// then with 64 ns sleeps up to the context's limit (default 2^19 polls: a wait gives up well
// within a second; a context may lower it, down to 0, so that tests can make a wait run out)

// Lanes per row in the sweeps: the largest power of two G <= 32 with G nc <= 512, so a
// row's G lanes are adjacent in one warp and meet by shuffles.
__host__ __device__ __forceinline__ int sweep_group(int nc) {
    int G = 32;
    while (G > 1 && G * nc > kSweepThreads) G >>= 1;
    return G;
}

// Factor entries of one sweep element held in registers.  Thread t = G r + g (g < G)
// handles row r of the columns c = g + G j.
template <class T>
struct SweepRegs {
    T fv[kMaxF][kMaxJ];  // blocks 1 + f (L or U)
    T dv[kMaxJ];         // block 0, inv(U_ii) (backward sweep)
    int4 nb;             // neighbours taking part (-1: none)
    int i;               // element, -1: nothing loaded
};

// issue the loads of element i's factor entries (they do not depend on the sweep values,
// so they are in flight while the element waits for its neighbours)
template <class T>
__device__ __forceinline__ void sweep_load(int nc, int nf, int G, const T* __restrict__ F, int i, int4 nbi, bool withD,
                                           SweepRegs<T>& R) {
    const int t = threadIdx.x, nc2 = nc * nc;
    const int r = t / G, g = t - r * G;
    R.i = i;
    R.nb = nbi;
    const int nb[kMaxF] = {R.nb.x, R.nb.y, R.nb.z, R.nb.w};
    const T* Fi = F + (size_t)i * (1 + nf) * nc2;
#pragma unroll
    for (int f = 0; f < kMaxF; f++)
#pragma unroll
        for (int j = 0; j < kMaxJ; j++) {
            const int c = g + G * j;
            R.fv[f][j] = (r < nc && f < nf && nb[f] >= 0 && c < nc) ? Fi[(size_t)(1 + f) * nc2 + (size_t)c * nc + r] : T(0);
        }
    if (withD) {
#pragma unroll
        for (int j = 0; j < kMaxJ; j++) {
            const int c = g + G * j;
            R.dv[j] = (r < nc && c < nc) ? Fi[(size_t)c * nc + r] : T(0);
        }
    }
}

// sum over the G adjacent lanes of a row (every lane of the warp takes part)
__device__ __forceinline__ double group_sum(double v, int G) {
    for (int o = G >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sweep values are published element-major with the epoch of the application: word
// (i, c, h) holds half h (0 low, 1 high) of value c of element i in its low 32 bits and
// the epoch in its high 32 bits.  A consumer polls the words themselves, so a value is
// usable as soon as its own word is, with no completion flag and no release fence (an
// aligned 64-bit store is seen whole or not at all).
__device__ __forceinline__ unsigned long long pub_load(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void pub_store(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Bounded wait for one published word of this epoch; returns its payload.  A wait that
// runs out sets FP_DEV_TIMEOUT and the abort word, which ends every other wait of the
// launch at once; the sweep values are then garbage and the host reports the timeout.
__device__ __forceinline__ unsigned pub_wait(const unsigned long long* p, unsigned epoch, unsigned* abortw,
                                             unsigned* status, int maxPolls) {
    for (int it = 0; it < maxPolls; it++) {
        const unsigned long long v = pub_load(p);
        if ((unsigned)(v >> 32) == epoch) return (unsigned)v;
        if ((it & 31) == 31 && *(volatile unsigned*)abortw) return 0u;
        if (it >= kSpinPolls) __nanosleep(64);
    }
    atomicOr(status, (unsigned)FP_DEV_TIMEOUT);
    atomicExch(abortw, 1u);
    return 0u;
}

// The whole application in one persistent launch over the sweep program: position v <
// nE is the forward sweep (y = L^-1 b) in forward-level order, v >= nE the backward sweep
// (x = U^-1 y) in backward-level order; swEl[v] is the element at position v and swNb[v]
// the neighbours it multiplies (lower, then upper; -1 none).  Thread block g takes the
// positions g, g + gridDim.x, ... of each sweep.  An element waits only for the published
// values it multiplies (the neighbours' and, in the backward sweep, its own forward
// value), so consecutive levels overlap.  Every dependency lies in an earlier level,
// every block walks its positions in level order and all blocks are co-resident
// (cooperative launch), so each wait ends.  The block's next element is known one element
// ahead, so its factor entries are requested right after the current values are published.
//
// One element: thread t = 128 f + 2 c + h fetches half h of value c of the neighbour over
// face f into shared memory; thread t = G r + g forms the partial sums of row r over the
// columns g + G j (one per face, so the chains are short), the G lanes of the row add
// them by shuffles and out_i = in_i - sum_f B_f v_f, then, backward, out_i = inv(U_ii)
// (that).  The shared buffers alternate between consecutive elements, so one barrier
// (two backward) per element suffices.
__device__ __forceinline__ int sweep_next(int v, int nE) {
    const int w = v + (int)gridDim.x;
    if (v < nE) return w < nE ? w : nE + (int)blockIdx.x;  // the first backward position after the last forward one
    return w;
}

template <class T>
__global__ void __launch_bounds__(kSweepThreads)
    k_ilu_sweeps(int nc, int nf, int ld, int nE, const int* __restrict__ swEl, const int4* __restrict__ swNb,
                 const T* __restrict__ F, const double* __restrict__ b, double* __restrict__ x, unsigned long long* pubF,
                 unsigned long long* pubB, unsigned epoch, unsigned* abortw, unsigned* status, int maxPolls) {
    __shared__ double vsb[2][kMaxF * 64];  // the neighbours' values
    __shared__ double yob[2][kMaxNc];      // backward: the element's forward value
    __shared__ double tvb[2][kMaxNc];      // backward: value before inv(U_ii)
    const int t = threadIdx.x, G = sweep_group(nc);
    const int r = t / G, g = t - r * G;
    const int nV = 2 * nE;
    SweepRegs<T> R;
    int v = blockIdx.x;
    if (v >= nE) return;
    sweep_load<T>(nc, nf, G, F, swEl[v], swNb[v], false, R);
    int v1 = sweep_next(v, nE);
    int i1 = v1 < nV ? swEl[v1] : -1;
    int4 nb1 = v1 < nV ? swNb[v1] : make_int4(-1, -1, -1, -1);
    int par = 0;
    while (v < nV) {
        const bool bwd = v >= nE;
        unsigned long long* pub = bwd ? pubB : pubF;  // the neighbours' values and this element's
        double* vs = vsb[par];
        double* yo = yob[par];
        double* tv = tvb[par];
        const int i = R.i;
        const double a_in = (!bwd && g < 2 && r < nc) ? __ldcg(b + (size_t)r * ld + i) : 0.0;  // the two publishing lanes
        // factor entries in double before the wait (a no-op for FP64 factors)
        double fv[kMaxF][kMaxJ], dv[kMaxJ];
#pragma unroll
        for (int f = 0; f < kMaxF; f++)
#pragma unroll
            for (int j = 0; j < kMaxJ; j++) fv[f][j] = (double)R.fv[f][j];
#pragma unroll
        for (int j = 0; j < kMaxJ; j++) dv[j] = bwd ? (double)R.dv[j] : 0.0;
        {
            const int f = t >> 7, c = (t >> 1) & 63, h = t & 1;
            const int n = f == 0 ? R.nb.x : f == 1 ? R.nb.y : f == 2 ? R.nb.z : R.nb.w;
            unsigned w = 0u;
            if (f < nf && n >= 0 && c < nc) w = pub_wait(pub + ((size_t)n * nc + c) * 2 + h, epoch, abortw, status, maxPolls);
            reinterpret_cast<unsigned*>(vs)[t] = w;
        }
        if (bwd && t < 2 * nc)
            reinterpret_cast<unsigned*>(yo)[t] = pub_wait(pubF + (size_t)i * nc * 2 + t, epoch, abortw, status, maxPolls);
        __syncthreads();
        double sf[kMaxF];
#pragma unroll
        for (int f = 0; f < kMaxF; f++) {
            sf[f] = 0.0;
#pragma unroll
            for (int j = 0; j < kMaxJ; j++) {
                const int c = g + G * j;
                if (c < nc) sf[f] += fv[f][j] * vs[f * 64 + c];
            }
        }
        const double s = group_sum((sf[0] + sf[1]) + (sf[2] + sf[3]), G);
        double a;
        if (!bwd) {
            a = a_in - s;
        } else {
            if (g == 0 && r < nc) tv[r] = yo[r] - s;
            __syncthreads();
            double d = 0.0;
#pragma unroll
            for (int j = 0; j < kMaxJ; j++) {
                const int c = g + G * j;
                if (c < nc) d += dv[j] * tv[c];
            }
            a = group_sum(d, G);
            if (g == 0 && r < nc) x[(size_t)r * ld + i] = a;
        }
        if (g < 2 && r < nc) {
            const unsigned long long e = (unsigned long long)epoch << 32;
            pub_store(pub + ((size_t)i * nc + r) * 2 + g, e | (unsigned)(g == 0 ? __double2loint(a) : __double2hiint(a)));
        }
        // the next element's factor entries, then the element after it
        if (v1 < nV) sweep_load<T>(nc, nf, G, F, i1, nb1, v1 >= nE, R);
        v = v1;
        v1 = v < nV ? sweep_next(v, nE) : nV;
        if (v1 < nV) {
            i1 = swEl[v1];
            nb1 = swNb[v1];
        }
        par ^= 1;
    }
}

// levels, neighbour sets and the per-element factorisation program (host, once per mesh)
int ilu_build(fp_ctx* c) {
    const HostMesh& h = c->hm;
    const int nE = h.nElem, nf = h.nf, ld = h.ld;
    const std::vector<int>& rank = h.rank;
    auto nb = [&](int e, int k) { return h.tt[(size_t)k * ld + e]; };
    std::vector<int> levF(nE, 0), levB(nE, 0);
    for (int r = 0; r < nE; r++) {
        const int i = h.order[r];
        for (int k = 0; k < nf; k++) {
            const int j = nb(i, k);
            if (j > -1 && rank[j] < r) levF[i] = std::max(levF[i], levF[j] + 1);
        }
    }
    for (int r = nE - 1; r >= 0; r--) {
        const int i = h.order[r];
        for (int k = 0; k < nf; k++) {
            const int j = nb(i, k);
            if (j > -1 && rank[j] > r) levB[i] = std::max(levB[i], levB[j] + 1);
        }
    }
    auto group = [&](const std::vector<int>& lev, std::vector<int>& el, std::vector<int>& ptr) {
        const int nl = nE ? *std::max_element(lev.begin(), lev.end()) + 1 : 0;
        ptr.assign(nl + 1, 0);
        for (int e = 0; e < nE; e++) ptr[lev[e] + 1]++;
        for (int l = 0; l < nl; l++) ptr[l + 1] += ptr[l];
        el.assign(nE, 0);
        std::vector<int> pos(ptr.begin(), ptr.end() - 1);
        for (int r = 0; r < nE; r++) el[pos[lev[h.order[r]]]++] = h.order[r];
    };
    std::vector<int> elF, elB;
    group(levF, elF, c->lvlF_ptr);
    std::vector<int> ptrB;
    group(levB, elB, ptrB);
    std::vector<int4> nbLow(nE), nbUp(nE);
    for (int i = 0; i < nE; i++) {
        int lo[4] = {-1, -1, -1, -1}, up[4] = {-1, -1, -1, -1};
        for (int f = 0; f < nf; f++) {
            const int j = nb(i, f);
            if (j > -1 && rank[j] < rank[i]) lo[f] = j;
            if (j > -1 && rank[j] > rank[i]) up[f] = j;
        }
        nbLow[i] = make_int4(lo[0], lo[1], lo[2], lo[3]);
        nbUp[i] = make_int4(up[0], up[1], up[2], up[3]);
    }
    // sweep program: forward positions, then backward positions
    std::vector<int> swEl(2 * (size_t)nE);
    std::vector<int4> swNb(2 * (size_t)nE);
    for (int q = 0; q < nE; q++) {
        swEl[q] = elF[q];
        swNb[q] = nbLow[elF[q]];
        swEl[nE + q] = elB[q];
        swNb[nE + q] = nbUp[elB[q]];
    }
    // factorisation program: per lower neighbour k in rank order an L step, then the
    // updates of every column j > k of row i that row k also has (j = i always)
    std::vector<int> opPtr(nE + 1, 0);
    std::vector<int4> ops;
    for (int i = 0; i < nE; i++) {
        opPtr[i] = (int)ops.size();
        std::vector<std::pair<int, int>> lower;  // (rank, face)
        for (int f = 0; f < nf; f++) {
            const int k = nb(i, f);
            if (k > -1 && rank[k] < rank[i]) lower.push_back({rank[k], f});
        }
        std::sort(lower.begin(), lower.end());
        for (auto& lf : lower) {
            const int f = lf.second, k = nb(i, f);
            ops.push_back(make_int4(0, f, k, 0));
            // columns of row i right of k, in rank order: i itself and its other neighbours
            std::vector<std::pair<int, int>> cols;  // (rank, slot)
            cols.push_back({rank[i], 0});
            for (int g = 0; g < nf; g++) {
                const int j = nb(i, g);
                if (j > -1 && rank[j] > rank[k]) cols.push_back({rank[j], 1 + g});
            }
            std::sort(cols.begin(), cols.end());
            for (auto& cs : cols) {
                const int j = cs.second == 0 ? i : nb(i, cs.second - 1);
                for (int hk = 0; hk < nf; hk++)
                    if (nb(k, hk) == j) {
                        ops.push_back(make_int4(1, cs.second, k, hk));
                        break;
                    }
            }
        }
    }
    opPtr[nE] = (int)ops.size();
    int rc;
    if ((rc = ialloc(c, &c->d_lvlF, nE)) || (rc = ialloc(c, &c->d_opPtr, nE + 1)) ||
        (rc = ialloc(c, &c->d_ops, ops.size())) || (rc = ialloc(c, &c->d_swEl, 2 * (size_t)nE)) ||
        (rc = ialloc(c, &c->d_swNb, 2 * (size_t)nE)) ||
        (rc = ialloc(c, &c->d_iluFlags, 2 + (size_t)nE)) || (rc = ialloc(c, &c->d_ilu_pub, 4 * (size_t)nE * c->nc)) ||
        (rc = ialloc(c, &c->d_ilu_sing, (size_t)nE)))
        return rc;
    cudaStream_t s = c->stream;
    auto up = [&](void* d, const void* hsrc, size_t bytes) {
        return cuda_check(c, cudaMemcpyAsync(d, hsrc, bytes, cudaMemcpyHostToDevice, s), "upload");
    };
    if ((rc = up(c->d_lvlF, elF.data(), nE * sizeof(int))) ||
        (rc = up(c->d_opPtr, opPtr.data(), (nE + 1) * sizeof(int))) ||
        (rc = up(c->d_ops, ops.data(), ops.size() * sizeof(int4))) ||
        (rc = up(c->d_swEl, swEl.data(), 2 * (size_t)nE * sizeof(int))) ||
        (rc = up(c->d_swNb, swNb.data(), 2 * (size_t)nE * sizeof(int4))) ||
        (rc = cuda_check(c, cudaMemsetAsync(c->d_iluFlags, 0, (2 + (size_t)nE) * sizeof(unsigned), s), "memset")) ||
        (rc = cuda_check(c, cudaMemsetAsync(c->d_ilu_pub, 0, 4 * (size_t)nE * c->nc * sizeof(unsigned long long), s),
                         "memset")) ||
        (rc = cuda_check(c, cudaStreamSynchronize(s), "sync")))
        return rc;
    // persistent sweep grid: every block co-resident (cooperative launch)
    int dev = 0, nsm = 0, perSm = 0, perSm32 = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    if ((rc = cuda_check(c, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, k_ilu_sweeps<double>, kSweepThreads, 0),
                         "occupancy")) ||
        (rc = cuda_check(c, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm32, k_ilu_sweeps<float>, kSweepThreads, 0),
                         "occupancy")))
        return rc;
    c->sweep_grid = std::max(1, std::min(nE, nsm * std::max(1, std::min(perSm, perSm32))));
    c->ilu_epoch = 0;
    c->ilu_fepoch = 0;
    c->pub_words = fp_ctx::PUB_REGISTER;  // cleared above
    c->ring_parity = 0;
    c->ilu_built = true;
    return FP_OK;
}

// factor storage of one precision, allocated on first use (the full 3D p = 2 case holds
// 69 GB of FP64 or 35 GB of FP32 factors, so only the precision in use exists)
template <class T>
int ilu_storage(fp_ctx* c, T** out);
template <>
int ilu_storage<double>(fp_ctx* c, double** out) {
    int rc;
    if (!c->d_iluF64 && (rc = ialloc(c, &c->d_iluF64, (size_t)c->hm.nElem * (1 + c->hm.nf) * c->nc * c->nc))) return rc;
    *out = c->d_iluF64;
    return FP_OK;
}
template <>
int ilu_storage<float>(fp_ctx* c, float** out) {
    int rc;
    if (!c->d_iluF32 && (rc = ialloc(c, &c->d_iluF32, (size_t)c->hm.nElem * (1 + c->hm.nf) * c->nc * c->nc))) return rc;
    *out = c->d_iluF32;
    return FP_OK;
}

int ilu_check_sizes(fp_ctx* c) {
    if (c->nc > kMaxNc || c->hm.nf > kMaxF)
        return set_err(c, FP_ERR_UNSUPPORTED, "block ILU(0): more than 64 unknowns per element");
    const size_t nc2 = (size_t)c->nc * c->nc;
    if (((size_t)(1 + c->hm.nf) * nc2 + 2 * nc2) * sizeof(double) > 227 * 1024)
        return set_err(c, FP_ERR_UNSUPPORTED, "block ILU(0): element blocks exceed shared memory");
    return FP_OK;
}

// the persistent factorisation of the blocks already in F (T precision), in place
template <class T>
int ilu_factor_run(fp_ctx* c, T* F) {
    int rc;
    const int nE = c->hm.nElem;
    if ((rc = cuda_check(c, cudaMemsetAsync(c->d_status, 0, sizeof(unsigned), c->stream), "memset"))) return rc;
    unsigned* abortw = c->d_iluFlags;
    unsigned epoch = ++c->ilu_fepoch;
    if (epoch == 0) {  // wrapped: clear the row flags and start again
        if ((rc = cuda_check(c, cudaMemsetAsync(c->d_iluFlags + 2, 0, (size_t)nE * sizeof(unsigned), c->stream), "memset")))
            return rc;
        epoch = c->ilu_fepoch = 1;
    }
    if ((rc = cuda_check(c, cudaMemsetAsync(c->d_ilu_sing, 0, (size_t)nE * sizeof(unsigned), c->stream), "memset")) ||
        (rc = ilu_rows(c, F, sizeof(T) == sizeof(float), epoch)))
        return rc;
    unsigned st = 0;
    if ((rc = cuda_check(c, cudaMemcpyAsync(&st, c->d_status, sizeof(unsigned), cudaMemcpyDeviceToHost, c->stream), "copy")) ||
        (rc = cuda_check(c, cudaStreamSynchronize(c->stream), "sync")))
        return rc;
    if (st & FP_DEV_TIMEOUT) {
        cudaMemsetAsync(abortw, 0, sizeof(unsigned), c->stream);
        c->ilu_prec = -1;
        return set_err(c, FP_ERR_TIMEOUT, "block ILU(0) factorisation: a dependency wait gave up");
    }
    if (st & FP_DEV_SINGULAR) {
        c->ilu_prec = -1;
        return set_err(c, FP_ERR_SINGULAR, "singular pivot block in block ILU(0)");
    }
    return FP_OK;
}

template <class T>
int ilu_factor_t(fp_ctx* c, bool gather) {
    int rc;
    T* F = nullptr;
    if ((rc = ilu_storage<T>(c, &F))) return rc;
    if (gather) {
        if (!c->d_Adiag) return set_err(c, FP_ERR_STATE, "block ILU(0): no assembled blocks");
        const int nc = c->nc, nf = c->hm.nf, nE = c->hm.nElem, ld = c->hm.ld;
        dim3 gg((nE + 31) / 32, 1 + nf);
        k_ilu_gather<T><<<gg, 256, 0, c->stream>>>(nE, ld, nc, nf, c->d_Adiag, c->d_Aneigh, c->d_tt, F);
        if ((rc = cuda_check(c, cudaGetLastError(), "ILU gather"))) return rc;
    }
    return ilu_factor_run<T>(c, F);
}

}  // namespace

void ilu_release(fp_ctx* c) {
    c->ilu_built = false;
    c->ilu_prec = -1;
    c->d_iluF64 = nullptr;
    c->d_iluF32 = nullptr;
    c->d_lvlF = c->d_opPtr = nullptr;
    c->d_iluFlags = nullptr;
    c->d_ilu_sing = nullptr;
    c->ilu_epoch = 0;
    c->ilu_fepoch = 0;
    c->d_ops = c->d_swNb = nullptr;
    c->d_swEl = nullptr;
    c->d_ilu_pub = nullptr;
    c->sweep_grid = 0;
    c->ring_grid[0] = c->ring_grid[1] = 0;
    c->pub_words = fp_ctx::PUB_UNKNOWN;
    c->ring_parity = 0;
    c->lvlF_ptr.clear();
}


int ilu_factor(fp_ctx* c, int precision) {
    int rc;
    if ((rc = ilu_check_sizes(c))) return rc;
    if (!c->ilu_built && (rc = ilu_build(c))) return rc;
    rc = precision == FP_PREC_FP32 ? ilu_factor_t<float>(c, true) : ilu_factor_t<double>(c, true);
    if (rc) return rc;
    c->ilu_prec = precision;
    return FP_OK;
}

int ilu_prepare_direct(fp_ctx* c, int precision, void** F) {
    int rc;
    if ((rc = ilu_check_sizes(c))) return rc;
    if (!c->ilu_built && (rc = ilu_build(c))) return rc;
    c->ilu_prec = -1;  // the storage is about to be overwritten
    if (precision == FP_PREC_FP32) {
        float* p = nullptr;
        rc = ilu_storage<float>(c, &p);
        *F = p;
    } else {
        double* p = nullptr;
        rc = ilu_storage<double>(c, &p);
        *F = p;
    }
    return rc;
}

int ilu_factor_direct(fp_ctx* c, int precision) {
    int rc = precision == FP_PREC_FP32 ? ilu_factor_run<float>(c, c->d_iluF32) : ilu_factor_run<double>(c, c->d_iluF64);
    if (rc) return rc;
    c->ilu_prec = precision;
    return FP_OK;
}

// the register kernel (odd numbers of unknowns, and fp_set_ilu_sweep(ctx, 1))
template <class T>
static int launch_register(fp_ctx* c, const T* F, const double* b, double* xx) {
    int nc = c->nc, nf = c->hm.nf, ld = c->hm.ld, nE = c->hm.nElem;
    const size_t words = 2 * (size_t)nE * nc;
    unsigned epoch = ++c->ilu_epoch;
    if (epoch == 0 || c->pub_words != fp_ctx::PUB_REGISTER) {  // wrapped, or not its own words: clear them and start again
        int rc = cuda_check(c, cudaMemsetAsync(c->d_ilu_pub, 0, 2 * words * sizeof(unsigned long long), c->stream), "memset");
        if (rc) return rc;
        epoch = c->ilu_epoch = 1;
        c->pub_words = fp_ctx::PUB_REGISTER;
    }
    unsigned long long* pubF = c->d_ilu_pub;
    unsigned long long* pubB = c->d_ilu_pub + words;
    unsigned* abortw = c->d_iluFlags;
    unsigned* status = abortw + 1;
    int polls = c->ilu_max_polls;
    void* args[] = {&nc, &nf, &ld, &nE, &c->d_swEl, &c->d_swNb, (void*)&F, (void*)&b, &xx, &pubF, &pubB, &epoch,
                    &abortw, &status, &polls};
    return cuda_check(c,
                      cudaLaunchCooperativeKernel((const void*)k_ilu_sweeps<T>, dim3(c->sweep_grid), dim3(kSweepThreads), args, 0,
                                                  c->stream),
                      "ILU sweeps");
}

// Elements in flight per thread block that fp_set_ilu_sweep(ctx, 2 .. 6) may ask for, as the interface
// states it: a power of two up to 16 for nc <= 16, 8 for nc <= 32, else 4, and no more than a budget of
// whole positions (all 1 + nf blocks) in shared memory, 208 KB above 32 unknowns, 100 KB below, divides
// into.  The ring itself would take any number up to its groups of warps; what was refused stays refused.
static bool sweep_groups_allowed(fp_ctx* c, int precision, int NG) {
    const int nc = c->nc, most = nc <= 16 ? 16 : nc <= 32 ? 8 : 4;
    const size_t slot = (size_t)(1 + c->hm.nf) * nc * nc * (precision == FP_PREC_FP32 ? sizeof(float) : sizeof(double));
    const int S = (int)std::min<size_t>(32, (size_t)(nc > 32 ? 208 : 100) * 1024 / slot);
    int p = 2;
    while (2 * p <= std::min(S, most)) p *= 2;
    return NG <= most && (S - S % p) % NG == 0;
}

int ilu_apply(fp_ctx* c, const double* x, double* y) {
    if (c->ilu_prec != FP_PREC_FP32 && c->ilu_prec != FP_PREC_FP64) return set_err(c, FP_ERR_STATE, "block ILU(0): not factorised");
    if (c->sweep_variant != 1 && ring_sweep_applies(c->nc)) {
        const int NG = c->sweep_variant >= 2 ? 1 << (c->sweep_variant - 2) : 0;
        if (NG && !sweep_groups_allowed(c, c->ilu_prec, NG))
            return set_err(c, FP_ERR_UNSUPPORTED, "ILU sweeps: group count above the slots or the block size allows");
        return ring_sweep(c, c->ilu_prec, x, y, NG);
    }
    if (c->ilu_prec == FP_PREC_FP32) return launch_register<float>(c, c->d_iluF32, x, y);
    return launch_register<double>(c, c->d_iluF64, x, y);
}

int ilu_check(fp_ctx* c) {
    if (!c->ilu_built) return FP_OK;
    unsigned* words = c->d_iluFlags;
    unsigned h[2] = {0, 0};
    int rc;
    if ((rc = cuda_check(c, cudaMemcpyAsync(h, words, sizeof(h), cudaMemcpyDeviceToHost, c->stream), "copy")) ||
        (rc = cuda_check(c, cudaStreamSynchronize(c->stream), "sync")))
        return rc;
    if (h[0] || h[1]) {
        cudaMemsetAsync(words, 0, sizeof(h), c->stream);
        c->pub_words = fp_ctx::PUB_UNKNOWN;
        return set_err(c, FP_ERR_TIMEOUT, "block ILU(0) sweep: a dependency wait gave up");
    }
    return FP_OK;
}

}  // namespace fp
