// Block ILU(0) application (BlockILU0.apply, BlockILU0.java:187-243) with the factor blocks
// streamed through shared memory: y = L^-1 b in forward-level order, then x = U^-1 y in
// backward-level order, one persistent cooperative launch per application.
//
// What bounds it.  On large meshes, the bytes of the factors (18,000 tetrahedra of 50 unknowns:
// 1.8 GB in FP64, 0.28 ms at the measured copy rate); on small and two-dimensional ones the
// dependency chain: a level cannot start before the values of the level before it have crossed
// the L2, and the levels of a mesh (127 + 127 on that box, several hundred on a channel) follow
// one another.  So everything between the arrival of the last neighbour's value and the
// publication of the element's own value is kept short (1,600 to 2,200 cycles at 50 unknowns,
// 1,000 to 1,400 at 12; it was 4,500 and 2,800):
//   * the number of unknowns NC is a compile-time constant: the block products are unrolled and each
//     lane holds two adjacent rows (one 16-byte shared load per column and two multiply-adds);
//   * a warp fetches only the values of the columns it multiplies and keeps them in its own
//     shared memory, so one barrier of the element's 1, 2 or 4 warps per block product is left;
//   * a warp leaves its wait as a whole: lanes that left one by one ran all that follows in
//     several passes, which was the largest part (950 -> 460 us an application on that box);
//   * a published value is one 64-bit word: the buffers of the coming application are filled
//     with a NaN pattern (the elements of the running one do that as they publish), and a word
//     that differs from it is the value.  Half the words of a value/epoch pair to poll.
//
// Measured per application, us, before (staged whole positions, the groups' number timed on the
// first application) and now: 18,000 tetrahedra of 50 unknowns FP64 950 -> 420, 86,700 FP32
// 2,200 -> 1,005 (4.3 GB: 4.3 TB/s), 8,832 triangles of 30 unknowns FP32 725 -> 434, 12 merged cases
// of 12 unknowns 1,050 -> 571, 4 of 40 unknowns 1,250 -> 583; 80 merged cases of 12 unknowns, 1.28
// million triangles, over 100 pseudo-time steps with the finished ones passing through 1,900 -> 1,100.
//
// A producer warp requests the factor blocks of the coming positions as single bulk copies into
// a ring of blocks in position order, as far ahead as the ring has room (10 blocks of 50 x 50 in
// FP64): what a position does not multiply takes no room.
//
// The order of a row's sum depends on NC alone, so the values do not depend on the number of
// elements in flight per thread block.  Needs an even NC (the blocks are then whole multiples of 16 bytes,
// as the bulk copies require); odd ones take the register kernel of fp_ilu.cu.
#include <algorithm>
#include <type_traits>

#include "fp_ctx.h"
#include "fp_ring_rule.h"

namespace fp {

namespace {

constexpr int kMaxBlocks = 128;  // blocks of the ring
constexpr int kFaces = 4;
constexpr unsigned long long kEmpty = ~0ull;  // an unpublished word: a NaN no arithmetic produces
constexpr int kSpin = 1 << 12;    // polls back to back before the sleeping ones
constexpr int kBarPolls = 1 << 22;

// The sum of a row: columns g, g + G, ... of every face in one chain of multiply-adds each,
// (face 0 + face 1) + (face 2 + face 3), then the G sums pairwise.  A part of a row is one g and, for
// G = 2, one half of the faces.  FP64 factors keep two chains a face, the order that the
// finite-difference solves have always had (their Jacobian turns a rounding of the state into 1e-8 of
// a block); FP32 factors, which serve the exact tangent, take four: the longest chain of a position
// is shorter and no lane waits for the other half's faces (an application of 8,832 triangles of 30
// unknowns 574 -> 434 us, of the 12 merged cases of 12 unknowns 722 -> 571 us).
template <class T, int NC>
struct Cfg {
    static constexpr int G = NC <= 4 ? 8 : NC <= 8 || sizeof(T) == 4 ? 4 : 2;  // column strides of a row
    static constexpr int H = G == 2 ? 2 : 1;                     // halves of the faces
    static constexpr int P = G * H;                              // parts of a row, g * H + h
    static constexpr int WG = NC <= 16 ? 1 : NC <= 32 ? 2 : 4;   // warps of an element
    static constexpr int CPW = P / WG;                           // parts of a warp
    static constexpr int CW = (NC + G - 1) / G;                  // columns of a part
    static constexpr int RL = NC / 2;                            // lanes of a part: two rows each
    static constexpr int GPW = CPW <= H ? 1 : CPW / H;           // strides of a warp
    static constexpr int FPW = CPW < H ? kFaces / 2 : kFaces;    // faces of a warp
    static constexpr int WC = GPW * CW;                          // columns of a warp
    static constexpr int WARPS = 16;                             // consumer warps (one more is the producer)
    static constexpr int GROUPS = WARPS / WG;                    // elements in flight per thread block
    static_assert(GROUPS <= kRingSlots / 2, "the producer keeps at least as many positions ahead as are in work");
    static constexpr int ROUNDS = ((FPW + 1) * WC + 31) / 32;    // words a lane fetches
    static constexpr int WV = (FPW + 2) * WC;                    // a warp's values: faces, own, before inv(U_ii)
    static constexpr int PART = 2 * P * NC;                      // partial sums of an element, two buffers
    static_assert(NC % 2 == 0 && RL * CPW <= 32 && NC <= 32 * WG && P % WG == 0, "lanes of the row split");
    // two thread blocks per SM for the small blocks, whose positions are short
    static constexpr int CTAS = NC <= 32 ? 2 : 1;
    static constexpr size_t WORK = ((size_t)GROUPS * PART + (size_t)WARPS * WV) * sizeof(double);  // sums and values
    // blocks of the ring: what is left of 226 KB (one thread block per SM) or 112 KB (two) beside
    // the work arrays and the static shared memory; a position takes up to 1 + nf blocks
    static constexpr int PB = (int)std::min<size_t>(kMaxBlocks, ((CTAS == 1 ? 224 : 110) * 1024 - WORK) / ((size_t)NC * NC * sizeof(T)));
    static_assert(PB >= 1 + kFaces, "the ring holds a position");
    static constexpr size_t RING = ((size_t)PB * NC * NC * sizeof(T) + 15) & ~(size_t)15;
    static constexpr size_t SMEM = RING + WORK;
    // the G sums of a row (p: [P][NC] partial sums, h halves added), in the order of the chains above
    __device__ static __forceinline__ double row(const double* p, int r) {
        if constexpr (G == 2) return (p[r] + p[NC + r]) + (p[2 * NC + r] + p[3 * NC + r]);
        if constexpr (G == 4) return (p[r] + p[2 * NC + r]) + (p[NC + r] + p[3 * NC + r]);
        return ((p[r] + p[4 * NC + r]) + (p[2 * NC + r] + p[6 * NC + r])) +
               ((p[NC + r] + p[5 * NC + r]) + (p[3 * NC + r] + p[7 * NC + r]));
    }
};

__device__ __forceinline__ unsigned sa(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bar_init(unsigned long long* b) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sa(b)) : "memory");
}
__device__ __forceinline__ void bar_expect(unsigned long long* b, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(sa(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bar_arrive(unsigned long long* b) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(sa(b)) : "memory");
}
__device__ __forceinline__ bool bar_test(unsigned long long* b, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(sa(b)), "r"(parity)
        : "memory");
    return ok != 0;
}
// the same without suspending the thread
__device__ __forceinline__ bool bar_passed(unsigned long long* b, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(sa(b)), "r"(parity)
        : "memory");
    return ok != 0;
}
// global -> shared bulk copy (multiple of 16 bytes, both addresses 16-byte aligned)
__device__ __forceinline__ void copy_block(void* dst, const void* src, unsigned bytes, unsigned long long* b) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(sa(dst)),
                 "l"(src), "r"(bytes), "r"(sa(b))
                 : "memory");
}
__device__ __forceinline__ unsigned long long word_load(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void word_store(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// k-th position of this thread block: forward b, b + GB, ... (< nE), then backward nE + b, ...;
// 2 nE past the end
__device__ __forceinline__ int position(int k, int nE) {
    const int b = (int)blockIdx.x, GB = (int)gridDim.x;
    const int Jf = b < nE ? (nE - 1 - b) / GB + 1 : 0;
    if (k < Jf) return b + k * GB;
    const int v = nE + b + (k - Jf) * GB;
    return v < 2 * nE ? v : 2 * nE;
}

struct SweepArgs {
    int nf, ld, nE, NG;       // NG: elements in flight per thread block
    const int* swEl;          // [2 nE] element at a position
    const int4* swNb;         // [2 nE] neighbours multiplied there (-1 none)
    const double* b;          // [NC][ld]
    double* x;                // [NC][ld]
    unsigned long long *fwd, *bwd;            // [nE][NC] words of this application
    unsigned long long *fwdNext, *bwdNext;    // the next application's, emptied on the way
    unsigned *abortw, *status;
    int maxPolls;
    const int *caseOf, *live;  // batched cases: positions of cases with live 0 only pass through
};

// loads that stay where they are written: the compiler would move a load down to its use, behind
// the wait for the neighbours' values (2,800 instead of 900 cycles from there to the publication)
__device__ __forceinline__ double early(const double* p) {
    double v;
    asm volatile("ld.global.cg.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ int early(const int* p) {
    int v;
    asm volatile("ld.global.nc.s32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ int4 early(const int4* p) {
    int4 v;
    asm volatile("ld.global.nc.v4.s32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

// rows r, r + 1 (ROWS 2) or r (ROWS 1) of a block times the columns g, g + G, ...  (Measured and
// dropped: the rows of two blocks in registers at once, and inv(U_ii) loaded before the warps
// meet; both were slower, 459 -> 489 us an application of 18,000 tetrahedra in FP64.)
template <class T, int NC, int ROWS>
__device__ __forceinline__ void rows_times(const T* B, const double* v, int r, int g, double* s) {
    using C = Cfg<T, NC>;
    B += g * NC + r;
#pragma unroll
    for (int j = 0; j < C::CW; j++) {
        if (C::G * (j + 1) <= NC || g + C::G * j < NC) {
            const double vj = v[j];
            if constexpr (ROWS == 1) {
                s[0] += (double)B[C::G * j * NC] * vj;
            } else {
                double b0, b1;
                if constexpr (sizeof(T) == 8) {
                    const double2 q = *reinterpret_cast<const double2*>(B + C::G * j * NC);
                    b0 = q.x;
                    b1 = q.y;
                } else {
                    const float2 q = *reinterpret_cast<const float2*>(B + C::G * j * NC);
                    b0 = (double)q.x;
                    b1 = (double)q.y;
                }
                s[0] += b0 * vj;
                s[1] += b1 * vj;
            }
        }
    }
}

template <class T, int NC>
__device__ __forceinline__ void group_sync(int grp) {
    if constexpr (Cfg<T, NC>::WG == 1)
        __syncwarp();
    else
        asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "r"(32 * Cfg<T, NC>::WG) : "memory");
}

// Shared memory: the ring's blocks, a full and an empty mbarrier and the first block of each
// position in flight, then per element in flight its partial sums and per warp its values.
//
// Waits: every dependency lies in an earlier level, a thread block takes its positions in level
// order, requests their blocks in that order and releases them in bounded time, and all thread
// blocks are co-resident (cooperative launch), so each wait ends; each is bounded all the same.
// A wait for a value that gives up sets FP_DEV_TIMEOUT and the abort word, which ends every other
// one; the sweep then runs to its end with garbage.  The waits on the ring's barriers (kBarPolls: for
// blocks on their way, and the producer's for a position to be released, which includes that
// position's waits for values) do the same and set `dead`: the producer requests nothing more, and
// the consumers pass the remaining positions without reading blocks that were not requested for them.
template <class T, int NC>
__global__ void __launch_bounds__(32 * (Cfg<T, NC>::WARPS + 1), Cfg<T, NC>::CTAS) k_sweep_ring(SweepArgs A, const T* __restrict__ F) {
    using C = Cfg<T, NC>;
    constexpr int NC2 = NC * NC, PB = C::PB;
    extern __shared__ __align__(128) unsigned char ring_smem[];
    __shared__ __align__(8) unsigned long long full[kRingSlots], empty[kRingSlots];
    __shared__ int first[kRingSlots];
    __shared__ int cnts[kRingSlots];  // producer's own: blocks of each position
    __shared__ volatile int dead;
    T* ring = reinterpret_cast<T*>(ring_smem);
    double* work = reinterpret_cast<double*>(ring_smem + C::RING);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nE = A.nE, nf = A.nf, nV = 2 * nE;
    if ((int)blockIdx.x >= nE) return;
    if (threadIdx.x == 0) {
        dead = 0;
        for (int q = 0; q < kRingSlots; q++) {
            bar_init(full + q);
            bar_init(empty + q);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

    if (warp == C::WARPS) {  // ------------------------------------------------ producer
        // A trip takes all positions that have been released since the last one: lane l tests the barrier of
        // position tail + l, their blocks are added up, one proxy fence, and as many of the next 32
        // positions as now fit are requested, a lane each.  With one position a trip the producer
        // bounded large meshes of small blocks at 1,150 cycles a position (an application, all cases live,
        // ms: 1.28 million triangles of 12 unknowns 5.09 -> 2.05, 1.34 million of 24 5.35 -> 3.33; the 100
        // pseudo-time steps of the former 43.6 -> 20.3 s).
        const int ns = 1 + nf;
        int head = 0, tail = 0;        // positions requested, released
        int used = 0, next = 0;        // blocks in use, first free block
        bool more = true, fail = false;
        int i_next = 0;
        int4 nb_next = make_int4(-1, -1, -1, -1);
        auto fetch = [&](int k) {  // the program entry of position k, used a trip later
            const int v = position(k, nE);
            if (v >= nV) return;
            i_next = early(A.swEl + v);
            nb_next = early(A.swNb + v);
        };
        fetch(lane);
        while (more && !fail) {
            const int k = head + lane, v = position(k, nE);
            const bool have = v < nV;
            const int i = i_next;
            const int4 nb = nb_next;
            fetch(k + 32);
            int cnt = 0;
            if (have && !(A.live && !A.live[A.caseOf[i]]))
                cnt = (v >= nE) + (nb.x >= 0) + (nb.y >= 0) + (nb.z >= 0) + (nb.w >= 0);
            int sum = cnt;  // blocks up to and with this position
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(~0u, sum, o);
                if (lane >= o) sum += t;
            }
            const int n = __popc(__ballot_sync(~0u, have));
            const int total = __shfl_sync(~0u, sum, 31);
            int done = 0, freed = 0;  // of these 32: requested; blocks released meanwhile
            while (true) {
                const bool ok = have && lane >= done && used + sum - freed <= PB && ring_may_request(k, tail, A.NG);
                const unsigned m = __ballot_sync(~0u, ok);
                if (ok) {
                    const int q = k % kRingSlots;
                    int blk = (next + sum - cnt) % PB;
                    first[q] = blk;
                    cnts[q] = cnt;
                    bar_expect(full + q, (unsigned)(cnt * NC2 * sizeof(T)));
                    if (cnt > 0) {
                        const T* src = F + (size_t)i * ns * NC2;
                        const int nbs[kFaces] = {nb.x, nb.y, nb.z, nb.w};
#pragma unroll
                        for (int f = -1; f < kFaces; f++)
                            if (f < 0 ? v >= nE : nbs[f < 0 ? 0 : f] >= 0) {
                                copy_block(ring + (size_t)blk * NC2, src + (size_t)(1 + f) * NC2, NC2 * sizeof(T), full + q);
                                blk = blk + 1 == PB ? 0 : blk + 1;
                            }
                    }
                }
                __syncwarp();
                done += __popc(m);
                if (done == n) break;
                // no room for the next one: wait for the oldest position in flight, then take all those that
                // follow it and are released (polling the 32 barriers for the first of them cost the
                // other warps 5 % where the chain of levels bounds: shared memory is theirs)
                bool got = false;
                for (int it = 0; it < kBarPolls && !got; it++) {
                    got = __all_sync(~0u, bar_test(empty + tail % kRingSlots, ring_lap_parity(tail)));
                    if (__any_sync(~0u, dead != 0)) break;
                }
                if (!got) {
                    fail = true;
                    break;
                }
                const int t = tail + lane;
                const bool rel = t < head + done && bar_passed(empty + t % kRingSlots, ring_lap_parity(t));
                int run = __ffs(~__ballot_sync(~0u, rel)) - 1;  // -1: all 32
                if (run < 0) run = 32;
                freed += __reduce_add_sync(~0u, lane < run ? cnts[(tail + lane) % kRingSlots] : 0);
                tail += run;
                // the positions' shared reads come before the copies that reuse their blocks
                __syncwarp();
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            }
            used += total - freed;
            next = (next + total) % PB;
            head += done;
            more = n == 32;
        }
        if (fail) {
            if (lane == 0) {
                dead = 1;
                atomicOr(A.status, (unsigned)FP_DEV_TIMEOUT);
                atomicExch(A.abortw, 1u);
            }
        }
        // no copy may be in flight when the thread block ends
        for (int k = tail; k < head; k++)
            for (int it = 0; it < kBarPolls && !bar_test(full + k % kRingSlots, ring_lap_parity(k)); it++) {
            }
        return;
    }

    // -------------------------------------------------------------------------- consumers
    const int grp = warp / C::WG, gw = warp - grp * C::WG;
    if (grp >= A.NG) return;
    const int gt = gw * 32 + lane;             // thread of the element: row of the final sums
    const int cl = lane / C::RL, rl = lane - cl * C::RL;
    const bool act = cl < C::CPW;
    const int pt = act ? gw * C::CPW + cl : 0, g = pt / C::H, h = pt - g * C::H;  // this lane's part
    const int g0 = gw * C::CPW / C::H;                           // first stride of this warp
    const int f0 = C::CPW < C::H ? (gw & 1) * C::FPW : 0;           // and its first face
    double* part = work + (size_t)grp * C::PART;
    double* wv = work + (size_t)C::GROUPS * C::PART + (size_t)warp * C::WV;
    int buf = 0;                               // partial-sum buffer, alternating at every barrier
    int k = grp, v = position(k, nE);
    int i_cur = v < nV ? early(A.swEl + v) : 0;
    int4 nb_cur = v < nV ? early(A.swNb + v) : make_int4(-1, -1, -1, -1);
    while (v < nV) {
        const bool bwd = v >= nE;
        const int i = i_cur, q = k % kRingSlots;
        const int4 nbv = nb_cur;
        const int vn = position(k + A.NG, nE);
        if (vn < nV) {  // the next program entry, in flight during this position
            i_cur = early(A.swEl + vn);
            nb_cur = early(A.swNb + vn);
        }
        const bool skip = A.live && !A.live[A.caseOf[i]];
        unsigned long long* pub = bwd ? A.bwd : A.fwd;
        const double a_in = (!skip && !bwd && gt < NC) ? early(A.b + (size_t)gt * A.ld + i) : 0.0;
        // the words this warp multiplies: its columns of every neighbour and, backward, of the
        // element's own forward value
        unsigned pw[C::ROUNDS];  // index of the word
        unsigned long long pv[C::ROUNDS];
        auto word = [&](int r, unsigned at) { return word_load(((r * 32 + lane) / C::WC == C::FPW ? A.fwd : pub) + at); };
#pragma unroll
        for (int r = 0; r < C::ROUNDS; r++) {
            const int u = r * 32 + lane, fl = u / C::WC, f = fl == C::FPW ? kFaces : f0 + fl;
            const int c = g0 + (u - fl * C::WC) / C::CW + C::G * ((u - fl * C::WC) % C::CW);
            int n = f == 0 ? nbv.x : f == 1 ? nbv.y : f == 2 ? nbv.z : f == 3 ? nbv.w : bwd ? i : -1;
            if (fl > C::FPW || c >= NC || skip) n = -1;
            pw[r] = n < 0 ? 0u : (unsigned)n * NC + c;
            pv[r] = n >= 0 ? word(r, pw[r]) : 0ull;
        }
        // the position's blocks have arrived
        bool got = false;
        for (int it = 0; it < kBarPolls && !got; it++) {
            got = __all_sync(~0u, bar_test(full + q, ring_lap_parity(k)));
            if (__any_sync(~0u, dead != 0)) {
                got = false;
                break;
            }
        }
        if (!got) {
            dead = 1;
            atomicOr(A.status, (unsigned)FP_DEV_TIMEOUT);
            atomicExch(A.abortw, 1u);
        }
        for (int it = 0;; it++) {
            bool miss = false;
#pragma unroll
            for (int r = 0; r < C::ROUNDS; r++) miss = miss || pv[r] == kEmpty;
            // the whole warp leaves together: lanes that left one by one would run what follows in
            // as many passes
            if (!__any_sync(~0u, miss)) break;
            if (it >= A.maxPolls) {
                if (miss) {
                    atomicOr(A.status, (unsigned)FP_DEV_TIMEOUT);
                    atomicExch(A.abortw, 1u);
                }
                break;
            }
            if ((it & 31) == 31 && __any_sync(~0u, *(volatile unsigned*)A.abortw != 0u)) break;
            if (it >= kSpin) __nanosleep(64);
#pragma unroll
            for (int r = 0; r < C::ROUNDS; r++)
                if (pv[r] == kEmpty) pv[r] = word(r, pw[r]);
        }
        __syncwarp();
#pragma unroll
        for (int r = 0; r < C::ROUNDS; r++)
            if (r * 32 + lane < (C::FPW + 1) * C::WC)
                wv[r * 32 + lane] = pv[r] == kEmpty ? 0.0 : __longlong_as_double((long long)pv[r]);  // empty: given up
        __syncwarp();
        int blk = first[q];
        const T* D = ring + (size_t)blk * NC2;
        if (bwd) blk = blk + 1 == PB ? 0 : blk + 1;
        if (!skip) {
            // the position's blocks follow one another in the ring, in the order of the faces
            double sf[kFaces][2] = {{0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}};
            const int nbs[kFaces] = {nbv.x, nbv.y, nbv.z, nbv.w};
#pragma unroll
            for (int f = 0; f < kFaces; f++)
                if (nbs[f] >= 0) {
                    if (act && got && (C::H == 1 || f / 2 == h))
                        rows_times<T, NC, 2>(ring + (size_t)blk * NC2, wv + (f - f0) * C::WC + (g - g0) * C::CW, 2 * rl, g, sf[f]);
                    blk = blk + 1 == PB ? 0 : blk + 1;
                }
            double* p = part + buf * C::P * NC;
            buf ^= 1;
            if (act)
                *reinterpret_cast<double2*>(p + pt * NC + 2 * rl) =
                    C::H == 1 ? make_double2((sf[0][0] + sf[1][0]) + (sf[2][0] + sf[3][0]),
                                             (sf[0][1] + sf[1][1]) + (sf[2][1] + sf[3][1]))
                    : h == 0  ? make_double2(sf[0][0] + sf[1][0], sf[0][1] + sf[1][1])
                              : make_double2(sf[2][0] + sf[3][0], sf[2][1] + sf[3][1]);
            group_sync<T, NC>(grp);
            double a = 0.0;
            if (!bwd) {
                if (gt < NC) a = a_in - C::row(p, gt);
            } else {
                // this warp's columns of the value before inv(U_ii), then the product with it: one
                // row a lane where two halves share a stride
                double* tv = wv + (C::FPW + 1) * C::WC;
                for (int u = lane; u < C::WC; u += 32) {
                    const int c = g0 + u / C::CW + C::G * (u % C::CW);
                    if (c < NC) tv[u] = wv[C::FPW * C::WC + u] - C::row(p, c);
                }
                __syncwarp();
                double d[2] = {0.0, 0.0};
                p = part + buf * C::P * NC;
                buf ^= 1;
                if (C::H == 2) {
                    if (act && got) rows_times<T, NC, 1>(D, tv + (g - g0) * C::CW, h * C::RL + rl, g, d);
                    if (act) p[g * NC + h * C::RL + rl] = d[0];
                } else {
                    if (act && got) rows_times<T, NC, 2>(D, tv + (g - g0) * C::CW, 2 * rl, g, d);
                    if (act) *reinterpret_cast<double2*>(p + g * NC + 2 * rl) = make_double2(d[0], d[1]);
                }
                group_sync<T, NC>(grp);
                if (gt < NC) a = C::H == 2 ? p[gt] + p[NC + gt] : C::row(p, gt);
            }
            if (gt < NC) {
                unsigned long long w = (unsigned long long)__double_as_longlong(a);
                if (w == kEmpty) w = 0x7ff8000000000000ull;
                word_store(pub + (size_t)i * NC + gt, w);
                if (bwd) A.x[(size_t)gt * A.ld + i] = a;
            }
        } else {
            group_sync<T, NC>(grp);  // every warp has passed the full barrier before the slot is reused
        }
        // the barrier above ends the reads of the blocks
        if (gt == 0) bar_arrive(empty + q);
        if (gt < NC) (bwd ? A.bwdNext : A.fwdNext)[(size_t)i * NC + gt] = kEmpty;
        v = vn;
        k += A.NG;
    }
}

template <class T, int NC>
struct Ring {
    using C = Cfg<T, NC>;
    static int configure(fp_ctx* c, int pi) {
        constexpr size_t sm = C::SMEM;
        int rc, dev = 0, nsm = 0, perSm = 0;
        if ((rc = cuda_check(c, cudaFuncSetAttribute(k_sweep_ring<T, NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm),
                             "smem")))
            return rc;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
        if ((rc = cuda_check(c, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, k_sweep_ring<T, NC>, 32 * (C::WARPS + 1), sm),
                             "occupancy")))
            return rc;
        if (perSm < 1) return set_err(c, FP_ERR_UNSUPPORTED, "block ILU(0): the sweep does not fit an SM");
        c->ring_grid[pi] = std::max(1, std::min(c->hm.nElem, nsm * perSm));
        return FP_OK;
    }
    static cudaError_t launch(fp_ctx* c, int pi, SweepArgs& a, const T* F) {
        if (a.NG <= 0) {
            // elements in flight for six levels of average width: with more, the warps that wait
            // several levels ahead poll the L2 for nothing (8,832 triangles of 30 unknowns, 62 a
            // level: 434 us with 1 or 2 a thread block, 508 with 8; 53,400 of 12 unknowns, 196 a
            // level: 775, 571 and 594 us with 1, 4 and 16).  Large meshes keep every warp busy: 1.28
            // million of 12 unknowns 4.23, 2.45 and 2.05 ms with 4, 8 and 16, 1.34 million of 24 4.54 and
            // 3.33 with 4 and 8.
            const double width = (double)a.nE / std::max<size_t>(1, c->lvlF_ptr.size() - 1);
            a.NG = 1 + (int)std::min(64.0, 6.0 * width / c->ring_grid[pi]);
        }
        a.NG = std::min(a.NG, C::GROUPS);
        void* args[] = {&a, (void*)&F};
        return cudaLaunchCooperativeKernel((const void*)k_sweep_ring<T, NC>, dim3(c->ring_grid[pi]), dim3(32 * (C::WARPS + 1)), args,
                                           C::SMEM, c->stream);
    }
};

template <class T>
int run(fp_ctx* c, SweepArgs& a, const T* F) {
    const int pi = sizeof(T) == sizeof(float) ? 1 : 0;
#define FP_RING(N)                                                                   \
    case N: {                                                                        \
        int rc = c->ring_grid[pi] ? FP_OK : Ring<T, N>::configure(c, pi);            \
        return rc ? rc : cuda_check(c, Ring<T, N>::launch(c, pi, a, F), "ILU sweeps"); \
    }
    switch (c->nc) {  // every even number of unknowns of the compiled models and orders
        FP_RING(4) FP_RING(6) FP_RING(10) FP_RING(12) FP_RING(16) FP_RING(18) FP_RING(20) FP_RING(24) FP_RING(30) FP_RING(40)
        FP_RING(50)
    }
#undef FP_RING
    return set_err(c, FP_ERR_UNSUPPORTED, "block ILU(0): no staged sweep for this number of unknowns");
}

}  // namespace

bool ring_sweep_applies(int nc) {
    for (int n : {4, 6, 10, 12, 16, 18, 20, 24, 30, 40, 50})
        if (nc == n) return true;
    return false;
}

int ring_sweep(fp_ctx* c, int precision, const double* b, double* x, int groups) {
    const size_t n = (size_t)c->hm.nElem * c->nc;
    unsigned long long* pub = c->d_ilu_pub;  // [2][forward, backward][nElem][nc]
    if (c->pub_words != fp_ctx::PUB_RING) {
        int rc = cuda_check(c, cudaMemsetAsync(pub, 0xff, 4 * n * sizeof(unsigned long long), c->stream), "memset");
        if (rc) return rc;
        c->pub_words = fp_ctx::PUB_RING;
    }
    const int par = c->ring_parity;
    c->ring_parity ^= 1;
    SweepArgs a{};
    a.nf = c->hm.nf;
    a.ld = c->hm.ld;
    a.nE = c->hm.nElem;
    a.NG = groups;
    a.swEl = c->d_swEl;
    a.swNb = c->d_swNb;
    a.b = b;
    a.x = x;
    a.fwd = pub + (size_t)(2 * par) * n;
    a.bwd = pub + (size_t)(2 * par + 1) * n;
    a.fwdNext = pub + (size_t)(2 * (par ^ 1)) * n;
    a.bwdNext = pub + (size_t)(2 * (par ^ 1) + 1) * n;
    a.abortw = c->d_iluFlags;
    a.status = c->d_iluFlags + 1;
    a.maxPolls = c->ilu_max_polls;
    a.caseOf = c->batch_mask ? c->d_case_of : nullptr;
    a.live = c->batch_mask ? c->d_blive : nullptr;
    const int rc = precision == FP_PREC_FP32 ? run<float>(c, a, c->d_iluF32) : run<double>(c, a, c->d_iluF64);
    if (rc) c->pub_words = fp_ctx::PUB_UNKNOWN;  // not launched: the other half has not been emptied
    return rc;
}

}  // namespace fp
