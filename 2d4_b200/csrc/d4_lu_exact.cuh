// d4_lu_exact.cuh: FP64 LU with exact partial pivoting in the oracle's
// operation order, by a group of CTAs (the grid of a cooperative launch, or one
// thread-block cluster).  Compiled with --fmad=false.
//
// Same result, bit for bit, as the oracle's right-looking Gaussian elimination
// with partial pivoting (first index of the largest |a_ik| wins; an exact zero
// pivot skips its column and marks the matrix singular), which stands in for
// umfpack_di_numeric (src/simulation.cpp:635-640).  Every entry keeps its
// update sequence: a_ij -= l_ik * u_kj for k ascending, product and difference
// rounded separately.
//
// Schedule, per block of 32 columns:
//   pass    Without pivoting, from the diagonal block's factors: the rows below
//           it (multipliers L21) and the columns right of it (U12 = L11^-1 A12),
//           4 lanes per row or column, both by all warps at once.  Starts from
//           a saved copy P0 of the block's columns with the swaps found so far
//           applied; U12 goes to a buffer, so a rejected pass has overwritten
//           nothing it reads.  Pre-division values go to Q; a 32-bit mask
//           records the columns where partial pivoting would have swapped (some
//           |a_ik| > |a_kk|) or met a zero pivot.  One group barrier.
//   decide  Every CTA reads the mask.  Empty: the pass is exact.  Otherwise the
//           first flagged column gets its exact pivot from Q (first max), the
//           swap (or the singular skip) joins the block's list, is applied to
//           the columns outside the block, and the pass repeats.  A row swap at
//           column k commutes with the updates of earlier columns, so applying
//           the list to P0 up front is exact.
//   update  A22 -= L21 U12 in tiles, the next tile's operands in flight while
//           one computes.  The tiles
//           that hold the next block's rows and columns come first and are
//           counted; the group's last CTA forms the next diagonal block itself
//           (the same operations in the same order as the tile that owns it),
//           eliminates it and publishes it.  The oracle skips an update whose
//           u_kj is exactly 0; here it is applied (x - l*0 == x for finite l,
//           and the multipliers of an accepted pass are finite, |l| <= 1, while the
//           elimination stays finite; the slow paths of a pass do skip).
// The next block's pass waits for that publication and those tiles only, so a
// block without swaps costs one group barrier.  Every wait is bounded.
//
// What bounds it.  At N <= 1024 the look-ahead's chain of one block, 26,500 cycles:
// its 32 rows and columns 5,500, their update 1,900, the elimination 8,800 (a
// reciprocal, a quotient, a product and a difference per column), loads, verdict and
// publication the rest; the others' chain (their rows and columns, the group
// barrier's 2,400, the strips) is 7,000 shorter.  At N = 4096 the update, at the
// rate of separate FP64 products and differences (64 lanes per clock and SM).
// One CTA of 256 threads per SM: the chains and the 8 x 4 update tiles need
// more than the 128 registers that 512 threads leave.
#pragma once
#include <cstddef>
#include <cstdint>

#include <cuda.h>

#include "d4_bulk.cuh"
#include "d4_internal.h"
#include "d4_qdiv.cuh"

namespace d4 {
namespace lux {

constexpr int NB = 32;
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kLanes = 4;            // lanes per row below / column right in a pass
constexpr int kHold = NB / kLanes;   // entries per lane
constexpr int kRows = 32 / kLanes;   // rows or columns per warp
constexpr int kBoxR = 64, kBoxC = 32;  // the update's tensor-copy boxes: rows x columns of A
constexpr int kDgWords = NB * (NB + 1) + NB;
constexpr long long kSpinLimit = 1ll << 22;  // polls of several hundred cycles: > 1 s

// Group-wide buffers of one factorisation (sizes in doubles, words or ints).
struct Args {
    int n;
    double *A;       // column-major n x n, factorised in place
    double *P0;      // n x 32, row-major: the block's columns before the block
    double *Q;       // 2 x (n x 32), row-major: pre-division values (double-buffered)
    double *U;       // 2 x (32 x n), row-major: U12 of a block (double-buffered)
    double *dg;      // kDgWords: the published diagonal block and its reciprocals
    unsigned *mask;  // one word per pass (zeroed before the launch): flagged columns
    unsigned *sched; // zeroed: per block kb the update's finished strip tiles [kb];
                     // [nblk] the last block whose diagonal block is published
    int *perm;       // n: original row of each position (receives the row swaps)
    int *piv;        // n pivot rows
    int *flags;      // kFlagSingular, kFlagBarrierTimeout, kFlagPasses, kFlagSwaps
    const CUtensorMap *map_a;  // A, boxes of kBoxR rows x kBoxC columns
    const CUtensorMap *map_u;  // U as 64 rows of n, boxes of kBoxC columns x NB rows
};

struct Smem {
    double lp[2][2][NB][kBoxR];     // [team][buffer]: a tile's L21 piece
    double up[2][2][2][NB][kBoxC];  // [team][buffer][column box]: its U12 piece
    double at[2][2][kBoxC][kBoxR];  // [team][column box]: the next tile's entries
    double s[NB][NB + 1];           // diagonal block (rows = positions k0..k0+31)
    double q[NB][NB + 1];           // its pre-division values
    double rs[NB];                  // RN(1 / pivot); 0 outside the quotient window
    double lcol[NB][NB];            // elimination: multipliers of each column
    uint64_t done[NB];              // elimination: mbarrier of each column
    uint64_t full[2][2];            // update: [team][buffer]: the copies have landed
    double red_v[kWarps];
    int red_i[kWarps];
    int sa[NB], sb[NB];             // swap list of the block (positions)
    unsigned skip;                  // singular columns (skipped)
    unsigned cta_mask;
    int ns;
    int dead;                       // a bounded wait gave up: stop waiting
    int stuck;                      // a wait of the elimination gave up
    unsigned parity;                // phase of the mbarriers' next elimination
    unsigned verdict;               // the pass's flagged columns, after the group barrier
    unsigned la_mask;               // look-ahead: flags of the published diagonal block
};
static_assert(offsetof(Smem, up) % 128 == 0 && offsetof(Smem, at) % 128 == 0, "alignment");
static_assert(sizeof(Smem) <= 227 * 1024, "shared memory of a CTA");

// The CTA's shared memory.  Every function names it itself: through a reference
// parameter the out-of-line ones would use generic loads (the rows' chain took
// 7,500 cycles with them).
__device__ __forceinline__ Smem &smem() {
    extern __shared__ __align__(128) unsigned char lux_smem[];
    return *reinterpret_cast<Smem *>(lux_smem);
}

__device__ __forceinline__ unsigned ld_acq(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_rel(unsigned *p, unsigned v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void red_rel(unsigned *p, unsigned v) {
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void named_bar(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// One thread: wait until *p >= target.  After kSpinLimit polls, or as soon as
// any CTA has given up (kFlagBarrierTimeout), it records the timeout and the
// CTA stops waiting for good, so the launch always ends.
__device__ __forceinline__ void wait_ge(const unsigned *p, unsigned target, int *flags,
                                        int *dead) {
    if (*dead) return;
    long long spins = 0;
    while ((int)(ld_acq(p) - target) < 0) {
        if ((++spins & 255) == 0 &&
            (spins > kSpinLimit || ld_acq((const unsigned *)&flags[kFlagBarrierTimeout]))) {
            atomicOr(&flags[kFlagBarrierTimeout], 1);
            *dead = 1;
            return;
        }
    }
}

// Orders this thread's writes before other CTAs' bulk copies, or writes it has
// seen before its own bulk copies (which go through another proxy).
__device__ __forceinline__ void fence_bulk() {
    asm volatile("fence.proxy.async;" ::: "memory");
}

// Tensor copy of the box at (x, y) into shared memory (x a multiple of 2: 16
// bytes); entries past the tensor's edges are zero.
__device__ __forceinline__ void box_load(void *dst, const CUtensorMap *map, int x, int y,
                                         uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], "
        "[%1, {%2, %3}], [%4];" ::"r"(bulk::smem_u32(dst)),
        "l"(map), "r"(x), "r"(y), "r"(bulk::smem_u32(bar))
        : "memory");
}

// Group barriers that also carry the pass's verdict.  arrive(flagged) ends a
// CTA's part of a pass (its flags, if any, are in the pass's mask word by
// then); wait(mask word) returns the flagged columns of all CTAs.  All threads
// call both.

// The CTAs of a cooperative launch.  *bar counts arrivals (low half) and
// flagged arrivals (high half), zeroed before the launch; the mask word is only
// read when the flagged count moved since this CTA's last barrier.  A count read
// after some CTA has arrived at the next barrier (the low half is past the
// target) may hold that barrier's flags: then this and the next barrier read the
// mask word whatever the count.
struct GridGroup {
    unsigned long long *bar;
    unsigned gen, flagged;
    bool unsure;
    __device__ int rank() const { return blockIdx.x; }
    __device__ int size() const { return gridDim.x; }
    __device__ void arrive(bool flag) {
        fence_bulk();
        __syncthreads();
        arrive_quiet(flag);
    }
    // ... where the caller has just synchronised; the release's fence holds up
    // one warp only, the last
    __device__ void arrive_quiet(bool flag) {
        if (threadIdx.x == kThreads - 1)
            asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(bar),
                         "l"(flag ? (1ull << 32) + 1ull : 1ull)
                         : "memory");
    }
    __device__ unsigned wait(const unsigned *mask, int *flags) {
        Smem &S = smem();
        if (threadIdx.x == 0) {
            const unsigned target = ++gen * gridDim.x;
            unsigned long long v = 0;
            long long spins = 0;
            while (!S.dead) {
                asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(bar) : "memory");
                if ((int)((unsigned)v - target) >= 0) break;
                if ((++spins & 255) == 0 &&
                    (spins > kSpinLimit || ld_acq((const unsigned *)&flags[kFlagBarrierTimeout]))) {
                    atomicOr(&flags[kFlagBarrierTimeout], 1);
                    S.dead = 1;
                }
            }
            const unsigned f = (unsigned)(v >> 32);
            const bool ahead = (unsigned)v != target;
            S.verdict = mask && (f != flagged || ahead || unsure) ? ld_acq(mask) : 0u;
            flagged = f;
            unsure = ahead;
        }
        __syncthreads();
        return S.verdict;
    }
};

// One thread-block cluster (all its CTAs run together by construction).
struct ClusterGroup {
    __device__ int rank() const {
        unsigned r;
        asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
        return (int)r;
    }
    __device__ int size() const {
        unsigned r;
        asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
        return (int)r;
    }
    __device__ void arrive(bool) {
        fence_bulk();
        __syncthreads();
        arrive_quiet(false);
    }
    __device__ void arrive_quiet(bool) {
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    }
    __device__ unsigned wait(const unsigned *mask, int *) {
        Smem &S = smem();
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        if (threadIdx.x == 0) S.verdict = mask ? ld_acq(mask) : 0u;
        __syncthreads();
        return S.verdict;
    }
};

// Source row in P0 of position r after the block's transpositions (applied in
// order to the arrangement): walk the list backwards.
__device__ __forceinline__ int src_row(int r, const int *sa, const int *sb, int ns) {
    for (int t = ns - 1; t >= 0; --t) {
        if (r == sa[t])
            r = sb[t];
        else if (r == sb[t])
            r = sa[t];
    }
    return r;
}

// A numerator of qdiv::fast whose divisor's reciprocal is known to be in window.
__device__ __forceinline__ bool value_ok(double a) { return qdiv::in_range(a) | (a == 0.0); }

// Reciprocal estimate (relative error about 2^-20), the seed of Newton steps.
__device__ __forceinline__ double rcp_seed(double d) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    return y;
}

// y = RN(1/d) from a seed: Newton steps y += y (1 - d y) with FMA residuals
// (Markstein 1990).  When the residual before the second step is below 2^-30,
// the second step's y is within an ulp of 1/d and the third step rounds
// correctly unless d's significand is all ones; recip_ok says that both hold and
// d is in qdiv's window.  (A branch-free chain: the compiler's division keeps a
// slow-path branch inside, which nothing can be scheduled across.)
__device__ __forceinline__ double recip_rn(double d, double y0, double &e2) {
    const double e1 = __fma_rn(-d, y0, 1.0), y1 = __fma_rn(y0, e1, y0);
    e2 = __fma_rn(-d, y1, 1.0);
    const double y2 = __fma_rn(y1, e2, y1);
    const double e3 = __fma_rn(-d, y2, 1.0);
    return __fma_rn(y2, e3, y2);
}
__device__ __forceinline__ bool recip_ok(double d, double e2) {
    const bool ones = __double2loint(d) == -1 && (__double2hiint(d) & 0xfffff) == 0xfffff;
    return qdiv::in_range(d) && fabs(e2) <= 0x1p-30 && !ones;
}

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_arrive(uint64_t *b) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(b)) : "memory");
}
// 0 when the wait gave up.  (The arrival is an earlier warp's of this CTA, within
// microseconds; a poll takes 1.5 us.  An elimination may run into 28 such waits, so
// their limit is short.)
__device__ __forceinline__ uint32_t mbar_wait(uint64_t *b, uint32_t parity) {
    uint32_t done = 0;
    for (long long k = 0; k < (1 << 16) && !done; ++k) {
        asm volatile(
            "{\n\t.reg .pred P1;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
            "selp.b32 %0, 1, 0, P1;\n\t}\n"
            : "=r"(done)
            : "r"(smem_u32(b)), "r"(parity)
            : "memory");
    }
    return done;
}

// Eliminates the 32 x 32 diagonal block without pivoting by warps 0..7: warp w
// holds columns 4w..4w+3, lane = row, in registers.  Column k's owner forms the
// multipliers and updates its own columns; the warps to its right take them
// from shared memory, one mbarrier per column, so the owner never waits.  The
// chain of a column is the pivot's reciprocal, the quotient of row k+1 and the
// next pivot's product and difference: every lane forms the next pivot itself
// from values broadcast a step early, and its reciprocal's seed starts from the
// uncorrected quotient, so no shuffle and no seed latency stays in the chain
// (275 cycles per column measured for the whole block, 406 with an IEEE
// division, a shuffle and a CTA barrier per column).  Pads (rows and columns
// >= kw) are those of an identity.  Returns the thread's flags: columns where a
// row has |a_ik| > |a_kk|, which for correctly rounded quotients is |l| > 1.
// `bad`: some quotient is outside the window; the caller redoes the block with
// eliminate_slow.  Writes S.s, S.q, S.rs; S.stuck when a wait gives up.
__device__ __forceinline__ unsigned eliminate(double (&c)[4], bool &bad) {
    Smem &S = smem();
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t par = S.parity;
    unsigned msk = 0;
    bool good = true;
    uint32_t arrived = 1;
#pragma unroll 1
    for (int o = 0; o < w; ++o) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int k = 4 * o + i;
            double u[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) u[j] = __shfl_sync(0xffffffffu, c[j], k);
            arrived &= mbar_wait(&S.done[k], par);
            const double l = S.lcol[k][lane];  // 0 for rows <= k
#pragma unroll
            for (int j = 0; j < 4; ++j) c[j] = c[j] - l * u[j];
        }
    }
    const int k0 = 4 * w;
    double d = __shfl_sync(0xffffffffu, c[0], k0), y0 = rcp_seed(d);
    double pre[4], piv[4], ys[4], e2s[4];  // checked and stored after the chain
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int k = k0 + i, in = i < 3 ? i + 1 : i;
        const double v = c[i];
        const double a10 = __shfl_sync(0xffffffffu, v, (k + 1) & 31);
        const double a11 = __shfl_sync(0xffffffffu, c[in], (k + 1) & 31);
        double u[4];
#pragma unroll
        for (int j = i + 1; j < 4; ++j) u[j] = __shfl_sync(0xffffffffu, c[j], k);
        const double y = recip_rn(d, y0, e2s[i]);
        double dn = 0.0, yn = 0.0;
        if (i < 3) {
            yn = rcp_seed(__fma_rn(-__dmul_rn(a10, y), u[in], a11));
            dn = a11 - qdiv::fast(a10, d, y) * u[in];
        }
        const double l = qdiv::fast(v, d, y);
        const bool low = lane > k;
        const double lz = low ? l : 0.0;
        S.lcol[k][lane] = lz;
        __syncwarp();
        if (lane == 0) mbar_arrive(&S.done[k]);
        pre[i] = v;
        piv[i] = d;
        ys[i] = y;
        c[i] = low ? l : v;
#pragma unroll
        for (int j = i + 1; j < 4; ++j) c[j] = c[j] - lz * u[j];
        d = dn;
        y0 = yn;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const bool low = lane > k0 + i;
        S.s[lane][k0 + i] = c[i];
        S.q[lane][k0 + i] = pre[i];
        if (lane == 0) S.rs[k0 + i] = ys[i];
        good = good && recip_ok(piv[i], e2s[i]) && (!low || value_ok(pre[i]));
        if (low && fabs(c[i]) > 1.0) msk |= 1u << (k0 + i);
    }
    if (!arrived) S.stuck = 1;
    bad = !good;
    return msk;
}

// The same elimination with IEEE divisions, for blocks with values outside the
// quotient window or zero pivots, and for passes that skip singular columns.  Its
// multipliers may be infinite or NaN, so it skips updates by a zero as the oracle does
// (and so do row_below_slow and col_slow).
// All threads call it (warps 0..7 pass their columns, the others idle).
static __device__ __noinline__ unsigned eliminate_slow(const double (&c0)[4], int kw,
                                                unsigned skip) {
    Smem &S = smem();
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned msk = 0;
    double c[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) c[i] = c0[i];
    for (int k = 0; k < NB; ++k) {
        if (w == k >> 2) {
            const int i = k & 3;
            const double v = i == 0 ? c[0] : i == 1 ? c[1] : i == 2 ? c[2] : c[3];
            const double d = __shfl_sync(0xffffffffu, v, k);
            S.q[lane][k] = v;
            double l = 0.0;
            if (!((skip >> k) & 1u)) {
                if (d == 0.0 && k < kw) msk |= 1u << k;
                if (lane > k) {
                    if (fabs(v) > fabs(d) && lane < kw) msk |= 1u << k;
                    l = v / d;
                }
            }
            S.lcol[k][lane] = l;
            S.s[lane][k] = (lane > k && !((skip >> k) & 1u)) ? l : v;
        }
        __syncthreads();
        if (w < 8 && !((skip >> k) & 1u)) {
            const double l = S.lcol[k][lane];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const double u = __shfl_sync(0xffffffffu, c[j], k);
                if (lane > k && 4 * w + j > k && u != 0.0) c[j] = c[j] - l * u;
            }
        }
    }
    __syncthreads();
    if (threadIdx.x < NB) S.rs[threadIdx.x] = qdiv::recip(S.s[threadIdx.x][threadIdx.x]);
    return msk;
}

// Eliminates c by the fast path, or the slow one where that has to be; all
// threads call it.  Afterwards S.s, S.q and S.rs are complete.  A wait that gave up
// is recorded in flags, and the CTA's later eliminations take the slow path, which has
// no such waits.
static __device__ __noinline__ unsigned eliminate_any(const double (&c0)[4], int kw,
                                                  unsigned skip, int *flags) {
    Smem &S = smem();
    unsigned msk = 0;
    bool bad = S.dead != 0;
    if (skip == 0 && !bad) {
        double c[4] = {c0[0], c0[1], c0[2], c0[3]};
        msk = eliminate(c, bad);
        bad = __syncthreads_or(bad);
        if (threadIdx.x == 0) {
            S.parity ^= 1u;
            if (S.stuck) {
                atomicOr(&flags[kFlagBarrierTimeout], 1);
                S.dead = 1;
            }
        }
    }
    if (skip != 0 || bad) msk = eliminate_slow(c0, kw, skip);
    __syncthreads();
    return msk;
}

// The diagonal block of a pass from P0 (block 0, and passes after a swap), in
// every CTA; CTA 0 stores the pre-division values.  All threads call it.
static __device__ __noinline__ unsigned diag_from_p0(const Args &a, double *Q, int k0, int kw,
                                              int ns, unsigned skip, bool write_q) {
    Smem &S = smem();
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    double c[4] = {0, 0, 0, 0};
    if (w < 8) {
        const bool ok = lane < kw;
        const int sr = ok ? src_row(k0 + lane, S.sa, S.sb, ns) : 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int k = 4 * w + i;
            c[i] = (ok && k < kw) ? a.P0[(size_t)sr * NB + k] : (lane == k ? 1.0 : 0.0);
        }
    }
    const unsigned msk = eliminate_any(c, kw, skip, a.flags);
    if (write_q)
        for (int t = tid; t < NB * NB; t += kThreads) {
            const int r = t / NB, k = t % NB;
            if (r >= k && r < kw) Q[(size_t)(k0 + r) * NB + k] = S.q[r][k];
        }
    __syncthreads();
    return msk;
}

// Rows below the diagonal block, kLanes lanes per row: lane q of a group holds
// the columns q, q + kLanes, ... in registers.  Every lane forms the multiplier
// (the IEEE quotient, from the pivot's reciprocal) and, from a value broadcast a
// step early, the next column's value, so the chain of a column is five FMA
// steps, a product and a difference (about 90 cycles; 192 with the broadcast
// and a window branch in the chain).  4 lanes per row: with 8 a lone row is
// faster (71 cycles a column) but every lane repeats the quotient, and the
// look-ahead's 32 rows and 32 columns on one SM took 6,400 cycles.
// Pre-division values to Q, multipliers to A.
__device__ __forceinline__ void row_store(const Args &a, double *Q, int r_pos, int k0,
                                          const double (&pre)[kHold], const double (&c)[kHold]) {
    const int q = threadIdx.x % kLanes;
#pragma unroll
    for (int t = 0; t < kHold; ++t) {
        Q[(size_t)r_pos * NB + q + kLanes * t] = pre[t];
        a.A[(size_t)r_pos + (size_t)(k0 + q + kLanes * t) * a.n] = c[t];
    }
}

// A row with IEEE divisions, for values outside the quotient window and passes
// that skip singular columns.  Returns the row's flags.
static __device__ __noinline__ unsigned row_below_slow(const Args &a, double *Q, int r_pos, int sr, int k0,
                                                unsigned skip, bool active) {
    Smem &S = smem();
    const int lane = threadIdx.x & 31, q = lane % kLanes, gb = lane - q;
    unsigned msk = 0;
    double c[kHold], pre[kHold];
#pragma unroll
    for (int t = 0; t < kHold; ++t) c[t] = active ? a.P0[(size_t)sr * NB + q + kLanes * t] : 0.0;
#pragma unroll
    for (int s = 0; s < kHold; ++s) {
#pragma unroll 1
        for (int own = 0; own < kLanes; ++own) {
            const int k = kLanes * s + own;
            const double v = __shfl_sync(0xffffffffu, c[s], gb + own);
            if (q == own) pre[s] = v;
            if ((skip >> k) & 1u) continue;
            const double d = S.s[k][k];
            if (fabs(v) > fabs(d)) msk |= 1u << k;
            const double l = v / d, us = S.s[k][q + kLanes * s];
            c[s] = q == own ? l : (q > own && us != 0.0 ? c[s] - l * us : c[s]);
#pragma unroll
            for (int t = s + 1; t < kHold; ++t) {
                const double u = S.s[k][q + kLanes * t];
                if (u != 0.0) c[t] = c[t] - l * u;
            }
        }
    }
    if (active) row_store(a, Q, r_pos, k0, pre, c);
    return active ? msk : 0u;
}

// The chain of a row: c in, multipliers out, pre-division values to pre; false
// when some value is outside the quotient window.
__device__ __forceinline__ bool row_core(double (&c)[kHold], double (&pre)[kHold]) {
    Smem &S = smem();
    const int lane = threadIdx.x & 31, q = lane % kLanes, gb = lane - q;
    bool good = true;
#pragma unroll
    for (int t = 0; t < kHold; ++t) good = good && S.rs[q + kLanes * t] != 0.0;
    double v = __shfl_sync(0xffffffffu, c[0], gb);
#pragma unroll
    for (int s = 0; s < kHold; ++s) {
#pragma unroll
        for (int own = 0; own < kLanes; ++own) {
            const int k = kLanes * s + own, s1 = s < kHold - 1 ? s + 1 : s;
            const double vn = own < kLanes - 1 ? __shfl_sync(0xffffffffu, c[s], gb + own + 1)
                                               : __shfl_sync(0xffffffffu, c[s1], gb);
            const double l = qdiv::fast(v, S.s[k][k], S.rs[k]);
            if (q == own) pre[s] = v;
            v = vn - l * S.s[k][k < 31 ? k + 1 : 31];
            const double cs = c[s] - l * S.s[k][q + kLanes * s];
            c[s] = q == own ? l : (q > own ? cs : c[s]);
#pragma unroll
            for (int t = s + 1; t < kHold; ++t) c[t] = c[t] - l * S.s[k][q + kLanes * t];
        }
    }
#pragma unroll
    for (int t = 0; t < kHold; ++t) good = good && value_ok(pre[t]);
    return __all_sync(0xffffffffu, good);
}

// U12 of one column, kLanes lanes per column: lane q holds rows q, q + kLanes,
// ...; the next row's value is formed from a broadcast a step early, as above.
// False when some value is not finite: col_slow then solves the column.
__device__ __forceinline__ bool col_core(double (&c)[kHold]) {
    Smem &S = smem();
    const int lane = threadIdx.x & 31, q = lane % kLanes, gb = lane - q;
    double u = __shfl_sync(0xffffffffu, c[0], gb);
#pragma unroll
    for (int s = 0; s < kHold; ++s) {
#pragma unroll
        for (int own = 0; own < kLanes; ++own) {
            const int k = kLanes * s + own, s1 = s < kHold - 1 ? s + 1 : s;
            const double un = own < kLanes - 1 ? __shfl_sync(0xffffffffu, c[s], gb + own + 1)
                                               : __shfl_sync(0xffffffffu, c[s1], gb);
            const double cs = c[s] - S.s[q + kLanes * s][k] * u;
            if (q > own) c[s] = cs;
#pragma unroll
            for (int t = s + 1; t < kHold; ++t) c[t] = c[t] - S.s[q + kLanes * t][k] * u;
            u = un - S.s[k < 31 ? k + 1 : 31][k] * u;
        }
    }
    bool good = true;
#pragma unroll
    for (int t = 0; t < kHold; ++t) good = good && isfinite(c[t]);
    return __all_sync(0xffffffffu, good);
}
static __device__ __noinline__ void col_slow(const Args &a, double *U, int pos, int k0,
                                             bool active) {
    Smem &S = smem();
    const int lane = threadIdx.x & 31, q = lane % kLanes, gb = lane - q;
    double c[kHold];
#pragma unroll
    for (int t = 0; t < kHold; ++t)
        c[t] = active ? a.A[(size_t)(k0 + q + kLanes * t) + (size_t)pos * a.n] : 0.0;
#pragma unroll
    for (int s = 0; s < kHold; ++s) {
#pragma unroll 1
        for (int own = 0; own < kLanes; ++own) {
            const int k = kLanes * s + own;
            const double u = __shfl_sync(0xffffffffu, c[s], gb + own);
            if (u != 0.0) {
                if (q > own) c[s] = c[s] - S.s[q + kLanes * s][k] * u;
#pragma unroll
                for (int t = s + 1; t < kHold; ++t) c[t] = c[t] - S.s[q + kLanes * t][k] * u;
            }
        }
    }
    if (active) {
#pragma unroll
        for (int t = 0; t < kHold; ++t) U[(size_t)(q + kLanes * t) * a.n + pos] = c[t];
    }
}

// Tile of update index t of tr x tc tiles: the first column of tiles, the rest
// of the first row, then the interior.
__device__ __forceinline__ void tile_at(int t, int tr, int tc, int &ti, int &tj) {
    if (t < tr) {
        ti = t;
        tj = 0;
    } else if (t < tr + tc - 1) {
        ti = 0;
        tj = t - tr + 1;
    } else {
        const int m = t - (tr + tc - 1);
        ti = 1 + m % (tr - 1);
        tj = 1 + m / (tr - 1);
    }
}

// Tiles of the update behind a block for a group of G CTAs: 64 x 64 by each of two
// teams per CTA; 64 x 32 by the whole CTA when every CTA gets at most one, where
// the tile's time is on the chain of the blocks.
struct Tiling {
    int teams;       // teams of a CTA
    int tr, tc;      // tiles along rows and columns
    int la_tiles;    // tiles a CTA finishes in the time of a look-ahead
    __device__ Tiling(int rest, int G) {
        tr = (rest + kBoxR - 1) / kBoxR;
        teams = 2 * tr * tr <= max(G - 1, 2) ? 1 : 2;
        tc = teams == 2 ? tr : (rest + kBoxC - 1) / kBoxC;
        la_tiles = 7;
    }
    __device__ int strips() const { return tr + tc - 1; }
};

// The next diagonal block from its entries c (warps 0..7: lane = row, columns
// 4w..4w+3), with L21 of its rows and U12 of its columns in shared memory
// ([k][row], [k][column]): the 32 updates in the order of the tile that owns
// it, then its elimination.  Leaves the updated entries in c.
__device__ __forceinline__ void next_diag(double (&c)[4], const double *Lp,
                                          const double *Up, int nkw, int *flags) {
    Smem &S = smem();
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (w < 8) {
#pragma unroll 8
        for (int k = 0; k < NB; ++k) {
            const double l = Lp[k * NB + lane];
            const double2 u0 = *reinterpret_cast<const double2 *>(Up + k * NB + 4 * w);
            const double2 u1 = *reinterpret_cast<const double2 *>(Up + k * NB + 4 * w + 2);
            c[0] = c[0] - l * u0.x;
            c[1] = c[1] - l * u0.y;
            c[2] = c[2] - l * u1.x;
            c[3] = c[3] - l * u1.y;
        }
        if (lane >= nkw) {  // pads: an identity
#pragma unroll
            for (int i = 0; i < 4; ++i) c[i] = lane == 4 * w + i ? 1.0 : 0.0;
        } else if (4 * w + 3 >= nkw) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (4 * w + i >= nkw) c[i] = 0.0;
        }
    }
    if (threadIdx.x == 0) S.la_mask = 0;
    const unsigned m = eliminate_any(c, nkw, 0u, flags);
    if (m) atomicOr(&S.la_mask, m);
}

// Publishes S.s, S.rs as the diagonal block of block kb + 1, and its entries
// before the elimination (c) as P0's rows.
__device__ __forceinline__ void publish(const Args &a, const double (&c)[4], int nk0,
                                        int nkw, int kb, int pass) {
    Smem &S = smem();
    const int n = a.n, tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    const int nblk = (n + NB - 1) / NB;
    double *Qn = a.Q + (size_t)(pass & 1) * n * NB;
    if (tid < NB) a.dg[NB * (NB + 1) + tid] = S.rs[tid];
    const double *sf = &S.s[0][0];
    for (int t = tid; t < NB * (NB + 1); t += kThreads) a.dg[t] = sf[t];
    if (w < 8 && lane < nkw) {
        double2 *dst = reinterpret_cast<double2 *>(a.P0 + (size_t)(nk0 + lane) * NB + 4 * w);
        dst[0] = make_double2(c[0], c[1]);
        dst[1] = make_double2(c[2], c[3]);
    }
    for (int t = tid; t < NB * NB; t += kThreads) {
        const int r = t / NB, k = t % NB;
        if (r >= k && r < nkw) Qn[(size_t)(nk0 + r) * NB + k] = S.q[r][k];
    }
    __syncthreads();
    if (tid == kThreads - 1) {
        if (S.la_mask) atomicOr(&a.mask[pass], S.la_mask);
        st_rel(a.sched + nblk, (unsigned)(kb + 1));
    }
}

// The look-ahead after a pass that needed a swap (or by a single CTA): L21 and
// U12 as the pass left them.
static __device__ __noinline__ void look_ahead(const Args &a, int k0, int kb, int pass,
                                        const double *U) {
    Smem &S = smem();
    const int n = a.n, tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    const int nk0 = k0 + NB, nkw = min(NB, n - nk0);
    double *Lp = &S.lp[0][0][0][0], *Up = &S.up[0][0][0][0][0];
    double c[4] = {0, 0, 0, 0};
    for (int t = tid; t < NB * NB; t += kThreads) {
        const int r = t % NB, k = t / NB;
        Lp[t] = r < nkw ? a.A[(size_t)(nk0 + r) + (size_t)(k0 + k) * n] : 0.0;
        Up[t] = r < nkw ? U[(size_t)k * n + nk0 + r] : 0.0;
    }
    if (w < 8) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int j = 4 * w + i;
            if (lane < nkw && j < nkw) c[i] = a.A[(size_t)(nk0 + lane) + (size_t)(nk0 + j) * n];
        }
    }
    __syncthreads();
    next_diag(c, Lp, Up, nkw, a.flags);
    publish(a, c, nk0, nkw, kb, pass);
}

// Trailing update: tiles first, first + stride, ... below `end`.  A team is all
// warps (64 x 32 tiles), or each half of them (64 x 64 tiles, team 1 takes every
// second one): then one team's waits, loads and stores run under the other's
// products.  The two take turns at the products (named barriers 3 and 4); left to
// themselves they fall in step and stand still together.  N=4096: 128 x 64 tiles by
// all warps 5.70 ms, two teams in step 5.61, in turns 5.15, with the operands of a
// step fetched during the step before 5.02 (the products alone: 2.6).  Four teams
// with 8 x 8 entries per thread and A read directly, in turns: 5.9 and more.
// A warp owns 8 RM x 4 RN entries, lane (lr, lc) of 8 x 4 the row pairs 2 lr + 16 p
// and column pairs 2 lc + 8 q of them, so every operand is read as 16-byte words
// without bank conflicts (8 x 4 entries per thread in the teams: in a bare loop 0.96
// of the product-difference rate by 8 warps, 0.88 by one team's 4; 4 x 4 0.91 and
// 0.69).  The next tile's L21 and U12 pieces and entries of A come by tensor copies
// of 64 x 32 boxes while a tile computes; as 16-byte cp.async by every thread the
// issue alone held up 128 x 64 entries 3,800 cycles of 15,300, as untiled bulk copies
// of whole columns 8,600 on the issuing warp.  `seq` counts the team's tiles (buffer
// and mbarrier phase).  The tiles of the first row also store U12 to A; tiles of the
// first column hold the next block's columns, whose new values go to P0, not A.
template <int kTeams>
static __device__ __noinline__ void update_tiles(const Args &a, int k0, int kb, const double *U,
                                              int ntr, int ntc, int first, int stride, int end,
                                              unsigned seq) {
    Smem &S = smem();
    constexpr int RM = 4 * kTeams, RN = 2 * kTeams, kTr = kBoxR, kTc = 32 * kTeams,
                  kTeam = kThreads / kTeams;
    const int team = kTeams > 1 ? threadIdx.x / kTeam : 0;
    const int n = a.n, tid = threadIdx.x % kTeam, warp = tid >> 5, lane = tid & 31;
    auto sync = [&] {
        if (kTeams > 1)
            named_bar(1 + team, kTeam);
        else
            __syncthreads();
    };
    uint64_t *full = S.full[team];
    const int base = k0 + NB;
    constexpr int kWr = kTr / (8 * RM);  // warps along a tile's rows
    const int lr = warp % kWr * 8 * RM + 2 * (lane & 7), lc = warp / kWr * 4 * RN + 2 * (lane >> 3);
    const int cbox = lc / kBoxC;
    // warp 0 fetches the L21 piece, warp 1 U12's, the next ones the entries' (a copy's
    // issue holds up its warp for some 300 cycles)
    auto stage = [&](int tile, unsigned buf) {
        constexpr int kCb = kTc / kBoxC;
        if (lane != 0) return;
        int ti, tj;
        tile_at(tile, ntr, ntc, ti, tj);
        const int i0 = base + ti * kTr, j0 = base + tj * kTc;
        uint64_t *bar = &full[buf];
        if (warp == 0) {
            bulk::arrive_expect_tx(bar, (uint32_t)sizeof(double) *
                                            (NB * kBoxR + kCb * NB * kBoxC + kCb * kBoxR * kBoxC));
            box_load(S.lp[team][buf], a.map_a, i0, k0, bar);
        } else if (warp == 1) {
#pragma unroll
            for (int c = 0; c < kCb; ++c)
                box_load(S.up[team][buf][c], a.map_u, j0 + c * kBoxC, U == a.U ? 0 : NB, bar);
        } else if (warp < 2 + kCb) {
            const int c = warp - 2;
            box_load(S.at[team][c], a.map_a, i0, j0 + c * kBoxC, bar);
        }
    };
    const int step = stride;  // from a tile to that of the other team's next turn
    bool wait_turn = kTeams > 1 && team;
    first += team * stride;
    stride *= kTeams;
    if (first < end) {
        fence_bulk();
        stage(first, seq & 1);
    }
    for (int tile = first; tile < end; tile += stride, ++seq) {
        int ti, tj;
        tile_at(tile, ntr, ntc, ti, tj);
        const int i0 = base + ti * kTr, j0 = base + tj * kTc;
        const unsigned buf = seq & 1;
        const double *Ls = &S.lp[team][buf][0][lr];
        const double *Us = &S.up[team][buf][cbox][0][lc % kBoxC];
        const double *At = &S.at[team][cbox][lc % kBoxC][lr];
        if (!bulk::wait(&full[buf], (seq >> 1) & 1)) atomicOr(&a.flags[kFlagBarrierTimeout], 1);
        double acc[RN][RM];  // [column][row]
#pragma unroll
        for (int q = 0; q < RN; ++q)
#pragma unroll
            for (int p = 0; p < RM / 2; ++p) {
                const double2 v = *reinterpret_cast<const double2 *>(
                    At + (8 * (q >> 1) + (q & 1)) * kBoxR + 16 * p);
                acc[q][2 * p] = v.x;
                acc[q][2 * p + 1] = v.y;
            }
        sync();  // the entries are in registers; the other buffer is free
        if (tile + stride < end) stage(tile + stride, buf ^ 1);
        if (kTeams > 1 && wait_turn) named_bar(3 + team, kThreads);
        wait_turn = true;
        double lv[2][RM], uv[2][RN];
        auto fetch = [&](int k, double (&l)[RM], double (&u)[RN]) {
#pragma unroll
            for (int p = 0; p < RM / 2; ++p) {
                const double2 v = *reinterpret_cast<const double2 *>(Ls + k * kBoxR + 16 * p);
                l[2 * p] = v.x;
                l[2 * p + 1] = v.y;
            }
#pragma unroll
            for (int q = 0; q < RN / 2; ++q) {
                const double2 v = *reinterpret_cast<const double2 *>(Us + k * kBoxC + 8 * q);
                u[2 * q] = v.x;
                u[2 * q + 1] = v.y;
            }
        };
        auto products = [&](const double (&l)[RM], const double (&u)[RN]) {
#pragma unroll
            for (int q = 0; q < RN; ++q)
#pragma unroll
                for (int p = 0; p < RM; ++p) acc[q][p] = acc[q][p] - l[p] * u[q];
        };
        fetch(0, lv[0], uv[0]);
#pragma unroll 4
        for (int k = 0; k < NB; k += 2) {
            fetch(k + 1, lv[1], uv[1]);
            products(lv[0], uv[0]);
            fetch((k + 2) % NB, lv[0], uv[0]);
            products(lv[1], uv[1]);
        }
        if (kTeams > 1 && tile + step < end)  // the other team's turn
            asm volatile("bar.arrive %0, %1;" ::"r"(4 - team), "r"(kThreads) : "memory");
#pragma unroll
        for (int q = 0; q < RN; q += 2) {
            const int lj = lc + 4 * q, gj = j0 + lj;
            if (gj >= n) continue;
            const bool next_cols = tj == 0 && lj < NB;  // the next block's columns
#pragma unroll
            for (int p = 0; p < RM; p += 2) {
                const int li = lr + 8 * p, gi = i0 + li;
                if (gi >= n) continue;
                if (!next_cols) {
                    double2 *dst = reinterpret_cast<double2 *>(a.A + (size_t)gi + (size_t)gj * n);
                    dst[0] = make_double2(acc[q][p], acc[q][p + 1]);
                    dst[n / 2] = make_double2(acc[q + 1][p], acc[q + 1][p + 1]);
                } else if (ti > 0 || li >= NB) {  // the next diagonal block is the look-ahead's
                    double2 *dst = reinterpret_cast<double2 *>(a.P0 + (size_t)gi * NB + lj);
                    dst[0] = make_double2(acc[q][p], acc[q + 1][p]);
                    dst[NB / 2] = make_double2(acc[q][p + 1], acc[q + 1][p + 1]);
                }
            }
        }
        // products done with this buffer before it is refilled; a strip tile's
        // stores are in before it is counted
        sync();
        if (tile < ntr + ntc - 1 && tid == kTeam - 1) red_rel(a.sched + kb, 1u);
        if (ti == 0) {
            // U12 to A, from this buffer (not refilled before the next barrier)
#pragma unroll
            for (int r = 0; r < NB * kTc / 2 / kTeam; ++r) {
                const int t = tid + r * kTeam, k = t % NB, jj = 2 * (t / NB);
                if (j0 + jj < n) {
                    const double2 v = *reinterpret_cast<const double2 *>(
                        &S.up[team][buf][jj / kBoxC][k][jj % kBoxC]);
                    double *dst = a.A + (size_t)(k0 + k) + (size_t)(j0 + jj) * n;
                    dst[0] = v.x;
                    dst[n] = v.y;
                }
            }
        }
    }
}

template <class Group>
__device__ __forceinline__ void factor(const Args &a, Group g) {
    Smem &S = smem();
    const int n = a.n, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int G = g.size(), cta = g.rank(), la = G - 1;
    const int nblk = (n + NB - 1) / NB;
    if (tid == 0) {
        S.dead = 0;
        S.stuck = 0;
        S.parity = 0;
    }
    if (tid < NB)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&S.done[tid]))
                     : "memory");
    if (tid < 4) bulk::init(&S.full[tid >> 1][tid & 1], 1);
    bulk::fence_init();
    for (int i = cta * kThreads + tid; i < n; i += G * kThreads) a.perm[i] = i;
    // P0 = the first block's columns
    for (int t = cta * kThreads + tid; t < n * NB; t += G * kThreads) {
        const int r = t % n, k = t / n;
        a.P0[(size_t)r * NB + k] = k < n ? a.A[(size_t)r + (size_t)k * n] : 0.0;
    }
    g.arrive(false);
    g.wait(nullptr, a.flags);

    const int Gt = G > 1 ? G - 1 : 1;  // CTAs that take rows, columns and most tiles
    const bool ahead = cta == la && G > 1;  // the look-ahead CTA
    bool stored = true;  // tiles of the last update stored by this CTA, for others' bulk copies
    int swaps = 0;  // row swaps so far
    unsigned seq0 = 0, seq1 = 0;  // update tiles of this CTA's teams so far
    int pass = 0;   // pass counter: mask word, and Q buffer by parity
    for (int kb = 0; kb < nblk; ++kb) {
        const int k0 = kb * NB, kw = min(NB, n - k0), rest = n - k0 - kw;
        double *U = a.U + (size_t)(kb & 1) * NB * n;
        if (tid == 0) {
            S.ns = 0;
            S.skip = 0;
            if (ahead && kb > 0) {
                // the look-ahead waits for the strips of the update here, while the
                // last warp's publication completes (N=1024 0.490 -> 0.476 ms)
                S.cta_mask = S.la_mask;
                wait_ge(a.sched + kb - 1, (unsigned)Tiling(n - k0, G).strips(), a.flags, &S.dead);
            }
        }
        __syncthreads();
        int scan_from = 0;
        bool early = false;  // the look-ahead CTA has the next diagonal block already
        double c_next[4];
        const int groups = (rest + kRows - 1) / kRows;  // rows below, columns right: per warp
        for (bool first = true;; first = false) {
            double *Q = a.Q + (size_t)(pass & 1) * n * NB;
            const int ns = S.ns;
            const unsigned skip = S.skip;
            unsigned my_mask = 0;
            if (kb > 0 && first) {
                // the published diagonal block, then the strips of the update
                if (cta != la) {
                    if (tid == 0) {
                        S.cta_mask = 0;
                        wait_ge(a.sched + nblk, (unsigned)kb, a.flags, &S.dead);
                    }
                    __syncthreads();
                    constexpr int kPer = (kDgWords + kThreads - 1) / kThreads;
                    double *sf = &S.s[0][0], v[kPer];
#pragma unroll
                    for (int e = 0; e < kPer; ++e) {
                        const int t = tid + e * kThreads;
                        v[e] = t < kDgWords ? __ldcg(a.dg + t) : 0.0;
                    }
#pragma unroll
                    for (int e = 0; e < kPer; ++e) {
                        const int t = tid + e * kThreads;
                        if (t < NB * (NB + 1))
                            sf[t] = v[e];
                        else if (t < kDgWords)
                            S.rs[t - NB * (NB + 1)] = v[e];
                    }
                }
                if (!ahead) {
                    if (tid == 0) {
                        if (cta == la) S.cta_mask = S.la_mask;
                        wait_ge(a.sched + kb - 1, (unsigned)Tiling(n - k0, G).strips(), a.flags,
                                &S.dead);
                    }
                    __syncthreads();
                }
            } else {
                if (tid == 0) S.cta_mask = 0;
                my_mask = diag_from_p0(a, Q, k0, kw, ns, skip, cta == 0);
            }
            // Rows below and columns right, kRows per warp, warps spread over the
            // CTAs.  The look-ahead CTA takes none: in a block's first pass it
            // forms L21 and U12 of the next block's 32 rows and columns itself
            // (the same operations as the CTAs that own them, into shared
            // memory) and from them the next diagonal block,
            // while the others are still in the pass and its barrier.  It loads
            // everything before it arrives at the barrier (afterwards the update
            // overwrites A); a rejected pass drops the result.
            const bool spec = cta == la && G > 1 && first && rest > 0;
            if (spec) {
                if (my_mask) atomicOr(&S.cta_mask, my_mask);
                __syncthreads();
            }
            bool good = true;
            double *Lp = &S.lp[0][0][0][0], *Up = &S.up[0][0][0][0][0];  // [k][row], [k][column]
            for (int t = spec ? warp : cta < Gt ? warp * Gt + cta : 2 * groups;
                 t < (spec ? kWarps : 2 * groups); t += spec ? kWarps : kWarps * Gt) {
                // (the look-ahead has 2 NB / kRows tasks; its other warps pass by)
                const int half = spec ? NB / kRows : groups, lim = spec ? min(NB, rest) : rest;
                const bool is_row = t < half;
                const int m = kRows * (is_row ? t : t - half) + lane / kLanes, q = lane % kLanes;
                const bool active = m < lim;
                const int pos = k0 + NB + (active ? m : 0);
                const int sr = is_row && active ? src_row(pos, S.sa, S.sb, ns) : pos;
                const double *src = is_row ? a.P0 + (size_t)sr * NB + q
                                           : a.A + (size_t)(k0 + q) + (size_t)pos * n;
                double c[kHold], pre[kHold];
#pragma unroll
                for (int e = 0; e < kHold; ++e) {
                    c[e] = active ? src[kLanes * e] : 0.0;
                    pre[e] = 0.0;
                }
                if (spec) {
                    double z = 0.0;
#pragma unroll
                    for (int e = 0; e < kHold; ++e) z += c[e];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        c_next[e] = 0.0;
                        if (warp < 8 && lane < lim && 4 * warp + e < lim)
                            c_next[e] = a.A[(size_t)(k0 + NB + lane) +
                                            (size_t)(k0 + NB + 4 * warp + e) * n];
                        z += c_next[e];
                    }
                    // the predicate depends on every load: all have returned
                    // before the arrival
                    if (stored) fence_bulk();
                    __syncthreads_or(z == 0.0);
                    if (tid == kThreads - 1 && S.cta_mask) atomicOr(&a.mask[pass], S.cta_mask);
                    g.arrive_quiet(S.cta_mask != 0);
                    if (t >= 2 * half) break;
                }
                if (is_row) {
                    good = skip == 0 && row_core(c, pre);
                    if (spec) {
#pragma unroll
                        for (int e = 0; e < kHold; ++e) Lp[(q + kLanes * e) * NB + m] = c[e];
                    } else if (!good) {
                        my_mask |= row_below_slow(a, Q, pos, sr, k0, skip, active);
                    } else if (active) {
#pragma unroll
                        for (int e = 0; e < kHold; ++e)
                            if (fabs(c[e]) > 1.0) my_mask |= 1u << (q + kLanes * e);
                        row_store(a, Q, pos, k0, pre, c);
                    }
                } else {
                    good = col_core(c);
                    if (!good && !spec) {
                        col_slow(a, U, pos, k0, active);
                        continue;
                    }
                    double *dst = spec ? Up + q * NB + m : U + (size_t)q * n + pos;
                    const size_t step = spec ? kLanes * NB : (size_t)kLanes * n;
                    if (active || spec) {
#pragma unroll
                        for (int e = 0; e < kHold; ++e) dst[e * step] = c[e];
                    }
                }
            }
            if (spec) {
                early = __syncthreads_and(good);
                if (early) next_diag(c_next, Lp, Up, min(NB, rest), a.flags);
            } else {
                if (my_mask) atomicOr(&S.cta_mask, my_mask);
                fence_bulk();
                __syncthreads();
                if (tid == kThreads - 1 && S.cta_mask) atomicOr(&a.mask[pass], S.cta_mask);
                g.arrive_quiet(S.cta_mask != 0);
            }
            const unsigned mw = g.wait(&a.mask[pass], a.flags);
            // ------------------------------------------------------- decide
            const unsigned m = scan_from >= 32 ? 0u : (mw >> scan_from) << scan_from;
            ++pass;
            if (m == 0 || S.dead) break;  // exact: this pass's values stand
            const int ks = __ffs(m) - 1;  // first flagged column
            const int kabs = k0 + ks;
            // exact first-max pivot over positions >= kabs of column ks
            double best = -1.0;
            int bi = n;
            for (int r = kabs + tid; r < n; r += kThreads) {
                const double v = fabs(Q[(size_t)r * NB + ks]);
                if (v > best) {
                    best = v;
                    bi = r;
                }
            }
            for (int o = 16; o > 0; o >>= 1) {
                const double ov = __shfl_down_sync(0xffffffffu, best, o);
                const int oi = __shfl_down_sync(0xffffffffu, bi, o);
                if (ov > best || (ov == best && oi < bi)) {
                    best = ov;
                    bi = oi;
                }
            }
            if (lane == 0) {
                S.red_v[warp] = best;
                S.red_i[warp] = bi;
            }
            __syncthreads();
            if (tid == 0) {
                for (int w = 1; w < kWarps; ++w)
                    if (S.red_v[w] > best || (S.red_v[w] == best && S.red_i[w] < bi)) {
                        best = S.red_v[w];
                        bi = S.red_i[w];
                    }
                const double dkk = Q[(size_t)kabs * NB + ks];
                const int p = best > fabs(dkk) ? bi : kabs;
                if (Q[(size_t)p * NB + ks] == 0.0) {
                    S.skip |= 1u << ks;
                    if (cta == 0) atomicOr(&a.flags[kFlagSingular], 1);
                } else {
                    S.sa[S.ns] = kabs;
                    S.sb[S.ns] = p;
                    S.ns = S.ns + 1;
                }
            }
            __syncthreads();
            if (S.ns > ns) {
                // the swap on the columns outside the block: right of it by the
                // warp that solves the column's U12 (it reads A again), left of
                // it by all threads
                const int p = S.sb[ns];
                if (p != kabs) {
                    auto swap_rows = [&](int j) {
                        double *cj = a.A + (size_t)j * n;
                        const double x = cj[kabs];
                        cj[kabs] = cj[p];
                        cj[p] = x;
                    };
                    if (cta < Gt)
                        for (int t = warp * Gt + cta; t < 2 * groups; t += kWarps * Gt) {
                            const int m2 = kRows * (t - groups) + lane;
                            if (t >= groups && lane < kRows && m2 < rest) swap_rows(k0 + kw + m2);
                        }
                    for (int j = cta * kThreads + tid; j < k0; j += G * kThreads) swap_rows(j);
                    __syncwarp();
                }
            }
            scan_from = ks + 1;
            early = false;  // formed without this swap
        }
        // ---------------------------------------------------------- finish
        const int ns = S.ns;
        swaps += ns;
        if (cta == 0) {
            for (int t = tid; t < NB * NB; t += kThreads) {
                const int r = t % NB, k = t / NB;
                if (r < kw && k < kw) a.A[(size_t)(k0 + r) + (size_t)(k0 + k) * n] = S.s[r][k];
            }
            for (int k = tid; k < kw; k += kThreads) {
                int p = k0 + k;
                for (int t = 0; t < ns; ++t)
                    if (S.sa[t] == k0 + k) p = S.sb[t];
                a.piv[k0 + k] = p;
            }
            if (tid == 0) {
                for (int t = 0; t < ns; ++t) {
                    const int x = a.perm[S.sa[t]];
                    a.perm[S.sa[t]] = a.perm[S.sb[t]];
                    a.perm[S.sb[t]] = x;
                }
            }
        }
        // ---------------------------------------------------------- update
        if (rest > 0) {
            const Tiling T(rest, G);
            // the look-ahead CTA takes fewer tiles, from the list's end
            const int tiles = T.tr * T.tc;
            const int quota = G > 1 ? max(0, tiles / G - T.la_tiles) : 0;
            const int split = tiles - quota;
            int first = cta, stride = Gt, end = split;
            if (cta == la) {
                if (early) {
                    publish(a, c_next, k0 + NB, min(NB, n - k0 - NB), kb, pass);
                } else {
                    __syncthreads();  // CTA 0 may be this one: S.s is stored before it changes
                    look_ahead(a, k0, kb, pass, U);
                }
                if (G > 1) {
                    first = split;
                    stride = 1;
                    end = tiles;
                }
            }
            const int mine = end > first ? (end - first + stride - 1) / stride : 0;
            stored = mine > 0;
            if (T.teams == 2) {
                update_tiles<2>(a, k0, kb, U, T.tr, T.tc, first, stride, end,
                                tid < kThreads / 2 ? seq0 : seq1);
                seq0 += (mine + 1) / 2;
                seq1 += mine / 2;
            } else {
                update_tiles<1>(a, k0, kb, U, T.tr, T.tc, first, stride, end, seq0);
                seq0 += mine;
            }
        }
    }
    if (cta == 0 && tid == 0) {
        a.flags[kFlagPasses] = pass;
        a.flags[kFlagSwaps] = swaps;
    }
}

}  // namespace lux
}  // namespace d4
