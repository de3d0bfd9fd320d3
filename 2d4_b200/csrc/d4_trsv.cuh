// d4_trsv.cuh: triangular solves with LU factors of element type T (double:
// plain form, exact order; float: mixed form inside refinement), by one
// thread-block cluster with distributed shared memory.
#pragma once
#include <cstdint>

#include "d4_internal.h"
#include "d4_qdiv.cuh"

namespace d4 {
namespace trsv {

struct GArgs {
    int gmode;
    double hval;
    const double *dvec, *s_end, *s_init, *x_new, *x_old, *g_in;
    const double *base;
    double *out;
    double *dx_out;
    int fix_singular;  // apply the zeroing of src/simulation.cpp:652-657
};

// Residual of the stage for row r (src/simulation.cpp:101,123,142,621).
__device__ __forceinline__ double g_of(const GArgs &ga, int r) {
    if (ga.gmode < 0) return ga.g_in[r];
    const double d = ga.dvec[r];
    const double X = (1 + d) * ga.s_end[r] + (1 - d) * ga.s_init[r];
    if (ga.gmode == kGBig) return -ga.hval * X / 2;
    if (ga.gmode == kGHalf) return -ga.hval / 2 * X / 2;
    return ga.x_new[r] - ga.x_old[r] - ga.hval * X / 2;
}

constexpr long long kSpinLimit = 1ll << 25;  // polls: > 1 s

// ---------------------------------------------------------------------------
// Triangular solves with LU factors of element type T (double: the plain form,
// exact order; float: the mixed form, inside refinement), by one thread-block
// cluster of kClusterCtas CTAs, one warp per 32-row block: block b belongs to
// warp b / C of CTA b % C (a warp takes further blocks b + C * warps when there
// are more blocks than warps).  A warp streams its block's factor tiles, the
// diagonal one last, through two shared-memory stages (cp.async: the next tile
// loads while the current one waits for its x values and is applied; loaded only
// after the previous tile was applied, each tile's memory latency stood in the
// chain of the blocks), then solves its diagonal block.  Every lane forms
// every x value of the block itself, from the right-hand side broadcast a step
// early, so the chain of a row is one product and difference (and the quotient
// where it divides) without a shuffle.  After each 8 rows the values go to every
// CTA's shared copy of x by asynchronous stores (st.async ...
// mbarrier::complete_tx) that count down the bytes which that CTA's mbarrier for
// the 8-row group expects.  A consumer waits on its own barrier (acquire) group by group, so it applies a
// block's first values while the last ones are still being formed.  With one
// shuffle per row in the chain, whole blocks handed over and a window branch
// around each quotient a row took 130 (forward) and 300 cycles (backward).  Each
// entry receives its updates in the oracle's order (forward: k ascending;
// backward: k descending, then the division), so the result equals the
// sequential substitution's.  The oracle skips updates with a zero value; here they
// are applied, as x - l*0 == x for finite l.  For a matrix of the caller's whose
// factors have overflowed (the engine's own are far from that) the kSkip form skips
// them; tests in the chain of the other form, or in its end, took 2 us (n = 64) to 18
// (4096).  Waits are bounded: after kSpinLimit polls a warp records err[0] and stops
// waiting (the host then discards the results).
// Before the final cluster barrier every CTA waits for all groups of its own
// copy of x.  An asynchronous store is complete only when its mbarrier says so (no
// CTA or cluster barrier orders it), and nobody has waited for the block solved
// last, whose values no other block applies: without this wait a CTA could exit,
// or a second pass set its barriers up again, with stores still on their way.
constexpr int kClusterCtas = 8;
constexpr int kClusterMaxWarps = 8;

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned cluster_size() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::
                     : "memory");
}
__device__ __forceinline__ uint32_t mapa(uint32_t addr, unsigned cta) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(cta));
    return r;
}
// Asynchronous store into another CTA's shared memory that completes
// sizeof(v) bytes of the transaction count of that CTA's mbarrier `mbar`.  No
// memory clobber: it orders nothing of this thread's, and would keep the chain's
// shared-memory operands from being loaded ahead.
__device__ __forceinline__ void st_async(uint32_t addr, double v, uint32_t mbar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f64 [%0], %1, [%2];" ::"r"(
                     addr),
                 "d"(v), "r"(mbar));
}
__device__ __forceinline__ void st_async(uint32_t addr, float v, uint32_t mbar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];" ::"r"(
                     addr),
                 "f"(v), "r"(mbar));
}
__device__ __forceinline__ void arrive_expect_tx(uint32_t mbar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool try_wait_cluster(uint32_t mbar) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred P1;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 P1, [%1], 0;\n\t"
        "selp.b32 %0, 1, 0, P1;\n\t}\n"
        : "=r"(done)
        : "r"(mbar)
        : "memory");
    return done != 0;
}

__host__ __device__ constexpr int cluster_warps(int n) {
    return ((n + 31) / 32 + kClusterCtas - 1) / kClusterCtas < kClusterMaxWarps
               ? ((n + 31) / 32 + kClusterCtas - 1) / kClusterCtas
               : kClusterMaxWarps;
}

// x (n values), four mbarriers (8-row groups) per 32-row block, and per warp two
// 32 x 32 tile stages and the diagonal's reciprocals.
template <typename T>
__host__ __device__ constexpr size_t cluster_smem_bytes(int n) {
    return ((sizeof(T) * (size_t)n + 15) / 16) * 16 + 32 * (size_t)((n + 31) / 32) +
           sizeof(T) * (2 * 32 * 32 + 32) * (size_t)kClusterMaxWarps;
}

// Tile (row block b, column block kb) of the factors into st[column][row] by one
// warp, asynchronously (element pairs; n is even, so pairs never straddle the
// edge, past which the tile is zero).
template <typename T>
__device__ __forceinline__ void tile_async(const T *__restrict__ LU, int n, int b, int kb, int lane,
                                           T (*st)[32]) {
    const int r = 2 * (lane & 15), row = b * 32 + r;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const int k = 2 * i + (lane >> 4), col = kb * 32 + k;
        const bool ok = row < n && col < n;
        const T *src = ok ? LU + (size_t)row + (size_t)col * n : LU;
        const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(&st[k][r]));
        if (sizeof(T) == 8)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src),
                         "r"(ok ? 16 : 0)
                         : "memory");
        else
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src),
                         "r"(ok ? 8 : 0)
                         : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// kTrans: the factors are given transposed (Lt = (LU)^T) and the system is
// A^T x = g (P A = L U, so A^T = U^T L^T P): the forward pass is U^T (lower,
// divided), the backward pass L^T (unit upper), g is taken unpermuted and the
// result scattered through perm at the end.
template <bool kFwd, typename T, bool kTrans, bool kSkip = false>
__device__ __forceinline__ void solve_pass(int n, const T *__restrict__ LU,
                                           const int *__restrict__ perm, const int *flags,
                                           const GArgs &ga, T *xg, const T *xin, int *err) {
    extern __shared__ __align__(16) unsigned char craw[];
    const int nblk = (n + 31) / 32;
    T *xall = reinterpret_cast<T *>(craw);
    uint64_t *mbar = reinterpret_cast<uint64_t *>(craw + ((sizeof(T) * (size_t)n + 15) / 16) * 16);
    T *slot = reinterpret_cast<T *>(mbar + 4 * (size_t)nblk);
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, nw = blockDim.x >> 5;
    const int C = (int)cluster_size(), c = (int)cluster_rank();
    // one barrier per 8-row group, expecting the group's values from their
    // producer's asynchronous stores
    for (int b = tid; b < 4 * nblk; b += blockDim.x) {
        const uint32_t ma = static_cast<uint32_t>(__cvta_generic_to_shared(mbar + b));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(ma) : "memory");
        if (b * 8 < n) arrive_expect_tx(ma, (uint32_t)(sizeof(T) * min(8, n - b * 8)));
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    __syncthreads();
    cluster_sync_all();
    bool aborted = false;
    slot += w * (2 * 32 * 32 + 32);
    T(*stage)[32][32] = reinterpret_cast<T(*)[32][32]>(slot);
    T *rec = slot + 2 * 32 * 32;
    // the CTAs this lane sends to
    const uint32_t xa = static_cast<uint32_t>(__cvta_generic_to_shared(xall));
    const uint32_t ma0 = static_cast<uint32_t>(__cvta_generic_to_shared(mbar));
    const unsigned p0 = min(lane >> 3, C - 1), p1 = min((lane >> 3) + 4, C - 1);
    const uint32_t xpeer0 = mapa(xa, p0), mpeer0 = mapa(ma0, p0);
    const uint32_t xpeer1 = mapa(xa, p1), mpeer1 = mapa(ma0, p1);
    // this warp's blocks, in solve order
    const int first = c + C * w, stride = C * nw;
    const int nmine = first < nblk ? (nblk - 1 - first) / stride + 1 : 0;
    for (int m = 0; m < nmine; ++m) {
        const int b = kFwd ? first + m * stride : first + (nmine - 1 - m) * stride;
        const int row = b * 32 + lane;
        const bool row_ok = row < n;
        T xi = row_ok ? (kFwd ? T(kTrans ? ga.g_in[row] : g_of(ga, perm[row])) : xin[row]) : T(0);
        const int napply = kFwd ? b : nblk - 1 - b;
        tile_async(LU, n, b, napply > 0 ? (kFwd ? 0 : nblk - 1) : b, lane, stage[0]);
        // the diagonal's reciprocals, formed before the chain (the quotient in
        // the chain is still the IEEE one; rows past the matrix are an identity's)
        rec[lane] = row_ok ? qdiv::recip(LU[(size_t)row + (size_t)row * n]) : T(1);
        for (int s = 0; s < napply; ++s) {
            const int kb = kFwd ? s : nblk - 1 - s;
            const int kw = min(32, n - kb * 32);
            tile_async(LU, n, b, kFwd ? s + 1 : nblk - 2 - s, lane, stage[(s + 1) & 1]);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncwarp();
            const T(*tl)[32] = stage[s & 1];
            const T *xb = xall + kb * 32;
#pragma unroll
            for (int gq = 0; gq < 4; ++gq) {
                const int g = kFwd ? gq : 3 - gq;
                if (g * 8 >= kw) continue;
                T l8[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) l8[e] = tl[8 * g + e][lane];
                if (!aborted) {
                    const uint32_t ma =
                        static_cast<uint32_t>(__cvta_generic_to_shared(mbar + kb * 4 + g));
                    long long spins = 0;
                    bool ok = true;
                    while (!try_wait_cluster(ma)) {
                        if (++spins > kSpinLimit) {
                            ok = false;
                            break;
                        }
                    }
                    if (!__all_sync(0xffffffffu, ok)) {
                        aborted = true;
                        if (lane == 0 && atomicCAS(err, 0, 1) == 0) {
                            err[1] = b;
                            err[2] = kb;
                            err[3] = -1;
                            err[4] = -1;
                        }
                    }
                }
                if (kw == 32 && !kSkip) {
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        const int k = kFwd ? 8 * g + e : 8 * g + 7 - e;
                        xi = xi - l8[k & 7] * xb[k];
                    }
                } else {
                    // the last block's: no product with what lies past it (and the
                    // kSkip form's: none with a zero)
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        const int k = kFwd ? 8 * g + e : 8 * g + 7 - e;
                        if (k < kw && (!kSkip || xb[k] != T(0))) xi = xi - l8[k & 7] * xb[k];
                    }
                }
            }
            __syncwarp();  // this stage is free for the tile after next
        }
        // diagonal block, 8 rows at a time: v is row k's right-hand side, then its
        // x value
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncwarp();
        T(*dt)[32] = stage[napply & 1];  // [column][row]
        if (!row_ok) dt[lane][lane] = T(1);
        __syncwarp();
        constexpr bool kDivides = kFwd == kTrans;
#pragma unroll 1
        for (int gq = 0; gq < 4; ++gq) {
            const int g8 = kFwd ? 8 * gq : 24 - 8 * gq;
            // where it divides, the chain's operands first (930 against 1000 cycles
            // a group; without the division the compiler's order is the better one)
            T own[8], nxt[8], dd[8], rr[8];
            if (kDivides) {
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const int k = kFwd ? g8 + e : g8 + 7 - e, kn = (kFwd ? k + 1 : k - 1) & 31;
                    own[e] = dt[k][lane];
                    nxt[e] = dt[k][kn];
                    dd[e] = dt[k][k];
                    rr[e] = rec[k];
                }
            }
            const T x0 = xi;
            T v = __shfl_sync(0xffffffffu, xi, kFwd ? g8 : g8 + 7), pre = T(0);
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const int k = kFwd ? g8 + e : g8 + 7 - e, kn = (kFwd ? k + 1 : k - 1) & 31;
                const T vn = __shfl_sync(0xffffffffu, xi, kn);
                if (kDivides) {
                    if (lane == k) pre = v;
                    v = qdiv::fast(v, dd[e], rr[e]);
                }
                const T t = xi - (kDivides ? own[e] : dt[k][lane]) * v;
                xi = lane == k ? v : ((kFwd ? lane > k : lane < k) ? t : xi);
                v = vn - (kDivides ? nxt[e] : dt[k][kn]) * v;
            }
            if (kSkip ||
                (kDivides && !__all_sync(0xffffffffu, qdiv::fast_ok(pre, rec[lane])))) {
                // outside the quotient window: the same rows with the division
                xi = x0;
#pragma unroll 1
                for (int e = 0; e < 8; ++e) {
                    const int k = kFwd ? g8 + e : g8 + 7 - e;
                    T x = __shfl_sync(0xffffffffu, xi, k);
                    if (kDivides) x = x / dt[k][k];
                    const T t = kSkip && x == T(0) ? xi : xi - dt[k][lane] * x;
                    xi = lane == k ? x : ((kFwd ? lane > k : lane < k) ? t : xi);
                }
            }
            // lane l sends row l % 8 of the group to CTAs l / 8 and l / 8 + 4
            const int r = b * 32 + g8 + (lane & 7);
            const T x = __shfl_sync(0xffffffffu, xi, g8 + (lane & 7));
            if (r < n) {
                const uint32_t xo = (uint32_t)(r * sizeof(T)), mo = (uint32_t)((r >> 3) * 8);
                if ((lane >> 3) < C) st_async(xpeer0 + xo, x, mpeer0 + mo);
                if ((lane >> 3) + 4 < C) st_async(xpeer1 + xo, x, mpeer1 + mo);
            }
        }
        __syncwarp();
        if (row_ok) {
            xg[(kTrans && !kFwd) ? perm[row] : row] = xi;
            if (!kFwd && !kTrans) {
                double d = (double)xi;
                if (ga.fix_singular && flags[kFlagSingular] && !((-1 < d) && (d < 1))) d = 0;
                if (ga.dx_out) ga.dx_out[row] = d;
                if (ga.out) ga.out[row] = ga.base[row] - d;
            }
        }
    }
    __syncthreads();
    bool gave_up = false;
    for (int b = tid; b * 8 < n; b += blockDim.x) {
        const uint32_t ma = static_cast<uint32_t>(__cvta_generic_to_shared(mbar + b));
        long long spins = 0;
        while (!gave_up && !try_wait_cluster(ma))
            if (++spins > kSpinLimit) {
                gave_up = true;
                if (atomicCAS(err, 0, 1) == 0) {
                    err[1] = -1;
                    err[2] = b >> 2;
                    err[3] = -1;
                    err[4] = -1;
                }
            }
    }
    cluster_sync_all();
}

// Between two passes of one launch by a lone CTA (all stores of the first pass have
// landed, see above): frees its barriers, so that the second can set them up again.
__device__ __forceinline__ void release_barriers(int n, size_t elem) {
    extern __shared__ __align__(16) unsigned char craw[];
    uint64_t *mbar = reinterpret_cast<uint64_t *>(craw + ((elem * (size_t)n + 15) / 16) * 16);
    for (int b = threadIdx.x; b < 4 * ((n + 31) / 32); b += blockDim.x)
        asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(
                         static_cast<uint32_t>(__cvta_generic_to_shared(mbar + b)))
                     : "memory");
    __syncthreads();
}

template <bool kFwd, typename T, bool kTrans, bool kSkip>
__global__ void __launch_bounds__(32 * kClusterMaxWarps) k_trsv_cluster(
    int n, const T *__restrict__ LU, const int *__restrict__ perm, const int *__restrict__ flags,
    GArgs ga, T *xg, const T *xin, int *err) {
    solve_pass<kFwd, T, kTrans, kSkip>(n, LU, perm, flags, ga, xg, xin, err);
}

// Forward then backward cluster solve on `stream`: x1 = forward result (global
// scratch), out = backward result.
template <typename T, bool kTrans = false, bool kSkip = false>
inline void launch_cluster_solve(int n, const T *LU, const int *perm, const int *flags,
                                 const GArgs &ga, T *x1, T *out, int *err, cudaStream_t stream) {
    const size_t bytes = cluster_smem_bytes<T>(n);
    const int warps = cluster_warps(n) > 0 ? cluster_warps(n) : 1;
    static bool attr_done = false;
    if (!attr_done) {
        const int maxb = (int)cluster_smem_bytes<T>(kMaxSolveN);
        D4_CUDA_OK(cudaFuncSetAttribute(k_trsv_cluster<true, T, kTrans, kSkip>,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize, maxb));
        D4_CUDA_OK(cudaFuncSetAttribute(k_trsv_cluster<false, T, kTrans, kSkip>,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize, maxb));
        attr_done = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kClusterCtas);
    cfg.blockDim = dim3(32 * warps);
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kClusterCtas;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const T *none = nullptr;
    D4_CUDA_OK(cudaLaunchKernelEx(&cfg, k_trsv_cluster<true, T, kTrans, kSkip>, n, LU, perm, flags, ga, x1,
                                  none, err));
    check_launch("k_trsv_cluster<fwd>");
    D4_CUDA_OK(cudaLaunchKernelEx(&cfg, k_trsv_cluster<false, T, kTrans, kSkip>, n, LU, perm, flags, ga,
                                  out, (const T *)x1, err));
    check_launch("k_trsv_cluster<bwd>");
}

}  // namespace trsv
}  // namespace d4
