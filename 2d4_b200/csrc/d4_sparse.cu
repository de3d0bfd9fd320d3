// d4_sparse.cu: the distant-pair cutoff path, the cutoff-sparse Jacobian solved
// by Jacobi-preconditioned restarted GMRES in FP64.
//
// Under the cutoff (src/simulation.cpp:461-478) the Jacobian keeps only pairs
// closer than the cutoff range (Heaviside, or the Gaussian tail out to 7 cutoff
// radii), about pi r^2 N entries per row, and the reference hands it to UMFPACK
// as a CSC matrix (src/simulation.cpp:635-659).  Here the matrix is still
// assembled densely by the pair kernels, so the row sums d_i and the row
// scaling keep the reference's order, and is then compressed to CSR:
//   k_csr_count  nonzeros per (row, 256-column chunk), chunk offsets inside the rows
//   k_csr_rows   the row-pointer scan (one CTA)
//   k_csr_fill   column indices and values in ascending column order
// Every solve of the step then runs GMRES(40) with right Jacobi preconditioning,
// classical Gram-Schmidt with one reorthogonalisation and Givens rotations, to a
// relative residual of 1e-13, as one cooperative kernel: each CTA owns a
// contiguous range of rows, the SpMV is 8 lanes per row (fixed lane split and
// butterfly, so results do not depend on timing), and each reduction goes
// through per-CTA partials (double-buffered) and a bounded grid barrier, three
// barriers per Krylov vector.  A solve that does not converge within the restart
// budget is reported to the host, which redoes it with the dense LU.
#include <algorithm>
#include <cstdint>

#include "d4_internal.h"
#include "d4_trsv.cuh"

namespace d4 {
namespace sp {

constexpr int kM = 40;            // Krylov dimension per restart
constexpr int kRestarts = 6;
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kStride = kM + 2;   // partials per CTA
constexpr int kChunk = 256;       // columns per counting chunk
constexpr int kCountChunks = 16;  // chunks counted at once
constexpr int kSpLanes = 8;       // lanes per row of the SpMV
constexpr int kRowsPer = 32;      // rows per CTA as long as the SMs suffice
constexpr long long kSpinLimit = 1ll << 22;  // polls of several hundred cycles: > 1 s
constexpr double kTol = 1e-13;

// The basis and w of the rows of a CTA.
constexpr size_t gmres_smem_bytes(int rows) { return sizeof(double) * (kM + 2) * rows; }

struct GmresArgs {
    int n;
    const int *rp, *ci;
    const double *val, *dinv;
    trsv::GArgs g;       // right-hand side
    const double *base;  // out = base - x (out null: no output but dx)
    double *out, *dx;    // written when the solve converged
    double *x;           // n: the iterate
    double *z;           // n: preconditioned vector fed to the SpMV
    double *part;        // 2 x kStride x G partial sums
    unsigned *bar;       // barrier counter (zeroed before the launch)
    int *flags;          // [0] barrier timeout, [1] not converged, [2] iterations
};

__device__ __forceinline__ unsigned ld_acq(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Barrier over all CTAs (a counter that only grows).  The wait gives up after
// kSpinLimit polls (or when another CTA gave up), sets flags[0] and marks the CTA
// dead, after which it no longer waits; the host turns flags[0] into an error.
__device__ __forceinline__ void grid_barrier(unsigned *bar, int *flags, unsigned &gen, int *dead) {
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned target = ++gen * gridDim.x;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
        long long spins = 0;
        while (!*dead && (int)(ld_acq(bar) - target) < 0) {
            if ((++spins & 255) == 0 &&
                (spins > kSpinLimit || ld_acq((const unsigned *)&flags[0]))) {
                atomicOr(&flags[0], 1);
                *dead = 1;
            }
        }
    }
    __syncthreads();
}

// w[r] = scale * (A src)[r0 + r] for the CTA's rows, kSpLanes lanes per row.
__device__ __forceinline__ void spmv_rows(const GmresArgs &a, int r0, int rows, const double *src,
                                          double scale, double *w) {
    const int l = threadIdx.x % kSpLanes;
    for (int b = 0; b < rows; b += kThreads / kSpLanes) {
        const int r = b + threadIdx.x / kSpLanes;
        double s = 0;
        if (r < rows) {
            const int q1 = a.rp[r0 + r + 1];
#pragma unroll 4
            for (int q = a.rp[r0 + r] + l; q < q1; q += kSpLanes)
                s += a.val[q] * __ldcg(src + a.ci[q]);
        }
        for (int o = kSpLanes / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (l == 0 && r < rows) w[r] = s * scale;
    }
    __syncthreads();
}

// Bound by the chain of a Krylov vector, 17 us at N = 4096: three reductions over 128
// CTAs, whose barriers take 1.3 us each, with the sums on both sides of them, and the
// SpMV's gathers.  32 rows per CTA, so that one pass of the SpMV
// covers them with 8 lanes a row, the basis in shared memory (rows of a CTA only), a
// warp per dot product and per total: N = 4096 486 -> 236 us a solve (128 rows per
// CTA with one warp per row, the basis in memory, every total a serial sum, and a
// sleeping barrier before).
__global__ void __launch_bounds__(kThreads, 1) k_gmres(GmresArgs a) {
    extern __shared__ double gm_smem[];
    __shared__ double H[kM + 1][kM];
    __shared__ double tot[kStride], hsum[kM], cs[kM], sn[kM], s[kM + 1], y[kM];
    __shared__ int dead, stop;
    const int n = a.n, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, G = gridDim.x;
    const int rows_per = (n + G - 1) / G;
    const int r0 = min(n, (int)blockIdx.x * rows_per), rows = min(n, r0 + rows_per) - r0;
    double *V = gm_smem;                         // (kM + 1) x rows_per
    double *w = V + (size_t)(kM + 1) * rows_per;  // rows_per
    unsigned gen = 0;
    int parity = 0;
    if (tid == 0) {
        dead = 0;
        stop = 0;
    }
    // Sums over all rows of w times basis vector k (of w's square where `square`) into
    // tot[0..cnt): a warp per sum over the CTA's rows, one partial per CTA, grid
    // barrier, then a warp per total over the CTAs (identical totals everywhere).
    auto reduce = [&](int cnt, bool square) {
        double *P = a.part + (size_t)parity * G * kStride;
        for (int k = wid; k < cnt; k += kWarps) {
            const double *u = square ? w : V + (size_t)k * rows_per;
            double v = 0;
            for (int r = lane; r < rows; r += 32) v += w[r] * u[r];
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0) P[(size_t)k * G + blockIdx.x] = v;
        }
        grid_barrier(a.bar, a.flags, gen, &dead);
        for (int k = wid; k < cnt; k += kWarps) {
            double v = 0;
#pragma unroll 5
            for (int b = lane; b < G; b += 32) v += __ldcg(P + (size_t)k * G + b);
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0) tot[k] = v;
        }
        __syncthreads();
        parity ^= 1;
    };
    // w -= V tot over the basis vectors 0..j
    auto subtract = [&](int j) {
        if (tid < rows) {
            double v = w[tid];
            for (int k = 0; k <= j; ++k) v -= tot[k] * V[(size_t)k * rows_per + tid];
            w[tid] = v;
        }
    };
    const int i = r0 + tid;  // the thread's row (rows_per <= kThreads)
    const bool own = tid < rows;
    const double gi = own ? trsv::g_of(a.g, i) : 0, di = own ? a.dinv[i] : 0;
    double xi = 0;
    if (own) w[tid] = gi;
    __syncthreads();
    reduce(1, true);
    const double gnorm = sqrt(tot[0]);
    int iters = 0;
    bool converged = !(gnorm > 0);
    for (int cycle = 0; cycle < kRestarts && !converged && !dead; ++cycle) {
        // r = g - A x -> V_0, beta = ||r||
        if (cycle > 0) spmv_rows(a, r0, rows, a.x, 1.0, w);
        if (own) w[tid] = cycle > 0 ? gi - w[tid] : gi;
        __syncthreads();
        reduce(1, true);
        const double beta = sqrt(tot[0]);
        if (!(beta > kTol * gnorm)) {
            converged = true;
            break;
        }
        if (own) {
            const double v = w[tid] / beta;
            V[tid] = v;
            a.z[i] = di * v;
        }
        if (tid == 0) {
            for (int k = 0; k <= kM; ++k) s[k] = 0;
            s[0] = beta;
        }
        grid_barrier(a.bar, a.flags, gen, &dead);
        double zscale = 1.0;  // z holds zscale * M^-1 V_j
        int jdone = 0;
        for (int j = 0; j < kM; ++j) {
            // w = A M^-1 V_j; first Gram-Schmidt pass
            spmv_rows(a, r0, rows, a.z, 1.0 / zscale, w);
            reduce(j + 1, false);
            subtract(j);
            if (tid <= j) hsum[tid] = tot[tid];
            __syncthreads();
            // reorthogonalisation
            reduce(j + 1, false);
            subtract(j);
            if (tid <= j) hsum[tid] += tot[tid];
            // ||w|| and the next (unnormalised) preconditioned vector share a barrier
            if (own) a.z[i] = di * w[tid];
            __syncthreads();
            reduce(1, true);
            const double nrm = sqrt(tot[0]);
            zscale = nrm > 0 ? nrm : 1.0;
            if (own) V[(size_t)(j + 1) * rows_per + tid] = nrm > 0 ? w[tid] / nrm : 0;
            if (tid == 0) {
                for (int k = 0; k <= j; ++k) H[k][j] = hsum[k];
                for (int k = 0; k < j; ++k) {
                    const double t = cs[k] * H[k][j] + sn[k] * H[k + 1][j];
                    H[k + 1][j] = -sn[k] * H[k][j] + cs[k] * H[k + 1][j];
                    H[k][j] = t;
                }
                const double d = sqrt(H[j][j] * H[j][j] + nrm * nrm);
                cs[j] = d > 0 ? H[j][j] / d : 1;
                sn[j] = d > 0 ? nrm / d : 0;
                H[j][j] = d;
                s[j + 1] = -sn[j] * s[j];
                s[j] = cs[j] * s[j];
                stop = (!(fabs(s[j + 1]) > kTol * gnorm) || !(nrm > 0)) ? 1 : 0;
            }
            __syncthreads();
            ++iters;
            jdone = j + 1;
            if (stop || dead) break;
        }
        converged = stop != 0;
        // y = H^-1 s (upper triangular); x += M^-1 V y
        if (tid == 0) {
            for (int k = jdone - 1; k >= 0; --k) {
                double t = s[k];
                for (int q = k + 1; q < jdone; ++q) t -= H[k][q] * y[q];
                y[k] = H[k][k] != 0 ? t / H[k][k] : 0;
            }
        }
        __syncthreads();
        if (own) {
            double u = 0;
            for (int k = 0; k < jdone; ++k) u += y[k] * V[(size_t)k * rows_per + tid];
            xi += di * u;
            a.x[i] = xi;
        }
        if (converged) break;
        grid_barrier(a.bar, a.flags, gen, &dead);
        if (tid == 0) stop = 0;
        __syncthreads();
    }
    if (own && converged && !dead) {
        a.dx[i] = xi;
        if (a.out) a.out[i] = a.base[i] - xi;
    }
    if (blockIdx.x == 0 && tid == 0) {
        if (!converged || dead) atomicOr(&a.flags[1], 1);
        a.flags[2] = iters;
    }
}

// Nonzeros per (row, column chunk) of 32 rows per block, one thread per row and chunk,
// 16 loads in flight (column-major matrix): chunk offsets off[ch][i] inside the row,
// row totals to rp[i].
template <typename T>
__global__ void __launch_bounds__(32 * kCountChunks) k_csr_count(int n, int nch,
                                                                 const T *__restrict__ A,
                                                                 int *__restrict__ off,
                                                                 int *__restrict__ rp) {
    __shared__ int cnt[kCountChunks][32];
    const int i = blockIdx.x * 32 + threadIdx.x, y = threadIdx.y;
    int run = 0;  // of the chunks before
    for (int ch0 = 0; ch0 < nch; ch0 += kCountChunks) {
        const int j0 = (ch0 + y) * kChunk, j1 = min(n, j0 + kChunk);
        int c = 0;
        if (i < n)
#pragma unroll 16
            for (int j = j0; j < j1; ++j) c += A[(size_t)i + (size_t)j * n] != T(0);
        cnt[y][threadIdx.x] = c;
        __syncthreads();
        int before = run;
        for (int q = 0; q < kCountChunks; ++q) {
            if (q == y) before = run;
            run += cnt[q][threadIdx.x];
        }
        if (i < n && ch0 + y < nch) off[(size_t)(ch0 + y) * n + i] = before;
        __syncthreads();
    }
    if (i < n && y == 0) rp[i] = run;
}

// The row pointer rp[0..n] from the row totals in it (one CTA of 1024:
// 5 us at n = 4096; 27 with the chunk offsets formed here too).
__global__ void __launch_bounds__(1024) k_csr_rows(int n, int *rp) {
    __shared__ int part[1024];
    const int tid = threadIdx.x;
    const int per = (n + 1023) / 1024;
    const int b0 = min(n, tid * per), b1 = min(n, b0 + per);
    int sum = 0;
#pragma unroll 4
    for (int i = b0; i < b1; ++i) sum += rp[i];
    part[tid] = sum;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {
        const int v = tid >= o ? part[tid - o] : 0;
        __syncthreads();
        part[tid] += v;
        __syncthreads();
    }
    int run = part[tid] - sum;
    for (int i = b0; i < b1; ++i) {
        const int t = rp[i];
        rp[i] = run;
        run += t;
    }
    if (tid == 1023) rp[n] = part[1023];
}

// Bound by the read of A: 16 loads in flight per thread (134 MB at n = 4096: 47 us;
// 73 with a load, a test and a store after each other).
template <typename T>
__global__ void k_csr_fill(int n, const T *__restrict__ A, const int *__restrict__ off,
                           const int *__restrict__ rp, int *__restrict__ ci,
                           double *__restrict__ val, double *__restrict__ dinv) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int ch = blockIdx.y;
    if (i >= n) return;
    const int j0 = ch * kChunk, j1 = min(n, j0 + kChunk);
    int q = rp[i] + off[(size_t)ch * n + i];
    for (int jb = j0; jb < j1; jb += 16) {
        T v[16];
#pragma unroll
        for (int u = 0; u < 16; ++u) v[u] = jb + u < j1 ? A[(size_t)i + (size_t)(jb + u) * n] : T(0);
#pragma unroll
        for (int u = 0; u < 16; ++u)
            if (v[u] != T(0)) {
                ci[q] = jb + u;
                val[q] = (double)v[u];
                ++q;
            }
    }
    if (i >= j0 && i < j1) {
        const double d = (double)A[(size_t)i + (size_t)i * n];
        dinv[i] = d != 0 ? 1 / d : 1.0;
    }
}

inline int nb(int n, int t) { return (n + t - 1) / t; }

}  // namespace sp

bool gmres_selected(const Ctx &c) {
    if (c.p.solver == D4_SOLVER_GMRES) return true;
    if (c.p.solver == D4_SOLVER_AUTO) return c.range_sq * c.cutoff_sq < 0.1;
    return false;
}

void sparse_alloc(Ctx &c) {
    const int n = c.n;
    int dev = 0, sms = 0;
    D4_CUDA_OK(cudaGetDevice(&dev));
    D4_CUDA_OK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    // kRowsPer rows per CTA while the SMs suffice (one row per thread at most): the
    // barriers cost little more over 128 CTAs than over 32, the SpMV a quarter
    c.sp_grid = std::max(1, std::min(sms, sp::nb(n, sp::kRowsPer)));
    if (sp::nb(n, c.sp_grid) > sp::kThreads) throw StateError("n too large for the GMRES grid");
    // for any number of rows per CTA: the limit is the process's, and other contexts
    // launch from other threads
    D4_CUDA_OK(cudaFuncSetAttribute(sp::k_gmres, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)sp::gmres_smem_bytes(sp::kThreads)));
    c.sp_nch = sp::nb(n, sp::kChunk);
    auto ialloc = [](int **p, size_t k) { D4_CUDA_OK(d4::dmalloc((void **)p, sizeof(int) * k)); };
    auto dalloc = [](double **p, size_t k) {
        D4_CUDA_OK(d4::dmalloc((void **)p, sizeof(double) * k));
    };
    ialloc(&c.sp_off, (size_t)c.sp_nch * n);
    ialloc(&c.sp_rp, (size_t)n + 1);
    D4_CUDA_OK(d4::dmalloc((void **)&c.sp_bar, sizeof(unsigned) * 64));
    c.sp_flags = (int *)(c.sp_bar + 32);
    dalloc(&c.sp_dinv, n);
    dalloc(&c.sp_z, n);
    dalloc(&c.sp_x, n);
    dalloc(&c.sp_part, (size_t)2 * c.sp_grid * sp::kStride);
    // initial CSR capacity: 64 entries per row, grown on demand
    c.sp_cap = 64 * n;
    ialloc(&c.sp_ci, (size_t)c.sp_cap);
    dalloc(&c.sp_val, (size_t)c.sp_cap);
}

void sparse_free(Ctx &c) {
    void *bufs[] = {c.sp_off, c.sp_rp, c.sp_bar, c.sp_dinv, c.sp_z, c.sp_x, c.sp_part, c.sp_ci, c.sp_val};
    for (void *b : bufs)
        if (b) cudaFree(b);
}

// CSR of the current matrix (the FP64 A of either form).  Reads the entry
// count back to size the index and value arrays (one host sync).
void sparse_prepare(Ctx &c) {
    const int n = c.n;
    const dim3 grid(sp::nb(n, 128), c.sp_nch);
    sp::k_csr_count<double><<<sp::nb(n, 32), dim3(32, sp::kCountChunks), 0, c.stream>>>(
        n, c.sp_nch, c.A, c.sp_off, c.sp_rp);
    check_launch("k_csr_count");
    sp::k_csr_rows<<<1, 1024, 0, c.stream>>>(n, c.sp_rp);
    check_launch("k_csr_rows");
    D4_CUDA_OK(cudaMemcpyAsync(c.h_flags, c.sp_rp + n, sizeof(int), cudaMemcpyDeviceToHost,
                               c.stream));
    D4_CUDA_OK(cudaStreamSynchronize(c.stream));
    const int nnz = c.h_flags[0];
    if (nnz > c.sp_cap) {
        D4_CUDA_OK(cudaFree(c.sp_ci));
        D4_CUDA_OK(cudaFree(c.sp_val));
        c.sp_ci = nullptr;
        c.sp_val = nullptr;
        c.sp_cap = nnz + nnz / 4 + 1024;
        D4_CUDA_OK(d4::dmalloc((void **)&c.sp_ci, sizeof(int) * (size_t)c.sp_cap));
        D4_CUDA_OK(d4::dmalloc((void **)&c.sp_val, sizeof(double) * (size_t)c.sp_cap));
    }
    c.sp_nnz = nnz;
    sp::k_csr_fill<double><<<grid, 128, 0, c.stream>>>(n, c.A, c.sp_off, c.sp_rp, c.sp_ci,
                                                       c.sp_val, c.sp_dinv);
    check_launch("k_csr_fill");
    c.sp_dense_ready = 0;
}

// One solve of the step by GMRES: g of the stage, x = A^-1 g, out = base - x.
// Returns false when GMRES did not converge (nothing written to out).
bool sparse_solve_update(Ctx &c, int gmode, double hval, const double *s_end,
                         const double *s_init, const double *x_new, const double *x_old,
                         const double *base, double *out) {
    const int n = c.n;
    trsv::GArgs ga{};
    ga.gmode = gmode;
    ga.hval = hval;
    ga.dvec = c.dvec;
    ga.s_end = s_end;
    ga.s_init = s_init;
    ga.x_new = x_new;
    ga.x_old = x_old;
    D4_CUDA_OK(cudaMemsetAsync(c.sp_bar, 0, sizeof(unsigned) * 64, c.stream));  // and sp_flags
    sp::GmresArgs a;
    a.n = n;
    a.rp = c.sp_rp;
    a.ci = c.sp_ci;
    a.val = c.sp_val;
    a.dinv = c.sp_dinv;
    a.g = ga;
    a.base = base;
    a.out = out;
    a.dx = c.dx;
    a.x = c.sp_x;
    a.z = c.sp_z;
    a.part = c.sp_part;
    a.bar = c.sp_bar;
    a.flags = c.sp_flags;
    void *args[] = {(void *)&a};
    const size_t smem = sp::gmres_smem_bytes(sp::nb(n, c.sp_grid));
    D4_CUDA_OK(cudaLaunchCooperativeKernel((const void *)sp::k_gmres, dim3(c.sp_grid),
                                           dim3(sp::kThreads), args, smem, c.stream));
    check_launch("k_gmres");
    D4_CUDA_OK(cudaMemcpyAsync(c.h_flags, c.sp_flags, sizeof(int) * 4, cudaMemcpyDeviceToHost,
                               c.stream));
    D4_CUDA_OK(cudaStreamSynchronize(c.stream));
    if (c.h_flags[0]) throw StateError("GMRES grid barrier timed out");
    c.sp_solves += 1;
    c.sp_iters += c.h_flags[2];
    if (c.h_flags[1]) {
        c.sp_fallbacks += 1;
        return false;
    }
    return true;
}

}  // namespace d4
