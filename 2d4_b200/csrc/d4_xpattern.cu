// d4_xpattern.cu: the direct-Fourier pattern analysis of a dislocation
// configuration (the reference's xpattern tool, method df,
// xpattern/xpattern.cpp:393-423).
//
// With K = res/2 + 1 and the four densities m = rho_t (weight 1), kappa
// (weight b), rho_p (b = +1 only) and rho_n (b = -1 only),
//     F_m(kx, ky) = sum_i w_m(b_i) exp(-2 pi i (kx x_i + ky y_i)),
//     S_m(kx)    += sum_ky |F_m(kx, ky)|^2.
// F_p and F_n (the sums over the b = +1 and the other dislocations; rho_t = F_p +
// F_n, kappa = F_p - F_n) are complex matrix products Ex^T Ey over their
// dislocations with E[i][k] = exp(-2 pi i k v_i).  k_xp_gemm forms both factors in
// shared memory (sincospi of 2 k v, so large k v keep their accuracy) and multiplies
// on the FP64 matrix units; k_xp_sum adds the four |F|^2 over ky (every 32nd per lane,
// then a tree) into the caller's running sums.  No atomics, fixed orders: the result
// repeats bit for bit.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>
#include <vector>

#include "d4_internal.h"

namespace d4 {
namespace {

constexpr int kXpTile = 64;   // edge of a tile of F (kx, ky)
constexpr int kXpThin = 16;   // thin tiles along a short remainder of K: kXpThin x kXpLong
constexpr int kXpLong = 128;
constexpr int kXpChunk = 32;  // dislocations staged per step
constexpr int kXpThreads = 512;
// the factors of a tile's rows and columns for one dislocation; 2 mod 8: no bank
// conflicts
__host__ __device__ constexpr int xp_row(int m, int n) { return m + n + 2; }
constexpr int kXpSmem = 2 * kXpChunk * xp_row(kXpThin, kXpLong) * (int)sizeof(double2);

// The tiles of F: `wide` x `wide` of kXpTile; what they leave of K (at most
// kXpThin) is covered by thin tiles, kx rows first, then ky columns.
struct XpTiles {
    int wide, rest, rows, cols;  // rows, cols: thin tiles along the last kx, the last ky
    __host__ __device__ explicit XpTiles(int K) {
        rest = K % kXpTile;
        if (rest > kXpThin || K < kXpTile) rest = 0;
        wide = rest ? K / kXpTile : (K + kXpTile - 1) / kXpTile;
        rows = rest ? (K + kXpLong - 1) / kXpLong : 0;
        cols = rest ? (wide * kXpTile + kXpLong - 1) / kXpLong : 0;
    }
    __host__ __device__ int count() const { return wide * wide + rows + cols; }
};

// Bound by the FP64 pipe, which the matrix products (64 fused multiply-adds per
// clock and SM: K = 513, n = 4096 276 us of the one wave's largest tiles) share with
// sincospi (a fifth on top; every tile forms its own factors, which costs less than
// tables in memory: they took 67 MB and an allocation each).  Half of the warps form
// the next chunk's factors first and multiply then, the others the other way round,
// so that both kinds of work are always in flight (0.45 ms; 0.71 ms with tables and
// 2 x 2 outputs per thread, 0.88 with one factor at a time per thread).  A remainder
// of K up to 16 (K is a power of two and one as a rule) gets thin tiles: padding to
// a whole tile costs 1.27 times the work at K = 513.
__device__ __forceinline__ void mma(double (&c)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(c[0]), "+d"(c[1])
        : "d"(a), "d"(b));
}

// One tile of kM x kN entries of F: rows from m0 (wave numbers of u), columns from
// c0 (of v), over the dislocations [beg, end).  Element (r, c), r < m_end, c < c_end, goes to
// out[r * rs + c * cs].
template <int kM, int kN>
__device__ __forceinline__ void xp_tile(int beg, int end, const double *u, const double *v, int m0,
                                        int m_end, int c0, int c_end, double2 *out, size_t rs,
                                        size_t cs) {
    extern __shared__ __align__(16) unsigned char xp_smem[];
    typedef double2 Stage[kXpChunk][xp_row(kM, kN)];  // [dislocation][rows, then columns]
    Stage *st = reinterpret_cast<Stage *>(xp_smem);
    constexpr int kWarpM = kM / 16, kWarpN = kXpThreads / 32 / kWarpM;  // warps along rows, columns
    constexpr int RM = kM / 8 / kWarpM, RN = kN / 8 / kWarpN;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int wm = warp / kWarpN * 8 * RM, wn = warp % kWarpN * 8 * RN;
    auto produce = [&](int i0, int buf) {
#pragma unroll 4
        for (int e = 0; e < kXpChunk * (kM + kN) / kXpThreads; ++e) {
            const int t = tid + e * kXpThreads, r = t / (kM + kN), col = t % (kM + kN);
            const double w = i0 + r < end ? (col < kM ? u : v)[i0 + r] : 0.0;
            const int k = col < kM ? m0 + col : c0 + col - kM;
            double s, c;
            sincospi(2.0 * w * (double)k, &s, &c);
            // (past the end: no contribution)
            st[buf][r][col] = i0 + r < end ? make_double2(c, -s) : make_double2(0.0, 0.0);
        }
    };
    double re[RM][RN][2], im[RM][RN][2];
#pragma unroll
    for (int a = 0; a < RM; ++a)
#pragma unroll
        for (int b = 0; b < RN; ++b)
            re[a][b][0] = re[a][b][1] = im[a][b][0] = im[a][b][1] = 0.0;
    auto consume = [&](int buf) {
#pragma unroll
        for (int r = 0; r < kXpChunk; r += 4) {
            double2 x[RM], y[RN];
#pragma unroll
            for (int a = 0; a < RM; ++a) x[a] = st[buf][r + (lane & 3)][wm + 8 * a + (lane >> 2)];
#pragma unroll
            for (int b = 0; b < RN; ++b) y[b] = st[buf][r + (lane & 3)][kM + wn + 8 * b + (lane >> 2)];
#pragma unroll
            for (int a = 0; a < RM; ++a)
#pragma unroll
                for (int b = 0; b < RN; ++b) {
                    mma(re[a][b], x[a].x, y[b].x);
                    mma(im[a][b], x[a].x, y[b].y);
                }
#pragma unroll
            for (int a = 0; a < RM; ++a)
#pragma unroll
                for (int b = 0; b < RN; ++b) {
                    mma(re[a][b], -x[a].y, y[b].y);
                    mma(im[a][b], x[a].y, y[b].x);
                }
        }
    };
    if (beg < end) produce(beg, 0);
    __syncthreads();
    int buf = 0;
    for (int i0 = beg; i0 < end; i0 += kXpChunk, buf ^= 1) {
        const bool more = i0 + kXpChunk < end;
        if (warp < kXpThreads / 64) {
            if (more) produce(i0 + kXpChunk, buf ^ 1);
            consume(buf);
        } else {
            consume(buf);
            if (more) produce(i0 + kXpChunk, buf ^ 1);
        }
        __syncthreads();
    }
#pragma unroll
    for (int a = 0; a < RM; ++a)
#pragma unroll
        for (int b = 0; b < RN; ++b)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int r = m0 + wm + 8 * a + (lane >> 2), c = c0 + wn + 8 * b + 2 * (lane & 3) + e;
                if (r < m_end && c < c_end) out[r * rs + c * cs] = make_double2(re[a][b][e], im[a][b][e]);
            }
}

// F[part * slices + slice][kx][ky] over slice `slice` of the dislocations of a part
// ([0, npos) and [npos, n)).  Block: tile x, slice y, part z.
__global__ void __launch_bounds__(kXpThreads)
    k_xp_gemm(int n, int npos, int K, const double *x, const double *y, double2 *F) {
    const XpTiles T(K);
    const int lo = blockIdx.z ? npos : 0, hi = blockIdx.z ? n : npos;
    const int per = ((hi - lo + gridDim.y - 1) / (int)gridDim.y + kXpChunk - 1) / kXpChunk * kXpChunk;
    const int beg = min(hi, lo + (int)blockIdx.y * per), end = min(hi, beg + per);
    double2 *out = F + (size_t)(blockIdx.z * gridDim.y + blockIdx.y) * K * K;
    int t = blockIdx.x;
    if (t < T.wide * T.wide) {
        xp_tile<kXpTile, kXpTile>(beg, end, x, y, t / T.wide * kXpTile, K, t % T.wide * kXpTile, K,
                                  out, K, 1);
        return;
    }
    t -= T.wide * T.wide;
    const int edge = T.wide * kXpTile;
    if (t < T.rows)  // the last kx, all ky
        xp_tile<kXpThin, kXpLong>(beg, end, x, y, edge, K, t * kXpLong, K, out, K, 1);
    else  // the last ky, the kx before
        xp_tile<kXpThin, kXpLong>(beg, end, y, x, edge, K, (t - T.rows) * kXpLong, edge, out, 1, K);
}

// acc[m][kx] += sum over ky of |F_m(kx, ky)|^2: one warp per kx, lane sums of every
// 32nd ky, then a fixed tree (18 us at K = 513; 73 us as one serial sum per thread).
__global__ void __launch_bounds__(128) k_xp_sum(int K, int slices, const double2 *F, double *acc) {
    const int kx = blockIdx.x * 4 + threadIdx.x / 32, lane = threadIdx.x & 31;
    if (kx >= K) return;
    const size_t KK = (size_t)K * K;
    double v[4] = {0, 0, 0, 0};
    for (int ky = lane; ky < K; ky += 32) {
        double2 f[2];
#pragma unroll
        for (int part = 0; part < 2; ++part) {
            f[part] = make_double2(0, 0);
            for (int s = 0; s < slices; ++s) {
                const double2 w = F[(size_t)(part * slices + s) * KK + (size_t)kx * K + ky];
                f[part].x += w.x;
                f[part].y += w.y;
            }
        }
        const double2 p = f[0], q = f[1];
        const double tr = p.x + q.x, ti = p.y + q.y;  // rho_t
        const double kr = p.x - q.x, ki = p.y - q.y;  // kappa
        v[0] += tr * tr + ti * ti;
        v[1] += kr * kr + ki * ki;
        v[2] += p.x * p.x + p.y * p.y;
        v[3] += q.x * q.x + q.y * q.y;
    }
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        for (int o = 16; o > 0; o >>= 1) v[m] += __shfl_down_sync(0xffffffffu, v[m], o);
        if (lane == 0) acc[(size_t)m * K + kx] += v[m];
    }
}

// The driver's process-wide unique number of the allocation at p; 0 when there is none
// or it cannot be queried.
unsigned long long buffer_id(const void *p) {
    using Fn = CUresult (*)(void *, CUpointer_attribute, CUdeviceptr);
    static const Fn fn = [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuPointerGetAttribute", &f, cudaEnableDefault, &q) !=
                cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            return (Fn) nullptr;
        return reinterpret_cast<Fn>(f);
    }();
    unsigned long long id = 0;
    if (!fn || fn(&id, CU_POINTER_ATTRIBUTE_BUFFER_ID, (CUdeviceptr)p) != CUDA_SUCCESS) return 0;
    return id;
}

// The device block kept between calls: allocating and freeing one took 0.6 of the
// 1.16 ms of a call (K = 513, n = 4096).  One block of at most kKeep bytes for the
// whole process; a call has it to itself from take to give (a second thread's call
// allocates its own), every call ends with its device work done, and another device,
// a larger size or a failed allocation of the library frees it (the process's end does
// by itself: the runtime must not be called after main).  A device reset by the host
// program frees it too, behind our back, and its address may become another
// allocation's: the block is ours only while its buffer number is the one noted.
class Spare {
  public:
    // *size: the block's own size, at least `bytes`; give gets it back.
    cudaError_t take(char **p, size_t bytes, size_t *size) {
        int dev = -1;
        cudaGetDevice(&dev);
        Block b = grab();
        if (b.p && b.dev == dev && b.size >= bytes) {
            *p = b.p;
            *size = b.size;
            return cudaSuccess;
        }
        if (b.p) cudaFree(b.p);
        *size = bytes;
        return dmalloc(p, bytes);
    }
    void give(char *p, size_t size, bool keep) {
        Block b{p, size, -1, 0};
        if (!p) return;
        if (keep && size <= kKeep && cudaGetDevice(&b.dev) == cudaSuccess &&
            (b.id = buffer_id(p)) != 0) {
            std::lock_guard<std::mutex> lock(m_);
            if (!b_.p) {
                b_ = b;
                return;
            }
        }
        cudaFree(p);
    }
    void release() {
        const Block b = grab();
        if (b.p) cudaFree(b.p);
    }

  private:
    struct Block {
        char *p;
        size_t size;
        int dev;
        unsigned long long id;
    };
    Block grab() {
        Block b{};
        {
            std::lock_guard<std::mutex> lock(m_);
            std::swap(b, b_);
        }
        if (b.p && buffer_id(b.p) != b.id) b = Block{};
        return b;
    }
    static constexpr size_t kKeep = 32u << 20;
    std::mutex m_;
    Block b_{};
};
Spare g_spare;

}  // namespace

void release_spare() { g_spare.release(); }

}  // namespace d4

extern "C" int d4_xpattern_df(int n, const double *x, const double *y, const int *b, int res,
                              double *acc) {
    using namespace d4;
    if (n < 0 || res < 2 || res > 65536 || (n > 0 && (!x || !y || !b)) || !acc) return D4_ERR_ARG;
    const int K = res / 2 + 1;
    if ((long long)K * K * 4 * 8 > (8ll << 30)) return D4_ERR_ARG;
    // one upload: x and y, positives first (stable), so each density's sum runs over
    // one range, then the running sums
    std::vector<double> h(2 * (size_t)n + 4 * (size_t)K);
    int npos = 0;
    for (int pass = 0, m = 0; pass < 2; ++pass) {
        for (int i = 0; i < n; ++i)
            if ((b[i] == 1) == (pass == 0)) {
                h[m] = x[i];
                h[(size_t)n + m] = y[i];
                ++m;
            }
        if (pass == 0) npos = m;
    }
    std::copy(acc, acc + 4 * (size_t)K, h.begin() + 2 * (size_t)n);
    const int tiles = XpTiles(K).count();
    int dev_no = 0, sms = 0;
    if (cudaGetDevice(&dev_no) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev_no) != cudaSuccess)
        return D4_ERR_CUDA;
    // few tiles: the dislocations are cut into slices, so that about one block runs
    // per SM, of at least four chunks each (below that the sums over the slices and
    // the first chunk's latency weigh as much as the products)
    const int slices = std::max(1, std::min(sms / (2 * tiles), n / (4 * kXpChunk)));
    const size_t vals = sizeof(double) * h.size(),
                 cells = sizeof(double2) * 2 * slices * (size_t)K * K;
    char *dev = nullptr;  // F, then the uploaded values
    size_t size = 0;
    int st = D4_OK;
    auto ok = [&](cudaError_t e) {
        if (e != cudaSuccess && st == D4_OK) st = D4_ERR_CUDA;
        return e == cudaSuccess;
    };
    if (ok(g_spare.take(&dev, cells + vals, &size))) {
        double2 *F = reinterpret_cast<double2 *>(dev);
        double *dv = reinterpret_cast<double *>(dev + cells), *dacc = dv + 2 * (size_t)n;
        ok(cudaMemcpy(dv, h.data(), vals, cudaMemcpyHostToDevice));
        ok(cudaFuncSetAttribute(k_xp_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, kXpSmem));
        if (st == D4_OK) {
            k_xp_gemm<<<dim3(tiles, slices, 2), kXpThreads, kXpSmem>>>(n, npos, K, dv, dv + n, F);
            k_xp_sum<<<(K + 3) / 4, 128>>>(K, slices, F, dacc);
            g_launches.fetch_add(2, std::memory_order_relaxed);
            ok(cudaGetLastError());
            ok(cudaMemcpy(acc, dacc, sizeof(double) * 4 * K, cudaMemcpyDeviceToHost));
        }
    }
    g_spare.give(dev, size, st == D4_OK);
    return st;
}
