// d4_lu_coop64.cu: host side of the FP64 LU with partial pivoting
// (d4_lu_exact.cuh, compiled with --fmad=false).

#include "d4_lu_exact.cuh"

namespace d4 {

namespace lux {

__global__ void __launch_bounds__(kThreads, 1)
    k_lu_grid(Args a, const __grid_constant__ LuMaps maps, unsigned long long *bar) {
    a.map_a = &maps.a;
    a.map_u = &maps.u;
    factor(a, GridGroup{bar, 0u, 0u, false});
}

// Self-test: an elimination whose columns' barriers lack an arrival.
__global__ void __launch_bounds__(kThreads, 1) k_elim_wait_selftest(int *flags) {
    Smem &S = smem();
    if (threadIdx.x == 0) {
        S.dead = 0;
        S.stuck = 0;
        S.parity = 0;
    }
    if (threadIdx.x < NB) bulk::init(&S.done[threadIdx.x], 2);
    bulk::fence_init();
    __syncthreads();
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double c[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) c[i] = lane == 4 * w + i ? 2.0 : 0.01;
    eliminate_any(c, NB, 0u, flags);
}

}  // namespace lux

void elim_wait_selftest(int *flags) {
    const int bytes = (int)sizeof(lux::Smem);
    D4_CUDA_OK(cudaFuncSetAttribute(lux::k_elim_wait_selftest,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    lux::k_elim_wait_selftest<<<1, lux::kThreads, bytes>>>(flags);
    check_launch("k_elim_wait_selftest");
}

// Tensor maps of a factorisation's buffers: A (n x n, column-major) and the two
// U12 halves (64 rows of n).
void lu_encode_maps(LuMaps &m, double *A, double *U, int n) {
    using Encode = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                                const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static const Encode encode = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) !=
                cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            return (Encode) nullptr;
        return reinterpret_cast<Encode>(p);
    }();
    if (!encode) throw StateError("cuTensorMapEncodeTiled not available");
    auto one = [&](CUtensorMap &t, double *base, int rows, int box_x, int box_y) {
        const cuuint64_t dims[2] = {(cuuint64_t)n, (cuuint64_t)rows};
        const cuuint64_t strides[1] = {(cuuint64_t)n * sizeof(double)};
        const cuuint32_t box[2] = {(cuuint32_t)box_x, (cuuint32_t)box_y}, step[2] = {1, 1};
        if (encode(&t, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, base, dims, strides, box, step,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            throw StateError("cuTensorMapEncodeTiled failed");
    };
    one(m.a, A, n, lux::kBoxR, lux::kBoxC);
    one(m.u, U, 2 * lux::NB, lux::kBoxC, lux::NB);
}

int coop_grid_size() {
    int dev = 0, sms = 0, per_sm = 0;
    D4_CUDA_OK(cudaGetDevice(&dev));
    D4_CUDA_OK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int bytes = (int)sizeof(lux::Smem);
    D4_CUDA_OK(cudaFuncSetAttribute(lux::k_lu_grid, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    bytes));
    D4_CUDA_OK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, lux::k_lu_grid,
                                                             lux::kThreads, bytes));
    return per_sm < 1 ? -1 : sms * per_sm;
}

// Factorises A into L.LU on `st` with `grid` CTAs, without waiting: flags
// (L.flags) are read by the caller later.  `after_copy` (may be null) is
// recorded once A has been copied, after which A may change.
void factor64_async(Ctx &c, const LuBufs &L, const double *A, int grid, cudaStream_t st,
                    cudaEvent_t after_copy) {
    const int n = c.n;
    const size_t bytes = sizeof(double) * (size_t)n * n;
    D4_CUDA_OK(cudaMemsetAsync(L.flags, 0, sizeof(int) * kFlagCount, st));
    D4_CUDA_OK(cudaMemsetAsync(L.bar, 0, sizeof(unsigned) * 64, st));
    D4_CUDA_OK(cudaMemsetAsync(L.mask, 0, sizeof(unsigned) * c.lu_mask_words, st));
    D4_CUDA_OK(cudaMemcpyAsync(L.LU, A, bytes, cudaMemcpyDeviceToDevice, st));
    if (after_copy) D4_CUDA_OK(cudaEventRecord(after_copy, st));
    lux::Args a;
    a.n = n;
    a.A = L.LU;
    a.P0 = L.P0;
    a.Q = L.Q;
    a.U = L.Q + (size_t)n * 64;
    a.dg = L.Q + (size_t)n * 128;
    a.mask = L.mask;
    a.sched = L.mask + lu_pass_words((n + kLuNb - 1) / kLuNb);
    a.perm = L.perm;
    a.piv = L.piv;
    a.flags = L.flags;
    unsigned long long *bar = reinterpret_cast<unsigned long long *>(L.bar);
    void *args[] = {(void *)&a, (void *)L.maps, (void *)&bar};
    D4_CUDA_OK(cudaLaunchCooperativeKernel((const void *)lux::k_lu_grid, dim3(grid),
                                           dim3(lux::kThreads), args, sizeof(lux::Smem), st));
    check_launch("k_lu_grid");
}

LuBufs primary_lu(Ctx &c) {
    LuBufs L;
    L.LU = c.LU;
    L.P0 = c.lu_p0;
    L.Q = c.lu_q;
    L.mask = c.lu_mask;
    L.bar = c.lu_bar;
    L.flags = c.flags;
    L.perm = c.perm;
    L.piv = c.piv;
    L.maps = &c.lu_maps;
    return L;
}

int factor64(Ctx &c) {
    factor64_async(c, primary_lu(c), c.A, c.lu_grid, c.stream, nullptr);
    D4_CUDA_OK(cudaMemcpyAsync(c.h_flags, c.flags, sizeof(int) * kFlagCount,
                               cudaMemcpyDeviceToHost, c.stream));
    D4_CUDA_OK(cudaStreamSynchronize(c.stream));
    if (c.h_flags[kFlagBarrierTimeout]) throw StateError("LU grid barrier timed out");
    count_lu(c, c.h_flags);
    c.factor_singular = c.h_flags[kFlagSingular] != 0;
    c.factor_pivoted = 0;
    return c.factor_singular ? D4_WARN_SINGULAR : D4_OK;
}

}  // namespace d4
