// Launches of the Hex20 gather (write_hex20.cuh).
#include <algorithm>

#include "write_hex20.cuh"

namespace fem {
namespace {

template <int kMode>
__global__ void __launch_bounds__(kWriteThreads, FEM_HEXW_CTAS)
    k_write_hex20(ListLayout L, HexRows h, const int* __restrict__ ucounts, const int* __restrict__ row_ptr,
                  int* __restrict__ col_idx, double* __restrict__ values, long long capacity) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    write_hex20<kMode>(L, h, ucounts, row_ptr, col_idx, values, capacity, blockIdx.x, gridDim.x,
                       *reinterpret_cast<WriteHexCta*>(smem_raw));
}

// Columns >= n of every row node: the sorted row's tail from the node itself on.
__global__ void __launch_bounds__(256) k_count_upper_hex20(ListLayout L, int* __restrict__ ucounts) {
    for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < L.N; n += gridDim.x * blockDim.x) {
        const int u = __ldg(L.counts + n), next = u > L.S1 ? __ldg(L.meta1 + (size_t)n * L.H1 + 1) : 0;
        int lo = 0, hi = u;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (__ldg(hex_col_word(L, n, next, mid)) - 1 < n) lo = mid + 1;
            else hi = mid;
        }
        ucounts[n] = u - lo;
    }
}

template <int kMode>
cudaError_t launch_mode(const ListLayout& L, const HexRows& h, const int* ucounts, const int* row_ptr, int* col_idx,
                        double* values, long long capacity, cudaStream_t s) {
    static DeviceCache cache;
    const size_t smem = sizeof(WriteHexCta);
    int per_sm = 0;
    const cudaError_t err = per_device(cache, [&](int& v) {
        cudaError_t e =
            cudaFuncSetAttribute(k_write_hex20<kMode>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (!e) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, k_write_hex20<kMode>, kWriteThreads, smem);
        return e;
    }, per_sm);
    if (err) return err;
    const long long want = ((long long)L.N + kWriteWarps - 1) / kWriteWarps;
    const int grid = (int)std::min<long long>(want, (long long)per_sm * sm_count());
    k_write_hex20<kMode><<<grid, kWriteThreads, smem, s>>>(L, h, ucounts, row_ptr, col_idx, values, capacity);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_count_upper_hex20(const ListLayout& L, int* ucounts, cudaStream_t s) {
    const int grid = (int)std::min<long long>(((long long)L.N + 255) / 256, (long long)sm_count() * 8);
    k_count_upper_hex20<<<grid, 256, 0, s>>>(L, ucounts);
    return cudaGetLastError();
}

cudaError_t launch_write_hex20(const ListLayout& L, const HexRows& h, int mode, const int* ucounts, const int* row_ptr,
                               int* col_idx, double* values, long long capacity, cudaStream_t s) {
    if (mode == kOutBsr) return launch_mode<kOutBsr>(L, h, ucounts, row_ptr, col_idx, values, capacity, s);
    if (mode == kOutUpper) return launch_mode<kOutUpper>(L, h, ucounts, row_ptr, col_idx, values, capacity, s);
    return launch_mode<kOutCsr>(L, h, ucounts, row_ptr, col_idx, values, capacity, s);
}

}  // namespace fem
