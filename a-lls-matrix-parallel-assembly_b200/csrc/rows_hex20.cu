// Launches of the Hex20 row-list kernels (rows_hex20.cuh).
#include <algorithm>

#include "rows_hex20.cuh"

namespace fem {
namespace {

__global__ void __launch_bounds__(kOccThreads) k_occ_count(MeshView m, HexRows h, int* __restrict__ cnt, DevInfo* info) {
    occ_count(m, h, cnt, info, blockIdx.x, gridDim.x);
}

__global__ void __launch_bounds__(kScanThreads) k_occ_sums(const int* __restrict__ cnt, int N,
                                                           long long* __restrict__ tiles) {
    __shared__ long long s_warp[kScanThreads / 32 + 1];
    occ_sums(cnt, N, tiles, blockIdx.x, s_warp);
}

__global__ void __launch_bounds__(kScanThreads) k_occ_offsets(const int* __restrict__ cnt, int N,
                                                              const long long* __restrict__ tiles,
                                                              int* __restrict__ off, DevInfo* info) {
    __shared__ OccSmem sm;
    occ_offsets(cnt, N, tiles, off, info, blockIdx.x, gridDim.x, sm);
}

__global__ void __launch_bounds__(kOccThreads) k_occ_fill(MeshView m, HexRows h) {
    occ_fill(m, h, blockIdx.x, gridDim.x);
}

__global__ void __launch_bounds__(kHexRowThreads, FEM_HEXR_CTAS)
    k_rows_hex20(const int* __restrict__ conn, ListLayout L, HexRows h, int* __restrict__ queue) {
    __shared__ HexRowSmem s_row[kHexRowWarps];
    rows_hex20(conn, L, h, queue, blockIdx.x, gridDim.x, s_row);
}

__global__ void __launch_bounds__(32) k_wide_rows_hex20(const int* __restrict__ conn, ListLayout L, HexRows h,
                                                        const int* __restrict__ queue) {
    __shared__ int s_uniq[kWideElems * 20];
    wide_rows_hex20(conn, L, h, queue, blockIdx.x, gridDim.x, s_uniq);
}

__global__ void __launch_bounds__(kHexRowThreads) k_long_rows_hex20(const int* __restrict__ conn, ListLayout L,
                                                                    HexRows h, const int* __restrict__ queue) {
    long_rows_hex20(conn, L, h, queue, blockIdx.x, gridDim.x);
}

}  // namespace

cudaError_t launch_occurrences(const MeshView& m, const ListLayout& L, const HexRows& h, int* cnt, long long* tiles,
                               cudaStream_t s) {
    const cudaError_t err = cudaMemsetAsync(cnt, 0, (size_t)m.N * sizeof(int), s);
    if (err) return err;
    const int ntiles = row_tiles(m.N), sms = sm_count();
    auto blocks = [&](long long work, int per_sm) {
        return (int)std::min<long long>((work + kOccThreads - 1) / kOccThreads, (long long)sms * per_sm);
    };
    if (m.E_count > 0) k_occ_count<<<blocks(m.E_count, 8), kOccThreads, 0, s>>>(m, h, cnt, L.info);
    k_occ_sums<<<ntiles, kScanThreads, 0, s>>>(cnt, m.N, tiles);
    k_occ_offsets<<<ntiles, kScanThreads, 0, s>>>(cnt, m.N, tiles, h.off, L.info);
    if (m.E_count > 0) k_occ_fill<<<blocks(20ll * m.E_count, 16), kOccThreads, 0, s>>>(m, h);
    return cudaGetLastError();
}

cudaError_t launch_rows_hex20(const MeshView& m, const ListLayout& L, const HexRows& h, int* queue, cudaStream_t s) {
    static DeviceCache cache;
    int per_sm = 0;
    const cudaError_t err = per_device(cache, [](int& v) {
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, k_rows_hex20, kHexRowThreads, 0);
    }, per_sm);
    if (err) return err;
    const long long want = ((long long)L.N + kHexRowWarps - 1) / kHexRowWarps;
    k_rows_hex20<<<(int)std::min<long long>(want, (long long)per_sm * sm_count()), kHexRowThreads, 0, s>>>(
        m.conn, L, h, queue);
    const int few = (int)std::min<long long>(L.N, 4 * sm_count());
    k_wide_rows_hex20<<<few, 32, 0, s>>>(m.conn, L, h, queue);
    k_long_rows_hex20<<<std::min(few, sm_count()), kHexRowThreads, 0, s>>>(m.conn, L, h, queue);
    return cudaGetLastError();
}

}  // namespace fem
