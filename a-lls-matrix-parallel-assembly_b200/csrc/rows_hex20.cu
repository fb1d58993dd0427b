// Launches of the Hex20 row-list kernels (rows_hex20.cuh).
#include <cooperative_groups.h>

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
                                                              int* __restrict__ off) {
    __shared__ OccSmem sm;
    occ_offsets(cnt, N, tiles, off, blockIdx.x, gridDim.x, sm);
}

__global__ void __launch_bounds__(kOccThreads) k_occ_fill(MeshView m, HexRows h) {
    occ_fill(m, h, blockIdx.x, gridDim.x);
}

__global__ void __launch_bounds__(kHexRowThreads, FEM_HEXR_CTAS)
    k_rows_hex20(const int* __restrict__ conn, ListLayout L, HexRows h, int* __restrict__ queue) {
    __shared__ HexRowSmem s_row[kHexRowWarps];
    rows_hex20(conn, L, h, queue, blockIdx.x, gridDim.x, s_row);
}

// Nodes with more than 8 elements: a warp each, or a CTA.
__global__ void __launch_bounds__(kHexRowThreads) k_long_rows_hex20(const int* __restrict__ conn, ListLayout L,
                                                                    HexRows h, const int* __restrict__ queue) {
    __shared__ union {
        int uniq[kHexRowWarps][kWideElems * 20];
        LongHexSmem longs;
    } sm;
    const int warp = threadIdx.x >> 5;
    wide_rows_hex20(conn, L, h, queue, blockIdx.x * kHexRowWarps + warp, gridDim.x * kHexRowWarps, sm.uniq[warp]);
    __syncthreads();
    long_rows_hex20(conn, L, h, queue, blockIdx.x, gridDim.x, sm.longs);
}

__global__ void __launch_bounds__(256) k_begin_hex20(ListLayout L, int* __restrict__ cnt) {
    lists_begin_hex20(L, cnt, blockIdx.x, gridDim.x);
}

// Everything up to the row lists of a small mesh (launch.h's kSmallNodes) in
// one cooperative launch: seven launches at about 4 us of the caller's time
// each become one and five grid barriers of 1 to 2 us.
static_assert(kOccThreads == kHexRowThreads && kScanThreads == kHexRowThreads, "one block shape");
__global__ void __launch_bounds__(kHexRowThreads, FEM_HEXR_CTAS)
    k_small_hex20(MeshView m, ListLayout L, HexRows h, int* __restrict__ cnt, int* __restrict__ queue) {
    __shared__ union Smem {
        HexRowSmem rows[kHexRowWarps];
        OccSmem occ;
        int uniq[kHexRowWarps][kWideElems * 20];
        LongHexSmem longs;
        __device__ Smem() {}
    } sm;
    const cooperative_groups::grid_group grid = cooperative_groups::this_grid();
    const int block = blockIdx.x, nblocks = gridDim.x, warp = threadIdx.x >> 5, tiles = (L.N + kRowTile - 1) / kRowTile;
    lists_begin_hex20(L, cnt, block, nblocks);
    grid.sync();
    occ_count(m, h, cnt, L.info, block, nblocks);
    grid.sync();
    for (int t = block; t < tiles; t += nblocks) occ_offsets(cnt, L.N, nullptr, h.off, t, tiles, sm.occ);
    grid.sync();
    occ_fill(m, h, block, nblocks);
    grid.sync();
    rows_hex20(m.conn, L, h, queue, block, nblocks, sm.rows);
    grid.sync();
    wide_rows_hex20(m.conn, L, h, queue, block * kHexRowWarps + warp, nblocks * kHexRowWarps, sm.uniq[warp]);
    __syncthreads();
    long_rows_hex20(m.conn, L, h, queue, block, nblocks, sm.longs);
}

}  // namespace

static cudaError_t launch_small(const MeshView& m, const ListLayout& L, const HexRows& h, int* cnt, int* queue,
                                cudaStream_t s) {
    static DeviceCache cache;
    int per_sm = 0;
    const cudaError_t err = per_device(cache, [](int& v) {
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, k_small_hex20, kHexRowThreads, 0);
    }, per_sm);
    if (err) return err;
    const long long want = ((long long)m.N + kHexRowWarps - 1) / kHexRowWarps;
    const int grid = (int)std::min<long long>(want, (long long)per_sm * sm_count());
    MeshView mv = m;
    ListLayout lv = L;
    HexRows hv = h;
    void* args[] = {&mv, &lv, &hv, &cnt, &queue};
    return cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(k_small_hex20), dim3(grid), dim3(kHexRowThreads), args,
                                       0, s);
}

cudaError_t launch_rows_hex20(const MeshView& m, const ListLayout& L, const HexRows& h, int* cnt, long long* tiles,
                              int* queue, cudaStream_t s) {
    if (m.N <= kSmallNodes && m.E_count <= kSmallNodes) return launch_small(m, L, h, cnt, queue, s);
    static DeviceCache cache;
    int per_sm = 0;
    const cudaError_t err = per_device(cache, [](int& v) {
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, k_rows_hex20, kHexRowThreads, 0);
    }, per_sm);
    if (err) return err;
    const int ntiles = row_tiles(m.N), sms = sm_count();
    auto blocks = [&](long long work, int threads, int most) {
        return (int)std::min<long long>((work + threads - 1) / threads, (long long)sms * most);
    };
    k_begin_hex20<<<blocks(m.N, 1024, 4), 256, 0, s>>>(L, cnt);
    if (m.E_count > 0) k_occ_count<<<blocks(m.E_count, kOccThreads, 8), kOccThreads, 0, s>>>(m, h, cnt, L.info);
    k_occ_sums<<<ntiles, kScanThreads, 0, s>>>(cnt, m.N, tiles);
    k_occ_offsets<<<ntiles, kScanThreads, 0, s>>>(cnt, m.N, tiles, h.off);
    if (m.E_count > 0) k_occ_fill<<<blocks(20ll * m.E_count, kOccThreads, 16), kOccThreads, 0, s>>>(m, h);
    k_rows_hex20<<<blocks(m.N, kHexRowWarps, per_sm), kHexRowThreads, 0, s>>>(m.conn, L, h, queue);
    k_long_rows_hex20<<<blocks(m.N, kHexRowWarps, 1), kHexRowThreads, 0, s>>>(m.conn, L, h, queue);
    return cudaGetLastError();
}

}  // namespace fem
