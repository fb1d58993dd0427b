// List -> CSR consolidation: per-row counts -> device scan -> row_ptr, then a
// per-row sort and coalesced write of col_idx / values.
//
// Replaces both the reference's host pattern build (buildCSRStructure,
// ALLS_Quad2D_Assembly_Accuracy_Analysis.cu:605-645; buildCSRStructureHex20,
// ALLS_Hex20_3D_Assembly_Performance.cu:364-392) and its convert kernels
// (convertALLStoCSRKernel, Q4A:471-501; ...FixedArray, H20:259-278), which walk
// each row's list and binary-search the host-built col_ind.
//
// The scatter inserts every column once per row and counts the entries of each
// row node in counts[n], so the CSR layout is known before any list is read:
//   k_tile_entries per tile of kRowTile nodes: sum of the nodes' entries
//   k_row_ptr      per tile: the sums of the tiles before it and a block scan
//                  of the counts -> row_ptr of all dpn rows; nnz, capacity check
//   k_write_sorted_2d  2-D CSR: the scatter's rows are sorted, so this copies
//                  each node's blocks into its two CSR rows
//   k_write_hex20  Hex20: the rows are sorted, their values summed from the
//                  elements' Ke as they are written (write_hex20.cu)
//   k_write        the other 2-D forms: a group of G lanes per row node: gather the node's non-empty
//                  hashed slots as 64-bit keys (col << 32 | slot), bitonic sort
//                  across the group, then write each dof row's entries
//                  (col*dpn + b, block value) with consecutive lanes on
//                  consecutive entries. Rows longer than the group's sort
//                  capacity take an exact slow path.
// Every dof row of node n holds {c*dpn + b : c in adj(n)} in increasing order,
// which is the reference's pattern. The same pass can write the node-block
// (BSR) form instead: one block row per node, the sorted column nodes and
// their dpn x dpn blocks; or the upper triangle only (columns >= row, the
// symmetric storage a Cholesky or symmetric solver reads): k_count_upper
// counts each node's columns >= the node, the scan and row pointers use those
// counts, and k_write keeps the tail of each sorted row.
#include <algorithm>

#include "consolidate.cuh"

namespace fem {
namespace {

template <int DPN, int kMode>
__global__ void __launch_bounds__(kScanThreads) k_tile_entries(const int* __restrict__ counts, int N,
                                                               long long* __restrict__ tile_sums) {
    __shared__ long long s_warp[kScanThreads / 32 + 1];
    tile_entries<DPN, kMode>(counts, N, tile_sums, blockIdx.x, s_warp);
}

template <int DPN, int kMode>
__global__ void __launch_bounds__(kScanThreads) k_row_ptr(const int* __restrict__ counts, int N,
                                                          const long long* __restrict__ tile_sums,
                                                          int* __restrict__ row_ptr, DevInfo* info,
                                                          long long capacity) {
    __shared__ RowPtrSmem sm;
    row_ptr_rows<DPN, kMode>(counts, N, tile_sums, row_ptr, info, capacity, blockIdx.x, gridDim.x, sm);
}

template <int G, int KPL, int kMode>
__global__ void __launch_bounds__(kBlockThreads, FEM_WRITE_MIN_CTAS_2D)
    k_write(ListLayout L, const int* __restrict__ row_ptr, int* __restrict__ col_idx, double* __restrict__ values,
            long long capacity, const int* __restrict__ ucounts) {
    constexpr int NPB = kBlockThreads / G;  // nodes per batch
    __shared__ WriteSmem<G, KPL> sm;
    write_batches<G, KPL, kMode>(L, row_ptr, col_idx, values, capacity, ucounts, (long long)blockIdx.x * NPB,
                                      (long long)gridDim.x * NPB, L.N, sm);
}

__global__ void __launch_bounds__(kBlockThreads) k_write_sorted_2d(ListLayout L, const int* __restrict__ row_ptr,
                                                                   int* __restrict__ col_idx,
                                                                   double* __restrict__ values, long long capacity) {
    __shared__ int s_stat[2 * (kBlockThreads / 32)];
    write_sorted_2d(L, row_ptr, col_idx, values, capacity, blockIdx.x, gridDim.x, s_stat);
}

// Persistent grid of k_write: the CTAs that fit on the GPU at once.
template <int G, int KPL, int kMode>
long long write_grid(long long batches) {
    static DeviceCache cache;
    int per_sm = 0;
    if (per_device(cache, [](int& v) {
            return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, k_write<G, KPL, kMode>, kBlockThreads, 0);
        }, per_sm))
        per_sm = 1;
    return std::max<long long>(1, std::min<long long>(batches, (long long)per_sm * sm_count()));
}

// counts: list columns per node (kOutUpper: columns >= the node); capacity in
// scalar entries (BSR: blocks * dpn^2).
template <int DPN, int kMode>
cudaError_t launch_mode(const ListLayout& L, const HexRows& hex, const int* counts, int* row_ptr, int* col_idx,
                        double* values, long long capacity, long long* tile_sums, cudaStream_t s) {
    const int tiles = row_tiles(L.N);
    if (L.N <= kSmallNodes) tile_sums = nullptr;
    else k_tile_entries<DPN, kMode><<<tiles, kScanThreads, 0, s>>>(counts, L.N, tile_sums);
    k_row_ptr<DPN, kMode><<<tiles, kScanThreads, 0, s>>>(counts, L.N, tile_sums, row_ptr, L.info, capacity);
    if (capacity <= 0) return cudaGetLastError();
    if constexpr (DPN == 3) {
        return launch_write_hex20(L, hex, kMode, counts, row_ptr, col_idx, values, capacity, s);
    } else {
        if (kMode == kOutCsr && wide_outputs(col_idx, values)) {
            static DeviceCache cache;
            int per_sm = 0;
            if (per_device(cache, [](int& v) {
                    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, k_write_sorted_2d, kBlockThreads, 0);
                }, per_sm))
                per_sm = 1;
            constexpr int kNodes = kBlockThreads / 16 * kCopyNodes;
            const long long want = ((long long)L.N + kNodes - 1) / kNodes;
            const int grid = (int)std::min<long long>(want, (long long)per_sm * sm_count());
            k_write_sorted_2d<<<grid, kBlockThreads, 0, s>>>(L, row_ptr, col_idx, values, capacity);
        } else {
            constexpr int G = 8, NPB = kBlockThreads / G;
            const long long batches = ((long long)L.N + NPB - 1) / NPB;
            k_write<G, 2, kMode><<<(int)write_grid<G, 2, kMode>(batches), kBlockThreads, 0, s>>>(
                L, row_ptr, col_idx, values, capacity, counts);
        }
        return cudaGetLastError();
    }
}

}  // namespace

cudaError_t launch_consolidate(const ListLayout& L, int dpn, const HexRows& hex, int* row_ptr, int* col_idx,
                               double* values, long long capacity, long long* tile_sums, cudaStream_t s) {
    if (dpn == 3) return launch_mode<3, kOutCsr>(L, hex, L.counts, row_ptr, col_idx, values, capacity, tile_sums, s);
    return launch_mode<2, kOutCsr>(L, hex, L.counts, row_ptr, col_idx, values, capacity, tile_sums, s);
}

cudaError_t launch_consolidate_upper(const ListLayout& L, int dpn, const HexRows& hex, int* ucounts, int* row_ptr,
                                     int* col_idx, double* values, long long capacity, long long* tile_sums,
                                     cudaStream_t s) {
    if (dpn == 3) {
        const cudaError_t err = launch_count_upper_hex20(L, ucounts, s);
        if (err) return err;
        return launch_mode<3, kOutUpper>(L, hex, ucounts, row_ptr, col_idx, values, capacity, tile_sums, s);
    }
    constexpr int G = 8, NPB = kBlockThreads / G;
    const long long batches = ((long long)L.N + NPB - 1) / NPB;
    const int grid = (int)std::max<long long>(1, std::min<long long>(batches, (long long)sm_count() * 8));
    k_count_upper<G><<<grid, kBlockThreads, 0, s>>>(L, ucounts);
    return launch_mode<2, kOutUpper>(L, hex, ucounts, row_ptr, col_idx, values, capacity, tile_sums, s);
}

cudaError_t launch_consolidate_bsr(const ListLayout& L, int dpn, const HexRows& hex, int* block_row_ptr,
                                   int* block_col_idx, double* block_values, long long capacity_blocks,
                                   long long* tile_sums, cudaStream_t s) {
    const long long cap = capacity_blocks * dpn * dpn;
    if (dpn == 3)
        return launch_mode<3, kOutBsr>(L, hex, L.counts, block_row_ptr, block_col_idx, block_values, cap, tile_sums, s);
    return launch_mode<2, kOutBsr>(L, hex, L.counts, block_row_ptr, block_col_idx, block_values, cap, tile_sums, s);
}

}  // namespace fem
