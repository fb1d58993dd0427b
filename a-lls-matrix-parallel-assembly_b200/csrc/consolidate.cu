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

// Entries of a node with c list columns (kOutUpper: c columns >= the node).
template <int DPN, int kMode>
__device__ __forceinline__ long long node_entries(int c) {
    return kMode == kOutUpper ? upper_node_entries<DPN>(c) : (long long)DPN * DPN * c;
}

// Entries of each tile of kRowTile nodes.
template <int DPN, int kMode>
__global__ void __launch_bounds__(kScanThreads) k_tile_entries(const int* __restrict__ counts, int N,
                                                               long long* __restrict__ tile_sums) {
    __shared__ long long s_warp[kScanThreads / 32 + 1];
    long long sum = 0;
#pragma unroll
    for (int i = 0; i < kRowTile / kScanThreads; i++) {
        const long long n = (long long)blockIdx.x * kRowTile + i * kScanThreads + threadIdx.x;
        if (n < N) sum += node_entries<DPN, kMode>(__ldg(counts + n));
    }
    long long total;
    block_exclusive_scan(sum, s_warp, total);
    if (threadIdx.x == 0) tile_sums[blockIdx.x] = total;
}

// row_ptr of a tile's rows (kOutBsr: block rows). Each CTA sums the tiles
// before its own itself (a few loads per thread: no launch in between), and
// writes its row pointers with consecutive threads on consecutive rows. The
// last CTA, which knows the total, clears what a consolidation pass owns in
// the info word (so the pass can be re-run on the same lists) and sets nnz.
template <int DPN, int kMode>
__global__ void __launch_bounds__(kScanThreads) k_row_ptr(const int* __restrict__ counts, int N,
                                                          const long long* __restrict__ tile_sums,
                                                          int* __restrict__ row_ptr, DevInfo* info,
                                                          long long capacity) {
    constexpr int kItems = kRowTile / kScanThreads, B = DPN * DPN;
    __shared__ long long s_warp[kScanThreads / 32 + 1];
    __shared__ int s_off[kRowTile], s_cnt[kRowTile];
    const int tid = threadIdx.x, tile = blockIdx.x;
    const long long first = (long long)tile * kRowTile;
#pragma unroll
    for (int i = 0; i < kItems; i++) {
        const long long n = first + i * kScanThreads + tid;
        s_cnt[i * kScanThreads + tid] = n < N ? __ldg(counts + n) : 0;
    }
    long long before = 0;
    for (int t = tid; t < tile; t += kScanThreads) before += __ldg(tile_sums + t);
    long long base;
    block_exclusive_scan(before, s_warp, base);
    long long sum = 0;
#pragma unroll
    for (int i = 0; i < kItems; i++) sum += node_entries<DPN, kMode>(s_cnt[tid * kItems + i]);
    long long total;
    long long off = block_exclusive_scan(sum, s_warp, total);
#pragma unroll
    for (int i = 0; i < kItems; i++) {
        s_off[tid * kItems + i] = (int)off;
        off += node_entries<DPN, kMode>(s_cnt[tid * kItems + i]);
    }
    __syncthreads();
    constexpr int R = kMode == kOutBsr ? 1 : DPN;  // rows per node
    const int rows = R * (int)min((long long)kRowTile, (long long)N - first);
    for (int r = tid; r < rows; r += kScanThreads) {
        const int i = r / R, a = r - i * R, c = s_cnt[i];
        long long p = base + s_off[i];
        if (kMode == kOutBsr) {
            p /= B;
        } else if (kMode == kOutUpper) {
#pragma unroll
            for (int k = 0; k < DPN - 1; k++) p += k < a ? upper_row_len<DPN>(c, k) : 0;
        } else {
            p += (long long)a * DPN * c;
        }
        row_ptr[first * R + r] = (int)p;
    }
    if (tile == gridDim.x - 1 && tid == 0) {
        constexpr int kOwned = (1 << FEM_ERR_CAPACITY) | (1 << FEM_ERR_RANGE) | (1 << FEM_ERR_INTERNAL);
        const long long nnz = base + total;
        int bits = info->status_bits & ~kOwned;
        if (nnz > 0x7FFFFFFFll) bits |= 1 << FEM_ERR_RANGE;
        if (nnz > capacity) bits |= 1 << FEM_ERR_CAPACITY;
        info->status_bits = bits;
        info->nnz = nnz;
        info->list_entries = 0;
        info->max_row_entries = 0;
        info->ticket = 0;
        row_ptr[(long long)N * R] = (int)(nnz / (kMode == kOutBsr ? B : 1));
    }
}

template <int DPN, int G, int KPL, int kMode>
__global__ void __launch_bounds__(kBlockThreads, DPN == 2 ? FEM_WRITE_MIN_CTAS_2D : FEM_WRITE_MIN_CTAS_3D)
    k_write(ListLayout L, const int* __restrict__ row_ptr, int* __restrict__ col_idx, double* __restrict__ values,
            long long capacity, const int* __restrict__ ucounts) {
    constexpr int NPB = kBlockThreads / G;  // nodes per batch
    __shared__ WriteSmem<DPN, G, KPL> sm;
    write_batches<DPN, G, KPL, kMode>(L, row_ptr, col_idx, values, capacity, ucounts, (long long)blockIdx.x * NPB,
                                      (long long)gridDim.x * NPB, L.N, sm);
}

// CSR of the 2-D lists whose rows the scatter left sorted (kRowSorted): 16
// lanes per node, lane 2k + i on row i of block k. A lane moves 16 bytes of
// values (a warp's loads are consecutive, its stores two runs per node) and 8
// bytes of columns; four nodes of a group are in flight. Hashed rows (fans)
// take the exact slow path.
constexpr int kCopyNodes = 4;
__global__ void __launch_bounds__(kBlockThreads) k_write_sorted_2d(ListLayout L, const int* __restrict__ row_ptr,
                                                                   int* __restrict__ col_idx,
                                                                   double* __restrict__ values, long long capacity) {
    constexpr int G = 16, NPB = kBlockThreads / G;
    __shared__ int s_sum[kBlockThreads / 32], s_max[kBlockThreads / 32];
    if (__ldg(&L.info->nnz) > capacity) return;  // FEM_ERR_CAPACITY already raised; write nothing
    const int tid = threadIdx.x, grp = tid / G, lane = tid % G, i = lane & 1;
    const unsigned gmask = 0xFFFFu << (((tid & 31) / G) * G);
    int t_sum = 0, t_max = 0;
    for (long long nb = (long long)blockIdx.x * NPB * kCopyNodes; nb < L.N; nb += (long long)gridDim.x * NPB * kCopyNodes) {
        int base[kCopyNodes], u[kCopyNodes], head[kCopyNodes];
#pragma unroll
        for (int q = 0; q < kCopyNodes; q++) {
            const long long n = nb + q * NPB + grp;
            base[q] = u[q] = 0;
            head[q] = kRowSorted;
            if (n < L.N) {
                base[q] = __ldg(row_ptr + 2 * n);
                u[q] = (__ldg(row_ptr + 2 * n + 1) - base[q]) / 2;
                head[q] = __ldg(L.meta1 + n * (k2DSlots + 2));
            }
        }
        double2 v[kCopyNodes][2];  // blocks k = lane / 2 and, in rows of more than 8, k + 8
        int c[kCopyNodes][2];
#pragma unroll
        for (int q = 0; q < kCopyNodes; q++) {
            const long long n = nb + q * NPB + grp;
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int p = lane + h * G;
                if (head[q] == kRowSorted && p < 2 * u[q]) {
                    v[q][h] = __ldg(reinterpret_cast<const double2*>(L.vals + n * (k2DSlots * 4)) + p);
                    c[q][h] = __ldg(L.meta1 + n * (k2DSlots + 2) + 2 + (p >> 1));
                }
            }
        }
#pragma unroll
        for (int q = 0; q < kCopyNodes; q++) {
            const long long n = nb + q * NPB + grp;
            t_sum += u[q];
            t_max = max(t_max, u[q]);
            if (head[q] == kRowSorted) {
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int k = (lane + h * G) >> 1;
                    if (k < u[q]) {
                        const long long p = base[q] + 2ll * i * u[q] + 2 * k;
                        *reinterpret_cast<double2*>(values + p) = v[q][h];
                        *reinterpret_cast<int2*>(col_idx + p) = make_int2(2 * c[q][h] - 2, 2 * c[q][h] - 1);
                    }
                }
            } else {
                long_row_write<2, G>(L, (int)n, u[q], base[q], lane, gmask, col_idx, values);
            }
        }
    }
    // list statistics (one atomic pair per CTA)
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        t_max = max(t_max, __shfl_xor_sync(0xFFFFFFFFu, t_max, d));
        t_sum += __shfl_xor_sync(0xFFFFFFFFu, t_sum, d);
    }
    if ((tid & 31) == 0) {
        s_sum[tid >> 5] = t_sum;
        s_max[tid >> 5] = t_max;
    }
    __syncthreads();
    if (tid == 0) {
        for (int w = 1; w < kBlockThreads / 32; w++) {
            t_sum += s_sum[w];
            t_max = max(t_max, s_max[w]);
        }
        atomicAdd(reinterpret_cast<unsigned long long*>(&L.info->list_entries), (unsigned long long)(t_sum / G));
        atomicMax(&L.info->max_row_entries, t_max);
    }
}

// Persistent grid of k_write: the CTAs that fit on the GPU at once.
template <int DPN, int G, int KPL, int kMode>
long long write_grid(long long batches) {
    static DeviceCache cache;
    int per_sm = 0;
    if (per_device(cache, [](int& v) {
            return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, k_write<DPN, G, KPL, kMode>, kBlockThreads, 0);
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
    k_tile_entries<DPN, kMode><<<tiles, kScanThreads, 0, s>>>(counts, L.N, tile_sums);
    k_row_ptr<DPN, kMode><<<tiles, kScanThreads, 0, s>>>(counts, L.N, tile_sums, row_ptr, L.info, capacity);
    if (capacity <= 0) return cudaGetLastError();
    if constexpr (DPN == 3) {
        return launch_write_hex20(L, hex, kMode, counts, row_ptr, col_idx, values, capacity, s);
    } else {
        // the copy kernel's 16-byte value and 8-byte column stores need outputs aligned to them (row starts are
        // multiples of 4 entries); other outputs take k_write, which stores entry by entry
        const bool wide = reinterpret_cast<uintptr_t>(values) % 16 == 0 && reinterpret_cast<uintptr_t>(col_idx) % 8 == 0;
        if (kMode == kOutCsr && wide) {
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
            k_write<DPN, G, 2, kMode><<<(int)write_grid<DPN, G, 2, kMode>(batches), kBlockThreads, 0, s>>>(
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
