// Device code of the list -> CSR consolidation (consolidate.cu), shared with
// the batch's merged launches (batched.cu): tile-level scan steps and the
// sorted write of a range of row-node batches. See consolidate.cu for the
// algorithm and the reference steps it replaces.
#pragma once

#include "launch.h"
#include "scan.cuh"

namespace fem {
namespace {

constexpr unsigned long long kEmptyKey = ~0ull;

__device__ __forceinline__ unsigned long long shfl_xor_u64(unsigned long long v, int m) {
    unsigned lo = (unsigned)v, hi = (unsigned)(v >> 32);
    lo = __shfl_xor_sync(0xFFFFFFFFu, lo, m);
    hi = __shfl_xor_sync(0xFFFFFFFFu, hi, m);
    return ((unsigned long long)hi << 32) | lo;
}

template <int G>
__device__ __forceinline__ unsigned group_mask(int grp_in_warp) {
    return G == 32 ? 0xFFFFFFFFu : (((1u << G) - 1u) << (grp_in_warp * G));
}

// Upper-triangle CSR: entries of node n's dof rows when u of its column nodes
// are >= n (the node itself among them): row a holds (dpn - a) entries of the
// diagonal block and dpn of each of the u - 1 later blocks.
template <int DPN>
__device__ __forceinline__ long long upper_row_len(int u, int a) {
    return u > 0 ? (long long)(u - 1) * DPN + (DPN - a) : 0;
}
template <int DPN>
__device__ __forceinline__ long long upper_node_entries(int u) {
    return u > 0 ? (long long)(u - 1) * DPN * DPN + DPN * (DPN + 1) / 2 : 0;
}

// Columns >= n in node n's list (a group of G lanes per node).
template <int G>
__global__ void __launch_bounds__(kBlockThreads) k_count_upper(ListLayout L, int* __restrict__ ucounts) {
    constexpr int NPB = kBlockThreads / G;
    const int tid = threadIdx.x, grp = tid / G, glane = tid % G;
    const unsigned gmask = group_mask<G>((tid & 31) / G);
    for (long long nb = (long long)blockIdx.x * NPB; nb < L.N; nb += (long long)gridDim.x * NPB) {
        const int n = (int)(nb + grp);
        int cnt = 0;
        if (n < L.N) {
            int c = n;
            for (int step = 0; step < kMaxChainSteps; step++) {
                const int* meta = chunk_meta(L, c);
                const int cap = chunk_cap(L, c);
                const int next = __ldg(meta + 1);
                for (int s = glane; s < cap; s += G) {
                    const int col = __ldg(meta + 2 + s) - 1;
                    cnt += col >= n;
                }
                if (next == 0) break;
                c = next - 1;
            }
        }
#pragma unroll
        for (int d = G / 2; d > 0; d >>= 1) cnt += __shfl_xor_sync(gmask, cnt, d);
        if (n < L.N && glane == 0) ucounts[n] = cnt;
    }
}

// Ascending bitonic sort of G*KPL keys held as keys[i] at position lane*KPL + i
// of a G-lane group. Every lane of the warp must call it.
template <int G, int KPL>
__device__ __forceinline__ void group_sort(unsigned long long (&keys)[KPL], int glane) {
    constexpr int N = G * KPL;
#pragma unroll
    for (int size = 2; size <= N; size <<= 1) {
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            if (stride >= KPL) {
                const int lstride = stride / KPL;
#pragma unroll
                for (int i = 0; i < KPL; i++) {
                    const int pos = glane * KPL + i;
                    const unsigned long long other = shfl_xor_u64(keys[i], lstride);
                    const bool up = (pos & size) == 0;
                    const bool lower = (pos & stride) == 0;
                    const unsigned long long mn = keys[i] < other ? keys[i] : other;
                    const unsigned long long mx = keys[i] < other ? other : keys[i];
                    keys[i] = (lower == up) ? mn : mx;
                }
            } else {
#pragma unroll
                for (int i = 0; i < KPL; i++) {
                    const int j = i ^ stride;
                    if (j > i) {
                        const int pos = glane * KPL + i;
                        const bool up = (pos & size) == 0;
                        const unsigned long long a = keys[i], b = keys[j];
                        const bool swap = up ? (a > b) : (a < b);
                        keys[i] = swap ? b : a;
                        keys[j] = swap ? a : b;
                    }
                }
            }
        }
    }
}

// Slow path for a row with more entries than a group can sort at once (a node
// of unusually high degree): iterated minimum extraction over the row's chunk
// chain. O(u * entries / G) work, exact for any row length.
template <int G>
__device__ int long_row_next_col(const ListLayout& L, int n, int after, int glane, unsigned mask) {
    int best = 0x7FFFFFFF;
    int c = n;
    for (int step = 0; step < kMaxChainSteps; step++) {
        const int* meta = chunk_meta(L, c);
        const int cap = chunk_cap(L, c);
        const int next = __ldg(meta + 1);
        for (int s = glane; s < cap; s += G) {
            const int col = __ldg(meta + 2 + s) - 1;
            if (col > after && col < best) best = col;
        }
        if (next == 0) break;
        c = next - 1;
    }
#pragma unroll
    for (int d = G / 2; d > 0; d >>= 1) best = min(best, __shfl_xor_sync(mask, best, d));
    return best;
}

// Returns whether the row has u columns.
template <int G>
__device__ bool long_row_write(const ListLayout& L, int n, int u, long long base, int glane, unsigned mask,
                               int* __restrict__ col_idx, double* __restrict__ values) {
    constexpr int DPN = 2, B = DPN * DPN;
    int last = -1;
    for (int k = 0;; k++) {
        const int col = long_row_next_col<G>(L, n, last, glane, mask);
        if (k == u || col == 0x7FFFFFFF) return k == u && col == 0x7FFFFFFF;
        last = col;
        double sum[B];
#pragma unroll
        for (int v = 0; v < B; v++) sum[v] = 0.0;
        int c = n;
        for (int step = 0; step < kMaxChainSteps; step++) {
            const int* meta = chunk_meta(L, c);
            const int cap = chunk_cap(L, c);
            const int next = __ldg(meta + 1);
            for (int s = glane; s < cap; s += G) {
                if (__ldg(meta + 2 + s) - 1 == col) {
                    const double* p = L.vals + (size_t)slot_gid(L, c, s) * B;
#pragma unroll
                    for (int v = 0; v < B; v++) sum[v] += __ldg(p + v);
                }
            }
            if (next == 0) break;
            c = next - 1;
        }
#pragma unroll
        for (int v = 0; v < B; v++) {
#pragma unroll
            for (int d = G / 2; d > 0; d >>= 1) sum[v] += __shfl_xor_sync(mask, sum[v], d);
        }
        if (glane == 0) {
#pragma unroll
            for (int a = 0; a < DPN; a++)
#pragma unroll
                for (int b = 0; b < DPN; b++) {
                    const long long pos = base + (long long)a * DPN * u + (long long)k * DPN + b;
                    col_idx[pos] = col * DPN + b;
                    values[pos] = sum[a * DPN + b];
                }
        }
    }
}

// Long-row slow path of the block (BSR) output: block k of the node's block row.
template <int G>
__device__ void long_row_write_bsr(const ListLayout& L, int n, int u, long long base, int glane, unsigned mask,
                                   int* __restrict__ col_idx, double* __restrict__ values) {
    constexpr int DPN = 2, B = DPN * DPN;
    int last = -1;
    for (int k = 0; k < u; k++) {
        const int col = long_row_next_col<G>(L, n, last, glane, mask);
        last = col;
        double sum[B];
#pragma unroll
        for (int v = 0; v < B; v++) sum[v] = 0.0;
        int c = n;
        for (int step = 0; step < kMaxChainSteps; step++) {
            const int* meta = chunk_meta(L, c);
            const int cap = chunk_cap(L, c);
            const int next = __ldg(meta + 1);
            for (int s = glane; s < cap; s += G) {
                if (__ldg(meta + 2 + s) - 1 == col) {
                    const double* p = L.vals + (size_t)slot_gid(L, c, s) * B;
#pragma unroll
                    for (int v = 0; v < B; v++) sum[v] += __ldg(p + v);
                }
            }
            if (next == 0) break;
            c = next - 1;
        }
#pragma unroll
        for (int v = 0; v < B; v++) {
#pragma unroll
            for (int d = G / 2; d > 0; d >>= 1) sum[v] += __shfl_xor_sync(mask, sum[v], d);
        }
        if (glane == 0) {
            col_idx[base + k] = col;
#pragma unroll
            for (int v = 0; v < B; v++) values[(base + k) * B + v] = sum[v];
        }
    }
}

// Long-row slow path of the upper-triangle output: the node's u column nodes
// >= n in increasing order (the first is n itself).
template <int G>
__device__ void long_row_write_upper(const ListLayout& L, int n, int u, const int* __restrict__ row_ptr, int glane,
                                     unsigned mask, int* __restrict__ col_idx, double* __restrict__ values) {
    constexpr int DPN = 2, B = DPN * DPN;
    int last = n - 1;
    for (int k = 0; k < u; k++) {
        const int col = long_row_next_col<G>(L, n, last, glane, mask);
        last = col;
        double sum[B];
#pragma unroll
        for (int v = 0; v < B; v++) sum[v] = 0.0;
        int c = n;
        for (int step = 0; step < kMaxChainSteps; step++) {
            const int* meta = chunk_meta(L, c);
            const int cap = chunk_cap(L, c);
            const int next = __ldg(meta + 1);
            for (int s = glane; s < cap; s += G) {
                if (__ldg(meta + 2 + s) - 1 == col) {
                    const double* p = L.vals + (size_t)slot_gid(L, c, s) * B;
#pragma unroll
                    for (int v = 0; v < B; v++) sum[v] += __ldg(p + v);
                }
            }
            if (next == 0) break;
            c = next - 1;
        }
#pragma unroll
        for (int v = 0; v < B; v++) {
#pragma unroll
            for (int d = G / 2; d > 0; d >>= 1) sum[v] += __shfl_xor_sync(mask, sum[v], d);
        }
        if (glane == 0) {
#pragma unroll
            for (int a = 0; a < DPN; a++) {
                const long long rbase = __ldg(row_ptr + (size_t)n * DPN + a);
#pragma unroll
                for (int b = 0; b < DPN; b++) {
                    if (k == 0 && b < a) continue;  // below the diagonal
                    const long long pos = k == 0 ? rbase + (b - a) : rbase + (DPN - a) + (long long)(k - 1) * DPN + b;
                    col_idx[pos] = col * DPN + b;
                    values[pos] = sum[a * DPN + b];
                }
            }
        }
    }
}

enum : int { kOutCsr = 0, kOutBsr = 1, kOutUpper = 2 };

// Whether the output is written: its entries fit the caller's buffers, and its row pointers (entries; kOutBsr: blocks)
// fit int32. Past either, FEM_ERR_CAPACITY / FEM_ERR_RANGE is raised already (row_ptr_rows) and nothing is stored: a
// wrapped row pointer would place rows in front of the buffers, whatever their capacity.
template <int DPN, int kMode>
__device__ __forceinline__ bool output_fits(const DevInfo* info, long long capacity) {
    constexpr long long kMost = 0x7FFFFFFFll * (kMode == kOutBsr ? DPN * DPN : 1);
    const long long nnz = __ldcg(&info->nnz);
    return nnz <= capacity && nnz <= kMost;
}

// Next link and slot words (kPre per lane of a G-lane group) of a node's first chunk.
template <int G, int kPre>
__device__ __forceinline__ void prefetch_first_chunk(const ListLayout& L, long long node, int glane, int (&w)[kPre],
                                                     int& next) {
    if (node < L.N) {
        const int* meta = chunk_meta(L, (int)node);
        next = __ldg(meta + 1);
#pragma unroll
        for (int q = 0; q < kPre; q++) {
            const int s = q * G + glane;
            w[q] = s < L.S1 ? __ldg(meta + 2 + s) : 0;
        }
    }
}

// Resident CTAs per SM the register budget of k_write is set for (build-time
// tuning knob, measured on B200).
#ifndef FEM_WRITE_MIN_CTAS_2D
#define FEM_WRITE_MIN_CTAS_2D 5
#endif

// Shared memory of the sorted write: each group's sort keys and the node's
// sorted 2x2 blocks, loaded together before the rows are written.
template <int G, int KPL>
struct WriteSmem {
    unsigned long long keys[kBlockThreads / G][G * KPL];
    double2 vals[kBlockThreads / G][G * KPL][2];
};

// The sorted write of the 2-D row nodes of batches nb = nb_first, nb_first +
// nb_stride, ... below nb_end (a batch: kBlockThreads / G consecutive nodes,
// one G-lane group each). Every thread of the CTA (kBlockThreads) calls it.
// kMode kOutBsr: block (BSR) output, one block row per node: block_col_idx =
// column node, block values dpn x dpn row-major; row_ptr is then the block row
// pointer. kOutUpper: the upper triangle in CSR (ucounts: columns >= n).
template <int G, int KPL, int kMode>
__device__ __forceinline__ void write_batches(const ListLayout& L, const int* __restrict__ row_ptr,
                                              int* __restrict__ col_idx, double* __restrict__ values,
                                              long long capacity, const int* __restrict__ ucounts, long long nb_first,
                                              long long nb_stride, long long nb_end, WriteSmem<G, KPL>& sm) {
    constexpr bool kBsr = kMode == kOutBsr;
    constexpr int NK = G * KPL;             // sort capacity per node
    constexpr int DPN = 2, B = DPN * DPN;
    constexpr int kPre = 16 / G;  // slot words of a node's first chunk per lane (14 slots)
    auto& s_keys = sm.keys;
    auto& s_vals = sm.vals;
    if (!output_fits<2, kMode>(L.info, capacity)) return;
    const int tid = threadIdx.x;
    const int grp = tid / G, glane = tid % G;
    const unsigned gmask = group_mask<G>((tid & 31) / G);
    const int gshift = G == 32 ? 0 : ((tid & 31) / G) * G;
    int t_sum = 0, t_max = 0;
    // the first chunk (next link and slot words) of the group's next node is
    // loaded while the current node is sorted and written
    int pre_w[kPre], pre_next = 0;
    prefetch_first_chunk<G, kPre>(L, nb_first + grp, glane, pre_w, pre_next);
    for (long long nb = nb_first; nb < nb_end; nb += nb_stride) {
        const int n = (int)(nb + grp);
        const bool valid = n < L.N;
        int u = 0;
        long long base = 0;
        if (valid) {
            if (kMode == kOutUpper) {
                u = __ldg(ucounts + n);  // columns >= n (the full row count is in L.counts)
            } else if (kBsr) {
                base = __ldg(row_ptr + n);
                u = __ldg(row_ptr + n + 1) - (int)base;
            } else {
                base = __ldg(row_ptr + (size_t)n * DPN);
                u = (__ldg(row_ptr + (size_t)n * DPN + 1) - (int)base) / DPN;
            }
        }
        // 1. gather the non-empty slots of the node's chunk chain (the first
        // chunk from the prefetched words)
        int T = 0;
        if (valid) {
#pragma unroll
            for (int q = 0; q < kPre; q++) {
                if (q * G < L.S1) {
                    const int s = q * G + glane;
                    const int col = s < L.S1 ? pre_w[q] : 0;
                    const unsigned used = (__ballot_sync(gmask, col != 0) >> gshift) & gmask >> gshift;
                    const int e = T + __popc(used & ((1u << glane) - 1u));
                    if (col != 0 && e < NK)
                        s_keys[grp][e] = ((unsigned long long)(unsigned)(col - 1) << 32) | slot_gid(L, n, s);
                    T += __popc(used);
                }
            }
            int next = pre_next;
            for (int step = 1; next != 0 && step < kMaxChainSteps; step++) {
                const int c = next - 1;
                const int* meta = chunk_meta(L, c);
                const int cap = chunk_cap(L, c);
                next = __ldg(meta + 1);
                for (int s0 = 0; s0 < cap; s0 += G) {
                    const int s = s0 + glane;
                    const int col = s < cap ? __ldg(meta + 2 + s) : 0;
                    const unsigned used = (__ballot_sync(gmask, col != 0) >> gshift) & gmask >> gshift;
                    const int e = T + __popc(used & ((1u << glane) - 1u));
                    if (col != 0 && e < NK)
                        s_keys[grp][e] = ((unsigned long long)(unsigned)(col - 1) << 32) | slot_gid(L, c, s);
                    T += __popc(used);
                }
            }
            const int expect = kMode == kOutUpper ? __ldg(L.counts + n) : u;
            if (glane == 0 && (T != expect || u > T)) raise_status(L.info, FEM_ERR_INTERNAL);
        }
        if (nb + nb_stride < nb_end) prefetch_first_chunk<G, kPre>(L, nb + nb_stride + grp, glane, pre_w, pre_next);
        t_sum += T;
        t_max = max(t_max, T);
        const bool long_row = T > NK;
        const int Ts = long_row ? 0 : min(T, kMode == kOutUpper ? T : u);
        __syncwarp();
        // 2. sort
        unsigned long long keys[KPL];
#pragma unroll
        for (int i = 0; i < KPL; i++) {
            const int p = glane * KPL + i;
            keys[i] = p < Ts ? s_keys[grp][p] : kEmptyKey;
        }
        group_sort<G, KPL>(keys, glane);
#pragma unroll
        for (int i = 0; i < KPL; i++) s_keys[grp][glane * KPL + i] = keys[i];
        __syncwarp();
        // all of the node's blocks in flight at once (two 16-byte loads each)
        for (int k = glane; k < Ts; k += G) {
            const double2* p = reinterpret_cast<const double2*>(L.vals + (size_t)(unsigned)s_keys[grp][k] * B);
            s_vals[grp][k][0] = __ldg(p);
            s_vals[grp][k][1] = __ldg(p + 1);
        }
        __syncwarp();
        // entry v of the node's k-th sorted block
        auto block_value = [&](int k, int v) { return reinterpret_cast<const double*>(&s_vals[grp][k][0])[v]; };
        // 3. write the dpn rows of the node (or its block row, or its upper rows)
        if (valid && kMode == kOutUpper) {
            if (long_row) {
                long_row_write_upper<G>(L, n, u, row_ptr, glane, gmask, col_idx, values);
            } else if (u > 0 && u <= Ts) {
                const int k0 = Ts - u;  // the sorted row's first column >= n (n itself)
                for (int a = 0; a < DPN; a++) {
                    const long long rbase = __ldg(row_ptr + (size_t)n * DPN + a);
                    const int len = (u - 1) * DPN + (DPN - a);
                    for (int r = glane; r < len; r += G) {
                        int k, b;
                        if (r < DPN - a) {
                            k = k0;
                            b = a + r;
                        } else {
                            const int q = r - (DPN - a);
                            k = k0 + 1 + q / DPN;
                            b = q - (q / DPN) * DPN;
                        }
                        const unsigned long long key = s_keys[grp][k];
                        col_idx[rbase + r] = (int)(key >> 32) * DPN + b;
                        values[rbase + r] = block_value(k, a * DPN + b);
                    }
                }
            }
        } else if (valid && kBsr) {
            if (long_row) {
                long_row_write_bsr<G>(L, n, u, base, glane, gmask, col_idx, values);
            } else {
                for (int k = glane; k < Ts; k += G) col_idx[base + k] = (int)(s_keys[grp][k] >> 32);
                for (int idx = glane; idx < Ts * B; idx += G) {
                    const int k = idx / B, v = idx - k * B;
                    values[base * B + idx] = block_value(k, v);
                }
            }
        } else if (valid) {
            if (long_row) {
                long_row_write<G>(L, n, u, base, glane, gmask, col_idx, values);
            } else {
                const int row_len = DPN * Ts;
                for (int a = 0; a < DPN; a++) {
                    const long long rbase = base + (long long)a * DPN * u;
                    for (int r = glane; r < row_len; r += G) {
                        const int k = r / DPN, b = r - k * DPN;
                        const unsigned long long key = s_keys[grp][k];
                        col_idx[rbase + r] = (int)(key >> 32) * DPN + b;
                        values[rbase + r] = block_value(k, a * DPN + b);
                    }
                }
            }
        }
        __syncwarp();
    }
    // list statistics (one atomic per warp)
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        t_max = max(t_max, __shfl_xor_sync(0xFFFFFFFFu, t_max, d));
        t_sum += __shfl_xor_sync(0xFFFFFFFFu, t_sum, d);
    }
    if ((tid & 31) == 0) {
        // every lane of a group counted the same rows: divide by G
        atomicAdd(reinterpret_cast<unsigned long long*>(&L.info->list_entries), (unsigned long long)(t_sum / G));
        atomicMax(&L.info->max_row_entries, t_max);
    }
}


// Entries of a node with c list columns (kOutUpper: c columns >= the node).
template <int DPN, int kMode>
__device__ __forceinline__ long long node_entries(int c) {
    return kMode == kOutUpper ? upper_node_entries<DPN>(c) : (long long)DPN * DPN * c;
}

// Entries of each tile of kRowTile nodes.
template <int DPN, int kMode>
__device__ __forceinline__ void tile_entries(const int* __restrict__ counts, int N, long long* __restrict__ tile_sums,
                                             int tile, long long* s_warp) {
    long long sum = 0;
#pragma unroll
    for (int i = 0; i < kRowTile / kScanThreads; i++) {
        const long long n = (long long)tile * kRowTile + i * kScanThreads + threadIdx.x;
        if (n < N) sum += node_entries<DPN, kMode>(__ldg(counts + n));
    }
    long long total;
    block_exclusive_scan(sum, s_warp, total);
    if (threadIdx.x == 0) tile_sums[tile] = total;
}

// row_ptr of a tile's rows (kOutBsr: block rows). Each CTA sums the tiles
// before its own itself (a few loads per thread: no launch in between), and
// writes its row pointers with consecutive threads on consecutive rows. The
// last CTA, which knows the total, clears what a consolidation pass owns in
// the info word (so the pass can be re-run on the same lists) and sets nnz.
struct RowPtrSmem {
    long long warp[kScanThreads / 32 + 1];
    int off[kRowTile], cnt[kRowTile];
};
template <int DPN, int kMode>
__device__ __forceinline__ void row_ptr_rows(const int* __restrict__ counts, int N,
                                             const long long* __restrict__ tile_sums, int* __restrict__ row_ptr,
                                             DevInfo* info, long long capacity, int tile, int ntiles, RowPtrSmem& sm) {
    constexpr int kItems = kRowTile / kScanThreads, B = DPN * DPN;
    long long* const s_warp = sm.warp;
    int* const s_off = sm.off;
    int* const s_cnt = sm.cnt;
    const int tid = threadIdx.x;
    const long long first = (long long)tile * kRowTile;
#pragma unroll
    for (int i = 0; i < kItems; i++) {
        const long long n = first + i * kScanThreads + tid;
        s_cnt[i * kScanThreads + tid] = n < N ? __ldg(counts + n) : 0;
    }
    long long before = 0;
    if (tile_sums) {
        for (int t = tid; t < tile; t += kScanThreads) before += __ldg(tile_sums + t);
    } else {  // a small mesh: the nodes before the tile
#pragma unroll 8
        for (int n = tid; n < (int)first; n += kScanThreads) before += node_entries<DPN, kMode>(__ldg(counts + n));
    }
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
    if (tile == ntiles - 1 && tid == 0) {
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
        info->done = 0;
        row_ptr[(long long)N * R] = (int)(nnz / (kMode == kOutBsr ? B : 1));
    }
}

// CSR of the 2-D lists whose rows the scatter left sorted (kRowSorted): 16
// lanes per node, lane 2k + i on row i of block k. A lane moves 16 bytes of
// values (a warp's loads are consecutive, its stores two runs per node) and 8
// bytes of columns; four nodes of a group are in flight. Hashed rows (fans)
// take the exact slow path, and so do rows whose header has another number of
// columns than the row pointers; a list without them raises FEM_ERR_INTERNAL.
constexpr int kCopyNodes = 4;
__device__ __forceinline__ void write_sorted_2d(const ListLayout& L, const int* __restrict__ row_ptr,
                                                int* __restrict__ col_idx, double* __restrict__ values,
                                                long long capacity, int block, int nblocks, int* s_stat) {
    constexpr int G = 16, NPB = kBlockThreads / G;
    int* const s_sum = s_stat;
    int* const s_max = s_stat + kBlockThreads / 32;
    if (!output_fits<2, kOutCsr>(L.info, capacity)) return;
    const int tid = threadIdx.x, grp = tid / G, lane = tid % G, i = lane & 1;
    const unsigned gmask = 0xFFFFu << (((tid & 31) / G) * G);
    int t_sum = 0, t_max = 0;
    int lowest = 1;  // lowest column word met; 0: a row whose list does not have the columns it is counted with
    for (long long nb = (long long)block * NPB * kCopyNodes; nb < L.N; nb += (long long)nblocks * NPB * kCopyNodes) {
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
                if (head[q] == kRowSorted + u[q] && p < 2 * u[q]) {
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
            if (head[q] == kRowSorted + u[q]) {
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int k = (lane + h * G) >> 1;
                    if (k < u[q]) {
                        lowest = min(lowest, c[q][h]);
                        const long long p = base[q] + 2ll * i * u[q] + 2 * k;
                        *reinterpret_cast<double2*>(values + p) = v[q][h];
                        *reinterpret_cast<int2*>(col_idx + p) = make_int2(2 * c[q][h] - 2, 2 * c[q][h] - 1);
                    }
                }
            } else {
                if (!long_row_write<G>(L, (int)n, u[q], base[q], lane, gmask, col_idx, values)) lowest = 0;
            }
        }
    }
    if (lowest <= 0) raise_status(L.info, FEM_ERR_INTERNAL);
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

}  // namespace
}  // namespace fem
