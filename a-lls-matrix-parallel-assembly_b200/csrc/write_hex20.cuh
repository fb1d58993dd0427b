// Device code of the Hex20 gather (write_hex20.cu, and the batch, batched.cu):
// row lists -> CSR, BSR or upper-triangle CSR, each row's element blocks
// are summed where they are written.
//
// Replaces the value half of assembleGlobalStiffnessKernelALLSFixedArray
// (ALLS_Hex20_3D_Assembly_Performance.cu:212-256, atomicAdd per entry) and
// convertALLStoCSRKernelFixedArray (H20:259-278). One warp per row node, the
// nodes taken by all CTAs together in an order that keeps neighbours close
// (launch_node_order), so that an element's Ke is read by its rows while it is
// in L2. The row's 3x3 blocks accumulate in shared memory (a window of kWindow
// columns at a time); for each of the node's occurrences (element e, position
// a) the lanes read the 20 blocks (a, b) of the packed Ke (180 doubles, a block
// below the diagonal from its transpose; the places come from a table) and add
// them at the ranks that the scatter recorded, one rank per lane handed out by
// shuffles, the next occurrence's loads in flight meanwhile. An element names a
// column node once, so the lanes' additions never meet; a repeated node's
// further blocks are added one by one. Then the rows leave with consecutive
// lanes on consecutive entries. No value is added atomically; a row's
// occurrences come in the order in which the scatter's counters dealt their
// places, so two runs differ in the sums' last bits.
//
// What bounds it: wavefronts of L1 and shared memory (six slab loads, table
// reads, sums read and written back per lane and occurrence: 88 % of the LSU
// data pipe at 32^3, DRAM 47 %). A 64^3 mesh has 4.0 GB of Ke to read and 6.7
// GB of CSR to write (1.6 ms at the measured copy rate). B200: 2.79 ms (4.02 ms with a fixed stride of nodes in
// their numbering, per-entry index arithmetic and no row headers in flight);
// the value pass into list blocks (stores and FP64 atomics) and the copy out of
// the lists that it replaces took 5.18 + 3.06 ms with the Ke computed inside.
// Streaming stores for the output measured the same (2.81 ms).
#pragma once

#include "consolidate.cuh"
#include "hex_rows.cuh"

namespace fem {
namespace {

// Warps per CTA and resident CTAs per SM: 24 warps in 191 KB of shared memory,
// which leaves 60 KB of L1 for the slabs that neighbouring rows share (64^3
// write: 2.79 ms; 3 x 8 warps in 207 KB 3.75, 2 x 14 in 218 KB 3.89, 2 x 10
// 2.90, 2 x 8 3.21 ms).
#ifndef FEM_HEXW_CTAS
#define FEM_HEXW_CTAS 2
#endif
#ifndef FEM_HEXW_WARPS
#define FEM_HEXW_WARPS 12
#endif
constexpr int kWriteWarps = FEM_HEXW_WARPS;
constexpr int kWriteThreads = kWriteWarps * 32;
constexpr int kWindow = 96;   // columns summed at once (an inner node of a regular mesh has 51 or 81)
static_assert(kWindow % 32 == 0, "whole lanes of columns");
constexpr int kItems = 6;     // entries of a 180-entry slab per lane

// Shared memory of a warp: the window's blocks, then one block that takes the
// additions outside the window.
constexpr int kBin = kWindow * 9;
struct alignas(16) WriteHexSmem {
    double acc[kBin + 10];
    int col[kWindow];
};
struct WriteHexCta {
    WriteHexSmem w[kWriteWarps];
    // entry x = 9 b + v of the slab of row position a: its place in the packed Ke
    unsigned short src[20][32 * kItems];
    int sum[kWriteWarps], max[kWriteWarps];
};
static_assert(sizeof(WriteHexSmem) % 16 == 0, "16-byte clears");

__device__ __forceinline__ int packed_block(int I, int J) { return I * 20 - I * (I - 1) / 2 + J - I; }

// What a warp knows of a row before it sums it.
struct RowHead {
    int n, u, lo, d;   // node (-1: no more), columns, first occurrence, occurrences
    int k0;            // first column written
    int word;          // occurrence `lane`
    long long base;    // the row's start in the output
};

// Runs as block `block` of `nblocks`.
template <int kMode>
__device__ __forceinline__ void write_hex20(const ListLayout& L, const HexRows& h, const int* __restrict__ ucounts,
                                            const int* __restrict__ row_ptr, int* __restrict__ col_idx,
                                            double* __restrict__ values, long long capacity, int block, int nblocks,
                                            WriteHexCta& cta) {
    int* const s_sum = cta.sum;
    int* const s_max = cta.max;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    WriteHexSmem& sm = cta.w[warp];
    if (!output_fits<3, kMode>(L.info, capacity)) return;
    for (int k = threadIdx.x; k < 20 * 32 * kItems; k += kWriteThreads) {
        const int a = k / (32 * kItems), x = k - a * 32 * kItems, b = min(x / 9, 19), v = x - 9 * (x / 9);
        (&cta.src[0][0])[k] =
            (unsigned short)(b >= a ? 9 * packed_block(a, b) + v : 9 * packed_block(b, a) + 3 * (v % 3) + v / 3);
    }
    __syncthreads();
    // entry i of this lane in a slab: block b(i), entry v(i) of it
    int sb[kItems], sv[kItems];
#pragma unroll
    for (int i = 0; i < kItems; i++) {
        const int x = lane + 32 * i;
        sb[i] = x / 9;
        sv[i] = x - 9 * sb[i];
    }
    int t_sum = 0, t_max = 0;
    bool bad = false;  // a row whose list lacks a column, or that an element has a further column for
    // The warps draw their nodes one by one from one counter, so that the rows in flight stay close in the visit order
    // however unevenly the SMs run (a fixed stride let them drift apart: Ke read 2.1 times from DRAM, 1.4 so). The
    // draws, the node ids and the headers of the next rows are in flight while a row is summed.
    // (A small mesh, without a visit order, is dealt at a fixed stride: about one node per warp, no drift.)
    int mine = (int)(block * kWriteWarps + warp);
    auto draw = [&]() {
        if (h.order) return lane == 0 ? atomicAdd(&L.info->ticket, 1) : 0;
        const int t = mine;
        mine = min(t, L.N) + nblocks * kWriteWarps;
        return t;
    };
    auto node_of = [&](int t) { return t < L.N ? (h.order ? __ldg(h.order + t) : t) : -1; };
    auto head_of = [&](int n) {
        RowHead r;
        r.n = n;
        r.u = r.lo = r.d = r.word = 0;
        r.k0 = 0;
        r.base = 0;
        if (n >= 0) {
            r.u = __ldg(L.counts + n);
            r.lo = __ldg(h.off + n);
            r.d = __ldg(h.off + n + 1);  // its end until `started`
            r.base = __ldg(row_ptr + (size_t)n * (kMode == kOutBsr ? 1 : 3));
            if (kMode == kOutUpper) r.k0 = __ldg(ucounts + n);
        }
        return r;
    };
    // the rest of a header, once its first loads are in: the row's first occurrences, one per lane
    auto started = [&](RowHead& r) {
        r.d -= r.lo;
        if (kMode == kOutUpper) r.k0 = r.u - r.k0;  // first column written: the node itself
        r.word = lane < r.d ? __ldg(h.inc + r.lo + lane) : 0;
    };
    RowHead cur = head_of(node_of(__shfl_sync(0xFFFFFFFFu, draw(), 0)));
    int n1 = node_of(__shfl_sync(0xFFFFFFFFu, draw(), 0)), t2 = draw();
    started(cur);
    while (cur.n >= 0) {
        RowHead nxt = head_of(n1);
        n1 = node_of(__shfl_sync(0xFFFFFFFFu, t2, 0));
        t2 = draw();
        const int n = cur.n, u = cur.u, lo = cur.lo, d = cur.d, k0 = cur.k0;
        const long long base = cur.base;
        const int next = u > L.S1 ? __ldg(L.meta1 + (size_t)n * L.H1 + 1) : 0;
        t_sum += u;
        t_max = max(t_max, u);
        bool first = true;
        for (int w0 = k0; w0 < u || first; w0 += kWindow) {
            const int uw = min(kWindow, u - w0);
            int col[kWindow / 32];
#pragma unroll
            for (int q = 0; q < kWindow / 32; q++) {
                const int k = lane + 32 * q;
                col[q] = k < uw ? __ldg(hex_col_word(L, n, next, w0 + k)) - 1 : 0;
                bad |= (unsigned)col[q] >= (unsigned)L.N;
            }
            double val[kItems];
            unsigned rk = 0;  // lane b < 20: rank of the occurrence's column node b
            int word = 0;
            auto fetch = [&](int t) {
                word = t < 32 ? __shfl_sync(0xFFFFFFFFu, cur.word, t) : __ldg(h.inc + lo + t);
                const unsigned o = occ_of(word), e = o / 20;
                const double* ke = h.ke + (size_t)e * kPackedHex20;
                const unsigned short* src = cta.src[o - 20 * e] + lane;
                if (lane < 20) rk = __ldg(h.map + (size_t)o * 20 + lane);
#pragma unroll
                for (int i = 0; i < kItems; i++) val[i] = __ldg(ke + src[32 * i]);
            };
            if (d > 0) fetch(0);
            for (int x = lane; 2 * x < uw * 9; x += 32) reinterpret_cast<double2*>(sm.acc)[x] = make_double2(0.0, 0.0);
            if (first && nxt.n >= 0) started(nxt);
            first = false;
            __syncwarp();
            for (int t = 0; t < d; t++) {
                // where column node `lane`'s block goes: its rank in the window, or the bin
                const int place = (int)((rk - (unsigned)w0) & (kRankRange - 1));
                int to = lane < 20 && place < uw ? place * 9 : kBin;
                bad |= lane < 20 && rk >= (unsigned)u && u != L.S1;  // S1 columns: cut when the pool overflowed
                if (u > kRankRange && to != kBin &&  // the rank is known up to a multiple of kRankRange only
                    __ldg(hex_col_word(L, n, next, w0 + place)) - 1 !=
                        __ldg(h.conn + (size_t)(occ_of(word) / 20) * 20 + lane))
                    to = kBin;
                unsigned later = 0;  // column nodes that the element has at an earlier position too
                const int again = to;
                if (word < 0) {
                    const unsigned same = __match_any_sync(0xFFFFFFFFu, to);
                    const bool dup = to != kBin && (same & ((1u << lane) - 1u));
                    later = __ballot_sync(0xFFFFFFFFu, dup);
                    if (dup) to = kBin;
                }
                int at[kItems];
                double x[kItems];
#pragma unroll
                for (int i = 0; i < kItems; i++) {
                    at[i] = __shfl_sync(0xFFFFFFFFu, to, sb[i]) + sv[i];
                    x[i] = val[i];
                }
                if (t + 1 < d) fetch(t + 1);
                double y[kItems];
#pragma unroll
                for (int i = 0; i < kItems; i++) y[i] = sm.acc[at[i]];
#pragma unroll
                for (int i = 0; i < kItems; i++) sm.acc[at[i]] = y[i] + x[i];
                __syncwarp();
                while (later) {  // a repeated node's further blocks, one at a time
                    const int b = __ffs(later) - 1, r9 = __shfl_sync(0xFFFFFFFFu, again, b);
                    later &= later - 1;
#pragma unroll
                    for (int i = 0; i < kItems; i++)
                        if (sb[i] == b) sm.acc[r9 + sv[i]] += x[i];
                    __syncwarp();
                }
            }
#pragma unroll
            for (int q = 0; q < kWindow / 32; q++) sm.col[lane + 32 * q] = col[q];
            __syncwarp();
            if (kMode == kOutBsr) {
                for (int k = lane; k < uw; k += 32) col_idx[base + w0 + k] = sm.col[k];
                for (int x = lane; x < uw * 9; x += 32) values[(base + w0) * 9 + x] = sm.acc[x];
            } else {
                for (int r = lane; r < 3 * uw; r += 32) {
                    const int k = r / 3, j = r - 3 * k, c = 3 * sm.col[k] + j;
                    const double* b = sm.acc + 9 * k + j;
                    if (kMode == kOutCsr) {
                        const long long p = base + 3 * w0 + r;
#pragma unroll
                        for (int i = 0; i < 3; i++) {
                            col_idx[p + 3ll * i * u] = c;
                            values[p + 3ll * i * u] = b[3 * i];
                        }
                    } else {
                        // row i starts i (3 len - 1) - i (i - 1) / 2 ... after row 0 and skips i entries of the diagonal block
                        const int q = 3 * (w0 - k0) + r, len = 3 * (u - k0);
#pragma unroll
                        for (int i = 0; i < 3; i++) {
                            if (q < i) continue;  // below the diagonal
                            const long long p = base + (long long)i * len - i * (i - 1) / 2 + (q - i);
                            col_idx[p] = c;
                            values[p] = b[3 * i];
                        }
                    }
                }
            }
            __syncwarp();
        }
        cur = nxt;
    }
    if (bad) raise_status(L.info, FEM_ERR_INTERNAL);
    // list statistics (one atomic pair per CTA)
    if (lane == 0) {
        s_sum[warp] = t_sum;
        s_max[warp] = t_max;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < kWriteWarps; w++) {
            t_sum += s_sum[w];
            t_max = max(t_max, s_max[w]);
        }
        atomicAdd(reinterpret_cast<unsigned long long*>(&L.info->list_entries), (unsigned long long)t_sum);
        atomicMax(&L.info->max_row_entries, t_max);
    }
}

}  // namespace
}  // namespace fem
