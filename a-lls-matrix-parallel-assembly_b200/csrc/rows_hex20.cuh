// Device code of the Hex20 row lists (rows_hex20.cu, and the batch, batched.cu):
// the pattern half of the A-LLS scatter.
//
// Replaces the insert half of assembleGlobalStiffnessKernelALLSFixedArray
// (ALLS_Hex20_3D_Assembly_Performance.cu:226-256: a linear scan of the row's
// columns, a slot claimed with atomicAdd on the row count, no fence), whose
// racing inserts duplicate or drop columns. Here a row belongs to the warp
// that builds it, from the node's occurrences (occ_* below), so nothing
// races, and the row comes out sorted:
//   k_rows_hex20       one warp per node with at most 8 elements (every inner
//                      node of a regular mesh): its elements' up to 160 node
//                      ids are loaded, up to five per lane, and inserted into
//                      a hash table in shared memory (128 entries for up to 4
//                      elements, the nodes inside an edge, 256 for 5 to 8);
//                      the distinct ones are compacted and sorted (bitonic, in
//                      registers: 64, 128 or 256 keys), written to the list
//                      chunks, and their ranks go back through the table to
//                      the rank map.
//   k_long_rows_hex20  nodes with up to 32 elements, one warp each: repeated
//                      minimum over the candidates, which stay in registers;
//                      then nodes with more, one CTA each: sorted in shared
//                      memory.
// A row past its first chunk takes consecutive overflow chunks from the pool.
//
// What bounds it: instruction issue (660 warp instructions a node in hash, sort
// and rank look-ups; ALU 58 %, 2.5 instructions per cycle) and waits for
// instructions and shared memory; DRAM is at 2 %. B200, 64^3 (1.09 M nodes):
// 1.02 ms, where five single-word loads per lane and a 256-entry table for
// every node took 1.13 ms, and the CAS claims of element groups 4.36 ms.
// CTAs per SM: 4 / 5 / 6 1.03 / 1.02 / 1.01 ms at 64^3, 9^3 call 70.7 / 70.9 /
// 73.6 us, batch of 16 meshes 1.73 / 1.69 / 1.73 ms. Listing new nodes as they
// are inserted, with the table entry packed into the sort key (no table scan,
// no second look-up), is 1.34 ms: the ballots after each insertion make the
// warps wait out each other's probes and the code no longer fits the
// instruction cache; so does a copy of the sorts for each of the two forms
// (batch 1.73 ms).
#pragma once

#include "hex_rows.cuh"
#include "scan.cuh"

namespace fem {
namespace {

// ---- occurrences: node -> (element, position) lists -----------------------------
//   occ_count  thread per element: one counter atomic per node; the position it
//              returns is kept (pos), so the fill needs no atomics. An element
//              with a bad node id has no occurrence (pos kNoOcc); the
//              occurrences of an element that repeats a node carry kOccRepeats.
//   occ_sums   sum of the counts per tile of kRowTile nodes
//   occ_offsets  exclusive prefix: each tile sums the tiles before it
//   occ_fill   thread per occurrence: inc[off[node] + pos] = 20 e + a

constexpr int kOccThreads = 256;
constexpr int kNoOcc = 0x7FFFFFFF;

__device__ __forceinline__ int* occ_pos(const HexRows& h) { return reinterpret_cast<int*>(h.map); }  // 80 of 800 bytes an element

// Clears a scatter's info word and occurrence counters.
__device__ __forceinline__ void lists_begin_hex20(const ListLayout& L, int* __restrict__ cnt, int block, int nblocks) {
    for (int i = block * blockDim.x + threadIdx.x; i < L.N; i += nblocks * blockDim.x) cnt[i] = 0;
    if (block == 0 && threadIdx.x == 0) {
        DevInfo d{};
        d.pool_chunks = L.cap2;
        *L.info = d;
    }
}

__device__ __forceinline__ void occ_count(const MeshView& m, const HexRows& h, int* __restrict__ cnt, DevInfo* info,
                                          int block, int nblocks) {
    int* pos = occ_pos(h);
    for (int e = block * kOccThreads + threadIdx.x; e < m.E_count; e += nblocks * kOccThreads) {
        const size_t o = (size_t)e * 20;
        int n[20];
        bool bad = false, rep = false;
#pragma unroll
        for (int k = 0; k < 20; k++) {
            n[k] = __ldg(m.conn + o + k);
            bad |= n[k] < 0 || n[k] >= m.N;
#pragma unroll
            for (int j = 0; j < k; j++) rep |= n[j] == n[k];
        }
        if (bad) raise_status(info, FEM_ERR_BAD_MESH);
        int p[20];
#pragma unroll
        for (int k = 0; k < 20; k++) p[k] = bad ? kNoOcc : atomicAdd(cnt + n[k], 1);
#pragma unroll
        for (int k = 0; k < 20; k++) pos[o + k] = rep && !bad ? (int)((unsigned)p[k] | kOccRepeats) : p[k];
    }
}

__device__ __forceinline__ void occ_sums(const int* __restrict__ cnt, int N, long long* __restrict__ tiles, int tile,
                                         long long* s_warp) {
    long long sum = 0;
#pragma unroll
    for (int i = 0; i < kRowTile / kScanThreads; i++) {
        const long long n = (long long)tile * kRowTile + i * kScanThreads + threadIdx.x;
        if (n < N) sum += __ldcg(cnt + n);
    }
    long long total;
    block_exclusive_scan(sum, s_warp, total);
    if (threadIdx.x == 0) tiles[tile] = total;
}

struct OccSmem {
    long long warp[kScanThreads / 32 + 1];
    int cnt[kRowTile];
};

// tiles NULL (small meshes): the counts before the tile are summed directly.
__device__ __forceinline__ void occ_offsets(const int* __restrict__ cnt, int N, const long long* __restrict__ tiles,
                                            int* __restrict__ off, int tile, int ntiles, OccSmem& sm) {
    constexpr int kItems = kRowTile / kScanThreads;
    const int tid = threadIdx.x;
    const long long first = (long long)tile * kRowTile;
#pragma unroll
    for (int i = 0; i < kItems; i++) {
        const long long n = first + i * kScanThreads + tid;
        sm.cnt[i * kScanThreads + tid] = n < N ? __ldcg(cnt + n) : 0;
    }
    long long before = 0, base, total;
    if (tiles) {
        for (int t = tid; t < tile; t += kScanThreads) before += __ldcg(tiles + t);
    } else {
#pragma unroll 8
        for (int n = tid; n < (int)first; n += kScanThreads) before += __ldcg(cnt + n);
    }
    block_exclusive_scan(before, sm.warp, base);
    int c[kItems];
    long long sum = 0;
#pragma unroll
    for (int i = 0; i < kItems; i++) {
        c[i] = sm.cnt[tid * kItems + i];
        sum += c[i];
    }
    long long o = base + block_exclusive_scan(sum, sm.warp, total);
#pragma unroll
    for (int i = 0; i < kItems; i++) {
        sm.cnt[tid * kItems + i] = (int)o;
        o += c[i];
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kItems; i++) {
        const long long n = first + i * kScanThreads + tid;
        if (n < N) off[n] = sm.cnt[i * kScanThreads + tid];
    }
    if (tile == ntiles - 1 && tid == 0) off[N] = (int)(base + total);
}

__device__ __forceinline__ void occ_fill(const MeshView& m, const HexRows& h, int block, int nblocks) {
    const int* pos = occ_pos(h);
    const long long count = 20ll * m.E_count;
    for (long long o = (long long)block * kOccThreads + threadIdx.x; o < count; o += (long long)nblocks * kOccThreads) {
        const int p = __ldcg(pos + o);
        if (p == kNoOcc) continue;
        const unsigned flag = (unsigned)p & kOccRepeats;
        h.inc[__ldcg(h.off + __ldg(m.conn + o)) + (int)((unsigned)p & ~kOccRepeats)] = (int)((unsigned)o | flag);
    }
}

// ---- rows -------------------------------------------------------------------------

// Resident CTAs per SM that the registers are set for.
#ifndef FEM_HEXR_CTAS
#define FEM_HEXR_CTAS 5
#endif
constexpr int kHexRowWarps = 8;
constexpr int kHexRowThreads = kHexRowWarps * 32;
constexpr int kMaxElems = 8;               // elements of a node in the main pass
constexpr int kTable = 256;
constexpr int kWideElems = 32;
constexpr int kWideCand = kWideElems * 20 / 32;

struct alignas(16) HexRowSmem {  // cleared with 16-byte stores
    int table[kTable];                 // distinct column nodes, -1 = empty
    int uniq[kTable];                  // compacted, then sorted
    unsigned short rank[kTable];       // rank of a table entry
};

// Overflow chunks of a row of u columns (called by one lane): returns the
// chain's first chunk id + 1 (0: none needed); a pool that is out cuts the row
// at its first chunk (FEM_ERR_POOL_OVERFLOW).
__device__ __forceinline__ int take_chunks(const ListLayout& L, int& u) {
    if (u <= L.S1) return 0;
    const int need = (u - L.S1 + L.S2 - 1) / L.S2;
    const int k = atomicAdd(&L.info->overflow_chunks, need);
    if (k < 0 || k + need > L.cap2) {
        raise_status(L.info, FEM_ERR_POOL_OVERFLOW);
        u = L.S1;
        return 0;
    }
    for (int i = 0; i < need; i++) {
        int* m = L.meta2 + (size_t)(k + i) * L.H2;
        m[0] = 0;
        m[1] = i + 1 < need ? L.N + k + i + 2 : 0;
    }
    return L.N + k + 1;
}

// Header of row n's first chunk and its column count.
__device__ __forceinline__ void finish_row(const ListLayout& L, int n, int u, int next) {
    *reinterpret_cast<int2*>(L.meta1 + (size_t)n * L.H1) = make_int2(0, next);
    L.counts[n] = u;
}

// Sorts the u keys of uniq (KPL per lane, padded) by a bitonic network.
template <int KPL>
__device__ __forceinline__ void sort_keys(int* uniq, int u, int lane) {
    int key[KPL];
#pragma unroll
    for (int i = 0; i < KPL; i++) key[i] = lane * KPL + i < u ? uniq[lane * KPL + i] : 0x7FFFFFFF;
#pragma unroll
    for (int size = 2; size <= 32 * KPL; size <<= 1) {
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            if (stride >= KPL) {
                const bool lower = ((lane * KPL) & stride) == 0;
#pragma unroll
                for (int i = 0; i < KPL; i++) {
                    const bool up = ((lane * KPL + i) & size) == 0;
                    const int o = __shfl_xor_sync(0xFFFFFFFFu, key[i], stride / KPL);
                    key[i] = lower == up ? min(key[i], o) : max(key[i], o);
                }
            } else {
#pragma unroll
                for (int i = 0; i < KPL; i++) {
                    const int j = i ^ stride;
                    if (j > i) {
                        const bool up = ((lane * KPL + i) & size) == 0;
                        const int lo = min(key[i], key[j]), hi = max(key[i], key[j]);
                        key[i] = up ? lo : hi;
                        key[j] = up ? hi : lo;
                    }
                }
            }
        }
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < KPL; i++)
        if (lane * KPL + i < u) uniq[lane * KPL + i] = key[i];
    __syncwarp();
}

// The row of node n with d <= 8 elements; o: lane t < d holds its occurrence t.
// Four lanes take an element's node ids (up to 4 elements: eight lanes): 16 in
// one load of four (two) words each, and the last four. conn16: conn is 16-byte
// aligned. The sorts are shared by both forms: at twice the code the warps wait for instructions.
__device__ __forceinline__ void row_hex20(const int* __restrict__ conn, bool conn16, const ListLayout& L,
                                          unsigned short* __restrict__ map, int n, int d, int o, HexRowSmem& sm) {
    const bool many = d > 4;
    const int lane = threadIdx.x & 31, t = many ? lane >> 2 : lane >> 3, sub = many ? lane & 3 : lane & 7;
    const int tab = many ? kTable : kTable / 2, shift = many ? 24 : 25;  // at most 20/32 of the table fills
    auto start = [&](int node) { return (int)(((unsigned)node * 2654435761u) >> shift); };
    const bool has = t < d, last = has && sub < 4;
    const int ot = __shfl_sync(0xFFFFFFFFu, o, t);
    const int* src = conn + (size_t)(ot / 20) * 20;
    int node[5] = {-1, -1, -1, -1, -1}, slot[5];
    if (last) node[4] = __ldg(src + 16 + sub);
    if (has && many) {
        if (conn16) {
            const int4 v = __ldg(reinterpret_cast<const int4*>(src) + sub);
            node[0] = v.x, node[1] = v.y, node[2] = v.z, node[3] = v.w;
        } else {
#pragma unroll
            for (int i = 0; i < 4; i++) node[i] = __ldg(src + 4 * sub + i);
        }
    } else if (has) {
        if (conn16) {
            const int2 v = __ldg(reinterpret_cast<const int2*>(src) + sub);
            node[0] = v.x, node[1] = v.y;
        } else {
            node[0] = __ldg(src + 2 * sub), node[1] = __ldg(src + 2 * sub + 1);
        }
    }
    reinterpret_cast<int4*>(sm.table)[lane] = make_int4(-1, -1, -1, -1);
    if (many) reinterpret_cast<int4*>(sm.table)[lane + 32] = make_int4(-1, -1, -1, -1);
    __syncwarp();
    auto insert = [&](int i) {
        int at = start(node[i]);
        if (node[i] >= 0) {
            for (int k = 0; k < kTable; k++) {
                const int old = atomicCAS(&sm.table[at], -1, node[i]);
                if (old == -1 || old == node[i]) break;
                at = (at + 1) & (tab - 1);
            }
        }
        slot[i] = at;
    };
    insert(4), insert(0), insert(1);
    if (many) insert(2), insert(3);
    __syncwarp();
    int u = 0;
#pragma unroll 4
    for (int q = 0; q < tab; q += 32) {
        const int k = sm.table[lane + q];
        const unsigned used = __ballot_sync(0xFFFFFFFFu, k >= 0);
        if (k >= 0) sm.uniq[u + __popc(used & ((1u << lane) - 1u))] = k;
        u += __popc(used);
    }
    __syncwarp();
    if (u <= 64) sort_keys<2>(sm.uniq, u, lane);
    else if (u <= 128) sort_keys<4>(sm.uniq, u, lane);
    else sort_keys<8>(sm.uniq, u, lane);
    int kept = u, next = 0;
    if (u > L.S1) {
        if (lane == 0) next = take_chunks(L, kept);
        next = __shfl_sync(0xFFFFFFFFu, next, 0);
        kept = __shfl_sync(0xFFFFFFFFu, kept, 0);
    }
    for (int p = lane; p < u; p += 32) {
        const int k = sm.uniq[p];
        int at = start(k);
        while (sm.table[at] != k) at = (at + 1) & (tab - 1);
        sm.rank[at] = (unsigned short)p;
        if (p < kept) *hex_col_word(L, n, next, p) = k + 1;
    }
    if (lane == 0) finish_row(L, n, kept, next);
    __syncwarp();
    unsigned short* dst = map + (size_t)ot * 20;
    if (has && many)
        reinterpret_cast<ushort4*>(dst)[sub] =
            make_ushort4(sm.rank[slot[0]], sm.rank[slot[1]], sm.rank[slot[2]], sm.rank[slot[3]]);
    else if (has)
        reinterpret_cast<ushort2*>(dst)[sub] = make_ushort2(sm.rank[slot[0]], sm.rank[slot[1]]);
    if (last) dst[16 + sub] = sm.rank[slot[4]];
    __syncwarp();
}

// The bodies below run as block `block` of `nblocks` of their launch.
__device__ __forceinline__ void rows_hex20(const int* __restrict__ conn, const ListLayout& L, const HexRows& h,
                                           int* __restrict__ queue, int block, int nblocks,
                                           HexRowSmem (&s_row)[kHexRowWarps]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool conn16 = (reinterpret_cast<uintptr_t>(conn) & 15) == 0;
    HexRowSmem& sm = s_row[warp];
    const long long step = (long long)nblocks * kHexRowWarps;
    // the next node's occurrences are loaded while the current row is built
    auto bounds = [&](long long nn) { return nn < L.N ? make_int2(__ldcg(h.off + nn), __ldcg(h.off + nn + 1)) : make_int2(0, 0); };
    auto occ = [&](int2 r) { return lane < min(r.y - r.x, kMaxElems) ? (int)occ_of(__ldcg(h.inc + r.x + lane)) : 0; };
    long long nn = (long long)block * kHexRowWarps + warp;
    int2 r = bounds(nn), r1 = bounds(nn + step);
    int o = occ(r);
    for (; nn < L.N; nn += step) {
        const int n = (int)nn, d = r.y - r.x, o1 = occ(r1);
        r = r1;
        r1 = bounds(nn + 2 * step);
        if (d > kMaxElems) {
            if (lane == 0) queue[atomicAdd(&L.info->long_rows, 1)] = n;
        } else {
            row_hex20(conn, conn16, L, h.map, n, d, o, sm);
        }
        o = o1;
    }
}

// warp `warp` of `nwarps`; s_uniq: the warp's kWideElems * 20 words.
__device__ __forceinline__ void wide_rows_hex20(const int* __restrict__ conn, const ListLayout& L, const HexRows& h,
                                                const int* __restrict__ queue, int warp, int nwarps, int* s_uniq) {
    const int* __restrict__ off = h.off;
    const int* __restrict__ inc = h.inc;
    unsigned short* __restrict__ map = h.map;
    const int lane = threadIdx.x & 31, count = __ldcg(&L.info->long_rows);
    for (int k = warp; k < count; k += nwarps) {
        const int n = __ldcg(queue + k), lo = __ldcg(off + n), d = __ldcg(off + n + 1) - lo;
        if (d > kWideElems) continue;  // long_rows_hex20's
        const int o = lane < d ? (int)occ_of(__ldcg(inc + lo + lane)) : 0;
        int node[kWideCand];
#pragma unroll
        for (int q = 0; q < kWideCand; q++) {
            const int j = lane + 32 * q, t = j / 20, b = j - 20 * t;
            const int e = __shfl_sync(0xFFFFFFFFu, o, t) / 20;
            node[q] = j < 20 * d ? __ldg(conn + (size_t)e * 20 + b) : 0x7FFFFFFF;
        }
        int u = 0;
        for (int last = -1;;) {
            int m = 0x7FFFFFFF;
#pragma unroll
            for (int q = 0; q < kWideCand; q++) m = node[q] > last ? min(m, node[q]) : m;
            m = __reduce_min_sync(0xFFFFFFFFu, m);
            if (m == 0x7FFFFFFF) break;
#pragma unroll
            for (int q = 0; q < kWideCand; q++) {
                const int j = lane + 32 * q, t = j / 20, b = j - 20 * t;
                const int ot = __shfl_sync(0xFFFFFFFFu, o, t);
                if (node[q] == m) map[(size_t)ot * 20 + b] = (unsigned short)u;
            }
            if (lane == 0) s_uniq[u] = m;
            u++;
            last = m;
        }
        int kept = u, next = 0;
        if (lane == 0) next = take_chunks(L, kept);
        next = __shfl_sync(0xFFFFFFFFu, next, 0);
        kept = __shfl_sync(0xFFFFFFFFu, kept, 0);
        __syncwarp();
        for (int p = lane; p < kept; p += 32) *hex_col_word(L, n, next, p) = s_uniq[p] + 1;
        if (lane == 0) finish_row(L, n, kept, next);
        __syncwarp();
    }
}

// Shared memory of a long row's CTA.
constexpr int kLongKeys = 4096, kLongBins = 1024;
struct LongHexSmem {
    long long scan[kScanThreads / 32 + 1];
    int key[kLongKeys];   // a stretch of the row's columns: candidates, sorted, distinct
    int bin[kLongBins];   // candidates per value range
    int count, cut, kept, next;
};

// The row of a node with more than kWideElems elements, by the CTA. Its 20 d candidate columns are taken in stretches
// of the value range with at most kLongKeys candidates (one stretch up to 204 elements; else found by a histogram,
// a column of its own when one value alone has more): collected and sorted in shared memory, distinct ones numbered,
// and each candidate's rank looked up in them. So the work is linear in the candidates, times their number over
// kLongKeys; the repeated minimum over memory that this replaces read all candidates once per column. B200, scatter of
// 24^3 elements beside elements that share one node: 33 of them 1570 -> 251 us, 204 34.6 -> 0.31 ms, 1000 802 -> 1.6 ms.
__device__ __forceinline__ void long_row_hex20(const int* __restrict__ conn, const ListLayout& L, const HexRows& h, int n,
                                               int lo, int d, LongHexSmem& sm) {
    const int tid = threadIdx.x;
    const long long cand = 20ll * d;
    const bool single = cand <= kLongKeys;
    // f(place in the map, column) for this thread's candidates with a column in [a, b)
    auto each = [&](int a, int b, auto f) {
        for (long long j = tid; j < cand; j += kHexRowThreads) {
            const unsigned o = occ_of(__ldcg(h.inc + lo + (int)(j / 20)));
            const int k = (int)(j % 20), x = __ldg(conn + (size_t)(o / 20) * 20 + k);
            if (x >= a && x < b) f((size_t)o * 20 + k, x);
        }
    };
    // pass 0 counts the columns (their chunks are taken at once), pass 1 writes; a single stretch stays for both
    for (int pass = 0; pass < 2; pass++) {
        int u = 0;
        for (int a = 0; a < L.N;) {
            int b = L.N, s = 0;
            bool one = false;  // the stretch is the single column a
            if (!single) {
                for (;;) {  // at most four times: each range is a bin of the one before
                    const int width = (int)(((long long)b - a + kLongBins - 1) / kLongBins);
                    __syncthreads();
                    for (int k = tid; k < kLongBins; k += kHexRowThreads) sm.bin[k] = 0;
                    if (tid == 0) sm.cut = sm.count = 0;
                    __syncthreads();
                    each(a, b, [&](size_t, int x) { atomicAdd(&sm.bin[(x - a) / width], 1); });
                    __syncthreads();
                    // the bins from a on with at most kLongKeys candidates together
                    constexpr int kEach = kLongBins / kHexRowThreads;
                    int c[kEach];
                    long long sum = 0, total;
#pragma unroll
                    for (int k = 0; k < kEach; k++) sum += c[k] = sm.bin[tid * kEach + k];
                    long long before = block_exclusive_scan(sum, sm.scan, total);
#pragma unroll
                    for (int k = 0; k < kEach; k++) {
                        before += c[k];
                        if (before <= kLongKeys) atomicMax(&sm.cut, tid * kEach + k + 1), atomicMax(&sm.count, (int)before);
                    }
                    __syncthreads();
                    const int cut = sm.cut;
                    const bool some = sm.count > 0;
                    const long long edge = min((long long)b, a + (long long)cut * width);
                    if (some || cut == kLongBins) {
                        b = (int)edge;
                        break;
                    }
                    // only empty bins before one with too many
                    a = (int)edge;
                    b = (int)min((long long)b, (long long)a + width);
                    one = width == 1;
                    if (one) break;
                }
            }
            if (one) {
                if (tid == 0) sm.key[0] = a;
                s = 1;
                __syncthreads();
            } else if (!single || pass == 0) {
                __syncthreads();
                if (tid == 0) sm.count = 0;
                __syncthreads();
                each(a, b, [&](size_t, int x) { sm.key[atomicAdd(&sm.count, 1)] = x; });
                __syncthreads();
                const int count = sm.count;
                int size = 2;
                while (size < count) size *= 2;
                for (int k = count + tid; k < size; k += kHexRowThreads) sm.key[k] = 0x7FFFFFFF;
                for (int run = 2; run <= size; run *= 2)
                    for (int step = run / 2; step > 0; step /= 2) {
                        __syncthreads();
                        for (int k = tid; k < size / 2; k += kHexRowThreads) {
                            const int p = 2 * k - (k & (step - 1)), q = p + step;
                            const int x = sm.key[p], y = sm.key[q];
                            if ((x > y) == ((p & run) == 0)) sm.key[p] = y, sm.key[q] = x;
                        }
                    }
                __syncthreads();
                // the distinct ones move to the front, a strip of the CTA's threads at a time
                for (int k0 = 0; k0 < count; k0 += kHexRowThreads) {
                    const int k = k0 + tid, x = k < count ? sm.key[k] : 0;
                    const bool first = k < count && (k == 0 || sm.key[k - 1] != x);
                    long long total;
                    const long long at = block_exclusive_scan(first, sm.scan, total);
                    if (first) sm.key[s + at] = x;
                    s += (int)total;
                    __syncthreads();
                }
                if (tid == 0) sm.cut = s;
                __syncthreads();
            } else {
                s = sm.cut;
            }
            if (pass == 1) {
                for (int p = tid; p < s && u + p < sm.kept; p += kHexRowThreads)
                    *hex_col_word(L, n, sm.next, u + p) = sm.key[p] + 1;
                each(a, one ? a + 1 : b, [&](size_t at, int x) {
                    int f = 0, l = s;
                    while (f < l) {
                        const int mid = (f + l) >> 1;
                        if (sm.key[mid] < x) f = mid + 1;
                        else l = mid;
                    }
                    h.map[at] = (unsigned short)(u + f);
                });
            }
            u += s;
            a = one ? a + 1 : b;
        }
        if (pass == 0 && tid == 0) {
            sm.next = take_chunks(L, u);
            sm.kept = u;
            finish_row(L, n, u, sm.next);
        }
        __syncthreads();
    }
}

__device__ __forceinline__ void long_rows_hex20(const int* __restrict__ conn, const ListLayout& L, const HexRows& h,
                                                const int* __restrict__ queue, int block, int nblocks, LongHexSmem& sm) {
    const int count = __ldcg(&L.info->long_rows);
    for (int k = block; k < count; k += nblocks) {
        const int n = __ldcg(queue + k), lo = __ldcg(h.off + n), d = __ldcg(h.off + n + 1) - lo;
        if (d > kWideElems) long_row_hex20(conn, L, h, n, lo, d, sm);
    }
}

}  // namespace
}  // namespace fem
