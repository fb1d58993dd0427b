// Internal definitions shared by the kernels and the C ABI of the assembler.
//
// Row lists ("A-LLS" lists, after the reference's ALLSNode pool,
// ALLS_Quad2D_Assembly_Accuracy_Analysis.cu:63-67,384-391) live in a device
// pool of fixed-size chunks. Every node n owns chunk n (its "first chunk");
// further chunks come from an overflow pool through an atomic bump counter and
// are linked through the previous chunk's `next` word. A list entry (slot) holds
// one column NODE of a row node, so the dpn rows of a node share one list.
//
// Chunk metadata is a row of H = S + 2 int32 words:
//     word 0 = kRowSorted + columns for a 2-D row stored sorted and compact, else 0
//     word 1 = next  (chunk id + 1 of the next chunk, 0 = none)
//     word 2+s = slot s: 0 = empty, col+1 = column node col
// A row belongs to the thread, warp or CTA that builds it (rows2d.cuh,
// rows_hex20.cuh), so a column appears once, and rows are stored sorted: the
// first u slots of the chain. The exception are 2-D rows that do not fit their
// first chunk, whose slots are hashed (scatter2d.cuh).
// 2-D values: each slot's dpn x dpn block, vals[gid * 4], gid the global slot id
// (first-chunk slots first, then overflow-chunk slots): one 32-byte sector.
// Hex20 values stay in the elements' packed Ke (in the place of vals) until the
// consolidation sums them (write_hex20.cuh).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "fem_alls.h"

namespace fem {

constexpr int kBlockThreads = 256;
constexpr int kScanTile = 4096;  // nodes per scan tile (256 threads x 16)
constexpr int kRowTile = 1024;   // nodes per tile of the consolidation's row pointers
inline int row_tiles(int num_nodes) { return (num_nodes + kRowTile - 1) / kRowTile; }

// Device-resident info word; its first bytes are laid out exactly as fem_info.
struct DevInfo {
    long long nnz;
    long long list_entries;
    int status_bits;
    int overflow_chunks;   // overflow-pool bump counter (may overshoot the capacity)
    int pool_chunks;
    int max_row_entries;
    int long_rows;         // rows queued for the long-row kernels
    int ticket;            // consolidation: next row node to write
    int spilled;           // 2-D: entries of the spill list (may overshoot its capacity)
    int done;              // batch: blocks of the mesh's write that are done
    long long pad1[2];
};
static_assert(sizeof(DevInfo) == 64, "DevInfo size");
static_assert(offsetof(DevInfo, max_row_entries) == offsetof(fem_info, max_row_entries), "fem_info layout");

struct ListLayout {
    int N;          // nodes (= first chunks)
    int S1, S2;     // slots per first / overflow chunk
    int H1, H2;     // int32 words per first / overflow chunk meta row (S + 2)
    int B;          // values per slot (dpn^2)
    int cap2;       // overflow chunk capacity
    int* meta1;     // [N * H1]
    int* meta2;     // [cap2 * H2]
    double* vals;   // 2-D: [(N*S1 + cap2*S2) * B]
    int* counts;    // [N] list entries of each row node (2-D: elements of the node until its row is built)
    unsigned* spill;  // 2-D: [spill_cap] elements past those that a node's own list storage keeps (4 element + position)
    int spill_cap;    // 0: none
    DevInfo* info;
};

// Bits of DevInfo::status_bits are 1 << FEM_ERR_*.
__device__ __forceinline__ void raise_status(DevInfo* info, int code) {
    atomicOr(&info->status_bits, 1 << code);
}

__device__ __forceinline__ int* chunk_meta(const ListLayout& L, int c) {
    return c < L.N ? L.meta1 + (size_t)c * L.H1 : L.meta2 + (size_t)(c - L.N) * L.H2;
}
__device__ __forceinline__ int chunk_cap(const ListLayout& L, int c) { return c < L.N ? L.S1 : L.S2; }
__device__ __forceinline__ unsigned slot_gid(const ListLayout& L, int c, int s) {
    return c < L.N ? (unsigned)c * (unsigned)L.S1 + (unsigned)s
                   : (unsigned)L.N * (unsigned)L.S1 + (unsigned)(c - L.N) * (unsigned)L.S2 + (unsigned)s;
}
// L2-coherent loads (bypass L1: list words change under other SMs' writes).
__device__ __forceinline__ int ld_cg(const int* p) { return __ldcg(p); }
__device__ __forceinline__ int4 ld_cg4(const int* p) { return __ldcg(reinterpret_cast<const int4*>(p)); }

// Takes one chunk from the overflow pool and zeroes its meta row and its slots'
// values (all contributions are atomic adds). Returns the chunk id, or -1 (and
// raises FEM_ERR_POOL_OVERFLOW) when the pool is empty. The caller must
// __threadfence() before publishing the chunk.
__device__ __forceinline__ int alloc_chunk(const ListLayout& L) {
    int k = atomicAdd(&L.info->overflow_chunks, 1);
    if (k >= L.cap2) {
        raise_status(L.info, FEM_ERR_POOL_OVERFLOW);
        return -1;
    }
    int* m = L.meta2 + (size_t)k * L.H2;
    for (int i = 0; i < L.H2; i += 4) *reinterpret_cast<int4*>(m + i) = make_int4(0, 0, 0, 0);
    double2* v = reinterpret_cast<double2*>(L.vals + (size_t)slot_gid(L, L.N + k, 0) * L.B);
    for (int i = 0; i < L.S2 * L.B / 2; i++) v[i] = make_double2(0.0, 0.0);
    return L.N + k;
}

// Bound on the walk along a chunk chain; hitting it raises FEM_ERR_TIMEOUT.
constexpr int kMaxChainSteps = 1 << 20;

// Header word (word 0) of a 2-D first chunk whose row is complete in it: this plus the number of columns, which fill
// the first slots in increasing order (no next chunk). 0: the row is hashed (fans).
constexpr int kRowSorted = 1;

// Start of the probe sequence of column key `key` (col + 1) in a chunk of S slots.
__device__ __forceinline__ int probe_start(int key, int S) {
    return (int)__umulhi((unsigned)key * 2654435761u, (unsigned)S);
}

// Appends a chunk to a row's chain, whose last chunk is `tail` (one thread). Returns its id, or -1 on pool overflow
// (status raised).
__device__ __forceinline__ int append_chunk(const ListLayout& L, int tail) {
    const int c = alloc_chunk(L);
    if (c < 0) return -1;
    __threadfence();  // the zeroed meta row is visible before the link
    atomicExch(chunk_meta(L, tail) + 1, c + 1);
    return c;
}

// Host-side layout description (sizes in bytes, offsets from the workspace base).
struct HostLayout {
    int kind, dpn, B, N, E;
    int S1, S2, H1, H2, cap2;
    int num_tiles;  // scan tiles of kScanTile nodes
    size_t off_info, off_meta1, off_meta2, off_vals, off_counts, off_ucounts, off_tiles, off_elist, off_inc, off_map,
        total;
    size_t meta1_bytes;
};

}  // namespace fem
