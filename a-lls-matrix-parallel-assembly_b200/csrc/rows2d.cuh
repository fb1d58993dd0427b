// Device code of the 2-D row lists (rows2d.cu, and the batch, batched.cu): the
// row lists of a Q4 / T3 / mixed mesh, one thread per
// row node.
//
// Replaces assembleGlobalStiffnessKernelALLS
// (ALLS_Quad2D_Assembly_Accuracy_Analysis.cu:394-468,
//  ALLS_T3_Unstructed_Elements_Assemble_Performance.cu:227-290,
//  ALLS_Q4_T3_Mixed_Elements_Assembly_Performance.cu:248-312), which runs one
// thread per element and walks a pointer list for each of its ndof^2 entries.
//
// Two launches:
//   k_fill_2d  thread per element: appends the element to the element list of
//              each of its distinct nodes (one counter atomic per node). The
//              list sits in the node's own list storage until its row is
//              built: the 14 slot words of its first chunk, then the chunk's
//              value words (kIncWords elements), so it takes no memory.
//   k_rows_2d  thread per node: walks the node's elements (the next one's
//              coordinates and the one after's nodes in flight), computes the
//              node's row of each Ke (element2d.cuh, the element rotated so
//              that the row node comes first) and sums the blocks per column
//              node. The first kLow column keys live in registers (an
//              unrolled compare against every key), their 2x2 sums in shared
//              memory, the threads of a warp on consecutive doubles (no bank
//              conflicts), the diagonal block in registers; further columns
//              (up to the chunk's 14) in the row's own value blocks. The row
//              leaves the thread once, sorted by column and compact: its slot
//              words (header word kRowSorted + columns) and its blocks as 32-byte
//              stores, whole sectors.
// No value is ever added in global memory, so nothing is zeroed first, no
// element order is needed and the value blocks are written once.
//
// What bounds it: instruction issue and the latency of the gathered loads
// (element -> nodes -> coordinates) together, at the 12 to 14 warps per SM
// that the accumulators and registers leave. B200, 1000x1000 cells: T3
// (shuffled elements) fill 97 us + rows 253 us, where one lane per element
// block with CAS claims and FP64 atomics into zeroed lists took 722 us plus
// 132 us of element order and memsets; Q4 37 + 233 us; mixed 1500x1500 287 +
// 812 us (1809 + 300 us). A group of 4 or 8 lanes per node, lane = element,
// with an all-pairs column comparison measured 299 us (T3), 274 us (Q4) and
// 1650 us (mixed): more instructions in all.
//
// Row nodes with more than 14 elements or columns (a fan's hub) take the
// hashed chunk lists instead (k_long_rows_2d): a CTA inserts the row's
// contributions with CAS claims and FP64 atomics (resolve_2d, scatter2d.cuh),
// chaining overflow chunks; the element list comes from the node's list
// storage and, past its kIncWords elements, from one list of all such nodes'
// further elements (ListLayout::spill), or from a pass over the connectivity if
// that list ran out. B200, scatter of a T3 1000x1000 mesh (340 us) beside a fan:
// 126 triangles 414 us, 130 429, 360 720, 50 fans of 360 825, 2,000 4,790 us; with
// a pass over the connectivity for each such node and the chain walked from its
// head for every chunk 484 us, 13.4, 13.8, 12.5 and 26.4 ms.
#pragma once

#include "scatter2d.cuh"

namespace fem {
namespace {

// Resident CTAs per SM that the registers are set for (build-time tuning
// knobs; measured on B200: T3 6 / 7 / 8 CTAs 274 / 257 / 273 us, mixed 4 / 5 /
// 6 / 7 CTAs 1074 / 988 / 911 / 1406 us, the last one spilling).
#ifndef FEM_ROWS_T3_CTAS
#define FEM_ROWS_T3_CTAS 7
#endif
#ifndef FEM_ROWS_Q4_CTAS
#define FEM_ROWS_Q4_CTAS 6
#endif
constexpr int kFillThreads = 256;
constexpr int kRowThreads = 64;
constexpr int kValInc = k2DSlots * 4 * 2;     // elements that fit in a first chunk's value words
constexpr int kIncWords = k2DSlots + kValInc; // elements that fit in a node's list storage

template <int KIND>
__device__ __forceinline__ int elem_nodes(const MeshView& m, int e) {
    if (KIND == FEM_T3) return 3;
    if (KIND == FEM_Q4) return 4;
    return __ldg(m.types + e) == FEM_Q4 ? 4 : 3;
}

// The bodies below run as block `block` of `nblocks` of their launch.
template <int KIND>
__device__ __forceinline__ void fill_2d(const MeshView& m, const ListLayout& L, int block, int nblocks) {
    constexpr int NPE = KIND == FEM_T3 ? 3 : 4;
    for (int e = block * blockDim.x + threadIdx.x; e < m.E_count; e += nblocks * blockDim.x) {
        const int npe = elem_nodes<KIND>(m, e);
        int n[NPE];
        bool bad = false;
#pragma unroll
        for (int k = 0; k < NPE; k++) {
            n[k] = __ldg(m.conn + (size_t)e * m.stride + k);
            if (k < npe) bad |= n[k] < 0 || n[k] >= m.N;
        }
        if (bad) {
            raise_status(L.info, FEM_ERR_BAD_MESH);
            continue;
        }
        int pos[NPE];
#pragma unroll
        for (int k = 0; k < NPE; k++) {
            bool distinct = k < npe;
#pragma unroll
            for (int j = 0; j < k; j++) distinct &= n[j] != n[k];
            pos[k] = distinct ? atomicAdd(L.counts + n[k], 1) : -1;
        }
#pragma unroll
        for (int k = 0; k < NPE; k++) {
            if (pos[k] < 0) continue;
            if (pos[k] < k2DSlots) {
                L.meta1[(size_t)n[k] * (k2DSlots + 2) + 2 + pos[k]] = e;
            } else if (pos[k] < kIncWords) {
                reinterpret_cast<int*>(L.vals + (size_t)n[k] * (k2DSlots * 4))[pos[k] - k2DSlots] = e;
            } else if (L.spill_cap > 0) {
                const int i = atomicAdd(&L.info->spilled, 1);
                if (i < L.spill_cap) L.spill[i] = 4u * (unsigned)e + k;
            }
        }
    }
}

// Stores a 2x2 block (32-byte aligned) with one 32-byte store: whole sectors.
__device__ __forceinline__ void store_block(double* p, double a, double b, double c, double d) {
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(a), "d"(b), "d"(c), "d"(d) : "memory");
}

// An element of a row node, its nodes rotated so that the row node is first.
template <int NPE>
struct ElemData {
    int e, npe;
    int nodes[NPE];
    unsigned more;  // further positions of the row node in the element (a repeated node)
    double x[NPE], y[NPE], E, nu;
};

template <int KIND, int NPE>
__device__ __forceinline__ void load_nodes(const MeshView& m, int e, ElemData<NPE>& d) {
    d.e = e;
    d.npe = elem_nodes<KIND>(m, e);
#pragma unroll
    for (int k = 0; k < NPE; k++) d.nodes[k] = __ldg(m.conn + (size_t)e * m.stride + k);
}

// Rotates the element's nodes so that position a comes first.
template <int KIND, int NPE>
__device__ __forceinline__ void rotate(ElemData<NPE>& d, int a) {
    const int n0 = d.nodes[0], n1 = d.nodes[1], n2 = d.nodes[2];
    if constexpr (NPE == 3) {
        d.nodes[0] = a == 0 ? n0 : (a == 1 ? n1 : n2);
        d.nodes[1] = a == 0 ? n1 : (a == 1 ? n2 : n0);
        d.nodes[2] = a == 0 ? n2 : (a == 1 ? n0 : n1);
    } else {
        // a T3 of a mixed mesh keeps its third node in the fourth position too
        const bool q4 = KIND == FEM_Q4 || d.npe == 4;
        const int n3 = q4 ? d.nodes[3] : n0;
        d.nodes[0] = a == 0 ? n0 : (a == 1 ? n1 : (a == 2 ? n2 : n3));
        d.nodes[1] = a == 0 ? n1 : (a == 1 ? n2 : (a == 2 ? n3 : n0));
        d.nodes[2] = a == 0 ? n2 : (a == 1 ? n3 : (a == 2 ? (q4 ? n0 : n1) : n1));
        d.nodes[3] = !q4 ? d.nodes[2] : (a == 0 ? n3 : (a == 1 ? n0 : (a == 2 ? n1 : n2)));
    }
}

// Rotates row node n to the front and loads coordinates and material.
template <int KIND, int NPE>
__device__ __forceinline__ void load_rest(const MeshView& m, int n, ElemData<NPE>& d) {
    unsigned at = 0;
#pragma unroll
    for (int k = 0; k < NPE; k++) at |= (k < d.npe && d.nodes[k] == n ? 1u : 0u) << k;
    rotate<KIND>(d, __ffs(at) - 1);
    d.more = at & (at - 1);
#pragma unroll
    for (int k = 0; k < NPE; k++) {
        d.x[k] = __ldg(m.x + d.nodes[k]);
        d.y[k] = __ldg(m.y + d.nodes[k]);
    }
    d.E = m.E ? __ldg(m.E + d.e) : m.E0;
    d.nu = m.nu ? __ldg(m.nu + d.e) : m.nu0;
}

// The next of a repeated row node's positions (its bit leaves d.more).
template <int KIND, int NPE>
__device__ __forceinline__ void next_position(const MeshView& m, ElemData<NPE>& d) {
    const unsigned more = d.more & (d.more - 1);
    load_nodes<KIND>(m, d.e, d);
    rotate<KIND>(d, __ffs(d.more) - 1);
    d.more = more;
#pragma unroll
    for (int k = 0; k < NPE; k++) {
        d.x[k] = __ldg(m.x + d.nodes[k]);
        d.y[k] = __ldg(m.y + d.nodes[k]);
    }
}

// Blocks (nodes[0], nodes[b]) of one element, b < npe. Returns detJ.
template <int KIND, typename T, int NPE>
__device__ __forceinline__ double row_blocks(const ElemData<NPE>& d, double t, double (&k)[NPE][4]) {
    if constexpr (KIND != FEM_MIXED_2D) {
        return ke_row_2d<NPE, T>(d.x, d.y, d.E, d.nu, t, k);
    } else {
        if (d.npe == 4) return ke_row_2d<4, T>(d.x, d.y, d.E, d.nu, t, k);
        const double x3[3] = {d.x[0], d.x[1], d.x[2]}, y3[3] = {d.y[0], d.y[1], d.y[2]};
        double k3[3][4];
        const double det = ke_row_2d<3, T>(x3, y3, d.E, d.nu, t, k3);
#pragma unroll
        for (int b = 0; b < 3; b++)
#pragma unroll
            for (int v = 0; v < 4; v++) k[b][v] = k3[b][v];
        return det;
    }
}

constexpr int kOffDiag = k2DSlots - 1;  // columns besides the diagonal in a chunk
constexpr int kLow = 8;                 // columns summed in shared memory

struct RowSmem {
    double acc[kLow][4][kRowThreads];       // block sums of the first columns
    int words[k2DSlots + 2][kRowThreads];   // the node's element list, then its sorted slot words
};

// Adds a block to column c past the first kLow columns: its sum is kept in the
// row's own (not yet written) value blocks, its key in hi. Returns whether the
// chunk is full. Out of line, as few rows come here.
__device__ __noinline__ bool add_high(int* hi, double* vals, int c, int& u, double k0, double k1, double k2, double k3) {
    int s = u;
    for (int q = kLow; q < u; q++) s = hi[q - kLow] == c ? q : s;
    if (s >= kOffDiag) return true;
    double* p = vals + 4 * s;
    const bool old = s < u;
    hi[s - kLow] = c;
    p[0] = (old ? p[0] : 0.0) + k0;
    p[1] = (old ? p[1] : 0.0) + k1;
    p[2] = (old ? p[2] : 0.0) + k2;
    p[3] = (old ? p[3] : 0.0) + k3;
    u = max(u, s + 1);
    return false;
}

// Places the columns past the first ones in the sorted row: adds them to the
// ranks of the others, moves their blocks.
__device__ __noinline__ void place_high(const int* hi, int nh, double* vals, const int* low_key, int* low_add, int n,
                                        int* words, int stride) {
    int hr[kOffDiag - kLow];
    double hv[kOffDiag - kLow][4];
    for (int p = 0; p <= kLow; p++) low_add[p] = 0;
    for (int q = 0; q < nh; q++) {
        const int c = hi[q];
        int r = c > n;
        low_add[kLow] += c < n;
        for (int p = 0; p < kLow; p++) {
            r += low_key[p] < c;
            low_add[p] += c < low_key[p];
        }
        for (int p = 0; p < nh; p++) r += hi[p] < c;
        hr[q] = r;
        for (int v = 0; v < 4; v++) hv[q][v] = vals[4 * (kLow + q) + v];
    }
    for (int q = 0; q < nh; q++) {
        words[(2 + hr[q]) * stride] = hi[q] + 1;
        double2* p = reinterpret_cast<double2*>(vals + 4 * hr[q]);
        p[0] = make_double2(hv[q][0], hv[q][1]);
        p[1] = make_double2(hv[q][2], hv[q][3]);
    }
}

constexpr int kStrip = 16 * kRowThreads;  // elements searched at once when a list was too long to keep

struct LongSmem {
    double blk[4 * 4][kRowThreads];  // the threads' element blocks
    int last[4][kRowThreads];        // their columns' progress along the chain (resolve_2d)
    int elems[kStrip];
    int nelems, full, tail;
};

// The hashed row of a node with many elements or columns, built by the CTA:
// each thread takes an element, its columns go into the chunks there are, and
// while some column finds them full, one thread appends a chunk (so a row
// takes exactly the chunks its columns need).
template <int KIND, typename T>
__device__ __forceinline__ void long_row_2d(const MeshView& m, const ListLayout& L, int n, int d, LongSmem& sm) {
    constexpr int NPE = KIND == FEM_T3 ? 3 : 4;
    static_assert(kStrip >= kIncWords, "a kept element list fits");
    const int tid = threadIdx.x;
    int* elems = sm.elems;
    int* meta = L.meta1 + (size_t)n * (k2DSlots + 2);
    double* vals = L.vals + (size_t)n * (k2DSlots * 4);
    // the elements: the row's own list, then, past it, those of the spill list that are the node's, or, if that list ran
    // out, all of the connectivity instead of both; a strip at a time
    const int spilled = __ldcg(&L.info->spilled);
    const bool in_spill = d > kIncWords && L.spill_cap > 0 && spilled <= L.spill_cap;
    const long long search = d <= kIncWords ? 0 : (in_spill ? spilled : m.E_count);
    bool own = d <= kIncWords || in_spill;
    const int listed = own ? min(d, kIncWords) : 0;
    for (int k = tid; k < listed; k += kRowThreads)
        elems[k] = k < k2DSlots ? __ldcg(meta + 2 + k) : __ldcg(reinterpret_cast<const int*>(vals) + k - k2DSlots);
    __syncthreads();
    for (int k = tid; k < k2DSlots + 2; k += kRowThreads) meta[k] = 0;
    for (int k = tid; k < k2DSlots * 4; k += kRowThreads) vals[k] = 0.0;
    if (tid == 0) {
        L.counts[n] = 0;
        sm.nelems = listed;
        sm.full = 0;
        sm.tail = n;
    }
    __syncthreads();
    for (long long i0 = 0; own || i0 < search;) {
        if (!own) {
            for (long long i = i0 + tid; i < min(search, i0 + kStrip); i += kRowThreads) {
                int e = (int)i;
                if (in_spill) {
                    const unsigned w = __ldcg(L.spill + i);
                    e = (int)(w >> 2);
                    if (__ldg(m.conn + (size_t)e * m.stride + (w & 3u)) == n) elems[atomicAdd(&sm.nelems, 1)] = e;
                    continue;
                }
                ElemData<NPE> el;
                load_nodes<KIND>(m, e, el);
                bool has = false, bad = false;
#pragma unroll
                for (int k = 0; k < NPE; k++) {
                    if (k >= el.npe) continue;
                    has |= el.nodes[k] == n;
                    bad |= el.nodes[k] < 0 || el.nodes[k] >= m.N;
                }
                if (has && !bad) elems[atomicAdd(&sm.nelems, 1)] = e;
            }
            __syncthreads();
            i0 += kStrip;
        }
        own = false;
        const int nelems = sm.nelems;
        for (int j0 = 0; j0 < nelems; j0 += kRowThreads) {
            ElemData<NPE> el;
            el.more = 0;
            const bool mine = j0 + tid < nelems;
            if (mine) {
                load_nodes<KIND>(m, elems[j0 + tid], el);
                load_rest<KIND>(m, n, el);
            }
            bool again = mine;
            while (__syncthreads_or(again)) {  // once per position of the row node in the element
                unsigned todo = 0;
                if (again) {
                    double k[NPE][4];
                    if (!(row_blocks<KIND, T>(el, m.t, k) > 0.0)) raise_status(L.info, FEM_ERR_DETJ);
#pragma unroll
                    for (int b = 0; b < NPE; b++)
#pragma unroll
                        for (int v = 0; v < 4; v++) sm.blk[4 * b + v][tid] = k[b][v];
#pragma unroll
                    for (int b = 0; b < NPE; b++) sm.last[b][tid] = 0;
                    todo = (1u << el.npe) - 1u;
                }
                for (;;) {
#pragma unroll 1
                    for (int b = 0; b < NPE; b++) {
                        if (!((todo >> b) & 1u)) continue;
                        unsigned gid = 0;
                        int col = el.nodes[0];
#pragma unroll
                        for (int k = 1; k < NPE; k++) col = k == b ? el.nodes[k] : col;
                        const int state = resolve_2d(L, n, col + 1, sm.last[b][tid], gid);
                        if (state == kUnresolved) continue;
                        todo &= ~(1u << b);
                        if (state == kSkip) continue;
                        if (state == kClaimed) atomicAdd(L.counts + n, 1);
#pragma unroll
                        for (int v = 0; v < 4; v++)
                            atomicAdd(L.vals + (size_t)gid * 4 + v, sm.blk[4 * b + v][tid]);
                    }
                    if (!__syncthreads_or(todo)) break;
                    if (tid == 0 && !sm.full) {
                        const int c = append_chunk(L, sm.tail);
                        if (c < 0) sm.full = 1;  // pool overflow: raised, the blocks are dropped
                        else sm.tail = c;
                    }
                    __syncthreads();
                    if (sm.full) todo = 0;
                }
                again = again && el.more;
                if (again) next_position<KIND>(m, el);
            }
        }
        __syncthreads();
        if (tid == 0) sm.nelems = 0;
        __syncthreads();
    }
}

// The rows that rows_2d left (a kernel of its own: inside the rows kernel its
// registers cost the main path a third of its speed).
template <int KIND, typename T>
__device__ __forceinline__ void long_rows_2d(const MeshView& m, const ListLayout& L, const int* __restrict__ queue,
                                             int block, int nblocks, LongSmem& sm) {
    const int count = __ldcg(&L.info->long_rows);
    for (int k = block; k < count; k += nblocks) {
        const int n = __ldcg(queue + k);
        long_row_2d<KIND, T>(m, L, n, __ldcg(L.counts + n), sm);
    }
}

template <int KIND, typename T>
__device__ __forceinline__ void rows_2d(const MeshView& m, const ListLayout& L, int* __restrict__ queue, int block,
                                        int nblocks, RowSmem& sm) {
    constexpr int NPE = KIND == FEM_T3 ? 3 : 4;
    const int tid = threadIdx.x;
    for (long long tile = block; tile * kRowThreads < m.N; tile += nblocks) {
        const int n = (int)min(tile * kRowThreads + tid, (long long)m.N);
        if (n < m.N) {
            int* meta = L.meta1 + (size_t)n * (k2DSlots + 2);
            const int d = __ldcg(L.counts + n);
            bool long_row = d > k2DSlots;
            int u = 0;  // columns besides the diagonal
            if (d > 0 && !long_row) {
#pragma unroll
                for (int q = 0; q < (k2DSlots + 2) / 4; q++) {
                    if (4 * q < d + 2) {
                        const int4 w = ld_cg4(meta + 4 * q);
                        sm.words[4 * q][tid] = w.x;
                        sm.words[4 * q + 1][tid] = w.y;
                        sm.words[4 * q + 2][tid] = w.z;
                        sm.words[4 * q + 3][tid] = w.w;
                    }
                }
                int key[kLow], hi[kOffDiag - kLow];
#pragma unroll
                for (int q = 0; q < kLow; q++) key[q] = -1;
                double dg[4] = {0.0, 0.0, 0.0, 0.0};
                double* vals = L.vals + (size_t)n * (k2DSlots * 4);
                ElemData<NPE> cur, nxt;
                load_nodes<KIND>(m, sm.words[2][tid], cur);
                if (d > 1) load_nodes<KIND>(m, sm.words[3][tid], nxt);
                load_rest<KIND>(m, n, cur);
                for (int i = 0; i < d; i++) {
                    ElemData<NPE> far;
                    if (i + 1 < d) load_rest<KIND>(m, n, nxt);
                    if (i + 2 < d) load_nodes<KIND>(m, sm.words[i + 4][tid], far);
                    for (;;) {
                        double kb[NPE][4];
                        if (!(row_blocks<KIND, T>(cur, m.t, kb) > 0.0)) raise_status(L.info, FEM_ERR_DETJ);
#pragma unroll
                        for (int v = 0; v < 4; v++) dg[v] += kb[0][v];
                        // the columns' slots first, then all of the sums' loads together
                        int s[NPE];
                        int u1 = u;
#pragma unroll
                        for (int b = 1; b < NPE; b++) {
                            const int c = cur.nodes[b];
                            s[b] = u1;
#pragma unroll
                            for (int q = 0; q < kLow; q++) s[b] = key[q] == c ? q : s[b];
                            const bool off = (KIND != FEM_MIXED_2D || b < cur.npe) && c != n;
                            if (!off) s[b] = -1;
                            if (off && s[b] == u1 && u1 < kLow) {
#pragma unroll
                                for (int q = 0; q < kLow; q++) key[q] = q == u1 ? c : key[q];
                                u1++;
                            }
                        }
                        double old[NPE][4];
#pragma unroll
                        for (int b = 1; b < NPE; b++)
#pragma unroll
                            for (int v = 0; v < 4; v++)
                                old[b][v] = s[b] >= 0 && s[b] < u && s[b] < kLow ? sm.acc[s[b]][v][tid] : 0.0;
                        bool same = false;  // an element with a repeated node besides n
#pragma unroll
                        for (int b = 2; b < NPE; b++)
#pragma unroll
                            for (int q = 1; q < b; q++) same |= s[b] == s[q] && s[b] >= 0;
                        if (!same) {
#pragma unroll
                            for (int b = 1; b < NPE; b++) {
                                if (s[b] >= 0 && s[b] < kLow) {
#pragma unroll
                                    for (int v = 0; v < 4; v++) sm.acc[s[b]][v][tid] = old[b][v] + kb[b][v];
                                }
                            }
                        } else {
                            int seen = u;
                            for (int b = 1; b < NPE; b++) {
                                if (s[b] >= 0 && s[b] < kLow) {
                                    for (int v = 0; v < 4; v++)
                                        sm.acc[s[b]][v][tid] = (s[b] < seen ? sm.acc[s[b]][v][tid] : 0.0) + kb[b][v];
                                    seen = max(seen, s[b] + 1);
                                }
                            }
                        }
                        u = max(u, u1);
#pragma unroll
                        for (int b = 1; b < NPE; b++) {
                            if (KIND == FEM_MIXED_2D && b >= cur.npe) continue;
                            if (s[b] < 0) {  // a repeated node
#pragma unroll
                                for (int v = 0; v < 4; v++) dg[v] += kb[b][v];
                            } else if (s[b] >= kLow) {
                                long_row |= add_high(hi, vals, cur.nodes[b], u, kb[b][0], kb[b][1], kb[b][2], kb[b][3]);
                            }
                        }
                        if (!cur.more) break;
                        next_position<KIND>(m, cur);
                    }
                    cur = nxt;
                    nxt = far;
                }
                if (!long_row) {
                    const int low = min(u, kLow);
                    int rank[kLow], rd = 0;
#pragma unroll
                    for (int q = 0; q < kLow; q++) {
                        const bool on = q < low;
                        rank[q] = key[q] > n;
                        rd += on && key[q] < n;
#pragma unroll
                        for (int p = 0; p < q; p++) {
                            const bool less = key[p] < key[q];
                            rank[q] += less;
                            rank[p] += on && !less;
                        }
                    }
                    if (u > kLow) {
                        int lk[kLow], add[kLow + 1];
#pragma unroll
                        for (int q = 0; q < kLow; q++) lk[q] = key[q];
                        place_high(hi, u - kLow, vals, lk, add, n, &sm.words[0][tid], kRowThreads);
#pragma unroll
                        for (int q = 0; q < kLow; q++) rank[q] += add[q];
                        rd += add[kLow];
                    }
                    sm.words[2 + rd][tid] = n + 1;
                    store_block(vals + 4 * rd, dg[0], dg[1], dg[2], dg[3]);
#pragma unroll
                    for (int q = 0; q < kLow; q++) {
                        if (q < low) {
                            sm.words[2 + rank[q]][tid] = key[q] + 1;
                            store_block(vals + 4 * rank[q], sm.acc[q][0][tid], sm.acc[q][1][tid], sm.acc[q][2][tid],
                                        sm.acc[q][3][tid]);
                        }
                    }
                }
            }
            if (long_row) {
                queue[atomicAdd(&L.info->long_rows, 1)] = n;
            } else {
                const int total = d > 0 ? u + 1 : 0;
                L.counts[n] = total;
#pragma unroll
                for (int q = 0; q < (k2DSlots + 2) / 4; q++) {
                    int w[4];
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const int s = 4 * q + k - 2;
                        w[k] = s == -2 ? kRowSorted + total : (s >= 0 && s < total ? sm.words[4 * q + k][tid] : 0);
                    }
                    reinterpret_cast<int4*>(meta)[q] = make_int4(w[0], w[1], w[2], w[3]);
                }
            }
        }
    }
}

// Clears a scatter's counters and info word.
__device__ __forceinline__ void lists_begin(const ListLayout& L, int block, int nblocks) {
    for (int i = block * blockDim.x + threadIdx.x; i < L.N; i += nblocks * blockDim.x) L.counts[i] = 0;
    if (block == 0 && threadIdx.x == 0) {
        DevInfo d{};
        d.pool_chunks = L.cap2;
        *L.info = d;
    }
}

}  // namespace
}  // namespace fem
