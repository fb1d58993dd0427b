// Value-only re-assembly: a mesh whose connectivity is unchanged (new
// coordinates, E or nu, as in nonlinear or time-stepping solvers) is
// re-assembled into the CSR pattern of an earlier assembly without building
// any list.
//
// The reference has no such path: every assembly repeats the list build
// (assembleGlobalStiffnessKernelALLS, ALLS_Quad2D_Assembly_Accuracy_Analysis.cu:394-468)
// and, on the host, the pattern (buildCSRStructure, Q4A:605-645).
//
// 2-D kinds (k_rows_values_2d): the map holds, node by node, the node's
// occurrences (element e, local position a) and the ranks of the element's
// nodes in the node's sorted row. A thread owns a node: it computes the node's
// row of each of its elements' Ke and sums the blocks at their ranks in shared
// memory; the warp then writes its nodes' two CSR rows with consecutive lanes
// on consecutive entries. No zeroing, no atomics, and nothing is searched. Rows
// of more than 14 columns are added with FP64 atomics by their warp. What
// bounds it: the gathered loads (element -> nodes -> coordinates) and the
// instructions of the element rows. B200, T3 1001x699 (shuffled elements): 177
// us, where the block-position form took 301 us plus 28 us of zeroing.
//
// Block positions (Hex20, small 2-D meshes, whose time is the serial walk over a
// node's elements above (min_row_nodes in fem_api.cu), and 2-D meshes whose
// occurrences do not fit, mostly unconnected triangles): the map records, for every element node block (a, b),
// the CSR position of its first entry, position of block (a, b) of element e at
// e * G + a * npe + b, G = npe^2; the element blocks are added there with FP64
// atomics, in the element order of reorder.cu, which the map holds too. Entry
// (i, j) of block (a, b) lies at p + i * rowlen + j, rowlen being the length of
// the block's first CSR row (the dpn rows of a node have the same columns).
// Bound by the L2's FP64 atomics (about 180 G/s measured; adding the entries of
// a block row by neighbouring lanes changes little: 301 against 281 us).
#include <algorithm>

#include "element2d.cuh"
#include "launch.h"
#include "rows_hex20.cuh"

namespace fem {
namespace {

constexpr int kThreads = 256;

// Position of column col in CSR row r (sorted), or -1.
__device__ __forceinline__ int find_col(const int* __restrict__ row_ptr, const int* __restrict__ col_idx, int r,
                                        int col) {
    int lo = __ldg(row_ptr + r), hi = __ldg(row_ptr + r + 1) - 1;
    while (lo <= hi) {
        const int mid = (lo + hi) >> 1;
        const int c = __ldg(col_idx + mid);
        if (c == col) return mid;
        if (c < col) lo = mid + 1;
        else hi = mid - 1;
    }
    return -1;
}

__device__ __forceinline__ int npe_of(const MeshView& m, int e) {
    if (m.types) return __ldg(m.types + e) == FEM_Q4 ? 4 : 3;
    return m.stride == 20 ? 20 : m.stride;
}

// One thread per (element, block): binary search of the block's first column
// in its first row. Blocks past the element's nodes (T3 in a mixed mesh) get -1, and so do all blocks of an element
// with a bad node id: it takes no part, and the re-assembly reads the coordinates of every node of an element that does.
__global__ void k_build_map(MeshView m, int dpn, int npe_max, const int* __restrict__ row_ptr,
                            const int* __restrict__ col_idx, int* __restrict__ map, int* __restrict__ status,
                            const int* gate) {
    if (gate && __ldcg(gate) == 0) return;
    const int G = npe_max * npe_max;
    const long long total = (long long)m.E_count * G;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < total;
         t += (long long)gridDim.x * blockDim.x) {
        const int e = (int)(t / G), k = (int)(t - (long long)e * G);
        const int a = k / npe_max, b = k - a * npe_max;
        const int npe = npe_of(m, e);
        int pos = -1;
        if (a < npe && b < npe) {
            bool bad = false;
            for (int k = 0; k < npe; k++) {
                const int n = __ldg(m.conn + (size_t)e * m.stride + k);
                bad |= n < 0 || n >= m.N;
            }
            if (bad) {
                atomicOr(status, 1 << FEM_ERR_BAD_MESH);
            } else {
                const int na = __ldg(m.conn + (size_t)e * m.stride + a), nb = __ldg(m.conn + (size_t)e * m.stride + b);
                pos = find_col(row_ptr, col_idx, dpn * na, dpn * nb);
                if (pos < 0) atomicOr(status, 1 << FEM_ERR_INTERNAL);  // the pattern lacks the block
            }
        }
        map[t] = pos;
    }
}

// 2-D value-only assembly: one lane per element block (NPE^2 lanes per
// element), elements perm[range[0], range[1]), FP64 red.add into the values.
template <int NPE, typename T>
__device__ __forceinline__ void add_blocks_2d(const MeshView& m, const BlocksMap& b2, const int* __restrict__ range,
                                              const int* __restrict__ row_ptr, double* __restrict__ values,
                                              int* __restrict__ status) {
    constexpr int GL = NPE * NPE, EPW = 32 / GL;
    const int lane = threadIdx.x & 31;
    const int eslot = lane / GL, sub = lane - eslot * GL, a = sub / NPE, b = sub - (sub / NPE) * NPE;
    const int begin = range[0], count = range[1] - range[0];
    const long long warp_id = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long stride = (((long long)gridDim.x * blockDim.x) >> 5) * EPW;
    for (long long i = warp_id * EPW + eslot; i - eslot < count; i += stride) {
        if (eslot >= EPW || i >= count) continue;
        const int e = __ldg(b2.perm + begin + i);
        const int p = __ldg(b2.pos + (size_t)e * b2.G + a * (b2.G == 16 ? 4 : NPE) + b);
        if (p < 0) continue;  // bad node (reported when the map was built)
        int nodes[NPE];
#pragma unroll
        for (int k = 0; k < NPE; k++) nodes[k] = __ldg(m.conn + (size_t)e * m.stride + k);
        double xe[NPE], ye[NPE];
#pragma unroll
        for (int k = 0; k < NPE; k++) {
            xe[k] = __ldg(m.x + nodes[k]);
            ye[k] = __ldg(m.y + nodes[k]);
        }
        const double E = m.E ? __ldg(m.E + e) : m.E0;
        const double nu = m.nu ? __ldg(m.nu + e) : m.nu0;
        double kv[4];
        const double det = ke_block_2d<NPE, T>(xe, ye, E, nu, m.t, a, b, kv);
        if (sub == 0 && !(det > 0.0)) atomicOr(status, 1 << FEM_ERR_DETJ);
        int row = nodes[0];
#pragma unroll
        for (int k = 1; k < NPE; k++) row = a == k ? nodes[k] : row;
        const int len = __ldg(row_ptr + 2 * row + 1) - __ldg(row_ptr + 2 * row);
        atomicAdd(values + p, kv[0]);
        atomicAdd(values + p + 1, kv[1]);
        atomicAdd(values + p + len, kv[2]);
        atomicAdd(values + p + len + 1, kv[3]);
    }
}

template <int NPE, typename T>
__global__ void __launch_bounds__(kThreads) k_reassemble_2d(MeshView m, BlocksMap b2, const int* __restrict__ range,
                                                            const int* __restrict__ row_ptr,
                                                            double* __restrict__ values, int* __restrict__ status) {
    add_blocks_2d<NPE, T>(m, b2, range, row_ptr, values, status);
}

// ---- 2-D rows ---------------------------------------------------------------------

template <int KIND>
__device__ __forceinline__ int elem_nodes(const MeshView& m, int e) {
    if (KIND == FEM_T3) return 3;
    if (KIND == FEM_Q4) return 4;
    return __ldg(m.types + e) == FEM_Q4 ? 4 : 3;
}

template <int KIND>
__device__ __forceinline__ bool bad_nodes(const MeshView& m, int e, int npe) {
    bool bad = false;
    for (int k = 0; k < npe; k++) {
        const int n = __ldg(m.conn + (size_t)e * m.stride + k);
        bad |= n < 0 || n >= m.N;
    }
    return bad;
}

template <int KIND>
__global__ void __launch_bounds__(kThreads) k_map_count(MeshView m, int* __restrict__ cnt, int* __restrict__ status) {
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < m.E_count; e += gridDim.x * blockDim.x) {
        const int npe = elem_nodes<KIND>(m, e);
        if (bad_nodes<KIND>(m, e, npe)) {
            atomicOr(status, 1 << FEM_ERR_BAD_MESH);
            continue;
        }
        for (int k = 0; k < npe; k++) atomicAdd(cnt + __ldg(m.conn + (size_t)e * m.stride + k), 1);
    }
}

__global__ void __launch_bounds__(kScanThreads) k_map_sums(const int* __restrict__ cnt, int N,
                                                           long long* __restrict__ tiles) {
    __shared__ long long s_warp[kScanThreads / 32 + 1];
    occ_sums(cnt, N, tiles, blockIdx.x, s_warp);
}

__global__ void __launch_bounds__(kScanThreads) k_map_offsets(const int* __restrict__ cnt, int N,
                                                              const long long* __restrict__ tiles,
                                                              int* __restrict__ off) {
    __shared__ OccSmem sm;
    occ_offsets(cnt, N, tiles, off, blockIdx.x, gridDim.x, sm);
}

// The occurrences of every node (cnt counts down to zero).
template <int KIND>
__global__ void __launch_bounds__(kThreads) k_map_fill(MeshView m, const int* __restrict__ off, int* __restrict__ cnt,
                                                       unsigned* __restrict__ occ) {
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < m.E_count; e += gridDim.x * blockDim.x) {
        const int npe = elem_nodes<KIND>(m, e);
        if (bad_nodes<KIND>(m, e, npe)) continue;
        for (int k = 0; k < npe; k++) {
            const int n = __ldg(m.conn + (size_t)e * m.stride + k);
            occ[__ldg(off + n) + atomicSub(cnt + n, 1) - 1] = ((unsigned)e << 2) | k;
        }
    }
}

// ranks[NPE * j + k]: rank in the row of occurrence j's node of the element's node k positions after it.
// blocks: set when the first row does not start at entry 0 (the rows would not cover the entries before it, and could
// start at odd places), a node's two rows differ in length or are odd, a column node's pair starts at an odd place, a
// rank passes 16 bits or the pattern lacks a block (a caller's own pattern: with further columns, or too small).
template <int KIND>
__global__ void __launch_bounds__(kThreads) k_map_ranks(MeshView m, const int* __restrict__ off,
                                                        const unsigned* __restrict__ occ,
                                                        const int* __restrict__ row_ptr,
                                                        const int* __restrict__ col_idx,
                                                        unsigned short* __restrict__ ranks, int* __restrict__ blocks) {
    constexpr int NPE = KIND == FEM_T3 ? 3 : 4;
    const int total = __ldg(off + m.N);
    bool other = false;
    for (long long n = blockIdx.x * blockDim.x + threadIdx.x; n < m.N; n += gridDim.x * blockDim.x) {
        const int r0 = __ldg(row_ptr + 2 * n), r1 = __ldg(row_ptr + 2 * n + 1), r2 = __ldg(row_ptr + 2 * n + 2);
        other |= r2 - r1 != r1 - r0 || ((r1 - r0) & 1) || (n == 0 && r0 != 0);
    }
    for (long long j = blockIdx.x * blockDim.x + threadIdx.x; j < total; j += gridDim.x * blockDim.x) {
        const unsigned w = __ldg(occ + j);
        const int e = (int)(w >> 2), a = (int)(w & 3u), npe = elem_nodes<KIND>(m, e);
        const int n = __ldg(m.conn + (size_t)e * m.stride + a);
        for (int k = 0; k < npe; k++) {
            const int b = a + k < npe ? a + k : a + k - npe;
            const int p = find_col(row_ptr, col_idx, 2 * n, 2 * __ldg(m.conn + (size_t)e * m.stride + b));
            const int r = p - __ldg(row_ptr + 2 * n);
            other |= p < 0 || (r & 1) || r / 2 > 0xFFFF;
            ranks[(size_t)NPE * j + k] = (unsigned short)(r / 2);
        }
    }
    if (other) *blocks = 1;
}

constexpr int kRowThreads = 64;
constexpr int kRowPad = kRowThreads + 1;  // a node's entries on different banks, and a warp's nodes too
// Columns of a row summed in shared memory (T3 nodes of up to 9 triangles, quadrilateral nodes of up to 6), and the
// resident CTAs the registers are set for. T3: 8 CTAs of 21 KB leave L1 60 KB for the gathered loads (9 CTAs 223, 10
// CTAs 217 us; 14 columns, 7 CTAs 232 us).
#ifndef FEM_REROWS_T3
#define FEM_REROWS_T3 10
#define FEM_REROWS_T3_CTAS 8
#endif
#ifndef FEM_REROWS_Q4
#define FEM_REROWS_Q4 14
#define FEM_REROWS_Q4_CTAS 6
#endif
template <int KIND>
struct RowsShape {
    static constexpr int kCols = KIND == FEM_T3 ? FEM_REROWS_T3 : FEM_REROWS_Q4;
    static constexpr int kCtas = KIND == FEM_T3 ? FEM_REROWS_T3_CTAS : FEM_REROWS_Q4_CTAS;
};

template <int NPE>
struct OccData {
    int e, npe;
    int nodes[NPE];  // [0]: unused (the row node)
    double x[NPE], y[NPE], E, nu;
    unsigned short rank[NPE];
};

template <int KIND, int NPE>
__device__ __forceinline__ void load_occ(const MeshView& m, unsigned w, const unsigned short* ranks, int j,
                                         OccData<NPE>& d) {
    d.e = (int)(w >> 2);
    d.npe = elem_nodes<KIND>(m, d.e);
    const int a = (int)(w & 3u);
#pragma unroll
    for (int k = 1; k < NPE; k++) {
        const int b = a + k < d.npe ? a + k : a + k - d.npe;
        d.nodes[k] = __ldg(m.conn + (size_t)d.e * m.stride + (k < d.npe ? b : a));
    }
#pragma unroll
    for (int k = 0; k < NPE; k++) d.rank[k] = __ldg(ranks + (size_t)NPE * j + k);
}

template <int NPE>
__device__ __forceinline__ void load_geometry(const MeshView& m, OccData<NPE>& d) {
#pragma unroll
    for (int k = 1; k < NPE; k++) {
        d.x[k] = __ldg(m.x + d.nodes[k]);
        d.y[k] = __ldg(m.y + d.nodes[k]);
    }
    d.E = m.E ? __ldg(m.E + d.e) : m.E0;
    d.nu = m.nu ? __ldg(m.nu + d.e) : m.nu0;
}

// Blocks (row node, node k positions after it) of an occurrence, k < npe. Returns detJ.
template <int KIND, typename T, int NPE>
__device__ __forceinline__ double occ_blocks(const OccData<NPE>& d, double t, double (&k)[NPE][4]) {
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

// Clears the call's info word and the entries that no row of the mesh covers: those behind the rows or, for a pattern
// that is not in the form of rows, all of them.
__global__ void __launch_bounds__(kThreads) k_rows_begin_2d(DevInfo* info, const int* __restrict__ blocks,
                                                            const int* __restrict__ end, double* __restrict__ values,
                                                            long long nnz) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *info = DevInfo{};
    const long long first = __ldg(end), all = __ldg(blocks);
    for (long long i = (all ? 0 : first) + (long long)blockIdx.x * kThreads + threadIdx.x; i < nnz;
         i += (long long)gridDim.x * kThreads)
        values[i] = 0.0;
}

template <int KIND, typename T>
__global__ void __launch_bounds__(kRowThreads, RowsShape<KIND>::kCtas)
    k_rows_values_2d(MeshView m, const int* __restrict__ off, const unsigned* __restrict__ occ,
                     const unsigned short* __restrict__ ranks, const int* __restrict__ row_ptr,
                     double* __restrict__ values, bool wide, int* __restrict__ status,
                     const int* __restrict__ blocks, BlocksMap b2) {
    constexpr int NPE = KIND == FEM_T3 ? 3 : 4, kRowCols = RowsShape<KIND>::kCols;
    constexpr unsigned kFull = 0xFFFFFFFFu;
    __shared__ double acc[kRowCols][4][kRowPad];
    const int tid = threadIdx.x, lane = tid & 31, warp0 = tid & ~31;
    if (__ldg(blocks)) {  // the pattern is not in this form; the values are zero (k_rows_begin_2d)
        if constexpr (KIND != FEM_T3) add_blocks_2d<4, T>(m, b2, b2.ranges, row_ptr, values, status);
        if constexpr (KIND != FEM_Q4) add_blocks_2d<3, T>(m, b2, b2.ranges + 2, row_ptr, values, status);
        return;
    }
    for (long long tile = blockIdx.x; tile * kRowThreads < m.N; tile += gridDim.x) {
        const long long n = tile * kRowThreads + tid;
        int base = 0, u = 0, lo = 0, d = 0;
        if (n < m.N) {
            base = __ldg(row_ptr + 2 * n);
            u = (__ldg(row_ptr + 2 * n + 1) - base) / 2;
            lo = __ldg(off + n);
            d = __ldg(off + n + 1) - lo;
        }
        const bool fits = u <= kRowCols;
        if (fits) {
            for (int q = 0; q < u; q++)
#pragma unroll
                for (int v = 0; v < 4; v++) acc[q][v][tid] = 0.0;
        }
        if (fits && d > 0) {
            OccData<NPE> cur, nxt;
            const double xn = __ldg(m.x + n), yn = __ldg(m.y + n);
            double dg[4] = {0.0, 0.0, 0.0, 0.0};
            load_occ<KIND>(m, __ldg(occ + lo), ranks, lo, cur);
            unsigned w1 = d > 1 ? __ldg(occ + lo + 1) : 0;
            load_geometry(m, cur);
            int diag = 0;
            for (int i = 0; i < d; i++) {
                // the next occurrence's nodes and the one after's word are in flight
                if (i + 1 < d) load_occ<KIND>(m, w1, ranks, lo + i + 1, nxt);
                if (i + 2 < d) w1 = __ldg(occ + lo + i + 2);
                cur.x[0] = xn;
                cur.y[0] = yn;
                double kb[NPE][4];
                if (!(occ_blocks<KIND, T>(cur, m.t, kb) > 0.0)) atomicOr(status, 1 << FEM_ERR_DETJ);
                if (i + 1 < d) load_geometry(m, nxt);
                diag = cur.rank[0];
#pragma unroll
                for (int v = 0; v < 4; v++) dg[v] += kb[0][v];
                bool same = false;  // a repeated node
#pragma unroll
                for (int b = 2; b < NPE; b++)
#pragma unroll
                    for (int q = 1; q < b; q++) same |= b < cur.npe && cur.rank[b] == cur.rank[q];
                if (!same) {
                    double old[NPE][4];
#pragma unroll
                    for (int b = 1; b < NPE; b++)
                        if (b < cur.npe)
#pragma unroll
                            for (int v = 0; v < 4; v++) old[b][v] = acc[cur.rank[b]][v][tid];
#pragma unroll
                    for (int b = 1; b < NPE; b++)
                        if (b < cur.npe)
#pragma unroll
                            for (int v = 0; v < 4; v++) acc[cur.rank[b]][v][tid] = old[b][v] + kb[b][v];
                } else {
#pragma unroll
                    for (int b = 1; b < NPE; b++)
                        if (b < cur.npe)
#pragma unroll
                            for (int v = 0; v < 4; v++) acc[cur.rank[b]][v][tid] += kb[b][v];
                }
                cur = nxt;
            }
#pragma unroll
            for (int v = 0; v < 4; v++) acc[diag][v][tid] += dg[v];
        }
        __syncwarp();
        // the warp's nodes: 2 rows of 2 u entries each
        if (wide) {  // two nodes at a time, 16 lanes each, two entries per lane and store
            const int half = lane >> 4, hl = lane & 15;
#pragma unroll 4
            for (int j = 0; j < 32; j += 2) {
                const int uj = __shfl_sync(kFull, fits ? u : 0, j + half), bj = __shfl_sync(kFull, base, j + half);
                for (int x = hl; x < 2 * uj; x += 16) {
                    const int i = x >= uj, q = x - (i ? uj : 0);
                    const double* a = &acc[q][2 * i][warp0 + j + half];
                    *reinterpret_cast<double2*>(values + (long long)bj + 2 * x) = make_double2(a[0], a[kRowPad]);
                }
            }
        } else {
            for (int j = 0; j < 32; j++) {
                const int uj = __shfl_sync(kFull, fits ? u : 0, j), bj = __shfl_sync(kFull, base, j);
                for (int x = lane; x < 4 * uj; x += 32) {
                    const int i = x >= 2 * uj, c = x - i * 2 * uj;
                    values[(long long)bj + x] = acc[c >> 1][2 * i + (c & 1)][warp0 + j];
                }
            }
        }
        // rows too long for the shared memory: the warp's lanes on the node's occurrences
        for (unsigned longs = __ballot_sync(kFull, !fits); longs; longs &= longs - 1) {
            const int src = __ffs(longs) - 1;
            const long long nl = tile * kRowThreads + warp0 + src;
            const int ul = __shfl_sync(kFull, u, src), bl = __shfl_sync(kFull, base, src);
            const int ll = __shfl_sync(kFull, lo, src), dl = __shfl_sync(kFull, d, src);
            for (int x = lane; x < 4 * ul; x += 32) values[(long long)bl + x] = 0.0;
            __syncwarp();
            for (int i = lane; i < dl; i += 32) {
                OccData<NPE> el;
                load_occ<KIND>(m, __ldg(occ + ll + i), ranks, ll + i, el);
                load_geometry(m, el);
                el.x[0] = __ldg(m.x + nl);
                el.y[0] = __ldg(m.y + nl);
                double kb[NPE][4];
                if (!(occ_blocks<KIND, T>(el, m.t, kb) > 0.0)) atomicOr(status, 1 << FEM_ERR_DETJ);
#pragma unroll
                for (int b = 0; b < NPE; b++) {
                    if (b >= el.npe) continue;
                    double* p = values + bl + 2 * el.rank[b];
                    atomicAdd(p, kb[b][0]);
                    atomicAdd(p + 1, kb[b][1]);
                    atomicAdd(p + 2 * ul, kb[b][2]);
                    atomicAdd(p + 2 * ul + 1, kb[b][3]);
                }
            }
            __syncwarp();
        }
        __syncwarp();
    }
}

template <int KIND>
cudaError_t build_rows_map(const MeshView& m, const int* row_ptr, const int* col_idx, const RowsMap& r, int* cnt,
                           long long* tiles, DevInfo* info, cudaStream_t s) {
    const cudaError_t err = cudaMemsetAsync(cnt, 0, (size_t)m.N * sizeof(int), s);
    if (err) return err;
    const int ntiles = row_tiles(m.N);
    const int grid = (int)std::min<long long>(((long long)m.E_count + kThreads - 1) / kThreads, (long long)sm_count() * 8);
    int* status = &info->status_bits;
    k_map_count<KIND><<<grid, kThreads, 0, s>>>(m, cnt, status);
    k_map_sums<<<ntiles, kScanThreads, 0, s>>>(cnt, m.N, tiles);
    k_map_offsets<<<ntiles, kScanThreads, 0, s>>>(cnt, m.N, tiles, r.off);
    k_map_fill<KIND><<<grid, kThreads, 0, s>>>(m, r.off, cnt, r.occ);
    k_map_ranks<KIND><<<(int)std::min<long long>(3ll * grid, (long long)sm_count() * 16), kThreads, 0, s>>>(
        m, r.off, r.occ, row_ptr, col_idx, r.ranks, r.blocks);
    return cudaGetLastError();
}

template <int KIND, typename T>
cudaError_t rows_values(const MeshView& m, const RowsMap& r, const BlocksMap& b2, const int* row_ptr, double* values,
                        int* status, cudaStream_t s) {
    static DeviceCache cache;
    int per_sm = 0;
    const cudaError_t err = per_device(cache, [](int& v) {
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, k_rows_values_2d<KIND, T>, kRowThreads, 0);
    }, per_sm);
    if (err) return err;
    const long long tiles = ((long long)m.N + kRowThreads - 1) / kRowThreads;
    k_rows_values_2d<KIND, T><<<(int)std::min<long long>(tiles, (long long)per_sm * sm_count()), kRowThreads, 0, s>>>(
        m, r.off, r.occ, r.ranks, row_ptr, values, reinterpret_cast<uintptr_t>(values) % 16 == 0, status, r.blocks, b2);
    return cudaGetLastError();
}

template <typename T>
cudaError_t rows_values_kind(const MeshView& m, int kind, const RowsMap& r, const BlocksMap& b2, const int* row_ptr,
                             double* values, int* status, cudaStream_t s) {
    if (kind == FEM_T3) return rows_values<FEM_T3, T>(m, r, b2, row_ptr, values, status, s);
    if (kind == FEM_Q4) return rows_values<FEM_Q4, T>(m, r, b2, row_ptr, values, status, s);
    return rows_values<FEM_MIXED_2D, T>(m, r, b2, row_ptr, values, status, s);
}

}  // namespace

cudaError_t launch_build_map(const MeshView& m, int kind, const int* row_ptr, const int* col_idx, int* map,
                             int* status, cudaStream_t s, const int* gate) {
    const int npe_max = kind == FEM_HEX20 ? 20 : (kind == FEM_T3 ? 3 : 4);
    const int dpn = kind == FEM_HEX20 ? 3 : 2;
    const long long total = (long long)m.E_count * npe_max * npe_max;
    if (total == 0) return cudaSuccess;
    const int grid = (int)std::min<long long>((total + kThreads - 1) / kThreads, (long long)sm_count() * 16);
    k_build_map<<<grid, kThreads, 0, s>>>(m, dpn, npe_max, row_ptr, col_idx, map, status, gate);
    return cudaGetLastError();
}

template <typename T>
void reassemble_2d_t(const MeshView& m, const BlocksMap& b2, const int* row_ptr, double* values, int* status,
                     cudaStream_t s) {
    const bool has_q4 = m.types || m.stride == 4, has_t3 = m.types || m.stride == 3;
    const long long warps = ((long long)m.E_count + 1) / 2;
    const int grid = (int)std::min<long long>((warps * 32 + kThreads - 1) / kThreads, (long long)sm_count() * 8);
    if (has_q4)
        k_reassemble_2d<4, T><<<grid > 0 ? grid : 1, kThreads, 0, s>>>(m, b2, b2.ranges, row_ptr, values, status);
    if (has_t3)
        k_reassemble_2d<3, T><<<grid > 0 ? grid : 1, kThreads, 0, s>>>(m, b2, b2.ranges + 2, row_ptr, values, status);
}

cudaError_t launch_reassemble_2d(const MeshView& m, int precision, const BlocksMap& b2, const int* row_ptr,
                                 double* values, int* status, cudaStream_t s) {
    if (precision == FEM_PREC_FP32)
        reassemble_2d_t<float>(m, b2, row_ptr, values, status, s);
    else
        reassemble_2d_t<double>(m, b2, row_ptr, values, status, s);
    return cudaGetLastError();
}

cudaError_t launch_build_rows_map(const MeshView& m, int kind, const int* row_ptr, const int* col_idx, const RowsMap& r,
                                  int* cnt, long long* tiles, DevInfo* info, cudaStream_t s) {
    if (kind == FEM_T3) return build_rows_map<FEM_T3>(m, row_ptr, col_idx, r, cnt, tiles, info, s);
    if (kind == FEM_Q4) return build_rows_map<FEM_Q4>(m, row_ptr, col_idx, r, cnt, tiles, info, s);
    return build_rows_map<FEM_MIXED_2D>(m, row_ptr, col_idx, r, cnt, tiles, info, s);
}

cudaError_t launch_rows_values_2d(const MeshView& m, int kind, int precision, const RowsMap& r, const BlocksMap& b2,
                                  const int* row_ptr, double* values, long long nnz, DevInfo* info, cudaStream_t s) {
    const int grid = (int)std::min<long long>((nnz + 4 * kThreads - 1) / (4 * kThreads) + 1, 2ll * sm_count());
    k_rows_begin_2d<<<grid, kThreads, 0, s>>>(info, r.blocks, row_ptr + 2 * (size_t)m.N, values, nnz);
    int* status = &info->status_bits;
    return precision == FEM_PREC_FP32 ? rows_values_kind<float>(m, kind, r, b2, row_ptr, values, status, s)
                                      : rows_values_kind<double>(m, kind, r, b2, row_ptr, values, status, s);
}

}  // namespace fem
