// Hex20 row lists -> CSR, BSR or upper-triangle CSR: each row's element blocks
// are summed where they are written.
//
// Replaces the value half of assembleGlobalStiffnessKernelALLSFixedArray
// (ALLS_Hex20_3D_Assembly_Performance.cu:212-256, atomicAdd per entry) and
// convertALLStoCSRKernelFixedArray (H20:259-278). One warp per row node, the
// nodes taken in order by all CTAs together (neighbouring rows read the same
// elements' Ke while it is in L2). The row's 3x3 blocks accumulate in shared
// memory (a window of kWindow columns at a time); for each of the node's
// occurrences (element e, position a) the lanes read the 20 blocks (a, b) of
// the packed Ke (180 doubles, a block below the diagonal from its transpose)
// and add them at the ranks that the scatter recorded, the next occurrence's
// loads in flight meanwhile. An element names a column node once, so the
// lanes' additions never meet; a repeated node's further blocks are added one
// by one. Then the rows leave with consecutive lanes on consecutive entries.
// No value is added atomically and the sums do not depend on timing.
//
// A 64^3 mesh moves 4.0 GB of Ke in and 6.7 GB of CSR out. B200: 4.02 ms; the
// value pass into list blocks (stores and FP64 atomics) and the copy out of the
// lists that this replaces took 5.18 + 3.06 ms with the Ke computed inside.
#include <algorithm>

#include "consolidate.cuh"
#include "rows_hex20.cuh"

namespace fem {
namespace {

// Resident CTAs per SM that the registers are set for (4 spill).
#ifndef FEM_HEXW_CTAS
#define FEM_HEXW_CTAS 3
#endif
constexpr int kWarps = 8;
constexpr int kThreads = kWarps * 32;
constexpr int kWindow = 96;   // columns summed at once (an inner node of a regular mesh has 51 or 81)
constexpr int kItems = 6;     // entries of a 180-entry slab per lane

struct WriteHexSmem {
    double acc[kWindow * 9];
    int col[kWindow];
};

__device__ __forceinline__ int packed_block(int I, int J) { return I * 20 - I * (I - 1) / 2 + J - I; }

template <int kMode>
__global__ void __launch_bounds__(kThreads, FEM_HEXW_CTAS)
    k_write_hex20(ListLayout L, HexRows h, const int* __restrict__ ucounts, const int* __restrict__ row_ptr,
                  int* __restrict__ col_idx, double* __restrict__ values, long long capacity) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int s_sum[kWarps], s_max[kWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    WriteHexSmem& sm = reinterpret_cast<WriteHexSmem*>(smem_raw)[warp];
    if (__ldg(&L.info->nnz) > capacity) return;  // FEM_ERR_CAPACITY already raised; write nothing
    // entry i of this lane in a slab: block b(i), entry v(i) of it
    int sb[kItems], sv[kItems], st[kItems];
#pragma unroll
    for (int i = 0; i < kItems; i++) {
        const int x = lane + 32 * i;
        sb[i] = x / 9;
        sv[i] = x - 9 * sb[i];
        st[i] = (sv[i] % 3) * 3 + sv[i] / 3;  // the transposed entry
    }
    int t_sum = 0, t_max = 0;
    for (long long nn = (long long)blockIdx.x * kWarps + warp; nn < L.N; nn += (long long)gridDim.x * kWarps) {
        const int n = (int)nn, u = __ldg(L.counts + n), lo = __ldg(h.off + n), d = __ldg(h.off + n + 1) - lo;
        const int next = u > L.S1 ? __ldg(L.meta1 + (size_t)n * L.H1 + 1) : 0;
        // first column written (upper: the node itself)
        const int k0 = kMode == kOutUpper ? u - __ldg(ucounts + n) : 0;
        t_sum += u;
        t_max = max(t_max, u);
        const long long base = __ldg(row_ptr + (size_t)n * (kMode == kOutBsr ? 1 : 3));
        for (int w0 = k0; w0 < u; w0 += kWindow) {
            const int uw = min(kWindow, u - w0);
            for (int k = lane; k < uw; k += 32) sm.col[k] = __ldg(hex_col_word(L, n, next, w0 + k)) - 1;
            for (int x = lane; x < uw * 9; x += 32) sm.acc[x] = 0.0;
            double val[kItems];
            unsigned rk[kItems];
            auto fetch = [&](int t) {
                const unsigned o = (unsigned)__ldg(h.inc + lo + t), e = o / 20, a = o - 20 * e;
                const double* ke = h.ke + (size_t)e * kPackedHex20;
                const unsigned short* mp = h.map + (size_t)o * 20;
#pragma unroll
                for (int i = 0; i < kItems; i++) {
                    if (i < kItems - 1 || lane < 20) {
                        const int b = sb[i];
                        const bool up = b >= (int)a;
                        rk[i] = __ldg(mp + b);
                        val[i] = __ldg(ke + 9 * (up ? packed_block(a, b) : packed_block(b, a)) + (up ? sv[i] : st[i]));
                    } else {
                        rk[i] = kRankMask;
                        val[i] = 0.0;
                    }
                }
            };
            if (d > 0) fetch(0);
            __syncwarp();
            for (int t = 0; t < d; t++) {
                int at[kItems];
                double x[kItems];
                bool dup = false;
#pragma unroll
                for (int i = 0; i < kItems; i++) {
                    const int r = (int)(rk[i] & kRankMask) - w0;
                    const bool in = (unsigned)r < (unsigned)uw;
                    at[i] = in ? r * 9 + sv[i] : -1;
                    x[i] = val[i];
                    if (rk[i] & kRankDup) {
                        dup |= in;
                        at[i] = in ? -2 - at[i] : -1;
                    }
                }
                if (t + 1 < d) fetch(t + 1);
                double y[kItems];
#pragma unroll
                for (int i = 0; i < kItems; i++) y[i] = at[i] >= 0 ? sm.acc[at[i]] : 0.0;
#pragma unroll
                for (int i = 0; i < kItems; i++)
                    if (at[i] >= 0) sm.acc[at[i]] = y[i] + x[i];
                __syncwarp();
                if (__any_sync(0xFFFFFFFFu, dup)) {  // a repeated node's further blocks, one at a time
                    for (int b = 1; b < 20; b++) {
#pragma unroll
                        for (int i = 0; i < kItems; i++)
                            if (at[i] < -1 && sb[i] == b) sm.acc[-2 - at[i]] += x[i];
                        __syncwarp();
                    }
                }
            }
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
    }
    // list statistics (one atomic pair per CTA)
    if (lane == 0) {
        s_sum[warp] = t_sum;
        s_max[warp] = t_max;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < kWarps; w++) {
            t_sum += s_sum[w];
            t_max = max(t_max, s_max[w]);
        }
        atomicAdd(reinterpret_cast<unsigned long long*>(&L.info->list_entries), (unsigned long long)t_sum);
        atomicMax(&L.info->max_row_entries, t_max);
    }
}

// Columns >= n of every row node: the sorted row's tail from the node itself on.
__global__ void __launch_bounds__(256) k_count_upper_hex20(ListLayout L, int* __restrict__ ucounts) {
    for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < L.N; n += gridDim.x * blockDim.x) {
        const int u = __ldg(L.counts + n), next = u > L.S1 ? __ldg(L.meta1 + (size_t)n * L.H1 + 1) : 0;
        int lo = 0, hi = u;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (__ldg(hex_col_word(L, n, next, mid)) - 1 < n) lo = mid + 1;
            else hi = mid;
        }
        ucounts[n] = u - lo;
    }
}

template <int kMode>
cudaError_t launch_mode(const ListLayout& L, const HexRows& h, const int* ucounts, const int* row_ptr, int* col_idx,
                        double* values, long long capacity, cudaStream_t s) {
    static DeviceCache cache;
    const size_t smem = kWarps * sizeof(WriteHexSmem);
    int per_sm = 0;
    const cudaError_t err = per_device(cache, [&](int& v) {
        cudaError_t e =
            cudaFuncSetAttribute(k_write_hex20<kMode>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (!e) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, k_write_hex20<kMode>, kThreads, smem);
        return e;
    }, per_sm);
    if (err) return err;
    const long long want = ((long long)L.N + kWarps - 1) / kWarps;
    const int grid = (int)std::min<long long>(want, (long long)per_sm * sm_count());
    k_write_hex20<kMode><<<grid, kThreads, smem, s>>>(L, h, ucounts, row_ptr, col_idx, values, capacity);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_count_upper_hex20(const ListLayout& L, int* ucounts, cudaStream_t s) {
    const int grid = (int)std::min<long long>(((long long)L.N + 255) / 256, (long long)sm_count() * 8);
    k_count_upper_hex20<<<grid, 256, 0, s>>>(L, ucounts);
    return cudaGetLastError();
}

cudaError_t launch_write_hex20(const ListLayout& L, const HexRows& h, int mode, const int* ucounts, const int* row_ptr,
                               int* col_idx, double* values, long long capacity, cudaStream_t s) {
    if (mode == kOutBsr) return launch_mode<kOutBsr>(L, h, ucounts, row_ptr, col_idx, values, capacity, s);
    if (mode == kOutUpper) return launch_mode<kOutUpper>(L, h, ucounts, row_ptr, col_idx, values, capacity, s);
    return launch_mode<kOutCsr>(L, h, ucounts, row_ptr, col_idx, values, capacity, s);
}

}  // namespace fem
