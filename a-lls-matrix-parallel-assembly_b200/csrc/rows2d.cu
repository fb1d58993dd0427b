// K1 for 2-D meshes: launches of the row-list kernels (rows2d.cuh).
#include <cooperative_groups.h>

#include <algorithm>

#include "rows2d.cuh"

namespace fem {
namespace {

__global__ void __launch_bounds__(256) k_lists_begin(ListLayout L) { lists_begin(L, blockIdx.x, gridDim.x); }

template <int KIND>
__global__ void __launch_bounds__(kFillThreads) k_fill_2d(MeshView m, ListLayout L) {
    fill_2d<KIND>(m, L, blockIdx.x, gridDim.x);
}

template <int KIND, typename T>
__global__ void __launch_bounds__(kRowThreads, KIND == FEM_T3 ? FEM_ROWS_T3_CTAS : FEM_ROWS_Q4_CTAS)
    k_rows_2d(MeshView m, ListLayout L, int* __restrict__ queue) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    rows_2d<KIND, T>(m, L, queue, blockIdx.x, gridDim.x, *reinterpret_cast<RowSmem*>(smem_raw));
}

template <int KIND, typename T>
__global__ void __launch_bounds__(kRowThreads) k_long_rows_2d(MeshView m, ListLayout L, const int* __restrict__ queue) {
    __shared__ LongSmem sm;
    long_rows_2d<KIND, T>(m, L, queue, blockIdx.x, gridDim.x, sm);
}

// The whole scatter of a small mesh (launch.h's kSmallNodes) in one cooperative
// launch: a launch costs the caller about 4 us, a grid barrier 1 to 2 us, and
// the phases of such a mesh take 1 to 10 us each. The long rows' registers slow
// the rows down here (rows2d.cuh), by less than a launch.
template <int KIND, typename T>
__global__ void __launch_bounds__(kRowThreads, FEM_ROWS_Q4_CTAS)
    k_small_2d(MeshView m, ListLayout L, int* __restrict__ queue) {
    __shared__ union {
        RowSmem rows;
        LongSmem longs;
    } sm;
    const cooperative_groups::grid_group grid = cooperative_groups::this_grid();
    lists_begin(L, blockIdx.x, gridDim.x);
    grid.sync();
    fill_2d<KIND>(m, L, blockIdx.x, gridDim.x);
    grid.sync();
    rows_2d<KIND, T>(m, L, queue, blockIdx.x, gridDim.x, sm.rows);
    grid.sync();
    long_rows_2d<KIND, T>(m, L, queue, blockIdx.x, gridDim.x, sm.longs);
}

template <int KIND, typename T>
cudaError_t launch_small_t(const MeshView& m, const ListLayout& L, int* queue, int ctas_per_sm, cudaStream_t s) {
    static DeviceCache cache;
    int per_sm = 0;
    cudaError_t err = per_device(cache, [](int& v) {
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, k_small_2d<KIND, T>, kRowThreads, 0);
    }, per_sm);
    if (err) return err;
    const int use = ctas_per_sm > 0 ? std::min(ctas_per_sm, per_sm) : per_sm;
    const long long want = std::max(((long long)m.N + kRowThreads - 1) / kRowThreads,
                                    ((long long)m.E_count + kRowThreads - 1) / kRowThreads);
    const int grid = (int)std::min<long long>(want, (long long)use * sm_count());
    MeshView mv = m;
    ListLayout lv = L;
    void* args[] = {&mv, &lv, &queue};
    return cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(k_small_2d<KIND, T>), dim3(grid), dim3(kRowThreads),
                                       args, 0, s);
}

cudaError_t launch_lists_begin(const ListLayout& L, cudaStream_t s) {
    const int grid = (int)std::max<long long>(1, std::min<long long>(((long long)L.N + 1023) / 1024, sm_count() * 4));
    k_lists_begin<<<grid, 256, 0, s>>>(L);
    return cudaGetLastError();
}

template <int KIND, typename T>
cudaError_t launch_rows_t(const MeshView& m, const ListLayout& L, int* queue, int ctas_per_sm, cudaStream_t s) {
    if (m.N <= kSmallNodes && m.E_count <= 4 * kSmallNodes) return launch_small_t<KIND, T>(m, L, queue, ctas_per_sm, s);
    cudaError_t err0 = launch_lists_begin(L, s);
    if (err0) return err0;
    static DeviceCache cache;
    const size_t smem = sizeof(RowSmem);
    int per_sm = 0;
    const cudaError_t err = per_device(cache, [&](int& v) {
        cudaError_t e = cudaFuncSetAttribute(k_rows_2d<KIND, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (!e) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, k_rows_2d<KIND, T>, kRowThreads, smem);
        return e;
    }, per_sm);
    if (err) return err;
    const int use = ctas_per_sm > 0 ? std::min(ctas_per_sm, per_sm) : per_sm;
    if (m.E_count > 0) {
        const long long want = ((long long)m.E_count + kFillThreads - 1) / kFillThreads;
        k_fill_2d<KIND><<<(int)std::min<long long>(want, (long long)sm_count() * 8), kFillThreads, 0, s>>>(m, L);
    }
    const long long tiles = ((long long)m.N + kRowThreads - 1) / kRowThreads;
    k_rows_2d<KIND, T><<<(int)std::min<long long>(tiles, (long long)use * sm_count()), kRowThreads, smem, s>>>(m, L, queue);
    k_long_rows_2d<KIND, T><<<(int)std::min<long long>(tiles, 2 * sm_count()), kRowThreads, 0, s>>>(m, L, queue);
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_rows_kind(const MeshView& m, const ListLayout& L, int* queue, int kind, int ctas_per_sm, cudaStream_t s) {
    if (kind == FEM_T3) return launch_rows_t<FEM_T3, T>(m, L, queue, ctas_per_sm, s);
    if (kind == FEM_Q4) return launch_rows_t<FEM_Q4, T>(m, L, queue, ctas_per_sm, s);
    return launch_rows_t<FEM_MIXED_2D, T>(m, L, queue, ctas_per_sm, s);
}

}  // namespace

cudaError_t launch_rows_2d(const MeshView& m, const ListLayout& L, int* queue, int kind, int precision,
                           int ctas_per_sm, cudaStream_t s) {
    return precision == FEM_PREC_FP32 ? launch_rows_kind<float>(m, L, queue, kind, ctas_per_sm, s)
                                      : launch_rows_kind<double>(m, L, queue, kind, ctas_per_sm, s);
}

}  // namespace fem
