// Launch of the FP64 Hex20 element stiffness (ke_hex20.cuh).
#include <algorithm>

#include "ke_hex20.cuh"

namespace fem {
namespace {

__global__ void __launch_bounds__(kKeThreads, 1) k_ke_hex20(MeshView m, double* __restrict__ ke_out,
                                                            int* __restrict__ status, int bulk) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    ke_hex20(m, ke_out, status, bulk != 0, blockIdx.x, gridDim.x, *reinterpret_cast<KeHexSmem*>(smem_raw));
}

}  // namespace

cudaError_t launch_hex20_ke_dmma(const MeshView& m, double* ke_out, int* status, cudaStream_t s) {
    static DeviceCache cache;
    const size_t smem = sizeof(KeHexSmem);
    int per_sm = 0;
    const cudaError_t err = per_device(cache, [&](int& v) {
        cudaError_t e = cudaFuncSetAttribute(k_ke_hex20, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (!e) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, k_ke_hex20, kKeThreads, smem);
        return e;
    }, per_sm);
    if (err) return err;
    const int grid = (int)std::min<long long>(m.E_count, (long long)per_sm * sm_count());
    const int bulk = (reinterpret_cast<uintptr_t>(ke_out) & 15u) == 0;
    k_ke_hex20<<<grid, kKeThreads, smem, s>>>(m, ke_out, status, bulk);
    return cudaGetLastError();
}

}  // namespace fem
