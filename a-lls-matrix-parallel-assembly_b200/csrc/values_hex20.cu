// The CTA-cooperative Hex20 element pass (values_hex20.cuh): FP64 element
// stiffness added into a CSR, for the value-only re-assembly and the colouring
// baseline.
//
// Replaces the element routine computeElementStiffnessHex20
// (ALLS_Hex20_3D_Assembly_Performance.cu:130-195).
//
// Element stiffness in direction-major form. With G_a (20 x 27) the physical
// shape-function gradients along direction a at the Gauss points and
// w_g = gauss weight * detJ_g, the nine 20 x 20 node-pair matrices
//     M^{ab} = G_a diag(w) G_b^T                    (a, b in x, y, z)
// give every 3x3 node block of the isotropic stiffness entry by entry,
//     Ke_IJ[a][b] = lambda M^{ab}_IJ + mu M^{ba}_IJ + mu delta_ab (M^{xx} + M^{yy} + M^{zz})_IJ,
// which is the reference's per-Gauss-point block formula (H20:173-191) summed
// over the Gauss points. Padded to 24 x 24 (8x8 tiles) and K = 28, the upper
// triangle of the node grid is six tile positions, each with nine M^{ab}
// tiles on the FP64 tensor cores (mma.sync.m8n8k4.f64, seven k-steps), so a
// lane holds, for its two (I, J) node pairs of a tile, all nine M^{ab}_IJ and
// forms Ke_IJ without exchanging anything with other lanes.
//
// Element pass (k_values_hex20, kToCsrMap / kToCsrColour): one 6-warp CTA
// per element at a time, warp w owning tile position w; the shape-function
// derivatives at the 27 Gauss points (H20:95-128) are tabulated once per CTA
// and the next element's node ids and coordinates are loaded while the
// current one is computed.
//
// What bounds the re-assembly is the L2's FP64 atomics: 3,600 additions per
// element, 230 M for 40x40x40 elements, 1.33 ms of the 1.49 ms call (the
// clear of the values is the rest). At one fixed stride over the grid the CTAs drift
// apart in the visit order, so additions to the same rows no longer meet in L2 and
// the lines go to memory and back. So the CTAs take at most kMapRun elements
// each, a wave of resident CTAs sharing a stretch of the order, and the next
// CTAs start where the last ones end: the drift is bounded without any shared
// state (a map may be in use on several streams). Call, 40x40x40, at 4 CTAs per
// SM: one stride 1722 us; 2 / 4 / 8 / 16 elements 1538 / 1506 / 1487 / 1513;
// 20x20x20 215 (one stride), 211 / 202 / 210 / 212; a run of 4 consecutive
// elements per CTA 1506. One warp per element with its
// blocks staged in shared memory (ke_hex20.cuh's pass with additions in place of
// the packed store) has no barriers, but only 8 elements per SM in flight behind
// their additions: 1969 us.
// The colouring keeps the fixed stride (its elements share no rows): 32^3 with 2 / 3 / 4
// CTAs per SM 4.91 / 3.83 / 3.07 ms; 5.49 ms when the choice of the stride is made at run time.
#include <algorithm>

#include "values_hex20.cuh"

namespace fem {
namespace {

constexpr int kMapRun = 8;  // elements of one CTA of the re-assembly, at most
#ifndef FEM_VALUES_CTAS
#define FEM_VALUES_CTAS 4
#endif
constexpr int kThreads = kValueWarps * 32;

// kOut as values_cta (kToCsrMap: all elements in the order perm, scatter map
// row e; kToCsrColour: the elements perm[range[0], range[1]) of one colour).
template <int kOut>
__global__ void __launch_bounds__(kThreads, FEM_VALUES_CTAS)
    k_values_hex20(MeshView m, const int* __restrict__ perm, [[maybe_unused]] int i0, int i1, const int* __restrict__ range,
                   ValuesTarget t, int group, int run) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ValuesSmem& sm = *reinterpret_cast<ValuesSmem*>(smem_raw);
    if (range) {
        i0 = range[0];
        i1 = range[1];
    }
    values_init(sm);
    if constexpr (kOut == kToCsrMap) {
        const long long chunk = blockIdx.x / group * ((long long)group * run);
        values_cta<kOut>(m, perm, chunk + blockIdx.x % group, group, (int)min((long long)i1, chunk + (long long)group * run),
                         t, sm);
    } else {
        values_cta<kOut>(m, perm, (long long)i0 + blockIdx.x, gridDim.x, i1, t, sm);
    }
}

template <int kOut>
cudaError_t launch_values(const MeshView& m, const int* perm, int i0, int i1, const int* range, const ValuesTarget& t,
                          cudaStream_t s) {
    static DeviceCache cache;
    const size_t smem = sizeof(ValuesSmem);
    int per_sm = 0;
    const cudaError_t err = per_device(cache, [&](int& v) {
        cudaError_t e =
            cudaFuncSetAttribute(k_values_hex20<kOut>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (!e) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, k_values_hex20<kOut>, kThreads, smem);
        return e;
    }, per_sm);
    if (err) return err;
    const long long count = range ? m.E_count : i1 - i0;  // a colour's size is on the device: bound by E
    const long long fit = (long long)per_sm * sm_count();
    long long grid = std::max<long long>(1, std::min(count, fit));
    int run = 1;
    if (kOut == kToCsrMap && count > fit) {
        const long long waves = (count + fit * kMapRun - 1) / (fit * kMapRun);
        run = (int)((count + fit * waves - 1) / (fit * waves));
        grid = waves * fit;
    }
    k_values_hex20<kOut><<<(int)grid, kThreads, smem, s>>>(m, perm, i0, i1, range, t, (int)fit, run);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_reassemble_hex20(const MeshView& m, int precision, const int* perm, const MapTarget& mt,
                                    DevInfo* info, cudaStream_t s) {
    if (m.E_count <= 0) return cudaSuccess;
    if (precision == FEM_PREC_TC_F16X3) return launch_reassemble_hex20_tc(m, perm, mt, info, s);
    ValuesTarget t{};
    t.map = mt.map;
    t.row_ptr = mt.row_ptr;
    t.csr = mt.values;
    t.info = info;
    return launch_values<kToCsrMap>(m, perm, 0, m.E_count, nullptr, t, s);
}

cudaError_t launch_colour_hex20(const MeshView& m, const int* perm, const int* range, const MapTarget& mt,
                                DevInfo* info, cudaStream_t s) {
    ValuesTarget t{};
    t.row_ptr = mt.row_ptr;
    t.col_idx = mt.col_idx;
    t.csr = mt.values;
    t.info = info;
    return launch_values<kToCsrColour>(m, perm, 0, 0, range, t, s);
}

}  // namespace fem
