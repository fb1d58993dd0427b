// Batched assembly: many independent meshes of uneven sizes and element kinds
// in one stream-ordered, graph-capturable call.
//
// The reference assembles one mesh per program run (each driver's main, e.g.
// ALLS_Q4_T3_Mixed_Elements_Assembly_Performance.cu:742-854). Here the meshes
// are assembled in rounds of `slots` (the workspace holds that many meshes'
// lists at once), and a round runs phase by phase: one launch per phase covers
// all of the round's meshes (begin; 2-D fill and Hex20 occurrences; rows; Hex20
// Ke; row pointers; writes), its blocks dealt to the meshes in
// proportion to their work, each block running the device code of the
// single-mesh kernels. Phases follow each other in stream order, so nothing
// waits inside a kernel, small meshes share their launches, and large ones get
// the same kernels as on their own. A round's mesh descriptors travel as kernel
// parameters, so a captured CUDA graph holds them.
//
// What bounds it: the single-mesh kernels. A round costs 14 merged launches
// (two more if some outputs are not aligned or have no room) and, for each of its
// Hex20 meshes of 3,072 elements or more, a node order: a memset and five small
// kernels. B200, 16 meshes of 1,000 to 50,000 elements of all kinds in 4 slots:
// 1.69 ms, where one persistent kernel of dependent work items (CAS claims,
// element-wise atomics, no spatial order) took 8.0 ms.
#include <algorithm>
#include <numeric>
#include <vector>

#include "ke_hex20.cuh"
#include "rows2d.cuh"
#include "rows_hex20.cuh"
#include "write_hex20.cuh"

namespace fem {
namespace {

// Meshes per round launch: the descriptors are kernel parameters (at most 32 KB).
// Rounds of up to kRoundSmall meshes (the default is 4 slots) pass small ones.
constexpr int kRoundSmall = 8, kRoundLarge = 64;

template <int kMax>
struct BatchRound {
    int n;
    int first[kMax + 1];  // first block of each mesh in this launch
    BatchMesh mesh[kMax];
};
static_assert(sizeof(BatchRound<kRoundLarge>) < 32000, "kernel parameter size");

// The block's mesh, copied to shared memory; its block number and block count there.
template <int kMax>
__device__ __forceinline__ void block_mesh(const BatchRound<kMax>& r, BatchMesh& bm, int& block, int& nblocks) {
    int i = 0;
    while (i + 1 < r.n && r.first[i + 1] <= (int)blockIdx.x) i++;
    block = blockIdx.x - r.first[i];
    nblocks = r.first[i + 1] - r.first[i];
    constexpr int kWords = sizeof(BatchMesh) / 8;
    static_assert(sizeof(BatchMesh) % 8 == 0, "descriptor copy in 8-byte words");
    const unsigned long long* src = reinterpret_cast<const unsigned long long*>(&r.mesh[i]);
    for (int w = threadIdx.x; w < kWords; w += blockDim.x) reinterpret_cast<unsigned long long*>(&bm)[w] = src[w];
    __syncthreads();
}

__device__ __forceinline__ unsigned long long global_timer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

#define FEM_BATCH_KERNEL(...) template <int kMax> __global__ void __launch_bounds__(__VA_ARGS__)
#define FEM_BATCH_MESH                   \
    __shared__ BatchMesh bm;             \
    int block, nblocks;                  \
    block_mesh<kMax>(r, bm, block, nblocks)

FEM_BATCH_KERNEL(256) kb_begin(const __grid_constant__ BatchRound<kMax> r, unsigned long long* start) {
    FEM_BATCH_MESH;
    if (start && blockIdx.x == 0 && threadIdx.x == 0) *start = global_timer();
    if (bm.kind == FEM_HEX20) lists_begin_hex20(bm.L, bm.cnt, block, nblocks);
    else lists_begin(bm.L, block, nblocks);
}

static_assert(kFillThreads == kOccThreads, "one block shape for both");
FEM_BATCH_KERNEL(kFillThreads) kb_fill(const __grid_constant__ BatchRound<kMax> r) {
    FEM_BATCH_MESH;
    if (bm.kind == FEM_HEX20) occ_count(bm.m, bm.h, bm.cnt, bm.L.info, block, nblocks);
    else if (bm.kind == FEM_T3) fill_2d<FEM_T3>(bm.m, bm.L, block, nblocks);
    else if (bm.kind == FEM_Q4) fill_2d<FEM_Q4>(bm.m, bm.L, block, nblocks);
    else fill_2d<FEM_MIXED_2D>(bm.m, bm.L, block, nblocks);
}

FEM_BATCH_KERNEL(kScanThreads) kb_occ_sums(const __grid_constant__ BatchRound<kMax> r) {
    FEM_BATCH_MESH;
    __shared__ long long s_warp[kScanThreads / 32 + 1];
    occ_sums(bm.cnt, bm.L.N, bm.tiles, block, s_warp);
}

FEM_BATCH_KERNEL(kScanThreads) kb_occ_offsets(const __grid_constant__ BatchRound<kMax> r) {
    FEM_BATCH_MESH;
    __shared__ OccSmem sm;
    occ_offsets(bm.cnt, bm.L.N, bm.tiles, bm.h.off, block, nblocks, sm);
}

FEM_BATCH_KERNEL(kOccThreads) kb_occ_fill(const __grid_constant__ BatchRound<kMax> r) {
    FEM_BATCH_MESH;
    occ_fill(bm.m, bm.h, block, nblocks);
}

FEM_BATCH_KERNEL(kRowThreads, FEM_ROWS_Q4_CTAS) kb_rows_2d(const __grid_constant__ BatchRound<kMax> r) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    RowSmem& sm = *reinterpret_cast<RowSmem*>(smem_raw);
    FEM_BATCH_MESH;
    if (bm.kind == FEM_T3) rows_2d<FEM_T3, double>(bm.m, bm.L, bm.queue, block, nblocks, sm);
    else if (bm.kind == FEM_Q4) rows_2d<FEM_Q4, double>(bm.m, bm.L, bm.queue, block, nblocks, sm);
    else rows_2d<FEM_MIXED_2D, double>(bm.m, bm.L, bm.queue, block, nblocks, sm);
}

FEM_BATCH_KERNEL(kRowThreads) kb_long_rows_2d(const __grid_constant__ BatchRound<kMax> r) {
    FEM_BATCH_MESH;
    __shared__ LongSmem sm;
    if (bm.kind == FEM_T3) long_rows_2d<FEM_T3, double>(bm.m, bm.L, bm.queue, block, nblocks, sm);
    else if (bm.kind == FEM_Q4) long_rows_2d<FEM_Q4, double>(bm.m, bm.L, bm.queue, block, nblocks, sm);
    else long_rows_2d<FEM_MIXED_2D, double>(bm.m, bm.L, bm.queue, block, nblocks, sm);
}

FEM_BATCH_KERNEL(kHexRowThreads, FEM_HEXR_CTAS) kb_rows_hex20(const __grid_constant__ BatchRound<kMax> r) {
    FEM_BATCH_MESH;
    __shared__ HexRowSmem s_row[kHexRowWarps];
    rows_hex20(bm.m.conn, bm.L, bm.h, bm.queue, block, nblocks, s_row);
}

FEM_BATCH_KERNEL(kHexRowThreads) kb_long_rows_hex20(const __grid_constant__ BatchRound<kMax> r) {
    FEM_BATCH_MESH;
    __shared__ union {
        int uniq[kHexRowWarps][kWideElems * 20];
        LongHexSmem longs;
    } sm;
    const int warp = threadIdx.x >> 5;
    wide_rows_hex20(bm.m.conn, bm.L, bm.h, bm.queue, block * kHexRowWarps + warp, nblocks * kHexRowWarps, sm.uniq[warp]);
    __syncthreads();
    long_rows_hex20(bm.m.conn, bm.L, bm.h, bm.queue, block, nblocks, sm.longs);
}

FEM_BATCH_KERNEL(kKeThreads, 1) kb_ke_hex20(const __grid_constant__ BatchRound<kMax> r) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    FEM_BATCH_MESH;
    ke_hex20(bm.m, bm.h.ke, &bm.L.info->status_bits, true, block, nblocks, *reinterpret_cast<KeHexSmem*>(smem_raw));
}

FEM_BATCH_KERNEL(kScanThreads) kb_tile_entries(const __grid_constant__ BatchRound<kMax> r) {
    FEM_BATCH_MESH;
    __shared__ long long s_warp[kScanThreads / 32 + 1];
    if (bm.kind == FEM_HEX20) tile_entries<3, kOutCsr>(bm.L.counts, bm.L.N, bm.tiles, block, s_warp);
    else tile_entries<2, kOutCsr>(bm.L.counts, bm.L.N, bm.tiles, block, s_warp);
}

FEM_BATCH_KERNEL(kScanThreads) kb_row_ptr(const __grid_constant__ BatchRound<kMax> r) {
    FEM_BATCH_MESH;
    __shared__ RowPtrSmem sm;
    if (bm.kind == FEM_HEX20)
        row_ptr_rows<3, kOutCsr>(bm.L.counts, bm.L.N, bm.tiles, bm.row_ptr, bm.L.info, bm.capacity, block, nblocks, sm);
    else
        row_ptr_rows<2, kOutCsr>(bm.L.counts, bm.L.N, bm.tiles, bm.row_ptr, bm.L.info, bm.capacity, block, nblocks, sm);
}

// The info word to the caller's array and the completion stamp (one thread).
__device__ __forceinline__ void finish_mesh(const BatchMesh& bm) {
    static_assert(sizeof(fem_info) % 8 == 0, "copied in 8-byte words");
    for (int w = 0; w < (int)(sizeof(fem_info) / 8); w++)
        reinterpret_cast<unsigned long long*>(bm.info_out)[w] =
            __ldcg(reinterpret_cast<const unsigned long long*>(bm.L.info) + w);
    if (bm.stamp) *bm.stamp = global_timer();
}

// The end of a write block; the mesh's last one finishes the mesh.
__device__ __forceinline__ void write_done(const BatchMesh& bm, int nblocks) {
    __syncthreads();
    if (threadIdx.x != 0) return;
    __threadfence();  // the block's entries and statistics before its count
    if (atomicAdd(&bm.L.info->done, 1) != nblocks - 1) return;
    __threadfence();
    finish_mesh(bm);
}

FEM_BATCH_KERNEL(kBlockThreads) kb_write_2d(const __grid_constant__ BatchRound<kMax> r) {
    FEM_BATCH_MESH;
    __shared__ int s_stat[2 * (kBlockThreads / 32)];
    write_sorted_2d(bm.L, bm.row_ptr, bm.col_idx, bm.values, bm.capacity, block, nblocks, s_stat);
    write_done(bm, nblocks);
}

// The 2-D meshes whose outputs are not aligned for write_sorted_2d.
FEM_BATCH_KERNEL(kBlockThreads) kb_write_2d_entries(const __grid_constant__ BatchRound<kMax> r) {
    FEM_BATCH_MESH;
    __shared__ WriteSmem<8, 2> sm;
    constexpr int NPB = kBlockThreads / 8;
    write_batches<8, 2, kOutCsr>(bm.L, bm.row_ptr, bm.col_idx, bm.values, bm.capacity, nullptr,
                                    (long long)block * NPB, (long long)nblocks * NPB, bm.L.N, sm);
    write_done(bm, nblocks);
}

FEM_BATCH_KERNEL(kWriteThreads, FEM_HEXW_CTAS) kb_write_hex20(const __grid_constant__ BatchRound<kMax> r) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    FEM_BATCH_MESH;
    write_hex20<kOutCsr>(bm.L, bm.h, nullptr, bm.row_ptr, bm.col_idx, bm.values, bm.capacity, block, nblocks,
                         *reinterpret_cast<WriteHexCta*>(smem_raw));
    write_done(bm, nblocks);
}

// The meshes without an output, one block each.
FEM_BATCH_KERNEL(32) kb_finish(const __grid_constant__ BatchRound<kMax> r) {
    FEM_BATCH_MESH;
    if (threadIdx.x == 0) finish_mesh(bm);
}

template <int kMax>
struct RoundLauncher {
    BatchRound<kMax> r;
    cudaStream_t s;
    cudaError_t err = cudaSuccess;

    // Launches `kernel` over the meshes with want(mesh) > 0 blocks; more than `cap` blocks in all are scaled down to
    // it (the kernels are persistent over their mesh's work; cap 0: exactly the wanted blocks).
    template <typename Kernel, typename Want, typename... Args>
    void run(Kernel kernel, int threads, size_t smem, long long cap, Want want, Args... args) {
        if (err) return;
        long long sum = 0;
        for (int i = 0; i < r.n; i++) sum += want(r.mesh[i]);
        if (sum == 0) return;
        long long at = 0;
        for (int i = 0; i < r.n; i++) {
            r.first[i] = (int)at;
            const long long w = want(r.mesh[i]);
            at += cap == 0 || sum <= cap ? w : (w > 0 ? std::max<long long>(1, w * cap / sum) : 0);
        }
        r.first[r.n] = (int)at;
        kernel<<<(unsigned)at, threads, smem, s>>>(r, args...);
        err = cudaGetLastError();
    }
};

long long blocks_of(long long work, long long per) { return (work + per - 1) / per; }

template <int kMax>
cudaError_t launch_round(const BatchMesh* meshes, int n, unsigned long long* start, int ctas_per_sm, cudaStream_t s) {
    static DeviceCache cache;
    int ready = 0;
    cudaError_t err = per_device(cache, [](int& v) {
        v = 1;
        cudaError_t e = cudaFuncSetAttribute(kb_rows_2d<kMax>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)sizeof(RowSmem));
        if (!e)
            e = cudaFuncSetAttribute(kb_ke_hex20<kMax>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)sizeof(KeHexSmem));
        if (!e)
            e = cudaFuncSetAttribute(kb_write_hex20<kMax>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)sizeof(WriteHexCta));
        return e;
    }, ready);
    if (err) return err;
    const int sms = sm_count();
    RoundLauncher<kMax> l;
    l.s = s;
    l.r.n = n;
    std::copy(meshes, meshes + n, l.r.mesh);
    using M = const BatchMesh&;
    auto hex = [](M b) { return b.kind == FEM_HEX20; };
    l.run(kb_begin<kMax>, 256, 0, 4 * sms, [](M b) { return blocks_of(b.L.N, 1024); }, start);
    l.run(kb_fill<kMax>, kFillThreads, 0, 8 * sms, [](M b) { return blocks_of(b.m.E_count, kFillThreads); });
    l.run(kb_occ_sums<kMax>, kScanThreads, 0, 0, [&](M b) { return hex(b) ? (long long)row_tiles(b.L.N) : 0; });
    l.run(kb_occ_offsets<kMax>, kScanThreads, 0, 0, [&](M b) { return hex(b) ? (long long)row_tiles(b.L.N) : 0; });
    l.run(kb_occ_fill<kMax>, kOccThreads, 0, 16 * sms,
          [&](M b) { return hex(b) ? blocks_of(20ll * b.m.E_count, kOccThreads) : 0; });
    l.run(kb_rows_2d<kMax>, kRowThreads, sizeof(RowSmem),
          (long long)(ctas_per_sm > 0 ? std::min(ctas_per_sm, FEM_ROWS_Q4_CTAS) : FEM_ROWS_Q4_CTAS) * sms,
          [&](M b) { return hex(b) ? 0 : blocks_of(b.L.N, kRowThreads); });
    l.run(kb_long_rows_2d<kMax>, kRowThreads, 0, 2 * sms, [&](M b) { return hex(b) ? 0 : blocks_of(b.L.N, kRowThreads); });
    l.run(kb_rows_hex20<kMax>, kHexRowThreads, 0, FEM_HEXR_CTAS * sms,
          [&](M b) { return hex(b) ? blocks_of(b.L.N, kHexRowWarps) : 0; });
    l.run(kb_long_rows_hex20<kMax>, kHexRowThreads, 0, sms,
          [&](M b) { return hex(b) ? blocks_of(b.L.N, kHexRowWarps) : 0; });
    for (int i = 0; i < n && !l.err; i++)
        if (hex(meshes[i]) && meshes[i].h.order)
            l.err = launch_node_order(meshes[i].m, meshes[i].hist, meshes[i].ranges, meshes[i].cnt, meshes[i].bbox, sms, s);
    l.run(kb_ke_hex20<kMax>, kKeThreads, sizeof(KeHexSmem), sms,
          [&](M b) { return hex(b) ? blocks_of(b.m.E_count, kKeWarps) : 0; });
    l.run(kb_tile_entries<kMax>, kScanThreads, 0, 0, [](M b) { return (long long)row_tiles(b.L.N); });
    l.run(kb_row_ptr<kMax>, kScanThreads, 0, 0, [](M b) { return (long long)row_tiles(b.L.N); });
    l.run(kb_write_2d<kMax>, kBlockThreads, 0, 4 * sms, [&](M b) {
        return !hex(b) && b.capacity > 0 && b.wide ? blocks_of(b.L.N, kBlockThreads / 16 * kCopyNodes) : 0;
    });
    l.run(kb_write_2d_entries<kMax>, kBlockThreads, 0, 4 * sms, [&](M b) {
        return !hex(b) && b.capacity > 0 && !b.wide ? blocks_of(b.L.N, kBlockThreads / 8) : 0;
    });
    l.run(kb_write_hex20<kMax>, kWriteThreads, sizeof(WriteHexCta), FEM_HEXW_CTAS * sms,
          [&](M b) { return hex(b) && b.capacity > 0 ? blocks_of(b.L.N, kWriteWarps) : 0; });
    l.run(kb_finish<kMax>, 32, 0, 0, [](M b) { return b.capacity > 0 ? 0ll : 1ll; });
    return l.err;
}

}  // namespace

double batch_cost(const fem_mesh& m) {
    const double w = m.kind == FEM_HEX20 ? 60.0 : (m.kind == FEM_T3 ? 1.0 : 1.4);
    return w * (double)m.num_elems + 1e3;
}

std::vector<int> batch_schedule(const fem_mesh* meshes, int n, int slots) {
    std::vector<int> order(n), slot_of(n, 0);
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(),
                     [&](int a, int b) { return batch_cost(meshes[a]) > batch_cost(meshes[b]); });
    std::vector<double> load(slots, 0.0);
    for (int i : order) {
        const int k = (int)(std::min_element(load.begin(), load.end()) - load.begin());
        slot_of[i] = k;
        load[k] += batch_cost(meshes[i]);
    }
    return slot_of;
}

cudaError_t launch_batch_round(const BatchMesh* meshes, int n, unsigned long long* start, int ctas_per_sm,
                               cudaStream_t s) {
    if (n <= kRoundSmall) return launch_round<kRoundSmall>(meshes, n, start, ctas_per_sm, s);
    for (int i = 0; i < n; i += kRoundLarge) {
        const cudaError_t err = launch_round<kRoundLarge>(meshes + i, std::min(kRoundLarge, n - i),
                                                          i == 0 ? start : nullptr, ctas_per_sm, s);
        if (err) return err;
    }
    return cudaSuccess;
}

}  // namespace fem
