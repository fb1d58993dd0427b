// Host-side launchers of the assembler kernels (internal to the library).
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <vector>

#include "fem_internal.cuh"

namespace fem {

// A launch-shape value (resident CTAs per SM, SM count) cached per device: it
// is computed on the first launch on each device (compute(int& v) sets v > 0),
// which also sets the kernel's per-device attributes. Devices past the table
// compute it every time.
constexpr int kMaxCachedDevices = 64;
struct DeviceCache {
    std::atomic<int> v[kMaxCachedDevices] = {};
};
template <typename F>
cudaError_t per_device(DeviceCache& cache, F&& compute, int& out) {
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err) return err;
    const bool cached = dev >= 0 && dev < kMaxCachedDevices;
    int v = cached ? cache.v[dev].load(std::memory_order_acquire) : 0;
    if (v <= 0) {
        if ((err = compute(v))) return err;
        if (v < 1) v = 1;
        if (cached) cache.v[dev].store(v, std::memory_order_release);
    }
    out = v;
    return cudaSuccess;
}

struct MeshView {
    const double* x;
    const double* y;
    const double* z;
    const int* conn;
    const unsigned char* types;
    const double* E;
    const double* nu;
    double E0, nu0, t;
    int N;       // nodes
    int E_count; // elements
    int stride;  // ints per connectivity row
};

// 2-D chunk rows are 16 int32 words (14 slots + fill + next).
constexpr int k2DSlots = 14;

// Meshes of at most this many nodes (and 2-D: 4 times as many elements) are scattered by one cooperative launch and
// scanned without a tile pass: their time is the launches'.
constexpr int kSmallNodes = 16384;
// The info word, counters and row lists of a 2-D mesh (rows2d.cu);
// precision FEM_PREC_FP64 or FEM_PREC_FP32 (the arithmetic of the Ke blocks).
// queue: N ints of scratch; ctas_per_sm: cap on the persistent grid's resident CTAs per SM (0 = all that fit).
cudaError_t launch_rows_2d(const MeshView& m, const ListLayout& L, int* queue, int kind, int precision,
                           int ctas_per_sm, cudaStream_t s);
// Node-local element order (perm) and the element ranges {q4 begin, q4 end, t3 begin, t3 end}.
int reorder_buckets(int num_nodes);
// gate: NULL, or a device word; 0 there when the sort's kernels run leaves the order as it is.
cudaError_t launch_reorder(const MeshView& m, int* hist, int* ranges, int* perm, int sms, cudaStream_t s,
                           const int* gate = nullptr);
int sm_count();
// Packed symmetric element stiffness (fem_element_stiffness): doubles per element.
constexpr int kPackedHex20 = 210 * 9;  // 210 upper 3x3 node blocks
constexpr int kPacked2D_Q4 = 10 * 4;   // 10 upper 2x2 node blocks (also the mixed-mesh stride)
constexpr int kPacked2D_T3 = 6 * 4;
// Element stiffness of every element, natural order; status gets 1 << FEM_ERR_* bits.
cudaError_t launch_element_stiffness(const MeshView& m, int kind, int precision, double* ke_out, int* status,
                                     long long wait_ns, cudaStream_t s);
// Hex20 element stiffness on the FP64 tensor cores, one warp per element (ke_hex20.cu).
cudaError_t launch_hex20_ke_dmma(const MeshView& m, double* ke_out, int* status, cudaStream_t s);
// Hex20 element stiffness with the contraction on the tcgen05 tensor cores
// (FEM_PREC_TC_F16X3), two elements per CTA step.
// wait_ns: bound on a CTA's wait for its products (< 0: no wait), see fem_opts.wait_limit_us.
cudaError_t launch_hex20_ke_tcgen05(const MeshView& m, double* ke_out, int* status, long long wait_ns,
                                    cudaStream_t s);
// fem_opts.wait_limit_us in nanoseconds: 0 -> 200 ms, > 0 -> that bound, < 0 -> -1 (no wait).
inline long long wait_ns_of(int wait_limit_us) {
    return wait_limit_us == 0 ? 200ll * 1000 * 1000 : (wait_limit_us > 0 ? 1000ll * wait_limit_us : -1);
}
// Target of a value-only re-assembly: CSR positions of every element block.
struct MapTarget {
    const int* map;      // [E * npe^2] position of block (a, b) of element e at e * npe^2 + a * npe + b
    const int* row_ptr;  // CSR row pointers of the pattern the map was built for
    double* values;      // CSR values (zeroed by the caller)
    const int* col_idx;  // CSR columns (the colouring baseline searches them)
};

// Scatter map of a mesh into a CSR pattern; status gets 1 << FEM_ERR_* bits. gate as launch_reorder's.
cudaError_t launch_build_map(const MeshView& m, int kind, const int* row_ptr, const int* col_idx, int* map,
                             int* status, cudaStream_t s, const int* gate = nullptr);
// Value-only re-assembly (atomics into values): 2-D kinds over perm ranges
// {q4 begin, q4 end, t3 begin, t3 end}; Hex20 over perm (status bits in info).
struct BlocksMap {
    const int* pos;     // [E * G] positions, -1: no block
    int G;              // npe^2
    const int* perm;    // element order
    const int* ranges;
};
cudaError_t launch_reassemble_2d(const MeshView& m, int precision, const BlocksMap& b, const int* row_ptr,
                                 double* values, int* status, cudaStream_t s);
// The same by row nodes (2-D): each node's occurrences (element << 2 | position) and the ranks of their nodes in its row.
struct RowsMap {
    int* off;               // [N + 1]
    unsigned* occ;          // [npe * E]
    unsigned short* ranks;  // [npe * npe * E]
    int* blocks;            // not 0: the pattern does not take this form, the map is the block positions
};
// cnt (N ints) and tiles (row_tiles(N) partials): scratch. *r.blocks (0 before) is set when the pattern is not one of
// node blocks that holds all of the mesh's, from entry 0 on, with rows of at most 65,536 columns.
cudaError_t launch_build_rows_map(const MeshView& m, int kind, const int* row_ptr, const int* col_idx, const RowsMap& r,
                                  int* cnt, long long* tiles, DevInfo* info, cudaStream_t s);
// Clears the info word; values[0, nnz): the rows and zeros behind them; by the block positions b where *r.blocks is set.
cudaError_t launch_rows_values_2d(const MeshView& m, int kind, int precision, const RowsMap& r, const BlocksMap& b,
                                  const int* row_ptr, double* values, long long nnz, DevInfo* info, cudaStream_t s);
// The tensor-core form of the Hex20 value-only re-assembly (ke_tcgen05.cu).
cudaError_t launch_reassemble_hex20_tc(const MeshView& m, const int* perm, const MapTarget& t, DevInfo* info,
                                       cudaStream_t s);
cudaError_t launch_reassemble_hex20(const MeshView& m, int precision, const int* perm, const MapTarget& t,
                                    DevInfo* info, cudaStream_t s);
// Colouring baseline for Hex20: elements perm[range[0], range[1]) (one colour),
// plain adds at binary-searched CSR positions (t.map unused); status bits in info.
cudaError_t launch_colour_hex20(const MeshView& m, const int* perm, const int* range, const MapTarget& t,
                                DevInfo* info, cudaStream_t s);

// Node -> element incidence lists (incidence.cu): cnt [N] (counts), off
// [N + 1], inc [sum of nodes per element], tiles [ceil(N / kScanTile)]
// scratch; status gets 1 << FEM_ERR_* bits.
cudaError_t launch_incidence(const MeshView& m, int* cnt, int* off, int* inc, long long* tiles, int* status, int sms,
                             cudaStream_t s);
// Mark of the occurrences of an element that repeats a node.
constexpr unsigned kOccRepeats = 0x80000000u;
// What a Hex20 scatter leaves besides the list chunks (hex_rows.cuh).
struct HexRows {
    double* ke;           // [E * kPackedHex20] packed element stiffness
    int* off;             // [N + 1] node -> occurrences
    int* inc;             // occurrences 20 e + a (bit 31: kOccRepeats)
    const int* order;     // [N] node visit order of the consolidation, or NULL: as numbered
    unsigned short* map;  // [E * 400] rank of column node b in row node a's list, at 20 (20 e + a) + b
    const int* conn;      // the mesh's connectivity (rows longer than a rank of the map)
};
// The info word, the occurrences (off / inc, of the elements without a bad node id), the sorted row lists and the
// rank map; cnt, queue: N ints, tiles: row_tiles(N) partials of scratch.
cudaError_t launch_rows_hex20(const MeshView& m, const ListLayout& L, const HexRows& h, int* cnt, long long* tiles,
                              int* queue, cudaStream_t s);
// Row lists -> CSR / BSR / upper triangle (mode: consolidate.cuh's kOut*; row_ptr already written).
cudaError_t launch_count_upper_hex20(const ListLayout& L, int* ucounts, cudaStream_t s);
cudaError_t launch_write_hex20(const ListLayout& L, const HexRows& h, int mode, const int* ucounts, const int* row_ptr,
                               int* col_idx, double* values, long long capacity, cudaStream_t s);
// Whether CSR outputs are aligned for the 2-D copy kernel's 16-byte value and 8-byte column stores (row starts are
// multiples of 4 entries); other outputs are stored entry by entry.
inline bool wide_outputs(const int* col_idx, const double* values) {
    return reinterpret_cast<uintptr_t>(values) % 16 == 0 && reinterpret_cast<uintptr_t>(col_idx) % 8 == 0;
}

// Spatial (3-D Morton bucket) element order; hist needs 1 << (3 * morton_bits(E)) ints, bbox 6 words.
int morton_bits(int num_elems);
// Nodes by the Morton code of their cell on a 2^kNodeOrderBits grid per axis (hist: one int per cell).
constexpr int kNodeOrderBits = 4;
cudaError_t launch_node_order(const MeshView& m, int* hist, int* ranges, int* order, unsigned long long* bbox, int sms,
                              cudaStream_t s);
cudaError_t launch_reorder_3d(const MeshView& m, int* hist, int* ranges, int* perm, unsigned long long* bbox, int sms,
                              cudaStream_t s);
// tile_sums: row_tiles(N) partials of scratch.
cudaError_t launch_consolidate(const ListLayout& L, int dpn, const HexRows& hex, int* row_ptr, int* col_idx, double* values,
                               long long capacity, long long* tile_sums, cudaStream_t s);
// Upper triangle (columns >= row, diagonal included) in CSR; ucounts: N ints of scratch.
cudaError_t launch_consolidate_upper(const ListLayout& L, int dpn, const HexRows& hex, int* ucounts, int* row_ptr,
                                     int* col_idx, double* values, long long capacity, long long* tile_sums,
                                     cudaStream_t s);
// Node-block (BSR) form of the consolidation; capacity in blocks.
cudaError_t launch_consolidate_bsr(const ListLayout& L, int dpn, const HexRows& hex, int* block_row_ptr,
                                   int* block_col_idx,
                                   double* block_values, long long capacity_blocks, long long* tile_sums,
                                   cudaStream_t s);

// ---- load vector and boundary conditions (loads.cu) ----
// f += body-force load vector (b: device [E * dim] or NULL for the uniform b0[dim], host values).
cudaError_t launch_body_force(const MeshView& m, int kind, const double* b, const double* b0, double* f, int* status,
                              cudaStream_t s);
// Symmetric elimination of fixed dofs in place on a CSR matrix (and f).
cudaError_t launch_dirichlet(int n_rows, const int* row_ptr, const int* col_idx, double* values, double* f,
                             const unsigned char* fixed, const double* u, cudaStream_t s);

// ---- batched assembly (batched.cu) ----
constexpr int kMaxBatchConcurrency = 256;  // meshes whose lists are live at once (workspace slots)
// Estimated work of a mesh (elements weighted by kind) and the slot of each
// mesh (largest first onto the least loaded slot).
double batch_cost(const fem_mesh& m);
std::vector<int> batch_schedule(const fem_mesh* meshes, int n, int slots);

// Everything the batched kernels need to know about one mesh (a kernel parameter).
struct BatchMesh {
    MeshView m;
    ListLayout L;
    HexRows h;
    int* cnt;                  // Hex20: occurrence counts, then the node order
    int* queue;                // long rows
    long long* tiles;          // scan partials
    int* hist;                 // Hex20: scratch of the node order
    int* ranges;
    unsigned long long* bbox;
    int* row_ptr;              // the caller's CSR
    int* col_idx;
    double* values;
    long long capacity;
    fem_info* info_out;        // the caller's info array entry
    unsigned long long* stamp; // completion stamp (may be NULL)
    int kind;
    int wide;                  // 2-D: the outputs are aligned for the copy kernel
};

// Assembles the meshes of one round (each in its own workspace slot), phase by
// phase on the stream; start: optional start stamp.
cudaError_t launch_batch_round(const BatchMesh* meshes, int n, unsigned long long* start, int ctas_per_sm,
                               cudaStream_t s);

// ---- element-colouring baseline (colour.cu) ----
constexpr int kMaxColours = 64;         // colours per mesh (a 64-bit mask of neighbour colours)
constexpr int kMaxColourRounds = 4096;  // bound on Jones-Plassmann rounds

struct ColourInfo {
    int num_colours;
    int status_bits;  // 1 << FEM_ERR_*
    int uncoloured;   // elements left after the last round
    int pad[13];
};
static_assert(sizeof(ColourInfo) == 64, "ColourInfo size");

// Device buffers of the colouring path (inside the caller's workspace).
struct ColourLayout {
    ColourInfo* info;
    int* cnt;        // [N] incidence counts, then fill cursors
    int* off;        // [N + 1] node -> element offsets
    int* inc;        // [sum of nodes per element] incidence lists
    int* colour;     // [E] round << 8 | colour, -1 = uncoloured
    int* perm;       // [E] elements grouped by (colour, type)
    int* hist;       // [2 * kMaxColours] counts, then cursors
    int* ranges;     // [2 * kMaxColours + 1] offsets of each (colour, type) group in perm
    long long* tiles;  // [ceil(N / kScanTile)] scan partials
};

// Incidence, colouring rounds (host loop, one sync per round) and grouping.
cudaError_t launch_colour_prepare(const MeshView& m, const ColourLayout& C, int sms, cudaStream_t s, int* num_colours,
                                  int* status_bits);
// out[e] = colour of element e.
cudaError_t launch_colour_export(const ColourLayout& C, int E, int* out, int sms, cudaStream_t s);
// values = 0, then one launch per (colour, type) group. Asynchronous.
cudaError_t launch_colour_assemble(const MeshView& m, const ColourLayout& C, int num_colours, const int* row_ptr,
                                   const int* col_idx, double* values, long long nnz, int sms, cudaStream_t s);


}  // namespace fem
