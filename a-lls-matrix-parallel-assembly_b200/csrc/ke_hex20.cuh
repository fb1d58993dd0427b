// Device code of the FP64 Hex20 element stiffness (ke_hex20.cu, and the batch,
// batched.cu): every element in FP64, packed (upper node blocks),
// one warp per element on the FP64 tensor cores. The Ke of fem_element_stiffness
// and of the Hex20 scatter (rows_hex20.cuh).
//
// Replaces computeElementStiffnessHex20
// (ALLS_Hex20_3D_Assembly_Performance.cu:130-195: a 60x60 FP32 Ke per thread in
// 14.9 KB of local memory).
//
// With the 60 rows P[(n, a)][g] = dN_n/dx_a at Gauss point g, M = P diag(w) P^T
// (w_g = weight * detJ_g) holds every 3x3 node block's products, and
//     Ke_IJ[a][b] = lambda M_IJ[a][b] + mu M_IJ[b][a] + mu delta_ab tr M_IJ.
// The rows are taken direction-major, as eight 8-row tiles of a 64-row
// operand (tile: nodes, directions):
//     0 1 2: nodes 0..7, x y z     3 4 5: nodes 8..15, x y z
//     6: nodes 16..19, x then y    7: nodes 16..19, z, then four zero rows
// so that the upper triangle of M is 36 8x8 tiles of seven k-steps each
// (mma.sync.m8n8k4.f64: 252 of them; three 8-node groups padded to 24 take
// 378). A lane's fragment entries are the same numbers for the A and the B
// operand (row 8 t + lane / 4, k = 4 s + lane % 4), so the gradients stay in
// registers (56 per lane). The products leave per pair of node groups:
//     (0..7, 8..15): nine tiles, all products of a lane's two node pairs in the lane;
//     (0..7, 0..7) and (8..15, 8..15): six tiles, M^{ba}_IJ = M^{ab}_JI by shuffles;
//     (0..7 or 8..15, 16..19): the x and y halves of tile 6 traded between lanes 2 apart;
//     (16..19, 16..19): through a 12x12 scratch.
// Each block is staged in shared memory in the packed order and the element's
// 15,120 bytes leave with one bulk copy while the warp works on the next
// element (plain stores when the output is not 16-byte aligned).
//
// What bounds it: the FP64 pipe (36.9 TFLOP/s measured for m8n8k4: 16 cycles
// each per SM quarter; 4,032 cycles of products and about 1,400 of Jacobians,
// gradients and blocks per element and quarter: 1.3 ms for 64^3), then the
// output (0.61 ms at the measured copy rate). B200, 64^3: 1.67 ms, where one
// 4-warp CTA per element with its fragments and products in shared memory took
// 3.65 ms; 39x41x40: 437 against 910 us. 10 warps 2.01 ms, two CTAs of 4 warps
// 1.73 ms. Warps of one CTA take elements a grid apart, so that few elements
// spread over all SMs, and the first element's loads are in flight while the
// derivative table is built: 8 elements 7.9 us (8.7 us by CTAs of 4 warps; 13.0
// us with a CTA's warps on consecutive elements), 512 9.3 (14.3; 13.4), 1,728
// 18.0 (33.4; 22.5).
#pragma once

#include "hex20.cuh"
#include "launch.h"

namespace fem {
namespace {

// Warps per CTA (one CTA per SM): 8 leave 255 registers a thread; 10 (168 registers) spill.
#ifndef FEM_KE_WARPS
#define FEM_KE_WARPS 8
#endif
constexpr int kKeWarps = FEM_KE_WARPS;
constexpr int kKeThreads = kKeWarps * 32;
constexpr int kKeStride = 28;  // Gauss points padded to seven k-steps; row stride of the tables (doubles)
constexpr unsigned kKeFull = 0xFFFFFFFFu;

struct alignas(16) KeWarpSmem {
    double ke[kPackedHex20];  // the element's blocks on their way out
    double X[20][3];
    double iJw[kKeStride][10];       // inverse Jacobian (9) and weight * detJ per Gauss point; row 27 zero
    double m12[12][13];       // products of nodes 16..19: row 4 a + I, column 4 b + J
};
struct KeHexSmem {
    double dN[3][20][kKeStride];     // dN_n / dxi_i at Gauss point g: [i][n][g]
    KeWarpSmem w[kKeWarps];
};
static_assert(sizeof(KeWarpSmem) % 16 == 0 && (3 * 20 * kKeStride * 8) % 16 == 0, "16-byte aligned bulk copies");

__device__ __forceinline__ void ke_dmma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

// Stages the block of node pair I <= J from its nine products m[a][b].
__device__ __forceinline__ void put_block(double* ke, int I, int J, const double (&m)[3][3], double lam, double mu) {
    double* d = ke + 9 * hex20::pair_index(I, J);
    const double tr = mu * (m[0][0] + m[1][1] + m[2][2]);
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
        for (int b = 0; b < 3; b++) d[3 * a + b] = fma(lam, m[a][b], fma(mu, m[b][a], a == b ? tr : 0.0));
}

// Runs as block `block` of `nblocks`. bulk: ke_out is 16-byte aligned.
__device__ __forceinline__ void ke_hex20(const MeshView& m, double* __restrict__ ke_out, int* __restrict__ status,
                                         bool bulk, int block, int nblocks, KeHexSmem& sm) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, fr = lane >> 2, fc = lane & 3;
    KeWarpSmem& ws = sm.w[warp];
    const long long stride = (long long)nblocks * kKeWarps;
    long long e = (long long)warp * nblocks + block;  // few elements: spread over the SMs
    // the next element's nodes, then its coordinates and material, are loaded ahead
    auto load_node = [&](long long el) { return el < m.E_count && lane < 20 ? __ldg(m.conn + el * 20 + lane) : 0; };
    double px = 0.0, py = 0.0, pz = 0.0;
    bool pbad = false;
    auto load_coords = [&](long long el, int n) {
        pbad = false;
        if (el >= m.E_count) return;
        if (lane < 20) {
            pbad = n < 0 || n >= m.N;
            if (!pbad) {
                px = __ldg(m.x + n);
                py = __ldg(m.y + n);
                pz = __ldg(m.z + n);
            }
        } else if (lane == 20) {
            px = m.E ? __ldg(m.E + el) : m.E0;
            py = m.nu ? __ldg(m.nu + el) : m.nu0;
        }
    };
    load_coords(e, load_node(e));
    int pnode = load_node(e + stride);
    for (int idx = tid; idx < 27 * 20; idx += kKeThreads) {
        const int g = idx / 20, n = idx - 20 * g;
        double dx, dy, dz;
        hex20::dshape_node(n, hex20::gauss3(g / 9), hex20::gauss3((g / 3) % 3), hex20::gauss3(g % 3), dx, dy, dz);
        sm.dN[0][n][g] = dx;
        sm.dN[1][n][g] = dy;
        sm.dN[2][n][g] = dz;
    }
    for (int idx = tid; idx < 3 * 20; idx += kKeThreads) sm.dN[idx / 20][idx % 20][27] = 0.0;
    for (int k = lane; k < 10; k += 32) ws.iJw[27][k] = 0.0;
    __syncthreads();
    for (; e < m.E_count; e += stride) {
        const bool bad = __any_sync(kKeFull, pbad);
        if (lane < 20) {
            ws.X[lane][0] = px;
            ws.X[lane][1] = py;
            ws.X[lane][2] = pz;
        }
        const double E = __shfl_sync(kKeFull, px, 20), nu = __shfl_sync(kKeFull, py, 20);
        const double lam = E * nu / ((1.0 + nu) * (1.0 - 2.0 * nu)), mu = E / (2.0 * (1.0 + nu));
        load_coords(e + stride, pnode);
        pnode = load_node(e + 2 * stride);
        __syncwarp();
        if (bad) {  // the element's Ke is zero
            if (lane == 0) {
                atomicOr(status, 1 << FEM_ERR_BAD_MESH);
                asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            }
            __syncwarp();
            for (int k = lane; k < kPackedHex20; k += 32) ke_out[(size_t)e * kPackedHex20 + k] = 0.0;
            continue;
        }
        if (lane < 27) {
            // Jacobian at Gauss point g = lane: J[3i + j] = sum_n dN[i][n][g] X[n][j]
            const int g = lane;
            double J[9];
#pragma unroll
            for (int r = 0; r < 9; r++) J[r] = 0.0;
#pragma unroll 4
            for (int n = 0; n < 20; n++) {
                const double d0 = sm.dN[0][n][g], d1 = sm.dN[1][n][g], d2 = sm.dN[2][n][g];
                const double x0 = ws.X[n][0], x1 = ws.X[n][1], x2 = ws.X[n][2];
                J[0] = fma(d0, x0, J[0]);
                J[1] = fma(d0, x1, J[1]);
                J[2] = fma(d0, x2, J[2]);
                J[3] = fma(d1, x0, J[3]);
                J[4] = fma(d1, x1, J[4]);
                J[5] = fma(d1, x2, J[5]);
                J[6] = fma(d2, x0, J[6]);
                J[7] = fma(d2, x1, J[7]);
                J[8] = fma(d2, x2, J[8]);
            }
            const double c0 = J[4] * J[8] - J[5] * J[7], c1 = J[5] * J[6] - J[3] * J[8], c2 = J[3] * J[7] - J[4] * J[6];
            const double det = J[0] * c0 + J[1] * c1 + J[2] * c2;
            if (!(det > 0.0)) atomicOr(status, 1 << FEM_ERR_DETJ);
            const double r = 1.0 / det;
            double* o = ws.iJw[g];
            o[0] = c0 * r;
            o[1] = (J[2] * J[7] - J[1] * J[8]) * r;
            o[2] = (J[1] * J[5] - J[2] * J[4]) * r;
            o[3] = c1 * r;
            o[4] = (J[0] * J[8] - J[2] * J[6]) * r;
            o[5] = (J[2] * J[3] - J[0] * J[5]) * r;
            o[6] = c2 * r;
            o[7] = (J[1] * J[6] - J[0] * J[7]) * r;
            o[8] = (J[0] * J[4] - J[1] * J[3]) * r;
            o[9] = hex20::weight3(g / 9) * hex20::weight3((g / 3) % 3) * hex20::weight3(g % 3) * det;
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // ke is free
        __syncwarp();
        // the lane's gradients: G[t][s] at row 8 t + fr, Gauss point 4 s + fc
        double G[8][7], w[7];
#pragma unroll
        for (int s = 0; s < 7; s++) {
            const int g = 4 * s + fc;
            const double* iJ = ws.iJw[g];
            w[s] = iJ[9];
#pragma unroll
            for (int q = 0; q < 2; q++) {
                const int n = 8 * q + fr;
                const double d0 = sm.dN[0][n][g], d1 = sm.dN[1][n][g], d2 = sm.dN[2][n][g];
#pragma unroll
                for (int a = 0; a < 3; a++)
                    G[3 * q + a][s] = fma(iJ[3 * a], d0, fma(iJ[3 * a + 1], d1, iJ[3 * a + 2] * d2));
            }
            const int n = 16 + (fr & 3);
            const double d0 = sm.dN[0][n][g], d1 = sm.dN[1][n][g], d2 = sm.dN[2][n][g];
            const double* iA = iJ + (fr < 4 ? 0 : 3);
            G[6][s] = fma(iA[0], d0, fma(iA[1], d1, iA[2] * d2));
            G[7][s] = fr < 4 ? fma(iJ[6], d0, fma(iJ[7], d1, iJ[8] * d2)) : 0.0;
        }
        // nodes 0..7 x 8..15
        {
            double c[3][3][2] = {};
#pragma unroll
            for (int s = 0; s < 7; s++)
#pragma unroll
                for (int a = 0; a < 3; a++) {
                    const double A = w[s] * G[a][s];
#pragma unroll
                    for (int b = 0; b < 3; b++) ke_dmma(c[a][b], A, G[3 + b][s]);
                }
#pragma unroll
            for (int h = 0; h < 2; h++) {
                double p[3][3];
#pragma unroll
                for (int a = 0; a < 3; a++)
#pragma unroll
                    for (int b = 0; b < 3; b++) p[a][b] = c[a][b][h];
                put_block(ws.ke, fr, 8 + 2 * fc + h, p, lam, mu);
            }
        }
        // nodes 0..7 and 8..15 with themselves: tiles a <= b
#pragma unroll
        for (int q = 0; q < 2; q++) {
            double c[6][2] = {};  // xx xy xz yy yz zz
#pragma unroll
            for (int s = 0; s < 7; s++) {
                const double A0 = w[s] * G[3 * q][s], A1 = w[s] * G[3 * q + 1][s], A2 = w[s] * G[3 * q + 2][s];
                ke_dmma(c[0], A0, G[3 * q][s]);
                ke_dmma(c[1], A0, G[3 * q + 1][s]);
                ke_dmma(c[2], A0, G[3 * q + 2][s]);
                ke_dmma(c[3], A1, G[3 * q + 1][s]);
                ke_dmma(c[4], A1, G[3 * q + 2][s]);
                ke_dmma(c[5], A2, G[3 * q + 2][s]);
            }
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int J = 2 * fc + h, src = 4 * J + (fr >> 1);  // the lane with entry (J, I)
                double p[3][3];
                auto other = [&](int k) {
                    const double v0 = __shfl_sync(kKeFull, c[k][0], src), v1 = __shfl_sync(kKeFull, c[k][1], src);
                    return fr & 1 ? v1 : v0;
                };
                p[0][0] = c[0][h];
                p[0][1] = c[1][h];
                p[0][2] = c[2][h];
                p[1][1] = c[3][h];
                p[1][2] = c[4][h];
                p[2][2] = c[5][h];
                p[1][0] = other(1);
                p[2][0] = other(2);
                p[2][1] = other(4);
                if (fr <= J) put_block(ws.ke, 8 * q + fr, 8 * q + J, p, lam, mu);
            }
        }
        // nodes 0..7 and 8..15 x 16..19: columns of tile 6 are x (fc < 2) and y of the same nodes, of tile 7 z (fc < 2)
#pragma unroll
        for (int q = 0; q < 2; q++) {
            double c[3][2][2] = {};
#pragma unroll
            for (int s = 0; s < 7; s++)
#pragma unroll
                for (int a = 0; a < 3; a++) {
                    const double A = w[s] * G[3 * q + a][s];
                    ke_dmma(c[a][0], A, G[6][s]);
                    ke_dmma(c[a][1], A, G[7][s]);
                }
            // lane fc < 2 takes node 16 + 2 fc, its partner (fc + 2) node 16 + 2 fc + 1
            const bool low = fc < 2;
            double p[3][3];
#pragma unroll
            for (int a = 0; a < 3; a++) {
                const double v1 = __shfl_xor_sync(kKeFull, low ? c[a][0][1] : c[a][0][0], 2);
                const double v2 = __shfl_xor_sync(kKeFull, c[a][1][1], 2);
                p[a][0] = low ? c[a][0][0] : v1;
                p[a][1] = low ? v1 : c[a][0][1];
                p[a][2] = low ? c[a][1][0] : v2;
            }
            put_block(ws.ke, 8 * q + fr, 16 + 2 * (fc & 1) + (low ? 0 : 1), p, lam, mu);
        }
        // nodes 16..19 with themselves
        {
            double c[3][2] = {};
#pragma unroll
            for (int s = 0; s < 7; s++) {
                const double A6 = w[s] * G[6][s];
                ke_dmma(c[0], A6, G[6][s]);
                ke_dmma(c[1], A6, G[7][s]);
                ke_dmma(c[2], w[s] * G[7][s], G[7][s]);
            }
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int col = 2 * fc + h;
                ws.m12[fr][col] = c[0][h];
                if (fc < 2) {
                    ws.m12[fr][8 + col] = c[1][h];
                    ws.m12[8 + col][fr] = c[1][h];  // (z, x) and (z, y) from the symmetry of M
                    if (fr < 4) ws.m12[8 + fr][8 + col] = c[2][h];
                }
            }
            __syncwarp();
            if (lane < 16) {
                const int I = lane >> 2, J = lane & 3;
                if (I <= J) {
                    double p[3][3];
#pragma unroll
                    for (int a = 0; a < 3; a++)
#pragma unroll
                        for (int b = 0; b < 3; b++) p[a][b] = ws.m12[4 * a + I][4 * b + J];
                    put_block(ws.ke, 16 + I, 16 + J, p, lam, mu);
                }
            }
        }
        double* out = ke_out + (size_t)e * kPackedHex20;
        if (bulk) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                const unsigned src = (unsigned)__cvta_generic_to_shared(ws.ke);
                asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(out), "r"(src),
                             "r"(kPackedHex20 * 8)
                             : "memory");
                asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            }
        } else {
            __syncwarp();
            for (int k = lane; k < kPackedHex20; k += 32) out[k] = ws.ke[k];
            __syncwarp();
        }
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

}  // namespace
}  // namespace fem
