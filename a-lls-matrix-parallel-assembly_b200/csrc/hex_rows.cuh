// Tables of the Hex20 row lists (rows_hex20.cuh) and of their gather into CSR /
// BSR / upper-triangle CSR (write_hex20.cuh).
//
// A Hex20 scatter leaves, per row node, its sorted column nodes in the list
// chunks, and the packed Ke of every element (fem_element_stiffness's layout);
// the consolidation sums each row's element blocks where it writes them. An
// element's block (a, b) meets its row through two tables: the node's
// occurrences (node -> element e and local position a, as o = 20 e + a) and
// the rank of column node b in row node a's sorted list, map[20 o + b] (its low
// 16 bits: in a row of more than 65,536 columns the gather compares the columns).
#pragma once

#include "launch.h"

namespace fem {
namespace {

constexpr int kRankRange = 0x10000;  // columns of a row that the rank map tells apart

__device__ __forceinline__ unsigned occ_of(int word) { return (unsigned)word & ~kOccRepeats; }

// Column word (column node + 1) k of row node n: the first chunk's slots, then
// the row's overflow chunks, which are consecutive from chunk id `next` - 1 on.
__device__ __forceinline__ int* hex_col_word(const ListLayout& L, int n, int next, int k) {
    if (k < L.S1) return L.meta1 + (size_t)n * L.H1 + 2 + k;
    const int q = k - L.S1, c = next - 1 - L.N + q / L.S2;
    return L.meta2 + (size_t)c * L.H2 + 2 + q % L.S2;
}

}  // namespace
}  // namespace fem
