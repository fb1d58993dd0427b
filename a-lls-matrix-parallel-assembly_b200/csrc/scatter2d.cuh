// Device code of the hashed 2-D A-LLS insertion, for the long rows of rows2d.cuh.
//
// A row's columns live in chunks of 14 hashed slots; a column is found, or
// claimed with atomicCAS(empty -> col) at the first empty slot of its probe
// sequence; a CAS that meets another column marks that slot taken in the
// caller's view and moves on along the sequence (slots are never freed, so a
// column is always found or placed at the first empty slot of its sequence,
// never twice). A chunk whose probe sequence is full continues in an overflow
// chunk. The values of every slot start at zero, so the claimer and every later
// contributor alike add their block with FP64 atomics: the claim publishes the
// column at once, with no pending state, no fence and no waiting on another
// thread. The reference's head insert can lose a contribution or insert a
// column twice (Q4A:452-463); this protocol does neither.
#pragma once

#include "element2d.cuh"
#include "launch.h"

namespace fem {
namespace {

enum SlotState : int { kUnresolved = 0, kFound = 1, kClaimed = 3, kSkip = 4 };
constexpr int kMask14 = (1 << k2DSlots) - 1;

__device__ __forceinline__ unsigned rot14(unsigned m, int h) {
    return ((m >> h) | (m << (k2DSlots - h))) & kMask14;
}

// Finds or claims the slot of column key `key` in the row list of node `row`.
// Returns the slot state (kFound or kClaimed; kSkip: the chain has no end); gid is
// the slot's global id. A column that needs a further chunk is left
// kUnresolved, and `last` is then the chain's last chunk + 1 (0 before the first
// call): the chunks up to it are full of other columns for good, so the next call
// goes on behind it.
__device__ __forceinline__ int resolve_2d(const ListLayout& L, int row, int key, int& last, unsigned& gid) {
    int c = last ? ld_cg(chunk_meta(L, last - 1) + 1) - 1 : row;
    if (c < 0) return kUnresolved;
    for (int step = 0; step < kMaxChainSteps; step++) {
        int* meta = chunk_meta(L, c);
        const int4 w0 = ld_cg4(meta), w1 = ld_cg4(meta + 4), w2 = ld_cg4(meta + 8), w3 = ld_cg4(meta + 12);
        const int cols[k2DSlots] = {w0.z, w0.w, w1.x, w1.y, w1.z, w1.w, w2.x,
                                    w2.y, w2.z, w2.w, w3.x, w3.y, w3.z, w3.w};
        unsigned empty = 0, match = 0;
#pragma unroll
        for (int s = 0; s < k2DSlots; s++) {
            empty |= (cols[s] == 0 ? 1u : 0u) << s;
            match |= (cols[s] == key ? 1u : 0u) << s;
        }
        int state = kUnresolved, pos = 0;
        if (match) {
            pos = __ffs(match) - 1;
            state = kFound;
        } else {
            const int h = probe_start(key, k2DSlots);
            for (int tries = 0; tries < k2DSlots; tries++) {
                const unsigned cand = rot14(empty, h);
                if (!cand) break;  // probe sequence full in this chunk: go on in the next one
                pos = h + __ffs(cand) - 1;
                pos -= pos >= k2DSlots ? k2DSlots : 0;
                const int old = atomicCAS(meta + 2 + pos, 0, key);
                if (old == 0) {
                    state = kClaimed;
                    break;
                }
                if (old == key) {
                    state = kFound;
                    break;
                }
                empty &= ~(1u << pos);  // taken by another column meanwhile
            }
        }
        if (state != kUnresolved) {
            gid = slot_gid(L, c, pos);
            return state;
        }
        last = c + 1;
        c = ld_cg(meta + 1) - 1;
        if (c < 0) return kUnresolved;
    }
    raise_status(L.info, FEM_ERR_TIMEOUT);
    return kSkip;
}

}  // namespace
}  // namespace fem
