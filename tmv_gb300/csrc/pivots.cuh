// pivots.cuh -- the interchanges of one panel as a row gather (device side).
#pragma once

#include "common.cuh"

namespace tmvg {

// Largest panel width any factorisation kernel uses.
constexpr int kPairsPanelMax = 128;

// ---------------------------------------------------------------------
// The interchanges of one panel as a row gather.  Applying
// swap(row k+t, row piv[t]) for t = 0..nb-1 in order moves row src[q] to
// row dst[q] for at most 2*nb pairs; only rows k..k+nb-1 and the pivot rows
// change.  One warp replays the swaps on row labels in shared memory: slots
// 0..nb-1 are the rows of the block, slot nb + t the row piv[t] outside it
// (only ever a pivot row; one above the block, which no factorisation
// produces, is handled the same way), shared by the steps that name the same
// row.  The slots each step exchanges are found beforehand, by all lanes, so
// that the replay is two loads and two stores per step (searching a list at
// every step took 19 us for 64 interchanges; this 4).  pairs[0] = count, then
// the dst and src arrays of kMaxPairs each.
// ---------------------------------------------------------------------
constexpr int kMaxPairs = 2 * kPairsPanelMax;

// (CAP: largest nb; MAXP: distance of the dst and src arrays)
template <int CAP = kPairsPanelMax, int MAXP = kMaxPairs>
__device__ inline void panel_row_pairs(int64_t k, int nb, const int* piv, int* pairs)
{
    __shared__ int lab[2 * CAP];  // the row whose content each slot holds
    __shared__ short slot[CAP];   // the slot step t exchanges with slot t
    const int lane = threadIdx.x & 31;
    for (int t = lane; t < nb; t += 32) {
        const int p = piv[t];
        lab[t] = (int)(k + t);
        lab[nb + t] = p;
        int s = (int)(p - k);
        if (p < k || p >= k + nb) {
            s = 0;
            while (piv[s] != p) ++s;  // the first step that names the row
            s += nb;
        }
        slot[t] = (short)s;
    }
    __syncwarp();
    if (lane == 0) {
        for (int t = 0; t < nb; ++t) {
            const int s = slot[t];
            const int a = lab[t], b = lab[s];
            lab[t] = b;
            lab[s] = a;
        }
    }
    __syncwarp();
    // emit the moved rows: row dst receives the old content of row src
    int np = 0;
    for (int s0 = 0; s0 < 2 * nb; s0 += 32) {
        const int s = s0 + lane;
        const int row = s < nb ? (int)(k + s) : s < 2 * nb ? piv[s - nb] : 0;
        // (slots that no step uses hold their own row)
        const bool moved = s < 2 * nb && lab[s] != row;
        const unsigned m = __ballot_sync(0xffffffffu, moved);
        if (moved) {
            const int q = np + __popc(m & ((1u << lane) - 1u));
            pairs[1 + q] = row;
            pairs[1 + MAXP + q] = lab[s];
        }
        np += __popc(m);
    }
    if (lane == 0) pairs[0] = np;
}

}  // namespace tmvg
