// Place of a particle inside its cell, for the reorder passes of both forms.
#pragma once

#include <cuda_runtime.h>

namespace tsg {
namespace {

// Rank of old index s among the particles perm[cb, ce) of its cell; every lane of the warp calls
// it, with on unset where there is nothing to rank.  Cells up to kRankWide (ordinary ones hold a
// few dozen) are read entry by entry.  Scenes of up to kSortAll particles come here with larger
// ones too (after a blow-up the out-of-grid bin holds nearly all of them), where that would be
// quadratic: the lanes of such a cell put their indices in order, every entry of the cell is
// counted once, in the gap between them that it falls into, and the sums over the gaps are the
// ranks.  sh: 64 ints of this warp.  Sort with 9,600 of 11,298 particles in one cell, FP64 /
// FP32-mixed: 57 / 60 us (180 / 183 us entry by entry; 68 / 60 us with a block sorting the cell in
// a launch of its own, which every healthy step would pay for too).
constexpr int kRankWide = 64;
__device__ __forceinline__ int rank_in_cell(const int* __restrict__ perm, int cb, int ce, int s, bool on, int* sh) {
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const bool wide = on && ce - cb > kRankWide;
    int r = 0;
    if (on && !wide)
        for (int q = cb; q < ce; ++q) r += perm[q] < s;
    int* gap = sh + 32;
    for (unsigned left = __ballot_sync(kAll, wide); left;) {  // one cell of the warp's at a time
        const int first = __ffs(left) - 1;
        const int b = __shfl_sync(kAll, cb, first), e = __shfl_sync(kAll, ce, first);
        const bool mine = wide && cb == b;
        left &= ~__ballot_sync(kAll, mine);
        const int key = mine ? s : 0x7fffffff;
        int place = 0;
        for (int o = 0; o < 32; ++o) {
            const int k = __shfl_sync(kAll, key, o);
            place += k < key || (k == key && o < lane);
        }
        sh[place] = key;
        gap[lane] = 0;
        __syncwarp();
        const int kth = sh[lane];
        constexpr int U = 8;  // chunks in flight
        for (int q0 = b; q0 < e; q0 += 32 * U) {
            int p[U], u[U];
#pragma unroll
            for (int c = 0; c < U; ++c) p[c] = q0 + 32 * c + lane < e ? perm[q0 + 32 * c + lane] : 0x7fffffff;
#pragma unroll
            for (int c = 0; c < U; ++c) {  // keys up to p
                u[c] = 0;
#pragma unroll
                for (int step = 16; step > 0; step >>= 1)
                    if (__shfl_sync(kAll, kth, u[c] + step - 1) <= p[c]) u[c] += step;
                if (__shfl_sync(kAll, kth, u[c]) <= p[c]) u[c] = 32;
            }
#pragma unroll
            for (int c = 0; c < U; ++c)
                if (u[c] < 32) atomicAdd(&gap[u[c]], 1);
        }
        __syncwarp();
        int below = gap[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int w = __shfl_up_sync(kAll, below, o);
            if (lane >= o) below += w;
        }
        __syncwarp();
        const int mine_below = __shfl_sync(kAll, below, place);
        if (mine) r = mine_below;
    }
    return r;
}

}  // namespace
}  // namespace tsg
