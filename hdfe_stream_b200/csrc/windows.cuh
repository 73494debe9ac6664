// Windows of rows: how the row passes give a sub-warp of BP lanes up to 32
// consecutive rows made of whole groups at a time.
#pragma once

#include "common.cuh"

namespace hdfe {

constexpr int kWin = 32;                // rows of a window
constexpr int kMaxChunk = 64;           // most groups a sub-warp takes at a time

__device__ __forceinline__ unsigned below(int n) { return n >= 32 ? 0xffffffffu : (1u << n) - 1u; }

// the next set bit of m after q, or n
__device__ __forceinline__ int next_bit(unsigned m, int q, int n)
{
    const unsigned r = q >= 31 ? 0u : m & ~below(q + 1);
    return r ? min(__ffs(r) - 1, n) : n;
}

// the place of the r-th set bit of m (r counts from 0)
__device__ __forceinline__ int nth_bit(unsigned m, int r)
{
    for (int k = 0; k < r; k++) m &= m - 1;
    return __ffs(m) - 1;
}

// A sub-warp's walk over its chunks of groups (lane j of BP, sub-warp `sub` of
// `subs` in the grid): window(g, i0, n, gheads, ng) for each window, groups g
// to g + ng - 1 and rows i0 to i0 + n - 1 with the groups' first rows in
// gheads, and lone(g, s, e) for a group of more than 32 rows or of none.
template <int BP, typename F, typename H>
__device__ __forceinline__ void walk_windows(const int64_t *starts, int64_t G, int64_t chunk,
                                             int64_t sub, int64_t subs, int j, unsigned mask,
                                             F window, H lone)
{
    for (int64_t ga = sub * chunk; ga < G; ga += subs * chunk) {
        const int64_t gb = min(ga + chunk, G);
        for (int64_t g = ga; g < gb;) {
            const int64_t s0 = starts[g];
            const int64_t e = g + j < gb ? starts[g + j + 1] : INT64_MAX;
            int64_t b = __shfl_up_sync(mask, e, 1, BP);
            if (j == 0) b = s0;
            const unsigned m =
                (__ballot_sync(mask, e - s0 <= kWin && e > b) & mask) >> ((threadIdx.x & 31) / BP * BP);
            const int ng = __ffs(~m) - 1 < 0 ? 32 : __ffs(~m) - 1;
            if (ng == 0) {
                lone(g, s0, starts[g + 1]);
                g++;
            } else {
                const int n = (int)(__shfl_sync(mask, e, ng - 1, BP) - s0);
                // group t + 1 of the window starts at the end of group t
                const unsigned gheads =
                    __reduce_or_sync(mask, j < ng - 1 ? 1u << (int)(e - s0) : 0u) | 1u;
                window(g, s0, n, gheads, ng);
                g += ng;
            }
            __syncwarp(mask);               // the next window reuses the staging
        }
    }
}

// Groups a sub-warp takes at a time: 64, fewer on panels that would leave
// sub-warps without a chunk.
inline int64_t window_chunk(int64_t G, int64_t subs)
{
    const int64_t chunk = (G + 2 * subs - 1) / (2 * subs);
    return chunk < 4 ? 4 : (chunk > kMaxChunk ? kMaxChunk : chunk);
}

}  // namespace hdfe
