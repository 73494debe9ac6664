#pragma once

#include "rows.cuh"
#include "windows.cuh"

namespace hdfe {
namespace rows {

// ------------------------------------------------------ Rademacher passes
//
// What bounds these passes is instruction issue (the centring pass: 71% of
// cycles) and, in the projection, the latency of a window's chain at 20 warps an
// SM (52%), not memory (3 and 6% of DRAM): N x B hashes and FP64 updates against
// N rows read once.  So per (row, draw) only what depends on both is left.  A
// sub-warp of BP lanes (lane j: draw j) takes a window of up to 32 rows made of
// whole groups, stages codes, covariates and weights lane-parallel in shared
// memory, and keeps each draw's signs of the window as one 32-bit word (bit q:
// row q).  Then, without weights, the sum of a run or a group is n - 2 popc(word
// & mask); the covariates' group sums are made once a window by lane (group,
// covariate); and U's row of a run of equal codes is gathered once, the window's
// first eight runs in flight during the hashing. The projection stores r o per
// (row, draw) in a padded tile (P = (r o)^2 and M = (1 - r o)^2 = (r - o)^2, r =
// +-1), and lane t then sums row t over the draws in draw order: one flush per 32
// rows rather than one per group, and coalesced.  A group of more than 32 rows is
// walked in chunks of 32, twice.
//
// 1M-worker panel (8.5M rows, 2 covariates, 32 draws): center 2.15 -> 0.82 ms,
// project with the five sums 5.30 -> 1.29 ms a block.

// The draw's sign by splitmix64 of seed ^ rterm ^ dterm (the row ordinal times
// kRowMul, the draw index times kDrawMul): the last step (x ^= x >> 31) leaves
// bit 63 alone, so the draw is -1 exactly when bit 63 is set before it.
__device__ __forceinline__ bool rad_negative(uint64_t seed, uint64_t rterm, uint64_t dterm)
{
    uint64_t x = seed ^ rterm ^ dterm;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return (x >> 63) != 0;
}

constexpr uint64_t kRowMul = 0x9E3779B97F4A7C15ull, kDrawMul = 0xBF58476D1CE4E5B9ull;

// shared memory of one sub-warp's window
template <int BP>
struct Win {
    static constexpr int kTileBytes = kWin * (BP + 1) * 8;
    // x (32 c), group sums (32 (c + 1)), weights (3 x 32) and codes (32 D)
    static __host__ __device__ int bytes(int c, int D, bool weights, bool tile)
    {
        const int b = kWin * c * 8 + kWin * (c + 1) * 8 + (weights ? 3 * kWin * 8 : 0) +
                      kWin * D * 4 + (tile ? kTileBytes : 0);
        return (b + 15) / 16 * 16;
    }
    double *x, *gx, *w, *wr, *root, *tile;
    uint32_t *codes;
    __device__ Win(char *p, int c, int D, bool weights, bool has_tile)
    {
        double *q = reinterpret_cast<double *>(p);
        tile = q;
        if (has_tile) q += kWin * (BP + 1);
        x = q;
        q += kWin * c;
        gx = q;
        q += kWin * (c + 1);
        w = q;
        wr = q + kWin;
        root = q + 2 * kWin;
        if (weights) q += 3 * kWin;
        codes = reinterpret_cast<uint32_t *>(q);
    }
};

// flip the sign of v when bit q of word is set
__device__ __forceinline__ double flip(double v, uint32_t word, int q)
{
    return __hiloint2double(__double2hiint(v) ^ (int)(((word >> q) & 1u) << 31),
                            __double2loint(v));
}

// Rows [i0, i0 + n) into the window; returns the run heads' mask (rows whose
// codes differ from the row before; row 0 always).  sq: this lane's part of
// sum w r^2 (null: not wanted).
template <int BP, int C, bool W>
__device__ __forceinline__ unsigned load_window(const Args &a, const Lanes<BP> &ln, Win<BP> &wn,
                                                int64_t i0, int n, double *sq)
{
    const int c = C < 0 ? a.c : C;
    for (int t = ln.j; t < n; t += BP) {
        const int64_t i = i0 + t;
        for (int d = 0; d < a.D; d++) {
            uint32_t code = a.codes[i * a.D + d];
            if ((int64_t)code >= a.nlev[d]) {
                if (a.status) atomicCAS(a.status, 0u, (unsigned)HDFE_ERR_BAD_CODE);
                code = 0;
            }
            wn.codes[t * a.D + d] = code;
        }
        for (int k = 0; k < c; k++) wn.x[t * c + k] = a.X[i * c + k];
        if (W) {
            const double w = a.w[i], ir = inv_root(a, w);
            wn.w[t] = w;
            wn.wr[t] = w * ir;
            if (a.sqrt_weights) wn.root[t] = sqrt(w);
            if (sq) *sq += w * ir * ir;
        } else if (sq) {
            *sq += 1.0;
        }
    }
    __syncwarp(ln.mask);
    unsigned heads = 0;
    for (int t = ln.j; t < n; t += BP) {
        bool head = t == 0;
        if (t > 0)
            for (int d = 0; d < a.D; d++)
                head |= wn.codes[t * a.D + d] != wn.codes[(t - 1) * a.D + d];
        heads |= (unsigned)head << t;
    }
    return __reduce_or_sync(ln.mask, heads);
}

// this lane's signs of rows [i0, i0 + n): bit q set when the draw is -1
__device__ __forceinline__ uint32_t window_signs(const Args &a, int64_t i0, int n, uint64_t dterm)
{
    uint32_t word = 0;
    uint64_t rterm = (uint64_t)(a.ordinal0 + i0) * kRowMul;
#pragma unroll 4
    for (int q = 0; q < n; q++) {
        word |= (uint32_t)rad_negative(a.seed, rterm, dterm) << q;
        rterm += kRowMul;
    }
    return word;
}

// gx[group, k] = the sum of w x_k over the group's rows (k < c) and of w (k =
// c), by lane (group, k); gheads: the groups' first rows, ng of them
template <int BP, int C, bool W>
__device__ __forceinline__ void group_sums(const Args &a, const Lanes<BP> &ln, Win<BP> &wn,
                                           unsigned gheads, int ng, int n)
{
    if constexpr (C != 0 || W) {
        const int c = C < 0 ? a.c : C, per = W ? c + 1 : c;
        for (int t = ln.j; t < ng * per; t += BP) {
            const int g = t / per, k = t - g * per;
            const int q0 = nth_bit(gheads, g), q1 = next_bit(gheads, q0, n);
            double v = 0.0;
            for (int q = q0; q < q1; q++) {
                const double xq = k < c ? wn.x[q * c + k] : 1.0;
                v += W ? wn.w[q] * xq : xq;
            }
            wn.gx[g * (c + 1) + k] = v;
        }
        __syncwarp(ln.mask);
    }
}

// the walk of this sub-warp
template <int BP, typename F, typename H>
__device__ __forceinline__ void walk(const Args &a, const Lanes<BP> &ln, F window, H lone)
{
    constexpr int SUBS = kPassThreads / BP;
    walk_windows<BP>(a.starts, a.G, a.chunk, (int64_t)blockIdx.x * SUBS + threadIdx.x / BP,
                     (int64_t)gridDim.x * SUBS, ln.j, ln.mask, window, lone);
}

// One Rademacher pass: the kernel for the block's width, the covariates' count
// (0 to 3 unrolled, else a loop to 8) and weights or none.  K<BP, C, W>::kernel
// is the kernel and K::kTile whether its windows have the tile.
template <template <int, int, bool> class K, int BP, int C, bool W>
int launch_draws(Args &a, cudaStream_t s)
{
    using Pass = K<BP, C, W>;
    constexpr int SUBS = kPassThreads / BP;
    const int smem = (Pass::kTile ? 0 : (int)((a.n_small * a.B * 8 + 15) / 16 * 16)) +
                     SUBS * Win<BP>::bytes(a.c, a.D, W, Pass::kTile);
    static hdfe_shared_limit limit;
    const int st = limit.raise((const void *)Pass::kernel(),
                               (Pass::kTile ? 0 : kSmallBytes) +
                                   SUBS * Win<BP>::bytes(C < 0 ? kMaxCov : C, HDFE_MAX_DIMS, true,
                                                         Pass::kTile));
    if (st != HDFE_OK) return st;
    const int64_t ctas = 148 * 5;
    a.chunk = window_chunk(a.G, ctas * SUBS);
    int64_t b = (a.G + a.chunk * SUBS - 1) / (a.chunk * SUBS);
    if (b > 2 * ctas) b = 2 * ctas;
    Pass::kernel()<<<(unsigned)(b > 0 ? b : 1), kPassThreads, smem, s>>>(a);
    return HDFE_OK;
}

template <template <int, int, bool> class K, int BP>
int launch_draws(Args &a, cudaStream_t s)
{
    const bool w = a.w != nullptr;
    switch (a.c) {
    case 0: return w ? launch_draws<K, BP, 0, true>(a, s) : launch_draws<K, BP, 0, false>(a, s);
    case 1: return w ? launch_draws<K, BP, 1, true>(a, s) : launch_draws<K, BP, 1, false>(a, s);
    case 2: return w ? launch_draws<K, BP, 2, true>(a, s) : launch_draws<K, BP, 2, false>(a, s);
    case 3: return w ? launch_draws<K, BP, 3, true>(a, s) : launch_draws<K, BP, 3, false>(a, s);
    default: return w ? launch_draws<K, BP, -1, true>(a, s) : launch_draws<K, BP, -1, false>(a, s);
    }
}

template <template <int, int, bool> class K>
int launch_draws(Args &a, cudaStream_t s)
{
    if (a.Bp == 8) return launch_draws<K, 8>(a, s);
    if (a.Bp == 16) return launch_draws<K, 16>(a, s);
    return launch_draws<K, 32>(a, s);
}

}  // namespace rows
}  // namespace hdfe
