// What the row passes share: their arguments and the sub-warp layout.
#pragma once

#include <cuda_runtime.h>

#include "common.cuh"

namespace hdfe {
namespace rows {

constexpr int kMaxCov = 8;

struct Args {
    const int64_t *starts;      // (G+1) row boundaries of the groups
    int64_t G;
    const uint32_t *codes;      // (N, D)
    int D;
    int64_t offs[HDFE_MAX_DIMS];
    int64_t nlev[HDFE_MAX_DIMS];
    int small[HDFE_MAX_DIMS];
    int64_t soff[HDFE_MAX_DIMS];
    int64_t n_small;
    int64_t L;
    const double *w;            // (N) or null (ones)
    const double *X;            // (N, c) covariates or null
    int c;
    const double *R;            // (N, B) explicit vectors, or null: Rademacher
    uint64_t seed;
    int64_t first_draw, ordinal0;
    int B, Bp;
    int sqrt_weights;
    int64_t chunk;              // groups a sub-warp takes at a time (the Rademacher passes)
    // center
    double *acc, *acc_x, *squares;
    // project
    const double *U, *C;        // (L, B), (c, B)
    double *out;                // (N, B) or null
    double *moments;            // (5, N) or null
    int64_t N;
    unsigned *status;
};

constexpr int kPassThreads = 128;
constexpr int kSmallBytes = 40 * 1024;    // small dimensions' level x draw sums per CTA

// a sub-warp of BP lanes: lane j holds draw j of the block (on: j < B)
template <int BP>
struct Lanes {
    int lane, j, sub;
    unsigned mask;
    bool on;
    __device__ Lanes(int B)
    {
        lane = threadIdx.x & 31;
        j = lane % BP;
        sub = lane / BP;
        mask = BP == 32 ? 0xffffffffu : (((1u << BP) - 1u) << (sub * BP));
        on = j < B;
    }
};

__device__ __forceinline__ double inv_root(const Args &a, double w)
{
    return a.sqrt_weights ? (w > 0.0 ? 1.0 / sqrt(w) : 0.0) : 1.0;
}

// The passes over Rademacher draws (a.R null); Bp, c, weights, D and the small
// dimensions' slots filled in.
int launch_center_draws(Args &a, cudaStream_t s);
int launch_project_draws(Args &a, cudaStream_t s);

}  // namespace rows
}  // namespace hdfe
