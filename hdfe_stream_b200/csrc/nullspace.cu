// The normal equations' null space taken out of coefficient-space vectors.
//
// Reference: inverse.py:376-428 `_null_space` (per connected component +1 on
// its groups and -1 on its levels of the first non-streamed dimension; per
// further dimension +1 across the first and -1 across it) and :445-460
// `_drop_null_component`.
//
// Every vector of that basis is constant on blocks of entries: a component's
// groups (block c of K), its levels of the first dimension (K + c), and each
// further dimension (2 K + d - 1).  So the projection needs the vectors' sums
// over the blocks, a correction per block, and one addition per entry: two
// reads and one write of the (G + L, B) block, which bounds it, instead of a
// dense (G + L, k) basis with its QR factorisation and products.  The sums of
// squares of what is left (the scale of the solve) come out of the same pass.
// 1.1M entries, 32 vectors: about 470 -> 216 us with the scale; the basis
// itself took a host QR (25 ms there), now a few counts.
#include <cuda_runtime.h>

#include "common.cuh"

namespace hdfe {
namespace nullspace {

constexpr int kThreads = 256;

struct Args {
    const double *levels, *streamed;        // (L, B), (G, B)
    int64_t L, G, n0;
    int B, D;
    const int32_t *comp_g, *comp_l;         // (G), (n0): 0 .. K - 1
    int64_t K;
    int64_t ends[HDFE_MAX_DIMS];            // past each dimension's last level
    const double *inv_size;                 // (K): 1 / (groups + levels of the component)
    const double *Q;                        // (2 K + D - 1, D - 1) orthonormal block values
    double *sums, *corr;                    // (2 K + D - 1, B) each
    double *out_levels, *out_streamed, *norm2;
};

__device__ __forceinline__ int64_t block_of(const Args &a, int64_t i)
{
    if (i < a.G) return a.K == 1 ? 0 : a.comp_g[i];
    const int64_t l = i - a.G;
    if (l < a.n0) return a.K + (a.K == 1 ? 0 : a.comp_l[l]);
    int d = 1;
    while (d < a.D - 1 && l >= a.ends[d]) d++;
    return 2 * a.K + d - 1;
}

// A thread holds column tid % B of rows tid / B, + rows per CTA, ...; its sum
// is added when the block of entries changes, and per CTA at the end when all
// of the CTA's threads end in one block.
__global__ void __launch_bounds__(kThreads) k_block_sums(Args a)
{
    __shared__ double s_sum[kThreads];
    const int per = kThreads / a.B;
    const int j = threadIdx.x % a.B, r = threadIdx.x / a.B;
    const int64_t n = a.G + a.L, step = (int64_t)gridDim.x * per;
    if (a.K == 1) {
        // the giant component alone: every block is one range of entries, whose
        // loop has no block to look up or flush
        int64_t lo = 0;
        for (int b = 0; b < 1 + a.D; b++) {
            const int64_t hi = b == 0 ? a.G : a.G + a.ends[b - 1];
            double t = 0.0;
            if (r < per) {
                const double *p = b == 0 ? a.streamed : a.levels - a.G * a.B;
#pragma unroll 8
                for (int64_t i = lo + (int64_t)blockIdx.x * per + r; i < hi; i += step)
                    t += p[i * a.B + j];
            }
            s_sum[threadIdx.x] = t;
            __syncthreads();
            if (threadIdx.x < a.B && lo + (int64_t)blockIdx.x * per < hi) {
                t = 0.0;
                for (int q = 0; q < per; q++) t += s_sum[q * a.B + threadIdx.x];
                atomicAdd(a.sums + b * a.B + threadIdx.x, t);
            }
            __syncthreads();
            lo = hi;
        }
        return;
    }
    int64_t at = -1;
    double sum = 0.0;
    if (r < per) {
        for (int64_t i = (int64_t)blockIdx.x * per + r; i < n; i += step) {
            const int64_t b = block_of(a, i);
            const double v = i < a.G ? a.streamed[i * a.B + j] : a.levels[(i - a.G) * a.B + j];
            if (b != at) {
                if (at >= 0) atomicAdd(a.sums + at * a.B + j, sum);
                at = b;
                sum = 0.0;
            }
            sum += v;
        }
    }
    // one block for the whole CTA (its first thread always has rows)
    __shared__ int64_t s_at;
    if (threadIdx.x == 0) s_at = at;
    s_sum[threadIdx.x] = sum;
    __syncthreads();
    const bool one = __syncthreads_and(r >= per || at == s_at || at < 0);
    if (one) {
        if (threadIdx.x < a.B && s_at >= 0) {
            double t = 0.0;
            for (int q = 0; q < per; q++) t += s_sum[q * a.B + threadIdx.x];
            atomicAdd(a.sums + s_at * a.B + threadIdx.x, t);
        }
    } else if (r < per && at >= 0) {
        atomicAdd(a.sums + at * a.B + j, sum);
    }
}

// corr = the null component's value on each block; one CTA
__global__ void __launch_bounds__(kThreads) k_correct(Args a)
{
    __shared__ double s_dot[(HDFE_MAX_DIMS - 1) * 32];
    const int64_t nb = 2 * a.K + a.D - 1;
    const int m = a.D - 1;
    for (int t = threadIdx.x >> 5; t < m * a.B; t += kThreads / 32) {
        const int d = t / a.B, j = t % a.B;
        double v = 0.0;
        for (int64_t b = threadIdx.x & 31; b < nb; b += 32) v += a.Q[b * m + d] * a.sums[b * a.B + j];
        v = warp_sum(v);
        if ((threadIdx.x & 31) == 0) s_dot[t] = v;
    }
    __syncthreads();
    for (int64_t t = threadIdx.x; t < nb * a.B; t += kThreads) {
        const int64_t b = t / a.B;
        const int j = (int)(t - b * a.B);
        double v = 0.0;
        if (b < 2 * a.K) {
            const int64_t c = b < a.K ? b : b - a.K;
            v = (a.sums[c * a.B + j] - a.sums[(a.K + c) * a.B + j]) * a.inv_size[c];
            if (b >= a.K) v = -v;
        }
        for (int d = 0; d < m; d++) v += a.Q[b * m + d] * s_dot[d * a.B + j];
        a.corr[t] = v;
    }
}

__global__ void __launch_bounds__(kThreads) k_apply(Args a)
{
    __shared__ double s_sum[kThreads];
    const int per = kThreads / a.B;
    const int j = threadIdx.x % a.B, r = threadIdx.x / a.B;
    const int64_t n = a.G + a.L, step = (int64_t)gridDim.x * per;
    double sq = 0.0;
    if (r < per) {
#pragma unroll 4
        for (int64_t i = (int64_t)blockIdx.x * per + r; i < n; i += step) {
            const double *in = i < a.G ? a.streamed + i * a.B : a.levels + (i - a.G) * a.B;
            double *out = i < a.G ? a.out_streamed + i * a.B : a.out_levels + (i - a.G) * a.B;
            const double v = in[j] - a.corr[block_of(a, i) * a.B + j];
            out[j] = v;
            sq += v * v;
        }
    }
    s_sum[threadIdx.x] = sq;
    __syncthreads();
    if (threadIdx.x < a.B) {
        double t = 0.0;
        for (int q = 0; q < per; q++) t += s_sum[q * a.B + threadIdx.x];
        atomicAdd(a.norm2 + threadIdx.x, t);
    }
}

}  // namespace nullspace
}  // namespace hdfe

using namespace hdfe;

extern "C" int64_t hdfe_drop_null_workspace_bytes(int64_t n_components, int32_t D, int32_t B)
{
    if (n_components < 1 || D < 1 || D > HDFE_MAX_DIMS || B < 1 || B > 32) return -1;
    return 2 * (2 * n_components + D - 1) * B * 8;
}

extern "C" int hdfe_drop_null(const double *levels, const double *streamed, int64_t n_groups,
                              int32_t B, int32_t D, const int64_t *n_levels,
                              const int32_t *comp_groups, const int32_t *comp_levels,
                              int64_t n_components, const double *inv_size, const double *Q,
                              double *out_levels, double *out_streamed, double *norm2,
                              void *workspace, int64_t workspace_bytes, void *stream)
{
    if (D < 1 || D > HDFE_MAX_DIMS || !n_levels || n_groups < 0 || B < 1 || B > 32 || !levels ||
        (n_groups > 0 && (!streamed || !out_streamed)) || !comp_groups || !comp_levels ||
        n_components < 1 || !inv_size || (D > 1 && !Q) || !out_levels || !norm2 || !workspace)
        return hdfe_set_arg_error("hdfe_drop_null: bad argument");
    if (workspace_bytes < hdfe_drop_null_workspace_bytes(n_components, D, B))
        return hdfe_set_error(HDFE_ERR_WORKSPACE, "hdfe_drop_null: workspace too small");
    nullspace::Args a{};
    a.levels = levels;
    a.streamed = streamed;
    a.G = n_groups;
    a.B = B;
    a.D = D;
    for (int d = 0; d < D; d++) {
        if (n_levels[d] < 1) return hdfe_set_arg_error("hdfe_drop_null: n_levels must be >= 1");
        a.L += n_levels[d];
        a.ends[d] = a.L;
    }
    a.n0 = n_levels[0];
    a.comp_g = comp_groups;
    a.comp_l = comp_levels;
    a.K = n_components;
    a.inv_size = inv_size;
    a.Q = Q;
    const int64_t nb = 2 * n_components + D - 1;
    a.sums = (double *)workspace;
    a.corr = a.sums + nb * B;
    a.out_levels = out_levels;
    a.out_streamed = out_streamed;
    a.norm2 = norm2;
    cudaStream_t s = (cudaStream_t)stream;
    HDFE_CUDA_TRY(cudaMemsetAsync(a.sums, 0, nb * B * 8, s));
    HDFE_CUDA_TRY(cudaMemsetAsync(norm2, 0, B * 8, s));
    const int64_t per = nullspace::kThreads / B;
    int64_t grid = (a.G + a.L + 4 * per - 1) / (4 * per);
    if (grid > 148 * 8) grid = 148 * 8;
    nullspace::k_block_sums<<<(unsigned)grid, nullspace::kThreads, 0, s>>>(a);
    nullspace::k_correct<<<1, nullspace::kThreads, 0, s>>>(a);
    nullspace::k_apply<<<(unsigned)grid, nullspace::kThreads, 0, s>>>(a);
    HDFE_CUDA_TRY(cudaGetLastError());
    hdfe_add_launches(3);
    return HDFE_OK;
}
