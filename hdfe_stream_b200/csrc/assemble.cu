// Steps 3-4 of a fit, as far as the KSS components read them.
//
// Reference: core/kernels_base.py:114-146 `_nb_residualize_rows` with
// core/inference.py:109-135 `_assemble` (V' W V of the fully residualised
// variables), core/kernels_base.py:544-615 `_nb_pass2` (residuals and the
// streamed effect, with gam_y = Gamma_y - Gamma_x beta, core/inference.py:
// 454-456) and the KSS pieces of leaveout.py: the plug-in moments' sums
// (:807-833) and sigma2 (:949-1016, stayers "own", weighted centring).
//
// A warp takes windows of up to 32 consecutive rows made of whole groups, a row
// a lane: the rows are read once and coalesced, the groups' sums are segmented
// sums over the lanes.  (A thread per group read its rows twice, 8 rows apart
// from its neighbours': 331 us for the moments of 3.4M rows of 3
// variables, 85 now; the bound is the latency of a window's chain,
// starts -> rows -> Gamma's gathers -> sums.)  Per-lane sums are combined per CTA
// in a fixed order and then over CTAs in a fixed order, and the windows are
// dealt statically, so the results are deterministic.
#include <cuda_runtime.h>

#include "windows.cuh"

namespace hdfe {
namespace assemble {

constexpr int kThreads = 256;
constexpr int kGrid = 148 * 4;
constexpr int kMaxM = 8;

struct Args {
    const int64_t *starts;
    int64_t G;
    const uint32_t *codes;
    int D;
    int64_t offs[HDFE_MAX_DIMS];
    int64_t nlev[HDFE_MAX_DIMS];
    const double *w;
    const double *V;        // (m, N): one row per variable
    int m;
    int64_t N;
    int64_t chunk;          // groups a warp takes at a time
    unsigned *status;
};

__device__ __forceinline__ int64_t level(const Args &a, int64_t i, int d)
{
    uint32_t c = a.codes[i * a.D + d];
    if ((int64_t)c >= a.nlev[d]) {
        if (a.status) atomicCAS(a.status, 0u, (unsigned)HDFE_ERR_BAD_CODE);
        c = 0;
    }
    return a.offs[d] + c;
}

// per CTA: thread values v[0..n) summed over the CTA in thread order
__device__ __forceinline__ void cta_sums(const double *v, int n, double *s_part, double *out)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int q = 0; q < n; q++) {
        const double t = warp_sum(v[q]);
        if (lane == 0) s_part[warp * n + q] = t;
    }
    __syncthreads();
    for (int q = threadIdx.x; q < n; q += kThreads) {
        double s = 0.0;
        for (int wv = 0; wv < kThreads / 32; wv++) s += s_part[wv * n + q];
        out[(int64_t)blockIdx.x * n + q] = s;
    }
}

// Row i's variables less their fixed-effect projections.
template <int M>
__device__ __forceinline__ void projected(const Args &a, const double *Gamma, int64_t i,
                                          double (&r)[M])
{
#pragma unroll
    for (int j = 0; j < M; j++) r[j] = a.V[(int64_t)j * a.N + i];
#pragma unroll 2
    for (int d = 0; d < a.D; d++) {
        const int64_t l = level(a, i, d);
#pragma unroll
        for (int j = 0; j < M; j++) r[j] -= Gamma[l * M + j];
    }
}

// x[q] summed over the lanes of this lane's segment (start .. last), the longest
// of the warp's `longest` lanes; every lane of it has the sum.
template <int NS>
__device__ __forceinline__ void segment_sums(double (&x)[NS], int start, int last, int longest)
{
    const int lane = threadIdx.x & 31;
    for (int o = 1; o < longest; o <<= 1) {
        const bool in = lane - o >= start;
#pragma unroll
        for (int q = 0; q < NS; q++) {
            const double y = __shfl_up_sync(0xffffffffu, x[q], o);
            if (in) x[q] += y;
        }
    }
#pragma unroll
    for (int q = 0; q < NS; q++) x[q] = __shfl_sync(0xffffffffu, x[q], last);
}

// The groups' rows, window by window:
//   load(i, w, r)            row i's values r[NR]
//   sums(w, r, x)            its terms of the group's sums x[NS]
//   use(i, w, r, x, z)       with the group's sums x: the row's part, and its
//                            terms z[NZ] of the group's second sums
//   done(g, x, z)            once a group, with both sums
// A group of more than 32 rows is read twice by the whole warp.
template <int NR, int NS, int NZ, typename Load, typename Sums, typename Use, typename Done>
__device__ __forceinline__ void group_rows(const Args &a, Load load, Sums sums, Use use, Done done)
{
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * kThreads + threadIdx.x) >> 5;
    const int64_t warps = ((int64_t)gridDim.x * kThreads) >> 5;
    walk_windows<32>(
        a.starts, a.G, a.chunk, warp, warps, lane, 0xffffffffu,
        [&](int64_t g, int64_t i0, int n, unsigned heads, int) {
            const bool have = lane < n;
            const int64_t i = i0 + lane;
            const int start = 31 - __clz(heads & below(lane + 1));
            const int last = next_bit(heads, lane, n) - 1;
            const int longest = __reduce_max_sync(0xffffffffu, have ? last - start + 1 : 0);
            double w = 0.0, r[NR], x[NS], z[NZ];
#pragma unroll
            for (int q = 0; q < NR; q++) r[q] = 0.0;
#pragma unroll
            for (int q = 0; q < NS; q++) x[q] = 0.0;
#pragma unroll
            for (int q = 0; q < NZ; q++) z[q] = 0.0;
            if (have) {
                w = a.w ? a.w[i] : 1.0;
                load(i, r);
                sums(w, r, x);
            }
            segment_sums(x, start, have ? last : lane, longest);
            if (have) use(i, w, r, x, z);
            if (NZ > 1) segment_sums(z, start, have ? last : lane, longest);
            if (have && lane == last) done(g + __popc(heads & below(lane + 1)) - 1, x, z);
        },
        [&](int64_t g, int64_t s, int64_t e) {
            double x[NS], z[NZ];
#pragma unroll
            for (int q = 0; q < NS; q++) x[q] = 0.0;
#pragma unroll
            for (int q = 0; q < NZ; q++) z[q] = 0.0;
            for (int64_t i = s + lane; i < e; i += 32) {
                double r[NR];
                load(i, r);
                double t[NS];
                sums(a.w ? a.w[i] : 1.0, r, t);
#pragma unroll
                for (int q = 0; q < NS; q++) x[q] += t[q];
            }
#pragma unroll
            for (int q = 0; q < NS; q++) x[q] = warp_sum(x[q]);
            for (int64_t i = s + lane; i < e; i += 32) {
                double r[NR], t[NZ];
                load(i, r);
                use(i, a.w ? a.w[i] : 1.0, r, x, t);
                if (NZ > 1) {
#pragma unroll
                    for (int q = 0; q < NZ; q++) z[q] += t[q];
                }
            }
            if (NZ > 1) {
#pragma unroll
                for (int q = 0; q < NZ; q++) z[q] = warp_sum(z[q]);
            }
            if (lane == 0) done(g, x, z);
        });
}

// V' W V of the residualised variables: per-CTA partials of its upper triangle,
// row by row
template <int M>
__global__ void __launch_bounds__(kThreads) k_moments(Args a, const double *Gamma, double *part)
{
    constexpr int T = M * (M + 1) / 2;
    __shared__ double s_part[(kThreads / 32) * T];
    double acc[T];
#pragma unroll
    for (int q = 0; q < T; q++) acc[q] = 0.0;
    group_rows<M, M + 1, 1>(
        a, [&](int64_t i, double (&r)[M]) { projected<M>(a, Gamma, i, r); },
        [&](double w, const double (&r)[M], double (&x)[M + 1]) {
            x[M] = w;
#pragma unroll
            for (int j = 0; j < M; j++) x[j] = w * r[j];
        },
        [&](int64_t, double w, const double (&r)[M], const double (&x)[M + 1], double (&)[1]) {
            double v[M];
#pragma unroll
            for (int j = 0; j < M; j++) v[j] = r[j] - (x[M] > 0.0 ? x[j] / x[M] : 0.0);
            int t = 0;
#pragma unroll
            for (int j = 0; j < M; j++)
#pragma unroll
                for (int k = j; k < M; k++, t++) acc[t] += w * v[j] * v[k];
        },
        [](int64_t, const double (&)[M + 1], const double (&)[1]) {});
    cta_sums(acc, T, s_part, part);
}

// The y-equation's residuals and streamed effect, and the sums the plug-in
// moments and the centring of sigma2 need: w, w y, w a, w b, w a^2, w b^2,
// w a b (a = the psi dimension's effect, b = the streamed effect).
template <int M>
__global__ void __launch_bounds__(kThreads) k_effects(Args a, int psi, const double *beta,
                                                      const double *gam_y, double *resid,
                                                      double *alpha, double *part)
{
    __shared__ double s_part[(kThreads / 32) * 7];
    double acc[7] = {0, 0, 0, 0, 0, 0, 0};
    double b[M > 1 ? M - 1 : 1];
#pragma unroll
    for (int j = 0; j + 1 < M; j++) b[j] = beta[j];
    auto mean = [](const double (&x)[2]) { return x[1] > 0.0 ? x[0] / x[1] : 0.0; };
    group_rows<3, 2, 1>(
        a,
        [&](int64_t i, double (&r)[3]) {        // the residual, y, the psi effect
            const double y = a.V[i];
            double u = y, ap = 0.0;
#pragma unroll
            for (int j = 0; j + 1 < M; j++) u -= a.V[(int64_t)(j + 1) * a.N + i] * b[j];
#pragma unroll 2
            for (int d = 0; d < a.D; d++) {
                const double t = gam_y[level(a, i, d)];
                u -= t;
                if (d == psi) ap = t;
            }
            r[0] = u;
            r[1] = y;
            r[2] = ap;
        },
        [&](double w, const double (&r)[3], double (&x)[2]) {
            x[0] = w * r[0];
            x[1] = w;
        },
        [&](int64_t i, double w, const double (&r)[3], const double (&x)[2], double (&)[1]) {
            const double mu = mean(x), ap = r[2];
            if (resid) resid[i] = r[0] - mu;
            acc[0] += w;
            acc[1] += w * r[1];
            acc[2] += w * ap;
            acc[3] += w * mu;
            acc[4] += w * ap * ap;
            acc[5] += w * mu * mu;
            acc[6] += w * ap * mu;
        },
        [&](int64_t g, const double (&x)[2], const double (&)[1]) {
            if (alpha) alpha[g] = mean(x);
        });
    cta_sums(acc, 7, s_part, part);
}

// The row pass of k_variance and k_scores: with h the residualised covariates
// (x less Gamma_x's projection and its weighted group mean) and e the residuals
// (the y equation's, as k_effects), use(i, w, e, h, z) per row and
// done(z) per group with the sums of the rows' z.
template <int M, int NZ, typename Use, typename Done>
__device__ __forceinline__ void residual_rows(const Args &a, const double *Gamma,
                                              const double *beta, Use use, Done done)
{
    constexpr int KX = M - 1;
    double b[KX];
#pragma unroll
    for (int j = 0; j < KX; j++) b[j] = beta[j];
    group_rows<M, M + 1, NZ>(
        a,
        [&](int64_t i, double (&r)[M]) {        // r[0] becomes y - x b
            projected<M>(a, Gamma, i, r);
#pragma unroll
            for (int j = 0; j < KX; j++) r[0] -= b[j] * r[j + 1];
        },
        [&](double w, const double (&r)[M], double (&x)[M + 1]) {
            x[M] = w;
#pragma unroll
            for (int j = 0; j < M; j++) x[j] = w * r[j];
        },
        [&](int64_t i, double w, const double (&r)[M], const double (&x)[M + 1],
            double (&z)[NZ]) {
            const double inv = x[M] > 0.0 ? 1.0 / x[M] : 0.0;
            double h[KX];
#pragma unroll
            for (int j = 0; j < KX; j++) h[j] = r[j + 1] - x[j + 1] * inv;
            use(i, w, r[0] - x[0] * inv, h, z);
        },
        [&](int64_t, const double (&)[M + 1], const double (&z)[NZ]) { done(z); });
}

// The sums of the variances of beta (core/inference.py:566-578, OLS with
// analytic weights), per CTA: the bread sum w h h', the meat sum
// (w e)^2 h h', the streamed groups' meat sum_g s_g s_g' (s_g the group's
// sum of w e h) -- each as its upper triangle, row by row -- and sum w e^2.
template <int M>
__global__ void __launch_bounds__(kThreads) k_variance(Args a, const double *Gamma,
                                                       const double *beta, double *part)
{
    constexpr int KX = M - 1;
    constexpr int T = KX * (KX + 1) / 2;
    constexpr int NQ = 3 * T + 1;
    constexpr int NZ = KX > 1 ? KX : 2;         // (one second sum means none)
    __shared__ double s_part[(kThreads / 32) * NQ];
    double acc[NQ];
#pragma unroll
    for (int q = 0; q < NQ; q++) acc[q] = 0.0;
    residual_rows<M, NZ>(
        a, Gamma, beta,
        [&](int64_t, double w, double e, const double (&h)[KX], double (&z)[NZ]) {
            const double we = w * e;
            int t = 0;
#pragma unroll
            for (int j1 = 0; j1 < KX; j1++)
#pragma unroll
                for (int j2 = j1; j2 < KX; j2++, t++) {
                    acc[t] += w * h[j1] * h[j2];
                    acc[T + t] += we * we * h[j1] * h[j2];
                }
            if (NZ > KX) z[NZ - 1] = 0.0;
#pragma unroll
            for (int j = 0; j < KX; j++) z[j] = we * h[j];
            acc[3 * T] += w * e * e;
        },
        [&](const double (&z)[NZ]) {
            int t = 0;
#pragma unroll
            for (int j1 = 0; j1 < KX; j1++)
#pragma unroll
                for (int j2 = j1; j2 < KX; j2++, t++) acc[2 * T + t] += z[j1] * z[j2];
        });
    cta_sums(acc, NQ, s_part, part);
}

// The per-row scores w e h (out (N, m - 1) row-major) from the same row pass
// as k_variance: core/inference.py:594-603, the rows that pass 2 scatters
// into the clusters of a CRV1 term that is not the streamed dimension.
template <int M>
__global__ void __launch_bounds__(kThreads) k_scores(Args a, const double *Gamma,
                                                     const double *beta, double *out,
                                                     double *h_out)
{
    constexpr int KX = M - 1;
    residual_rows<M, 1>(
        a, Gamma, beta,
        [&](int64_t i, double w, double e, const double (&h)[KX], double (&)[1]) {
            const double we = w * e;
#pragma unroll
            for (int j = 0; j < KX; j++) out[i * KX + j] = we * h[j];
            if (h_out) {
#pragma unroll
                for (int j = 0; j < KX; j++) h_out[i * KX + j] = h[j];
            }
        },
        [](const double (&)[1]) {});
}

// out[q] = sum over CTAs of part[., q], one warp per entry, fixed order; with m
// the entries are the upper triangle of an (m, m) matrix, row by row
__global__ void __launch_bounds__(kThreads) k_sum_parts(const double *part, int blocks, int n,
                                                        double *out, int m = 0)
{
    const int lane = threadIdx.x & 31;
    const int q = (int)(((int64_t)blockIdx.x * kThreads + threadIdx.x) >> 5);
    if (q >= n) return;
    double s = 0.0;
    for (int b = lane; b < blocks; b += 32) s += part[(int64_t)b * n + q];
    s = warp_sum(s);
    if (lane != 0) return;
    if (m == 0) {
        out[q] = s;
        return;
    }
    int j = 0, k = q;
    while (k >= m - j) k -= m - j++;
    out[j * m + j + k] = s;
    out[(j + k) * m + j] = s;
}

// sigma2_i = w_i (y_i - ybar) e_i / M_ii * factor_i (leaveout.py:1000-1003)
__global__ void __launch_bounds__(kThreads) k_sigma2(const double *y, const double *w,
                                                     const double *e, const double *comp,
                                                     const double *factor, double ybar,
                                                     int64_t N, double *out)
{
    for (int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x; i < N;
         i += (int64_t)gridDim.x * kThreads) {
        const double wi = w ? w[i] : 1.0;
        out[i] = wi * (y[i] - ybar) * e[i] / comp[i] * factor[i];
    }
}

int fill(Args &a, const int64_t *starts, int64_t G, const uint32_t *codes, int32_t D,
         const int64_t *n_levels, const double *w, const double *V, int32_t m, int64_t N,
         unsigned *status)
{
    if (D < 1 || D > HDFE_MAX_DIMS || G < 0 || !starts || !codes || !n_levels || !V || m < 1 ||
        m > kMaxM || N < 1)
        return hdfe_set_arg_error("hdfe_resid_moments/row_effects: bad argument (m <= 8)");
    a = Args{};
    a.starts = starts;
    a.G = G;
    a.codes = codes;
    a.D = D;
    int64_t L = 0;
    for (int d = 0; d < D; d++) {
        a.offs[d] = L;
        a.nlev[d] = n_levels[d];
        L += n_levels[d];
    }
    a.w = w;
    a.V = V;
    a.m = m;
    a.N = N;
    a.chunk = window_chunk(G, (int64_t)kGrid * (kThreads / 32));
    a.status = status;
    return HDFE_OK;
}

// a warp per chunk of groups
inline unsigned grid_for(const Args &a)
{
    const int64_t warps = (a.G + a.chunk - 1) / a.chunk;
    int64_t b = (warps + kThreads / 32 - 1) / (kThreads / 32);
    if (b > kGrid) b = kGrid;
    return (unsigned)(b > 0 ? b : 1);
}

}  // namespace assemble
}  // namespace hdfe

using namespace hdfe;

extern "C" int64_t hdfe_assemble_workspace_bytes(int32_t m)
{
    if (m < 1 || m > assemble::kMaxM) return -1;
    return (int64_t)assemble::kGrid * (m * m > 7 ? m * m : 7) * 8;
}

extern "C" int hdfe_resid_moments(const int64_t *starts, int64_t n_groups, const uint32_t *codes,
                                  int32_t D, const int64_t *n_levels, const double *w,
                                  const double *V, int32_t m, int64_t n_rows,
                                  const double *Gamma, double *out, void *workspace,
                                  int64_t workspace_bytes, void *status, void *stream)
{
    assemble::Args a;
    int st = assemble::fill(a, starts, n_groups, codes, D, n_levels, w, V, m, n_rows,
                            (unsigned *)status);
    if (st != HDFE_OK) return st;
    if (!Gamma || !out || !workspace || workspace_bytes < hdfe_assemble_workspace_bytes(m))
        return hdfe_set_arg_error("hdfe_resid_moments: bad argument");
    cudaStream_t s = (cudaStream_t)stream;
    const unsigned grid = assemble::grid_for(a);
    double *part = (double *)workspace;
    switch (m) {
    case 1: assemble::k_moments<1><<<grid, assemble::kThreads, 0, s>>>(a, Gamma, part); break;
    case 2: assemble::k_moments<2><<<grid, assemble::kThreads, 0, s>>>(a, Gamma, part); break;
    case 3: assemble::k_moments<3><<<grid, assemble::kThreads, 0, s>>>(a, Gamma, part); break;
    case 4: assemble::k_moments<4><<<grid, assemble::kThreads, 0, s>>>(a, Gamma, part); break;
    case 5: assemble::k_moments<5><<<grid, assemble::kThreads, 0, s>>>(a, Gamma, part); break;
    case 6: assemble::k_moments<6><<<grid, assemble::kThreads, 0, s>>>(a, Gamma, part); break;
    case 7: assemble::k_moments<7><<<grid, assemble::kThreads, 0, s>>>(a, Gamma, part); break;
    default: assemble::k_moments<8><<<grid, assemble::kThreads, 0, s>>>(a, Gamma, part); break;
    }
    const int nt = m * (m + 1) / 2;
    assemble::k_sum_parts<<<(unsigned)((nt * 32 + assemble::kThreads - 1) / assemble::kThreads),
                            assemble::kThreads, 0, s>>>(part, (int)grid, nt, out, m);
    HDFE_CUDA_TRY(cudaGetLastError());
    hdfe_add_launches(2);
    return HDFE_OK;
}

extern "C" int hdfe_row_effects(const int64_t *starts, int64_t n_groups, const uint32_t *codes,
                                int32_t D, const int64_t *n_levels, int32_t psi_column,
                                const double *w, const double *V, int32_t m, int64_t n_rows,
                                const double *beta, const double *gam_y, double *resid,
                                double *alpha, double *sums, void *workspace,
                                int64_t workspace_bytes, void *status, void *stream)
{
    assemble::Args a;
    int st = assemble::fill(a, starts, n_groups, codes, D, n_levels, w, V, m, n_rows,
                            (unsigned *)status);
    if (st != HDFE_OK) return st;
    if (psi_column < 0 || psi_column >= D || (m > 1 && !beta) || !gam_y || !sums ||
        !workspace || workspace_bytes < hdfe_assemble_workspace_bytes(m))
        return hdfe_set_arg_error("hdfe_row_effects: bad argument");
    cudaStream_t s = (cudaStream_t)stream;
    const unsigned grid = assemble::grid_for(a);
    double *part = (double *)workspace;
#define HDFE_EFFECTS(M) assemble::k_effects<M><<<grid, assemble::kThreads, 0, s>>>( \
        a, psi_column, beta, gam_y, resid, alpha, part)
    switch (m) {
    case 1: HDFE_EFFECTS(1); break;
    case 2: HDFE_EFFECTS(2); break;
    case 3: HDFE_EFFECTS(3); break;
    case 4: HDFE_EFFECTS(4); break;
    case 5: HDFE_EFFECTS(5); break;
    case 6: HDFE_EFFECTS(6); break;
    case 7: HDFE_EFFECTS(7); break;
    default: HDFE_EFFECTS(8); break;
    }
#undef HDFE_EFFECTS
    assemble::k_sum_parts<<<(unsigned)((7 * 32 + assemble::kThreads - 1) / assemble::kThreads),
                            assemble::kThreads, 0, s>>>(part, (int)grid, 7, sums);
    HDFE_CUDA_TRY(cudaGetLastError());
    hdfe_add_launches(2);
    return HDFE_OK;
}

extern "C" int hdfe_kss_sigma2(const double *y, const double *w, const double *resid,
                               const double *complement, const double *factor, double ybar,
                               int64_t n_rows, double *out, void *stream)
{
    if (!y || !resid || !complement || !factor || !out || n_rows < 0)
        return hdfe_set_arg_error("hdfe_kss_sigma2: bad argument");
    if (n_rows == 0) return HDFE_OK;
    int64_t b = (n_rows + assemble::kThreads - 1) / assemble::kThreads;
    if (b > 148 * 16) b = 148 * 16;
    assemble::k_sigma2<<<(unsigned)b, assemble::kThreads, 0, (cudaStream_t)stream>>>(
        y, w, resid, complement, factor, ybar, n_rows, out);
    HDFE_CUDA_TRY(cudaGetLastError());
    hdfe_add_launches(1);
    return HDFE_OK;
}

extern "C" int64_t hdfe_variance_sums_workspace_bytes(int32_t m)
{
    if (m < 2 || m > assemble::kMaxM) return -1;
    const int kx = m - 1, nq = 3 * kx * (kx + 1) / 2 + 1;
    return (int64_t)assemble::kGrid * nq * 8;
}

extern "C" int hdfe_variance_sums(const int64_t *starts, int64_t n_groups, const uint32_t *codes,
                                  int32_t D, const int64_t *n_levels, const double *w,
                                  const double *V, int32_t m, int64_t n_rows,
                                  const double *Gamma, const double *beta, double *out,
                                  void *workspace, int64_t workspace_bytes, void *status,
                                  void *stream)
{
    assemble::Args a;
    int st = assemble::fill(a, starts, n_groups, codes, D, n_levels, w, V, m, n_rows,
                            (unsigned *)status);
    if (st != HDFE_OK) return st;
    if (m < 2 || !Gamma || !beta || !out || !workspace ||
        workspace_bytes < hdfe_variance_sums_workspace_bytes(m))
        return hdfe_set_arg_error("hdfe_variance_sums: bad argument (2 <= m <= 8)");
    cudaStream_t s = (cudaStream_t)stream;
    const unsigned grid = assemble::grid_for(a);
    double *part = (double *)workspace;
    const int kx = m - 1, nq = 3 * kx * (kx + 1) / 2 + 1;
#define HDFE_VARIANCE(M) assemble::k_variance<M><<<grid, assemble::kThreads, 0, s>>>( \
        a, Gamma, beta, part)
    switch (m) {
    case 2: HDFE_VARIANCE(2); break;
    case 3: HDFE_VARIANCE(3); break;
    case 4: HDFE_VARIANCE(4); break;
    case 5: HDFE_VARIANCE(5); break;
    case 6: HDFE_VARIANCE(6); break;
    case 7: HDFE_VARIANCE(7); break;
    default: HDFE_VARIANCE(8); break;
    }
#undef HDFE_VARIANCE
    assemble::k_sum_parts<<<(unsigned)((nq * 32 + assemble::kThreads - 1) / assemble::kThreads),
                            assemble::kThreads, 0, s>>>(part, (int)grid, nq, out);
    HDFE_CUDA_TRY(cudaGetLastError());
    hdfe_add_launches(2);
    return HDFE_OK;
}

extern "C" int hdfe_row_scores(const int64_t *starts, int64_t n_groups, const uint32_t *codes,
                               int32_t D, const int64_t *n_levels, const double *w,
                               const double *V, int32_t m, int64_t n_rows, const double *Gamma,
                               const double *beta, double *out, double *h_out, void *status,
                               void *stream)
{
    assemble::Args a;
    int st = assemble::fill(a, starts, n_groups, codes, D, n_levels, w, V, m, n_rows,
                            (unsigned *)status);
    if (st != HDFE_OK) return st;
    if (m < 2 || !Gamma || !beta || !out)
        return hdfe_set_arg_error("hdfe_row_scores: bad argument (2 <= m <= 8)");
    cudaStream_t s = (cudaStream_t)stream;
    const unsigned grid = assemble::grid_for(a);
#define HDFE_SCORES(M) assemble::k_scores<M><<<grid, assemble::kThreads, 0, s>>>(a, Gamma, beta, out, \
                                                                                h_out)
    switch (m) {
    case 2: HDFE_SCORES(2); break;
    case 3: HDFE_SCORES(3); break;
    case 4: HDFE_SCORES(4); break;
    case 5: HDFE_SCORES(5); break;
    case 6: HDFE_SCORES(6); break;
    case 7: HDFE_SCORES(7); break;
    default: HDFE_SCORES(8); break;
    }
#undef HDFE_SCORES
    HDFE_CUDA_TRY(cudaGetLastError());
    hdfe_add_launches(1);
    return HDFE_OK;
}
