// Connected components of the levels of one non-streamed dimension (levels
// sharing an identifying group are connected), and the normalisation of the
// solved fixed effects.
//
// Components: core/kernels_base.py:156-174 `_nb_components`.  The device
// union-find links the larger root under the smaller with atomicCAS, so every
// component's root is its smallest level, whatever the order the unions run
// in -- the reference's root, exactly (its serial union-find also links
// toward the smaller index).  Ranking the roots into labels by rows
// (core/passes.py:933-950) is bookkeeping done by the caller.
//
// Unions alone are latency-bound: every thread walks parent chains that the
// others are still building and retries on the roots that all of them want
// (243 us for the 300k unions of a 400k-worker panel, 281 us on the 5M-worker
// one; a year dimension's ten roots see three million unions).  So the trees
// are first grown by rounds without walks or retries -- every pair hooks the
// larger of its two roots under the smaller by one atomicMin, then all trees
// are flattened -- over a sample of the groups, enough for the giant component
// to close (three rounds; a sample of one window in four still leaves a firm
// about four neighbours); the last pass unites what is left, and nearly every
// pair finds one common root with two loads.  One cooperative launch does all
// of it, grid barriers between the phases.
// Normalisation: core/solve.py:383-399 `_normalize`.  The first dimension's
// effects get obs-weighted mean zero within each component, every further
// dimension obs-weighted mean zero overall.  Within-component sums are
// carried along each thread's walk and combined per warp (lanes with the same
// root) before one atomic per root: the giant component of 500k levels sees
// about a thousand atomics a column.
#include <atomic>

#include <cuda_runtime.h>

#include "unionfind.cuh"

namespace hdfe {
namespace graph {

constexpr int kThreads = 256;
struct CompArgs {
    const int64_t *starts;
    int64_t G;
    const uint32_t *codes;
    int D, col;
    int64_t nlev;
    int32_t *parent;
    unsigned *status;
    unsigned long long *n_roots;
    GridBarrier bar;
    int sample;             // the rounds take every sample-th window
    // rows of two dimensions instead (walk_rows): G rows, vertices code[col] and
    // n_first + code[col2]
    int col2;
    int64_t n_first;
};

constexpr int kCompThreads = 512;
constexpr int kRounds = 3;

// The levels (dimension col) of each group joined into one component: a
// warp takes a window of 32 groups, reads their cells coalesced (one per lane,
// 32 at a time, the next 32 in flight) and calls join(prev, c) for each cell's
// level and the previous cell's of the same group where they differ -- a chain
// over the group, which connects what the reference's star over the group's
// first level connects (every root is the component's smallest level either
// way).
template <typename F>
__device__ __forceinline__ void walk_groups(const CompArgs &a, int sample, F join)
{
    const int lane = threadIdx.x & 31;
    const int64_t wid = ((int64_t)blockIdx.x * kCompThreads + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * kCompThreads) >> 5;
    for (int64_t g0 = wid * 32 * sample; g0 < a.G; g0 += nw * 32 * sample) {
        const int ng = (int)min((int64_t)32, a.G - g0);
        const int64_t gend = a.starts[g0 + ng];
        const int64_t st = lane < ng ? a.starts[g0 + lane] : gend;   // this lane's group start
        int64_t base = __shfl_sync(0xffffffffu, st, 0);
        uint32_t next = base + lane < gend ? a.codes[(base + lane) * a.D + a.col] : 0u;
        uint32_t last = 0;                  // the code before the chunk
        for (; base < gend; base += 32) {
            const uint32_t c = next;
            const int64_t i = base + lane;
            if (i + 32 < gend) next = a.codes[(i + 32) * a.D + a.col];
            const bool in = lane < ng && st >= base && st < base + 32;
            const unsigned heads = __reduce_or_sync(0xffffffffu, in ? 1u << (int)(st - base) : 0u);
            const bool valid = i < gend;
            uint32_t prev = __shfl_up_sync(0xffffffffu, c, 1);
            if (lane == 0) prev = last;     // a window begins with a head
            last = __shfl_sync(0xffffffffu, c, 31);
            const bool head = (heads >> lane) & 1u;
            if (valid && (int64_t)c >= a.nlev) atomicCAS(a.status, 0u, (unsigned)HDFE_ERR_BAD_CODE);
            if (!valid || head || c == prev || (int64_t)c >= a.nlev || (int64_t)prev >= a.nlev)
                continue;
            join((int32_t)prev, (int32_t)c);
        }
    }
}

// The two levels of each row (dimensions col and col2) joined, the second
// dimension's vertices after the first's: join(x, y), rows 32 to a warp.
template <typename F>
__device__ __forceinline__ void walk_rows(const CompArgs &a, int sample, F join)
{
    const int lane = threadIdx.x & 31;
    const int64_t wid = ((int64_t)blockIdx.x * kCompThreads + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * kCompThreads) >> 5;
    const int64_t n2 = a.nlev - a.n_first;
#pragma unroll 4
    for (int64_t i = wid * 32 * sample + lane; i < a.G; i += nw * 32 * sample) {
        const int64_t x = a.codes[i * a.D + a.col], y = a.codes[i * a.D + a.col2];
        if (x >= a.n_first || y >= n2) atomicCAS(a.status, 0u, (unsigned)HDFE_ERR_BAD_CODE);
        else join((int32_t)x, (int32_t)(a.n_first + y));
    }
}

// ROWS: vertices joined by rows (walk_rows), else by groups (walk_groups)
template <bool ROWS>
__global__ void __launch_bounds__(kCompThreads, 2) k_components(CompArgs a)
{
    auto walk = [](const CompArgs &c, int sample, auto join) {
        if constexpr (ROWS) walk_rows(c, sample, join);
        else walk_groups(c, sample, join);
    };
    const int64_t t0 = (int64_t)blockIdx.x * kCompThreads + threadIdx.x;
    const int64_t step = (int64_t)gridDim.x * kCompThreads;
    int32_t *parent = a.parent;
    if (t0 == 0) *a.n_roots = 0;
    for (int64_t i = t0; i < a.nlev; i += step) parent[i] = (int32_t)i;
    if (!a.bar.sync()) return;
    for (int r = 0; r < kRounds; r++) {
        walk(a, a.sample, [&](int32_t x, int32_t y) {
            const int32_t px = parent[x], py = parent[y];
            if (px != py) hook(parent, px, py);
        });
        if (!a.bar.sync()) return;
        for (int64_t i = t0; i < a.nlev; i += step) parent[i] = root_of(parent, (int32_t)i);
        if (!a.bar.sync()) return;
    }
    walk(a, 1, [&](int32_t x, int32_t y) {
        if (parent[x] != parent[y]) unite(parent, x, y, a.status);
    });
    if (!a.bar.sync()) return;
    unsigned long long roots = 0;
    for (int64_t i = t0; i < a.nlev; i += step) {
        const int32_t r = root_of(parent, (int32_t)i);
        parent[i] = r;
        roots += (r == (int32_t)i);
    }
    roots = warp_sum(roots);
    if ((threadIdx.x & 31) == 0 && roots) atomicAdd(a.n_roots, roots);
}

// ------------------------------------------------------------ nesting

// Whether every level lies within one cluster: each level keeps the first
// cluster seen, and a row of another one ends the question for the dimension
// (*loose).  The reference compares every level's least and greatest cluster;
// as two scatter reductions that was 1.9 ms each for ten year levels, whose
// addresses see 3.4M atomics, while most dimensions are loose within their
// first few rows.
__global__ void __launch_bounds__(kThreads) k_first_cluster(const int64_t *clusters, int64_t N,
                                                            const uint32_t *codes, int stride,
                                                            int64_t n_levels,
                                                            unsigned long long *first,
                                                            int32_t *loose)
{
    const int lane = threadIdx.x & 31;
    for (int64_t base = (int64_t)blockIdx.x * kThreads + (threadIdx.x & ~31); base < N;
         base += (int64_t)gridDim.x * kThreads) {
        if (__any_sync(0xffffffffu, *(volatile int32_t *)loose)) return;
        const int64_t i = base + lane;
        const int64_t l = i < N ? (int64_t)codes[i * stride] : -1;
        const bool valid = l >= 0 && l < n_levels;
        const unsigned long long c = valid ? (unsigned long long)clusters[i] : 0ull;
        // a lane per level and warp meets the others' clusters and the table
        const int leader = __ffs(__match_any_sync(0xffffffffu, l)) - 1;
        bool differ = c != __shfl_sync(0xffffffffu, c, leader);
        if (valid && lane == leader) {
            unsigned long long v = *(volatile unsigned long long *)(first + l);
            if (v == ~0ull) {
                v = atomicCAS(first + l, ~0ull, c);
                if (v == ~0ull) v = c;
            }
            differ = v != c;
        }
        if (differ && valid) *(volatile int32_t *)loose = 1;
    }
}

// a level without rows is in no cluster
__global__ void __launch_bounds__(kThreads) k_unseen(const int64_t *first, int64_t n_levels,
                                                     int32_t *loose)
{
    if (*(volatile int32_t *)loose) return;
    for (int64_t l = (int64_t)blockIdx.x * kThreads + threadIdx.x; l < n_levels;
         l += (int64_t)gridDim.x * kThreads)
        if (first[l] < 0) *(volatile int32_t *)loose = 1;
}

// ------------------------------------------------------------ normalise

// Sums per root: column j of the grid's second dimension, cw[root] += w (j 0)
// or cs[root, j - 1] += w * Gamma[l, j - 1].
__global__ void __launch_bounds__(kThreads) k_comp_sums(const int32_t *root, const double *w,
                                                        const double *gamma, int64_t nl, int m,
                                                        double *cw, double *cs)
{
    const int j = (int)blockIdx.y - 1;
    auto add = [&](int32_t r, double v) {
        atomicAdd(j < 0 ? cw + r : cs + (int64_t)r * m + j, v);
    };
    int32_t at = -1;                // the root of the carried sum
    double sum = 0.0;
    for (int64_t l = (int64_t)blockIdx.x * kThreads + threadIdx.x; l < nl;
         l += (int64_t)gridDim.x * kThreads) {
        const int32_t r = root[l];
        if (r != at) {
            if (at >= 0) add(at, sum);
            at = r;
            sum = 0.0;
        }
        sum += j < 0 ? w[l] : w[l] * gamma[l * m + j];
    }
    // the peers' sums added in lane order
    const unsigned peers = __match_any_sync(0xffffffffu, at);
    double total = 0.0;
    for (int q = 0; q < 32; q++) {
        const double v = __shfl_sync(0xffffffffu, sum, q);
        if ((peers >> q) & 1u) total += v;
    }
    if (at >= 0 && (int)(threadIdx.x & 31) == __ffs(peers) - 1) add(at, total);
}

__global__ void __launch_bounds__(kThreads) k_comp_apply(const int32_t *root, const double *cw,
                                                         const double *cs, int64_t nl, int m,
                                                         double *gamma)
{
    for (int64_t l = (int64_t)blockIdx.x * kThreads + threadIdx.x; l < nl;
         l += (int64_t)gridDim.x * kThreads) {
        const int32_t r = root[l];
        double c = cw[r];
        if (c == 0.0) c = 1.0;
        for (int j = 0; j < m; j++) gamma[l * m + j] -= cs[(int64_t)r * m + j] / c;
    }
}

// per-CTA partial sums of w and w * Gamma over one dimension's block
__global__ void __launch_bounds__(kThreads) k_dim_sums(const double *w, const double *gamma,
                                                       int64_t nl, int m, double *part)
{
    __shared__ double s_red[kThreads / 32];
    double sw = 0.0;
    for (int64_t l = (int64_t)blockIdx.x * kThreads + threadIdx.x; l < nl;
         l += (int64_t)gridDim.x * kThreads)
        sw += w[l];
    sw = block_sum(sw, s_red);
    if (threadIdx.x == 0) part[blockIdx.x * (1 + m)] = sw;
    for (int j = 0; j < m; j++) {
        double s = 0.0;
        for (int64_t l = (int64_t)blockIdx.x * kThreads + threadIdx.x; l < nl;
             l += (int64_t)gridDim.x * kThreads)
            s += w[l] * gamma[l * m + j];
        s = block_sum(s, s_red);
        if (threadIdx.x == 0) part[blockIdx.x * (1 + m) + 1 + j] = s;
    }
}

__global__ void __launch_bounds__(kThreads) k_dim_apply(const double *part, int nparts,
                                                        double *gamma, int64_t nl, int m)
{
    __shared__ double s_mean[HDFE_MAX_VARS];
    if (threadIdx.x < 32) {
        double sw = 0.0;
        for (int b = 0; b < nparts; b++) sw += part[b * (1 + m)];
        const double den = fmax(sw, 1.0);
        for (int j = (int)threadIdx.x; j < m; j += 32) {
            double s = 0.0;
            for (int b = 0; b < nparts; b++) s += part[b * (1 + m) + 1 + j];
            s_mean[j] = s / den;
        }
    }
    __syncthreads();
    for (int64_t l = (int64_t)blockIdx.x * kThreads + threadIdx.x; l < nl;
         l += (int64_t)gridDim.x * kThreads)
        for (int j = 0; j < m; j++) gamma[l * m + j] -= s_mean[j];
}

// ------------------------------------------------------------ solve set-up

// What step 2 does before its PCG, in two launches instead of ten array
// operations and a host read: dinv = 1 / diag (0 up to 1e-12, core/solve.py:
// 142-146), and per right-hand side the sum of squares, a CTA's columns in
// part[column * CTAs + CTA].
constexpr int kSetupCtas = 148;

__global__ void __launch_bounds__(kThreads) k_setup(const double *diag, const double *rhs,
                                                    int64_t L, int m, double *dinv, double *part)
{
    __shared__ double s_red[kThreads / 32];
    const int64_t t0 = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    const int64_t step = (int64_t)gridDim.x * kThreads;
    for (int64_t l = t0; l < L; l += step) {
        const double d = diag[l];
        dinv[l] = d > 1e-12 ? 1.0 / d : 0.0;
    }
    for (int j = 0; j < m; j++) {
        double s = 0.0;
        for (int64_t l = t0; l < L; l += step) {
            const double v = rhs[l * m + j];
            s += v * v;
        }
        s = block_sum(s, s_red);
        if (threadIdx.x == 0) part[j * gridDim.x + blockIdx.x] = s;
    }
}

// zero[j] = ||rhs_j|| <= tol sqrt(max(raw_ss_j, 0)) (core/solve.py:294-320), a
// warp per column, the CTAs in a fixed order
__global__ void __launch_bounds__(kThreads) k_zero_columns(const double *part, int ctas, int m,
                                                           const double *raw_ss, double tol,
                                                           uint8_t *zero)
{
    const int lane = threadIdx.x & 31;
    for (int j = threadIdx.x >> 5; j < m; j += kThreads / 32) {
        double s = 0.0;
        for (int b = lane; b < ctas; b += 32) s += part[j * ctas + b];
        s = warp_sum(s);
        const double ss = raw_ss[j] < 0.0 ? 0.0 : raw_ss[j];
        if (lane == 0) zero[j] = sqrt(s) <= tol * sqrt(ss) ? 1 : 0;
    }
}

// From this many windows of 32 groups the rounds take one in four: below, a
// window a warp is one wave and sampling saves nothing.
constexpr int64_t kSampleFrom = 16384;

// CTAs of k_components that the current device holds at once (0: an error)
template <bool ROWS>
int64_t resident_ctas()
{
    static std::atomic<int> known[64];
    int dev = 0, per = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (dev >= 0 && dev < 64 && (per = known[dev].load()) > 0) return per;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_components<ROWS>, kCompThreads, 0) !=
            cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 0;
    per *= sms;
    if (dev >= 0 && dev < 64) known[dev].store(per);
    return per;
}

inline unsigned grid_for(int64_t n)
{
    int64_t b = (n + kThreads - 1) / kThreads;
    if (b > 4096) b = 4096;
    return (unsigned)(b > 0 ? b : 1);
}

template <bool ROWS>
int launch_components(CompArgs &a, int64_t *n_components, void *workspace, cudaStream_t s)
{
    // the barrier's three words; its error word is the status, a bad code's too
    a.status = (unsigned *)workspace + 2;
    a.n_roots = (unsigned long long *)n_components;
    a.bar = GridBarrier{(unsigned *)workspace};
    HDFE_CUDA_TRY(cudaMemsetAsync(workspace, 0, 16, s));
    const int64_t windows = (a.G + 31) / 32;
    a.sample = windows >= kSampleFrom ? 4 : 1;
    const int64_t most = resident_ctas<ROWS>();
    if (most < 1) return hdfe_set_cuda_error(cudaGetLastError());
    // a warp per window and eight levels a thread fill the grid of small panels,
    // whose barriers then wait for fewer CTAs
    int64_t need = (windows * 32 + kCompThreads - 1) / kCompThreads;
    const int64_t by_level = (a.nlev + 8 * kCompThreads - 1) / (8 * kCompThreads);
    if (need < by_level) need = by_level;
    if (need < 1) need = 1;
    void *args[] = {&a};
    HDFE_CUDA_TRY(cudaLaunchCooperativeKernel((const void *)k_components<ROWS>,
                                              dim3((unsigned)(need < most ? need : most)),
                                              dim3(kCompThreads), args, 0, s));
    HDFE_CUDA_TRY(cudaGetLastError());
    hdfe_add_launches(1);
    // n_components[1] = the status and the zero word after it
    HDFE_CUDA_TRY(cudaMemcpyAsync(n_components + 1, a.status, 8, cudaMemcpyDeviceToDevice, s));
    return HDFE_OK;
}

}  // namespace graph
}  // namespace hdfe

using namespace hdfe;

extern "C" int64_t hdfe_components_workspace_bytes(void) { return 256; }

extern "C" int hdfe_components(const int64_t *starts, int64_t n_groups, const uint32_t *codes,
                               int32_t D, int32_t col, int64_t n_levels, int32_t *root,
                               int64_t *n_components, void *workspace, int64_t workspace_bytes,
                               void *stream)
{
    if (D < 1 || D > HDFE_MAX_DIMS || col < 0 || col >= D || n_levels < 1 ||
        n_levels >= INT32_MAX || n_groups < 0 || !starts || (n_groups > 0 && !codes) || !root ||
        !n_components || !workspace || workspace_bytes < 256)
        return hdfe_set_arg_error("hdfe_components: bad argument");
    graph::CompArgs a{};
    a.starts = starts;
    a.G = n_groups;
    a.codes = codes;
    a.D = D;
    a.col = col;
    a.nlev = n_levels;
    a.parent = root;
    return graph::launch_components<false>(a, n_components, workspace, (cudaStream_t)stream);
}

extern "C" int hdfe_code_components(const uint32_t *codes, int64_t n_rows, int32_t D,
                                    int32_t col1, int32_t col2, int64_t n1, int64_t n2,
                                    int32_t *root, int64_t *n_components, void *workspace,
                                    int64_t workspace_bytes, void *stream)
{
    if (D < 2 || D > HDFE_MAX_DIMS || col1 < 0 || col1 >= D || col2 < 0 || col2 >= D ||
        n1 < 1 || n2 < 1 || n1 + n2 >= INT32_MAX || n_rows < 0 || (n_rows > 0 && !codes) ||
        !root || !n_components || !workspace || workspace_bytes < 256)
        return hdfe_set_arg_error("hdfe_code_components: bad argument");
    graph::CompArgs a{};
    a.G = n_rows;
    a.codes = codes;
    a.D = D;
    a.col = col1;
    a.col2 = col2;
    a.nlev = n1 + n2;
    a.n_first = n1;
    a.parent = root;
    return graph::launch_components<true>(a, n_components, workspace, (cudaStream_t)stream);
}

extern "C" int hdfe_levels_nested(const int64_t *clusters, int64_t n_rows, const uint32_t *codes,
                                  int32_t stride, int64_t n_levels, int64_t *first, int32_t *loose,
                                  void *stream)
{
    if (n_rows < 0 || stride < 1 || n_levels < 1 || !first || !loose ||
        (n_rows > 0 && (!clusters || !codes)))
        return hdfe_set_arg_error("hdfe_levels_nested: bad argument");
    cudaStream_t s = (cudaStream_t)stream;
    HDFE_CUDA_TRY(cudaMemsetAsync(first, 0xff, n_levels * 8, s));
    HDFE_CUDA_TRY(cudaMemsetAsync(loose, 0, 4, s));
    const unsigned grid = graph::grid_for(n_rows) < 148 * 4 ? graph::grid_for(n_rows) : 148 * 4;
    unsigned long long *seen = reinterpret_cast<unsigned long long *>(first);
    // the first thousand rows by one CTA: they settle most questions, and put a
    // small dimension's levels in place before the whole grid would contend for
    // them (216 us otherwise for ten levels)
    graph::k_first_cluster<<<1, graph::kThreads, 0, s>>>(
        clusters, n_rows < 1024 ? n_rows : 1024, codes, stride, n_levels, seen, loose);
    graph::k_first_cluster<<<grid, graph::kThreads, 0, s>>>(clusters, n_rows, codes, stride,
                                                            n_levels, seen, loose);
    graph::k_unseen<<<graph::grid_for(n_levels), graph::kThreads, 0, s>>>(first, n_levels, loose);
    HDFE_CUDA_TRY(cudaGetLastError());
    hdfe_add_launches(3);
    return HDFE_OK;
}

extern "C" int64_t hdfe_solve_setup_workspace_bytes(int32_t m)
{
    if (m < 1) return -1;
    return (int64_t)graph::kSetupCtas * m * 8;
}

extern "C" int hdfe_solve_setup(const double *diag, const double *rhs, int64_t L, int32_t m,
                                const double *raw_ss, double tol, double *dinv, uint8_t *zero,
                                void *workspace, int64_t workspace_bytes, void *stream)
{
    if (!diag || !rhs || L < 1 || m < 1 || !raw_ss || !dinv || !zero ||
        !workspace)
        return hdfe_set_arg_error("hdfe_solve_setup: bad argument");
    if (workspace_bytes < hdfe_solve_setup_workspace_bytes(m))
        return hdfe_set_error(HDFE_ERR_WORKSPACE, "hdfe_solve_setup: workspace too small");
    cudaStream_t s = (cudaStream_t)stream;
    double *part = (double *)workspace;
    const unsigned g = graph::grid_for(L);
    const int ctas = g < graph::kSetupCtas ? (int)g : graph::kSetupCtas;
    graph::k_setup<<<ctas, graph::kThreads, 0, s>>>(diag, rhs, L, m, dinv, part);
    graph::k_zero_columns<<<1, graph::kThreads, 0, s>>>(part, ctas, m, raw_ss, tol, zero);
    HDFE_CUDA_TRY(cudaGetLastError());
    hdfe_add_launches(2);
    return HDFE_OK;
}

extern "C" int64_t hdfe_normalize_workspace_bytes(int64_t n_first, int32_t m)
{
    if (n_first < 0 || m < 1 || m > HDFE_MAX_VARS) return -1;
    return (n_first * (1 + (int64_t)m) + 4096 * (1 + (int64_t)m)) * 8 + 256;
}

extern "C" int hdfe_normalize(double *gamma, int32_t m, int32_t D, const int64_t *n_levels,
                              const double *obs, const int32_t *root, void *workspace,
                              int64_t workspace_bytes, void *stream)
{
    if (!gamma || m < 1 || m > HDFE_MAX_VARS || D < 1 || D > HDFE_MAX_DIMS || !n_levels ||
        !obs || !root || !workspace)
        return hdfe_set_arg_error("hdfe_normalize: bad argument");
    const int64_t n0 = n_levels[0];
    if (workspace_bytes < hdfe_normalize_workspace_bytes(n0, m))
        return hdfe_set_error(HDFE_ERR_WORKSPACE, "hdfe_normalize: workspace too small");
    cudaStream_t s = (cudaStream_t)stream;
    double *cw = (double *)workspace;
    double *cs = cw + n0;
    double *part = cs + n0 * m;
    HDFE_CUDA_TRY(cudaMemsetAsync(cw, 0, n0 * (1 + (int64_t)m) * 8, s));
    const unsigned nc = graph::grid_for(n0) < 148 ? graph::grid_for(n0) : 148;
    graph::k_comp_sums<<<dim3(nc, 1 + m), graph::kThreads, 0, s>>>(root, obs, gamma, n0, m, cw,
                                                                   cs);
    graph::k_comp_apply<<<graph::grid_for(n0), graph::kThreads, 0, s>>>(root, cw, cs, n0, m,
                                                                        gamma);
    int64_t off = n0;
    for (int d = 1; d < D; d++) {
        const int64_t nl = n_levels[d];
        const unsigned nb = graph::grid_for(nl) < 1024 ? graph::grid_for(nl) : 1024;
        graph::k_dim_sums<<<nb, graph::kThreads, 0, s>>>(obs + off, gamma + off * m, nl, m, part);
        graph::k_dim_apply<<<graph::grid_for(nl), graph::kThreads, 0, s>>>(part, (int)nb,
                                                                           gamma + off * m, nl, m);
        off += nl;
    }
    HDFE_CUDA_TRY(cudaGetLastError());
    hdfe_add_launches(2 + 2 * (D - 1));
    return HDFE_OK;
}
