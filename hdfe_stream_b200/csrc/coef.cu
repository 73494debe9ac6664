// Coefficient-space passes of the inverse operator, and the trace moments.
//
// Reference: inverse.py:311-374 `apply_inverse` with kernels_inverse.py:
// 112-130 `_nb_reduce_rows`, :134-152 `_nb_spread_groups`, :157-188
// `_nb_project_coef`; the Hutchinson trace's collect sink (leaveout.py:
// 423-431, with core/kernels_groups.py:17-27 `_nb_group_sums`) and
// kernels_inverse.py:192-231 `_nb_trace_moments`; the coefficient-space
// Rademacher vectors of `_trace_block` (core/kernels_groups.py:53-76).
//
//   reduce        acc[level, j] += w_i R_ij over the rows (no centring), where
//                 R is either explicit rows or the streamed block spread over
//                 its group (R_ij = streamed[g, j] / s_g, s_g = the group's
//                 weight); acc_x[c, j] += X_ic w_i R_ij; optionally the group
//                 sums of w_i R_ij.
//   project_coef  h_ij = sum_d U[level_d(i), j] + X_i . C[:, j]; u0[g, j] =
//                 weighted group mean of (rho - h); rows (A u)_ij = h + u0 and
//                 the groups' u0; optionally the collect sink in the same pass:
//                 v = w_i omega_i (A u)_ij reduced like `reduce`.
//   trace         per vector j the eight weighted sums of the psi-dimension
//                 values (a) and streamed values (b) of Z and U over rows, per
//                 CTA in a fixed order and then over CTAs in a fixed order.
//
// Blocks of vectors (more than four) take windows of up to 32 rows made of
// whole groups, a sub-warp of Bp lanes (the width rounded up to 8, 16 or 32),
// lane j vector j.  Within a run of rows with equal codes the values h differ
// by the covariates only, so everything but the rows' own output is linear in
// sums over the run that no vector enters: w, w omega and w omega X.  Those
// are made once a window by lane (run, sum), and a vector's work is per run
// (1.75 a worker rather than 8.5 rows): one gather of U's row, the window's
// first eight in flight, and a few FMAs.  The covariates' own block X' omega X
// C of the sink is per pass: each lane sums omega X X' over the rows it staged.
// 1M-worker panel, 32 vectors, 2 covariates: reduce 1.34 -> 0.45 ms,
// project_coef with the sink 3.23 -> 1.58 ms.
//
// Narrow blocks (one to four vectors, the adjoint's) have too few lanes for
// that: there a thread (or 2, 4) takes a group and walks its rows, 32 (16, 8)
// groups a warp.  Dimensions with few levels (the years) are added into a
// CTA's own copy in shared memory: ten addresses otherwise see every row's
// atomic (3.4M rows, one vector: reduce 2.37 -> 0.09 ms, project_coef
// 1.22 -> 0.13 ms).
#include <cuda_runtime.h>

#include "common.cuh"
#include "windows.cuh"

namespace hdfe {
namespace coef {

constexpr int kThreads = 128;
constexpr int kMaxCov = 8;
constexpr int kMaxGrid = 148 * 16;

struct Args {
    const int64_t *starts;
    int64_t G;
    const uint32_t *codes;
    int D;
    int64_t offs[HDFE_MAX_DIMS];
    int64_t nlev[HDFE_MAX_DIMS];
    int64_t L;
    const double *w;            // (N) or null (ones)
    const double *X;            // (N, c) or null
    int c;
    int B, Bp;
    const double *streamed;     // (G, B): spread over the rows, or null
    const double *R;            // (N, B) explicit rows (reduce), or null
    const double *U, *C;        // (L, B), (c, B)
    const double *omega;        // (N) or null: the collect sink's row weights (ones)
    bool collect;               // project_coef: run the collect sink
    double *rows;               // (N, B) or null
    double *groups;             // (G, B) or null
    double *acc, *acc_x;        // (L, B), (c, B): added into
    double *gsum;               // (G, B) or null
    unsigned *status;
    int64_t chunk;              // groups a sub-warp takes at a time (windows)
    // narrow passes: dimensions summed in shared memory first
    int small[HDFE_MAX_DIMS];
    int64_t soff[HDFE_MAX_DIMS];
    int64_t n_small;
};

template <int BP>
struct Lanes {
    int lane, j;
    unsigned mask;
    bool on;
    __device__ Lanes(int B)
    {
        lane = threadIdx.x & 31;
        j = lane % BP;
        const int sub = lane / BP;
        mask = BP == 32 ? 0xffffffffu : (((1u << BP) - 1u) << (sub * BP));
        on = j < B;
    }
};

// row i's codes, checked (an out-of-range code is reported and read as 0)
__device__ __forceinline__ void row_codes(const Args &a, int64_t i, uint32_t (&c)[HDFE_MAX_DIMS])
{
#pragma unroll
    for (int d = 0; d < HDFE_MAX_DIMS; d++) {
        if (d >= a.D) break;
        uint32_t v = __ldg(a.codes + i * a.D + d);
        if ((int64_t)v >= a.nlev[d]) {
            if (a.status) atomicCAS(a.status, 0u, (unsigned)HDFE_ERR_BAD_CODE);
            v = 0;
        }
        c[d] = v;
    }
}

__device__ __forceinline__ bool same(const Args &a, const uint32_t (&x)[HDFE_MAX_DIMS],
                                     const uint32_t (&y)[HDFE_MAX_DIMS])
{
    bool s = true;
#pragma unroll
    for (int d = 0; d < HDFE_MAX_DIMS; d++) {
        if (d >= a.D) break;
        s &= x[d] == y[d];
    }
    return s;
}

__device__ __forceinline__ double group_weight(const Args &a, int64_t s, int64_t e)
{
    double sw = 0.0;
    for (int64_t i = s; i < e; i++) sw += a.w ? __ldg(a.w + i) : 1.0;
    return sw;
}

// the run sums: v of consecutive rows with equal codes, added once per run
struct Runs {
    uint32_t codes[HDFE_MAX_DIMS];
    double v;
    bool have;
};

__device__ __forceinline__ void run_flush(const Args &a, const Runs &run, int j, double *s_acc)
{
#pragma unroll
    for (int d = 0; d < HDFE_MAX_DIMS; d++) {
        if (d >= a.D) break;
        if (a.small[d]) atomicAdd(s_acc + (a.soff[d] + run.codes[d]) * a.B + j, run.v);
        else atomicAdd(a.acc + (a.offs[d] + run.codes[d]) * a.B + j, run.v);
    }
}

// the shared sums of the small dimensions: cleared, and added to acc at the end
__device__ __forceinline__ void small_clear(const Args &a, double *s_acc)
{
    for (int64_t k = threadIdx.x; k < a.n_small * a.B; k += kThreads) s_acc[k] = 0.0;
    __syncthreads();
}

__device__ __forceinline__ void small_flush(const Args &a, const double *s_acc)
{
    if (a.n_small == 0) return;
    __syncthreads();
    for (int d = 0; d < a.D; d++) {
        if (!a.small[d]) continue;
        for (int64_t q = threadIdx.x; q < a.nlev[d] * a.B; q += kThreads) {
            const double v = s_acc[a.soff[d] * a.B + q];
            if (v != 0.0) atomicAdd(a.acc + a.offs[d] * a.B + q, v);
        }
    }
}

__device__ __forceinline__ void run_add(const Args &a, Runs &run, const uint32_t (&c)[HDFE_MAX_DIMS],
                                        double v, int j, bool on, double *s_acc)
{
    if (run.have && !same(a, run.codes, c)) {
        if (on) run_flush(a, run, j, s_acc);
        run.v = 0.0;
    }
#pragma unroll
    for (int d = 0; d < HDFE_MAX_DIMS; d++) {
        if (d >= a.D) break;
        run.codes[d] = c[d];
    }
    run.have = true;
    run.v += v;
}

// the covariate block: per lane of equal j in the warp, then per CTA, then one
// add per entry
template <int BP>
__device__ __forceinline__ void flush_cov(const Args &a, const double (&ax)[kMaxCov], double *s_ax,
                                          int j, bool on)
{
    for (int k = threadIdx.x; k < a.c * a.B; k += kThreads) s_ax[k] = 0.0;
    __syncthreads();
#pragma unroll
    for (int c = 0; c < kMaxCov; c++) {
        if (c >= a.c) break;
        double v = ax[c];
#pragma unroll
        for (int o = 16; o >= BP; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (on && (threadIdx.x & 31) < BP) atomicAdd(s_ax + c * a.B + j, v);
    }
    __syncthreads();
    for (int k = threadIdx.x; k < a.c * a.B; k += kThreads)
        if (s_ax[k] != 0.0) atomicAdd(a.acc_x + k, s_ax[k]);
}

template <int BP>
__global__ void __launch_bounds__(kThreads) k_reduce(Args a)
{
    constexpr int SUBS = kThreads / BP;
    extern __shared__ __align__(16) double s_acc[];
    __shared__ double s_ax[kMaxCov * 32];
    const Lanes<BP> ln(a.B);
    small_clear(a, s_acc);
    const int64_t g0 = (int64_t)blockIdx.x * SUBS + threadIdx.x / BP;
    const int64_t gstep = (int64_t)gridDim.x * SUBS;
    double ax[kMaxCov];
#pragma unroll
    for (int c = 0; c < kMaxCov; c++) ax[c] = 0.0;
    for (int64_t g = g0; g < a.G; g += gstep) {
        const int64_t s = a.starts[g], e = a.starts[g + 1];
        double rho = 0.0;
        if (a.streamed) {
            const double sw = group_weight(a, s, e);
            rho = (ln.on && sw > 0.0) ? a.streamed[g * a.B + ln.j] / sw : 0.0;
        }
        Runs run{};
        double gs = 0.0;
        for (int64_t i = s; i < e; i++) {
            uint32_t c[HDFE_MAX_DIMS];
            row_codes(a, i, c);
            const double wi = a.w ? __ldg(a.w + i) : 1.0;
            const double r = a.streamed ? rho : (ln.on ? a.R[i * a.B + ln.j] : 0.0);
            const double v = wi * r;
            run_add(a, run, c, v, ln.j, ln.on, s_acc);
            gs += v;
#pragma unroll
            for (int cc = 0; cc < kMaxCov; cc++) {
                if (cc >= a.c) break;
                ax[cc] += __ldg(a.X + i * a.c + cc) * v;
            }
        }
        if (run.have && ln.on) run_flush(a, run, ln.j, s_acc);
        if (a.gsum && ln.on) a.gsum[g * a.B + ln.j] = gs;
    }
    small_flush(a, s_acc);
    if (a.acc_x && a.c > 0) flush_cov<BP>(a, ax, s_ax, ln.j, ln.on);
}

template <int BP>
__global__ void __launch_bounds__(kThreads) k_project_coef(Args a)
{
    constexpr int SUBS = kThreads / BP;
    __shared__ double s_ax[kMaxCov * 32];
    __shared__ double s_C[kMaxCov * 32];
    extern __shared__ __align__(16) double s_acc[];
    const Lanes<BP> ln(a.B);
    for (int k = threadIdx.x; k < a.c * a.B; k += kThreads) s_C[k] = a.C[k];
    small_clear(a, s_acc);
    const int64_t g0 = (int64_t)blockIdx.x * SUBS + threadIdx.x / BP;
    const int64_t gstep = (int64_t)gridDim.x * SUBS;
    double ax[kMaxCov];
#pragma unroll
    for (int c = 0; c < kMaxCov; c++) ax[c] = 0.0;
    auto h_of = [&](int64_t i, const uint32_t (&c)[HDFE_MAX_DIMS], double &hU, Runs &key) {
        // sum_d U[level_d(i), j], read again only when the codes change
        if (!key.have || !same(a, key.codes, c)) {
            hU = 0.0;
            if (ln.on) {
#pragma unroll
                for (int d = 0; d < HDFE_MAX_DIMS; d++) {
                    if (d >= a.D) break;
                    hU += a.U[(a.offs[d] + c[d]) * a.B + ln.j];
                }
            }
#pragma unroll
            for (int d = 0; d < HDFE_MAX_DIMS; d++) {
                if (d >= a.D) break;
                key.codes[d] = c[d];
            }
            key.have = true;
        }
        double h = hU;
        if (ln.on)
            for (int cc = 0; cc < a.c; cc++) h += __ldg(a.X + i * a.c + cc) * s_C[cc * a.B + ln.j];
        return h;
    };
    for (int64_t g = g0; g < a.G; g += gstep) {
        const int64_t s = a.starts[g], e = a.starts[g + 1];
        const double sw = group_weight(a, s, e);
        const double rho = (a.streamed && ln.on && sw > 0.0) ? a.streamed[g * a.B + ln.j] / sw : 0.0;
        // pass 1: the group's mean of rho - h
        double tot = 0.0, hU = 0.0;
        Runs key{};
        for (int64_t i = s; i < e; i++) {
            uint32_t c[HDFE_MAX_DIMS];
            row_codes(a, i, c);
            const double wi = a.w ? __ldg(a.w + i) : 1.0;
            tot += wi * (rho - h_of(i, c, hU, key));
        }
        const double mean = sw > 0.0 ? tot / sw : 0.0;
        if (a.groups && ln.on) a.groups[g * a.B + ln.j] = mean;
        if (!a.rows && !a.collect) continue;
        // pass 2: the rows, and the collect sink
        key.have = false;
        Runs run{};
        double gs = 0.0;
        for (int64_t i = s; i < e; i++) {
            uint32_t c[HDFE_MAX_DIMS];
            row_codes(a, i, c);
            const double o = h_of(i, c, hU, key) + mean;
            if (a.rows && ln.on) a.rows[i * a.B + ln.j] = o;
            if (a.collect) {
                const double wi = a.w ? __ldg(a.w + i) : 1.0;
                const double v = wi * (a.omega ? __ldg(a.omega + i) : 1.0) * o;
                run_add(a, run, c, v, ln.j, ln.on, s_acc);
                gs += v;
#pragma unroll
                for (int cc = 0; cc < kMaxCov; cc++) {
                    if (cc >= a.c) break;
                    ax[cc] += __ldg(a.X + i * a.c + cc) * v;
                }
            }
        }
        if (a.collect) {
            if (run.have && ln.on) run_flush(a, run, ln.j, s_acc);
            if (a.gsum && ln.on) a.gsum[g * a.B + ln.j] = gs;
        }
    }
    if (a.collect) small_flush(a, s_acc);
    if (a.collect && a.acc_x && a.c > 0) flush_cov<BP>(a, ax, s_ax, ln.j, ln.on);
}

// ------------------------------------------------------ windows (wide blocks)

// one sub-warp's staging: rows (codes, covariates, weights, w omega), group
// sums, run sums, the groups' streamed values and U's rows of the runs
constexpr int kAhead = 8;               // runs and groups whose values are loaded ahead

template <int BP>
struct Win {
    static __host__ __device__ int bytes(int c, int D, bool weights, bool project, bool collect)
    {
        const int d = kWin * c + kWin * (c + 2) + (weights ? 2 * kWin : 0) +
                      (collect ? kWin + kWin * (c + 1) : 0) + kAhead * BP +
                      (project ? kWin * BP : 0);
        return (d * 8 + kWin * D * 4 + 15) / 16 * 16;
    }
    double *x, *gx, *w, *rw, *om, *ro, *st, *hu;
    uint32_t *codes;
    __device__ Win(char *p, int c, int D, bool weights, bool project, bool collect)
    {
        double *q = reinterpret_cast<double *>(p);
        auto take = [&](int n) { double *at = q; q += n; return at; };
        x = take(kWin * c);
        gx = take(kWin * (c + 2));                  // sums of w x, w; 1 / sum of w
        w = take(weights ? kWin : 0);
        rw = take(weights ? kWin : 0);              // by run head
        om = take(collect ? kWin : 0);
        ro = take(collect ? kWin * (c + 1) : 0);    // by run: sums of w omega, w omega x
        st = take(kAhead * BP);
        hu = take(project ? kWin * BP : 0);         // by run head
        codes = reinterpret_cast<uint32_t *>(q);
    }
};

// rows [i0, i0 + n) into the window; returns the run heads' mask.  xx: this
// lane's sums of w omega x_k x_l (k <= l) over the rows it staged.
template <int BP, int C, bool COLLECT>
__device__ __forceinline__ unsigned load_window(const Args &a, const Lanes<BP> &ln, Win<BP> &wn,
                                                int64_t i0, int n, double *xx)
{
    const int c = C < 0 ? a.c : C;
    const bool W = a.w != nullptr;
    constexpr int CM = C < 0 ? kMaxCov : (C > 0 ? C : 1);
    for (int t = ln.j; t < n; t += BP) {
        const int64_t i = i0 + t;
        uint32_t code[HDFE_MAX_DIMS];
        row_codes(a, i, code);
#pragma unroll
        for (int d = 0; d < HDFE_MAX_DIMS; d++) {
            if (d >= a.D) break;
            wn.codes[t * a.D + d] = code[d];
        }
        double x[CM];
#pragma unroll
        for (int k = 0; k < CM; k++) {
            if (k >= c) break;
            x[k] = __ldg(a.X + i * a.c + k);
            wn.x[t * c + k] = x[k];
        }
        const double w = W ? __ldg(a.w + i) : 1.0;
        if (W) wn.w[t] = w;
        if (COLLECT) {
            const double o = w * (a.omega ? __ldg(a.omega + i) : 1.0);
            wn.om[t] = o;
            if (xx) {
#pragma unroll
                for (int k = 0; k < CM; k++) {
                    if (k >= c) break;
#pragma unroll
                    for (int l = 0; l < CM; l++) {
                        if (l < k) continue;
                        if (l >= c) break;
                        xx[k * CM + l] += o * x[k] * x[l];
                    }
                }
            }
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

// the groups' sums of w x and w with the reciprocal weight, and the runs' sums
// of w, w omega and w omega x, each by one lane
template <int BP, int C, bool COLLECT>
__device__ __forceinline__ void window_sums(const Args &a, const Lanes<BP> &ln, Win<BP> &wn,
                                            unsigned gheads, int ng, unsigned heads, int n)
{
    const int c = C < 0 ? a.c : C;
    const bool W = a.w != nullptr;
    for (int t = ln.j; t < ng * (c + 1); t += BP) {
        const int g = t / (c + 1), k = t - g * (c + 1);
        const int q0 = nth_bit(gheads, g), q1 = next_bit(gheads, q0, n);
        double v = 0.0;
        if (k == c && !W) {
            v = (double)(q1 - q0);
        } else {
            for (int q = q0; q < q1; q++) {
                const double xq = k < c ? wn.x[q * c + k] : 1.0;
                v += W ? wn.w[q] * xq : xq;
            }
        }
        wn.gx[g * (c + 2) + k] = v;
        if (k == c) wn.gx[g * (c + 2) + c + 1] = v > 0.0 ? 1.0 / v : 0.0;
    }
    if (W || COLLECT) {
        const int nr = __popc(heads), per = (W ? 1 : 0) + (COLLECT ? c + 1 : 0);
        for (int t = ln.j; t < nr * per; t += BP) {
            const int r = t / per, k = t - r * per - (W ? 1 : 0);      // -1: the run's weight
            const int q0 = nth_bit(heads, r), q1 = next_bit(heads, q0, n);
            double v = 0.0;
            for (int q = q0; q < q1; q++)
                v += k < 0 ? wn.w[q] : (k == 0 ? wn.om[q] : wn.om[q] * wn.x[q * c + k - 1]);
            if (k < 0) wn.rw[q0] = v;
            else wn.ro[r * (c + 1) + k] = v;
        }
    }
    __syncwarp(ln.mask);
}

// the streamed values of the window's first groups (the rest is loaded when
// its turn comes)
template <int BP>
__device__ __forceinline__ void load_streamed(const Args &a, const Lanes<BP> &ln, Win<BP> &wn,
                                              int64_t g, int ng)
{
    double v[kAhead];
#pragma unroll
    for (int f = 0; f < kAhead; f++)
        v[f] = f < ng && ln.on && a.streamed ? a.streamed[(g + f) * a.B + ln.j] : 0.0;
#pragma unroll
    for (int f = 0; f < kAhead; f++)
        if (f < ng) wn.st[f * BP + ln.j] = v[f];
}

template <int BP>
__device__ __forceinline__ double streamed_of(const Args &a, const Lanes<BP> &ln,
                                              const Win<BP> &wn, int64_t g, int f)
{
    if (f < kAhead) return wn.st[f * BP + ln.j];
    return ln.on && a.streamed ? a.streamed[(g + f) * a.B + ln.j] : 0.0;
}

// v to row q's levels
template <int BP>
__device__ __forceinline__ void add_levels(const Args &a, const Lanes<BP> &ln, const Win<BP> &wn,
                                           int q, double v)
{
    if (!ln.on) return;
#pragma unroll
    for (int d = 0; d < HDFE_MAX_DIMS; d++) {
        if (d >= a.D) break;
        atomicAdd(a.acc + (a.offs[d] + wn.codes[q * a.D + d]) * a.B + ln.j, v);
    }
}

template <int BP, int CM>
__device__ __forceinline__ void add_cov(const Args &a, const Lanes<BP> &ln, const double (&ax)[CM],
                                        int c, double *s_ax)
{
    if (!a.acc_x || c == 0) return;
    for (int k = threadIdx.x; k < c * a.B; k += kThreads) s_ax[k] = 0.0;
    __syncthreads();
    if (ln.on) {
#pragma unroll
        for (int k = 0; k < CM; k++) {
            if (k >= c) break;
            atomicAdd(s_ax + k * a.B + ln.j, ax[k]);
        }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < c * a.B; k += kThreads)
        if (s_ax[k] != 0.0) atomicAdd(a.acc_x + k, s_ax[k]);
}

template <int BP, typename F, typename H>
__device__ __forceinline__ void walk(const Args &a, const Lanes<BP> &ln, F window, H lone)
{
    constexpr int SUBS = kThreads / BP;
    walk_windows<BP>(a.starts, a.G, a.chunk, (int64_t)blockIdx.x * SUBS + threadIdx.x / BP,
                     (int64_t)gridDim.x * SUBS, ln.j, ln.mask, window, lone);
}

// reduce of the streamed block
template <int BP, int C>
__global__ void __launch_bounds__(kThreads) k_spread_win(Args a)
{
    extern __shared__ __align__(16) char s_raw[];
    __shared__ double s_ax[kMaxCov * 32];
    const Lanes<BP> ln(a.B);
    const int c = C < 0 ? a.c : C;
    const bool W = a.w != nullptr;
    constexpr int CM = C < 0 ? kMaxCov : (C > 0 ? C : 1);
    Win<BP> wn(s_raw + (threadIdx.x / BP) * Win<BP>::bytes(c, a.D, W, false, false), c, a.D, W,
               false, false);
    double ax[CM];
#pragma unroll
    for (int k = 0; k < CM; k++) ax[k] = 0.0;
    // group f of the window, rows [q0, q1), rho its streamed value over its weight
    auto group = [&](int f, int q0, int q1, unsigned heads, double rho) {
#pragma unroll
        for (int k = 0; k < CM; k++) {
            if (k >= c) break;
            ax[k] += wn.gx[f * (c + 2) + k] * rho;
        }
        for (int p0 = q0; p0 < q1;) {
            const int p1 = next_bit(heads, p0, q1);
            add_levels(a, ln, wn, p0, (W ? wn.rw[p0] : (double)(p1 - p0)) * rho);
            p0 = p1;
        }
    };
    auto window = [&](int64_t g, int64_t i0, int n, unsigned gheads, int ng) {
        load_streamed(a, ln, wn, g, ng);
        const unsigned heads =
            load_window<BP, C, false>(a, ln, wn, i0, n, nullptr) | gheads;
        window_sums<BP, C, false>(a, ln, wn, gheads, ng, heads, n);
        int q0 = 0;
        for (int f = 0; f < ng; f++) {
            const int q1 = next_bit(gheads, q0, n);
            // (nothing of a group without weight: its value may be no number)
            const double *gx = wn.gx + f * (c + 2);
            group(f, q0, q1, heads,
                  gx[c] > 0.0 ? streamed_of(a, ln, wn, g, f) * gx[c + 1] : 0.0);
            q0 = q1;
        }
    };
    auto lone = [&](int64_t g, int64_t s, int64_t e) {
        const double sw = group_weight(a, s, e);
        const double rho = ln.on && sw > 0.0 ? a.streamed[g * a.B + ln.j] / sw : 0.0;
        for (int64_t i0 = s; i0 < e; i0 += kWin) {
            const int n = (int)min((int64_t)kWin, e - i0);
            const unsigned heads = load_window<BP, C, false>(a, ln, wn, i0, n, nullptr);
            window_sums<BP, C, false>(a, ln, wn, 1u, 1, heads, n);
            group(0, 0, n, heads, rho);
            __syncwarp(ln.mask);
        }
    };
    walk(a, ln, window, lone);
    add_cov<BP, CM>(a, ln, ax, c, s_ax);
}

template <int BP, int C, bool COLLECT>
__global__ void __launch_bounds__(kThreads) k_project_win(Args a)
{
    extern __shared__ __align__(16) char s_raw[];
    __shared__ double s_ax[kMaxCov * 32];
    const Lanes<BP> ln(a.B);
    const int c = C < 0 ? a.c : C;
    const bool W = a.w != nullptr;
    constexpr int CM = C < 0 ? kMaxCov : (C > 0 ? C : 1);
    Win<BP> wn(s_raw + (threadIdx.x / BP) * Win<BP>::bytes(c, a.D, W, true, COLLECT), c, a.D, W,
               true, COLLECT);
    double ax[CM], xx[COLLECT ? CM * CM : 1], Cj[CM];
#pragma unroll
    for (int k = 0; k < CM; k++) {
        ax[k] = 0.0;
        Cj[k] = k < c && ln.on ? a.C[k * a.B + ln.j] : 0.0;
    }
    if (COLLECT) {
#pragma unroll
        for (int k = 0; k < CM * CM; k++) xx[k] = 0.0;
    }
    auto gather = [&](int q) {                  // sum_d U[level_d, j] of row q's run
        double h = 0.0;
#pragma unroll
        for (int d = 0; d < HDFE_MAX_DIMS; d++) {
            if (d >= a.D) break;
            h += a.U[(a.offs[d] + wn.codes[q * a.D + d]) * a.B + ln.j];
        }
        return h;
    };
    // U's rows of the runs: the first kAhead loaded together
    auto load_runs = [&](unsigned heads) {
        double h[kAhead];
        unsigned m = heads;
#pragma unroll
        for (int f = 0; f < kAhead; f++) {
            h[f] = m && ln.on ? gather(__ffs(m) - 1) : 0.0;
            m &= m - 1;
        }
        unsigned m2 = heads;
#pragma unroll
        for (int f = 0; f < kAhead; f++) {
            if (m2) wn.hu[(__ffs(m2) - 1) * BP + ln.j] = h[f];
            m2 &= m2 - 1;
        }
        for (; m; m &= m - 1) {
            const int q = __ffs(m) - 1;
            wn.hu[q * BP + ln.j] = ln.on ? gather(q) : 0.0;
        }
    };
    // sum over the runs of [q0, q1) of w hU
    auto sum_h = [&](unsigned heads, int q0, int q1) {
        double t = 0.0;
        for (int p0 = q0; p0 < q1;) {
            const int p1 = next_bit(heads, p0, q1);
            t += (W ? wn.rw[p0] : (double)(p1 - p0)) * wn.hu[p0 * BP + ln.j];
            p0 = p1;
        }
        return t;
    };
    // the rows' output and the sink's sums of rows [q0, q1) of one group whose
    // first run is the window's r-th; returns the group sum
    auto emit = [&](unsigned heads, int64_t i0, int q0, int q1, int r, double mean) {
        double gs = 0.0;
        for (int p0 = q0; p0 < q1; r++) {
            const int p1 = next_bit(heads, p0, q1);
            const double base = wn.hu[p0 * BP + ln.j] + mean;
            if (a.rows) {
                for (int q = p0; q < p1; q++) {
                    double o = base;
#pragma unroll
                    for (int k = 0; k < CM; k++) {
                        if (k >= c) break;
                        o += wn.x[q * c + k] * Cj[k];
                    }
                    if (ln.on) a.rows[(i0 + q) * a.B + ln.j] = o;
                }
            }
            if (COLLECT) {
                const double *ro = wn.ro + r * (c + 1);
                double v = ro[0] * base;
#pragma unroll
                for (int k = 0; k < CM; k++) {
                    if (k >= c) break;
                    v += ro[1 + k] * Cj[k];
                    ax[k] += ro[1 + k] * base;
                }
                add_levels(a, ln, wn, p0, v);
                gs += v;
            }
            p0 = p1;
        }
        return gs;
    };
    auto window = [&](int64_t g, int64_t i0, int n, unsigned gheads, int ng) {
        load_streamed(a, ln, wn, g, ng);
        const unsigned heads = load_window<BP, C, COLLECT>(a, ln, wn, i0, n, xx) | gheads;
        load_runs(heads);
        window_sums<BP, C, COLLECT>(a, ln, wn, gheads, ng, heads, n);
        int q0 = 0, r = 0;
        for (int f = 0; f < ng; f++) {
            const int q1 = next_bit(gheads, q0, n);
            const double *gx = wn.gx + f * (c + 2);
            // the mean of rho - h, rho = streamed / sum of w
            double tot = (gx[c] > 0.0 ? streamed_of(a, ln, wn, g, f) : 0.0) - sum_h(heads, q0, q1);
#pragma unroll
            for (int k = 0; k < CM; k++) {
                if (k >= c) break;
                tot -= gx[k] * Cj[k];
            }
            const double mean = gx[c] > 0.0 ? tot * gx[c + 1] : 0.0;
            if (a.groups && ln.on) a.groups[(g + f) * a.B + ln.j] = mean;
            if (a.rows || COLLECT) {
                const double gs = emit(heads, i0, q0, q1, r, mean);
                if (COLLECT && a.gsum && ln.on) a.gsum[(g + f) * a.B + ln.j] = gs;
            }
            r += __popc(heads & below(q1) & ~below(q0));
            q0 = q1;
        }
    };
    auto lone = [&](int64_t g, int64_t s, int64_t e) {
        const double sw = group_weight(a, s, e);
        double tot = a.streamed && ln.on && sw > 0.0 ? a.streamed[g * a.B + ln.j] : 0.0, gs = 0.0;
        for (int64_t i0 = s; i0 < e; i0 += kWin) {
            const int n = (int)min((int64_t)kWin, e - i0);
            const unsigned heads = load_window<BP, C, COLLECT>(a, ln, wn, i0, n, nullptr);
            load_runs(heads);
            window_sums<BP, C, COLLECT>(a, ln, wn, 1u, 1, heads, n);
            tot -= sum_h(heads, 0, n);
#pragma unroll
            for (int k = 0; k < CM; k++) {
                if (k >= c) break;
                tot -= wn.gx[k] * Cj[k];
            }
            __syncwarp(ln.mask);
        }
        const double mean = sw > 0.0 ? tot / sw : 0.0;
        if (a.groups && ln.on) a.groups[g * a.B + ln.j] = mean;
        if (!a.rows && !COLLECT) return;
        for (int64_t i0 = s; i0 < e; i0 += kWin) {
            const int n = (int)min((int64_t)kWin, e - i0);
            const unsigned heads = load_window<BP, C, COLLECT>(a, ln, wn, i0, n, xx);
            load_runs(heads);
            window_sums<BP, C, COLLECT>(a, ln, wn, 1u, 1, heads, n);
            gs += emit(heads, i0, 0, n, 0, mean);
            __syncwarp(ln.mask);
        }
        if (COLLECT && a.gsum && ln.on) a.gsum[g * a.B + ln.j] = gs;
    };
    walk(a, ln, window, lone);
    if (COLLECT) {
        // the sub-warp's w omega X X' times C
#pragma unroll
        for (int k = 0; k < CM; k++) {
#pragma unroll
            for (int l = 0; l < CM; l++) {
                if (l < k || k >= c || l >= c) continue;
                double v = xx[k * CM + l];
#pragma unroll
                for (int o = BP / 2; o > 0; o >>= 1) v += __shfl_xor_sync(ln.mask, v, o, BP);
                ax[k] += v * Cj[l];
                if (l != k) ax[l] += v * Cj[k];
            }
        }
        add_cov<BP, CM>(a, ln, ax, c, s_ax);
    }
}

// ---------------------------------------------------------- trace moments

struct TraceArgs {
    const int64_t *starts;
    int64_t G;
    const uint32_t *codes;
    int D, psi_column;
    int64_t psi_offset, psi_levels;
    const double *w;
    const double *Zl, *Zg, *Ul, *Ug;     // (L, B), (G, B), (L, B), (G, B)
    int B;
    double *partial;                     // (gridDim, B, 8)
    unsigned *status;
    int64_t chunk;
};

// Per run of rows with one psi level, as the passes above (0.60 -> 0.45 ms
// for 32 vectors on the 1M-worker panel).
template <int BP>
__global__ void __launch_bounds__(kThreads) k_trace(TraceArgs a)
{
    constexpr int SUBS = kThreads / BP;
    __shared__ double s_m[SUBS][BP][8];
    __shared__ uint32_t s_code[SUBS][kWin];
    __shared__ double s_w[SUBS][kWin];
    const Lanes<BP> ln(a.B);
    const int sub = threadIdx.x / BP;
    uint32_t *code = s_code[sub];
    double *w = s_w[sub];
    double m[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    // rows [i0, i0 + n): their psi codes and weights; returns the run heads
    auto load = [&](int64_t i0, int n) {
        for (int t = ln.j; t < n; t += BP) {
            uint32_t v = __ldg(a.codes + (i0 + t) * a.D + a.psi_column);
            if ((int64_t)v >= a.psi_levels) {
                if (a.status) atomicCAS(a.status, 0u, (unsigned)HDFE_ERR_BAD_CODE);
                v = 0;
            }
            code[t] = v;
            if (a.w) w[t] = __ldg(a.w + i0 + t);
        }
        __syncwarp(ln.mask);
        unsigned heads = 0;
        for (int t = ln.j; t < n; t += BP)
            heads |= (unsigned)(t == 0 || code[t] != code[t - 1]) << t;
        return __reduce_or_sync(ln.mask, heads);
    };
    // the runs of rows [q0, q1), all of one group
    auto group = [&](unsigned heads, int q0, int q1, double b1, double b2) {
        for (int p0 = q0; p0 < q1;) {
            const int p1 = next_bit(heads, p0, q1);
            const int64_t lv = a.psi_offset + code[p0];
            const double a1 = ln.on ? a.Zl[lv * a.B + ln.j] : 0.0;
            const double a2 = ln.on ? a.Ul[lv * a.B + ln.j] : 0.0;
            double wt = (double)(p1 - p0);
            if (a.w) {
                wt = 0.0;
                for (int q = p0; q < p1; q++) wt += w[q];
            }
            m[0] += wt;
            m[1] += wt * a1 * a2;
            m[2] += wt * b1 * b2;
            m[3] += wt * (a1 * b2 + b1 * a2);
            m[4] += wt * a1;
            m[5] += wt * a2;
            m[6] += wt * b1;
            m[7] += wt * b2;
            p0 = p1;
        }
    };
    auto window = [&](int64_t g, int64_t i0, int n, unsigned gheads, int ng) {
        const unsigned heads = load(i0, n) | gheads;
        int q0 = 0;
        for (int f = 0; f < ng; f++) {
            const int q1 = next_bit(gheads, q0, n);
            group(heads, q0, q1, ln.on ? a.Zg[(g + f) * a.B + ln.j] : 0.0,
                  ln.on ? a.Ug[(g + f) * a.B + ln.j] : 0.0);
            q0 = q1;
        }
    };
    auto lone = [&](int64_t g, int64_t s, int64_t e) {
        const double b1 = ln.on && e > s ? a.Zg[g * a.B + ln.j] : 0.0;
        const double b2 = ln.on && e > s ? a.Ug[g * a.B + ln.j] : 0.0;
        for (int64_t i0 = s; i0 < e; i0 += kWin) {
            const int n = (int)min((int64_t)kWin, e - i0);
            group(load(i0, n), 0, n, b1, b2);
            __syncwarp(ln.mask);
        }
    };
    walk_windows<BP>(a.starts, a.G, a.chunk, (int64_t)blockIdx.x * SUBS + sub,
                     (int64_t)gridDim.x * SUBS, ln.j, ln.mask, window, lone);
#pragma unroll
    for (int k = 0; k < 8; k++) s_m[sub][ln.j][k] = m[k];
    __syncthreads();
    for (int t = threadIdx.x; t < a.B * 8; t += kThreads) {
        const int j = t / 8, k = t % 8;
        double sum = 0.0;
        for (int q = 0; q < SUBS; q++) sum += s_m[q][j][k];
        a.partial[((int64_t)blockIdx.x * a.B + j) * 8 + k] = sum;
    }
}

// out[j, k] = sum over CTAs of partial, one warp per entry, fixed order
__global__ void __launch_bounds__(kThreads) k_trace_reduce(const double *partial, int64_t blocks,
                                                           int B, double *out)
{
    const int lane = threadIdx.x & 31;
    const int64_t q = ((int64_t)blockIdx.x * kThreads + threadIdx.x) >> 5;
    if (q >= (int64_t)B * 8) return;
    double s = 0.0;
    for (int64_t b = lane; b < blocks; b += 32) s += partial[b * B * 8 + q];
    s = warp_sum(s);
    if (lane == 0) out[q] = s;
}

// ------------------------------------------------------- Rademacher draws

__global__ void __launch_bounds__(256) k_rademacher(double *out, int64_t n_rows, int64_t ordinal0,
                                                    int B, uint64_t seed, int64_t first_draw)
{
    const int64_t total = n_rows * B;
    for (int64_t t = (int64_t)blockIdx.x * 256 + threadIdx.x; t < total;
         t += (int64_t)gridDim.x * 256) {
        const int64_t i = t / B, j = t % B;
        uint64_t x = seed ^ ((uint64_t)(ordinal0 + i) * 0x9E3779B97F4A7C15ull) ^
                     ((uint64_t)(first_draw + j) * 0xBF58476D1CE4E5B9ull);
        x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
        x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
        x = x ^ (x >> 31);
        out[t] = (x >> 63) == 0 ? 1.0 : -1.0;
    }
}

int fill(Args &a, const int64_t *starts, int64_t G, const uint32_t *codes, int32_t D,
         const int64_t *n_levels, const double *w, const double *X, int32_t c, int32_t B,
         unsigned *status)
{
    if (D < 1 || D > HDFE_MAX_DIMS || G < 0 || !starts || !codes || !n_levels || B < 1 ||
        B > 32 || c < 0 || c > kMaxCov || (c > 0 && !X))
        return hdfe_set_arg_error("hdfe_rows_reduce/project_coef: bad argument");
    a = Args{};
    a.starts = starts;
    a.G = G;
    a.codes = codes;
    a.D = D;
    int64_t L = 0;
    for (int d = 0; d < D; d++) {
        if (n_levels[d] < 1) return hdfe_set_arg_error("hdfe_rows: n_levels must be >= 1");
        a.offs[d] = L;
        a.nlev[d] = n_levels[d];
        L += n_levels[d];
    }
    a.L = L;
    a.w = w;
    a.X = X;
    a.c = c;
    a.B = B;
    a.Bp = B <= 8 ? 8 : (B <= 16 ? 16 : 32);
    a.status = status;
    return HDFE_OK;
}

inline unsigned grid_for(int64_t G, int Bp)
{
    const int64_t per = kThreads / Bp;
    int64_t b = (G + per - 1) / per;
    if (b > kMaxGrid) b = kMaxGrid;
    return (unsigned)(b > 0 ? b : 1);
}

// CTAs of a window pass (sub-warps of Bp lanes), and its chunk of groups
inline unsigned window_grid(int64_t G, int Bp, int64_t *chunk)
{
    const int64_t ctas = 148 * 5, subs = kThreads / Bp;
    *chunk = window_chunk(G, ctas * subs);
    int64_t b = (G + *chunk * subs - 1) / (*chunk * subs);
    if (b > 2 * ctas) b = 2 * ctas;
    return (unsigned)(b > 0 ? b : 1);
}

// Blocks up to this many vectors take the narrow passes.  us of reduce / project
// with the sink, narrow against windows: 1M workers without years, 4 vectors 237 /
// 2194 against 346 / 1444, 8 vectors 432 / 2909 against 348 / 1468; 400k workers
// with ten years, 4 vectors 164 / 1109 against 3343 / 3441, 8 vectors 272 / 1645
// against 3387 / 3479.  (The windows add every run to the years' ten addresses by
// global atomics, which holds them up from the first vector on.)
constexpr int kNarrow = 4;
constexpr int64_t kSmallBytes = 32 * 1024;      // level sums in shared memory per CTA

// the dimensions a narrow pass sums in shared memory first; returns the bytes
inline int take_small(Args &a)
{
    int64_t slots = 0;
    for (int d = 0; d < a.D; d++) {
        if (a.nlev[d] <= 512 && (slots + a.nlev[d]) * a.B * 8 <= kSmallBytes) {
            a.small[d] = 1;
            a.soff[d] = slots;
            slots += a.nlev[d];
        }
    }
    a.n_small = slots;
    return (int)(slots * a.B * 8);
}

template <int BP, int C>
int launch_spread(Args &a, cudaStream_t s)
{
    constexpr int subs = kThreads / BP, most = C < 0 ? kMaxCov : C;
    static hdfe_shared_limit limit;
    const int st = limit.raise((const void *)k_spread_win<BP, C>,
                               subs * Win<BP>::bytes(most, HDFE_MAX_DIMS, true, false, false));
    if (st != HDFE_OK) return st;
    const unsigned grid = window_grid(a.G, BP, &a.chunk);
    k_spread_win<BP, C><<<grid, kThreads,
                          subs * Win<BP>::bytes(a.c, a.D, a.w != nullptr, false, false), s>>>(a);
    return HDFE_OK;
}

template <int BP>
int launch_spread(Args &a, cudaStream_t s)
{
    switch (a.c) {
    case 0: return launch_spread<BP, 0>(a, s);
    case 1: return launch_spread<BP, 1>(a, s);
    case 2: return launch_spread<BP, 2>(a, s);
    case 3: return launch_spread<BP, 3>(a, s);
    default: return launch_spread<BP, -1>(a, s);
    }
}

template <int BP, int C, bool COLLECT>
int launch_project(Args &a, cudaStream_t s)
{
    constexpr int subs = kThreads / BP, most = C < 0 ? kMaxCov : C;
    static hdfe_shared_limit limit;
    const int st = limit.raise((const void *)k_project_win<BP, C, COLLECT>,
                               subs * Win<BP>::bytes(most, HDFE_MAX_DIMS, true, true, COLLECT));
    if (st != HDFE_OK) return st;
    const unsigned grid = window_grid(a.G, BP, &a.chunk);
    k_project_win<BP, C, COLLECT>
        <<<grid, kThreads, subs * Win<BP>::bytes(a.c, a.D, a.w != nullptr, true, COLLECT), s>>>(a);
    return HDFE_OK;
}

template <int BP, bool COLLECT>
int launch_project(Args &a, cudaStream_t s)
{
    switch (a.c) {
    case 0: return launch_project<BP, 0, COLLECT>(a, s);
    case 1: return launch_project<BP, 1, COLLECT>(a, s);
    case 2: return launch_project<BP, 2, COLLECT>(a, s);
    case 3: return launch_project<BP, 3, COLLECT>(a, s);
    default: return launch_project<BP, -1, COLLECT>(a, s);
    }
}

template <int BP>
int launch_project(Args &a, cudaStream_t s)
{
    return a.collect ? launch_project<BP, true>(a, s) : launch_project<BP, false>(a, s);
}

// project_coef: narrow blocks by groups, the others by windows
int project(Args &a, cudaStream_t s)
{
    if (a.B <= kNarrow) {
        const int smem = a.collect ? take_small(a) : 0;
        if (a.B == 1) k_project_coef<1><<<grid_for(a.G, 1), kThreads, smem, s>>>(a);
        else if (a.B == 2) k_project_coef<2><<<grid_for(a.G, 2), kThreads, smem, s>>>(a);
        else k_project_coef<4><<<grid_for(a.G, 4), kThreads, smem, s>>>(a);
    } else {
        const int st = a.Bp == 8 ? launch_project<8>(a, s)
                                 : (a.Bp == 16 ? launch_project<16>(a, s) : launch_project<32>(a, s));
        if (st != HDFE_OK) return st;
    }
    HDFE_CUDA_TRY(cudaGetLastError());
    hdfe_add_launches(1);
    return HDFE_OK;
}

// reduce: explicit rows and narrow blocks by groups, the others by windows
int reduce(Args &a, cudaStream_t s)
{
    if (a.streamed && a.B > kNarrow) {
        const int st = a.Bp == 8 ? launch_spread<8>(a, s)
                                 : (a.Bp == 16 ? launch_spread<16>(a, s) : launch_spread<32>(a, s));
        if (st != HDFE_OK) return st;
    } else {
        const int smem = take_small(a);
        if (a.B == 1) k_reduce<1><<<grid_for(a.G, 1), kThreads, smem, s>>>(a);
        else if (a.B == 2) k_reduce<2><<<grid_for(a.G, 2), kThreads, smem, s>>>(a);
        else if (a.B <= 4) k_reduce<4><<<grid_for(a.G, 4), kThreads, smem, s>>>(a);
        else if (a.Bp == 8) k_reduce<8><<<grid_for(a.G, 8), kThreads, smem, s>>>(a);
        else if (a.Bp == 16) k_reduce<16><<<grid_for(a.G, 16), kThreads, smem, s>>>(a);
        else k_reduce<32><<<grid_for(a.G, 32), kThreads, smem, s>>>(a);
    }
    HDFE_CUDA_TRY(cudaGetLastError());
    hdfe_add_launches(1);
    return HDFE_OK;
}

}  // namespace coef
}  // namespace hdfe

using namespace hdfe;

extern "C" int hdfe_rows_reduce(const int64_t *starts, int64_t n_groups, const uint32_t *codes,
                                int32_t D, const int64_t *n_levels, const double *w,
                                const double *X, int32_t c, const double *streamed,
                                const double *R, int32_t B, double *acc, double *acc_x,
                                double *group_sums, void *status, void *stream)
{
    coef::Args a;
    int st = coef::fill(a, starts, n_groups, codes, D, n_levels, w, X, c, B, (unsigned *)status);
    if (st != HDFE_OK) return st;
    if ((streamed == nullptr) == (R == nullptr) || !acc || (c > 0 && !acc_x) ||
        (group_sums && streamed))
        return hdfe_set_arg_error("hdfe_rows_reduce: give exactly one of streamed and R "
                                  "(group sums with R only)");
    a.streamed = streamed;
    a.R = R;
    a.acc = acc;
    a.acc_x = acc_x;
    a.gsum = group_sums;
    return coef::reduce(a, (cudaStream_t)stream);
}

extern "C" int hdfe_rows_project_coef(const int64_t *starts, int64_t n_groups,
                                      const uint32_t *codes, int32_t D, const int64_t *n_levels,
                                      const double *w, const double *X, int32_t c,
                                      const double *C, const double *U, const double *streamed,
                                      int32_t B, double *rows, double *groups,
                                      const double *omega, double *acc, double *acc_x,
                                      double *group_sums, void *status, void *stream)
{
    coef::Args a;
    int st = coef::fill(a, starts, n_groups, codes, D, n_levels, w, X, c, B, (unsigned *)status);
    if (st != HDFE_OK) return st;
    if (!U || (c > 0 && !C) || (omega && (!acc || (c > 0 && !acc_x))))
        return hdfe_set_arg_error("hdfe_rows_project_coef: bad argument");
    a.U = U;
    a.C = C;
    a.streamed = streamed;
    a.rows = rows;
    a.groups = groups;
    a.omega = omega;
    a.collect = omega != nullptr;
    a.acc = acc;
    a.acc_x = acc_x;
    a.gsum = group_sums;
    return coef::project(a, (cudaStream_t)stream);
}

extern "C" int64_t hdfe_trace_moments_workspace_bytes(int32_t B)
{
    if (B < 1 || B > 32) return -1;
    return (int64_t)coef::kMaxGrid * B * 8 * 8;
}

extern "C" int hdfe_trace_moments(const int64_t *starts, int64_t n_groups, const uint32_t *codes,
                                  int32_t D, const int64_t *n_levels, int32_t psi_column,
                                  const double *w, const double *Z_levels,
                                  const double *Z_groups, const double *U_levels,
                                  const double *U_groups, int32_t B, double *out,
                                  void *workspace, int64_t workspace_bytes, void *status,
                                  void *stream)
{
    if (D < 1 || D > HDFE_MAX_DIMS || psi_column < 0 || psi_column >= D || n_groups < 0 ||
        !starts || !codes || !n_levels || !Z_levels || !Z_groups || !U_levels || !U_groups ||
        !out || B < 1 || B > 32 || !workspace)
        return hdfe_set_arg_error("hdfe_trace_moments: bad argument");
    if (workspace_bytes < hdfe_trace_moments_workspace_bytes(B))
        return hdfe_set_error(HDFE_ERR_WORKSPACE, "hdfe_trace_moments: workspace too small");
    coef::TraceArgs a{};
    a.starts = starts;
    a.G = n_groups;
    a.codes = codes;
    a.D = D;
    a.psi_column = psi_column;
    int64_t off = 0;
    for (int d = 0; d < psi_column; d++) off += n_levels[d];
    a.psi_offset = off;
    a.psi_levels = n_levels[psi_column];
    a.w = w;
    a.Zl = Z_levels;
    a.Zg = Z_groups;
    a.Ul = U_levels;
    a.Ug = U_groups;
    a.B = B;
    a.partial = (double *)workspace;
    a.status = (unsigned *)status;
    cudaStream_t s = (cudaStream_t)stream;
    const int Bp = B <= 8 ? 8 : (B <= 16 ? 16 : 32);
    const unsigned grid = coef::window_grid(n_groups, Bp, &a.chunk);
    if (Bp == 8) coef::k_trace<8><<<grid, coef::kThreads, 0, s>>>(a);
    else if (Bp == 16) coef::k_trace<16><<<grid, coef::kThreads, 0, s>>>(a);
    else coef::k_trace<32><<<grid, coef::kThreads, 0, s>>>(a);
    coef::k_trace_reduce<<<(unsigned)((B * 8 * 32 + coef::kThreads - 1) / coef::kThreads),
                           coef::kThreads, 0, s>>>(a.partial, grid, B, out);
    HDFE_CUDA_TRY(cudaGetLastError());
    hdfe_add_launches(2);
    return HDFE_OK;
}

extern "C" int hdfe_rademacher(double *out, int64_t n_rows, int64_t ordinal0, int32_t B,
                               uint64_t seed, int64_t first_draw, void *stream)
{
    if (!out || n_rows < 0 || B < 1) return hdfe_set_arg_error("hdfe_rademacher: bad argument");
    if (n_rows == 0) return HDFE_OK;
    int64_t blocks = (n_rows * B + 255) / 256;
    if (blocks > 148 * 32) blocks = 148 * 32;
    coef::k_rademacher<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(out, n_rows, ordinal0,
                                                                          B, seed, first_draw);
    HDFE_CUDA_TRY(cudaGetLastError());
    hdfe_add_launches(1);
    return HDFE_OK;
}

// (D_o' M_0 D_o) P from the identifying cells, without S: per group the
// n-weighted mean of h_i = sum_d P[level_d(i)] is taken off, and
// n_i (h_i - mean) is added to each of cell i's levels -- the projection pass
// with U = P, no streamed block, weights n and the collect sink's unit weights
// (core/kernels_base.py:478-507 `_nb_stream_matvec`).
extern "C" int hdfe_stream_matvec(const int64_t *starts, int64_t n_groups, const uint32_t *codes,
                                  int32_t D, const int64_t *n_levels, const double *n,
                                  const double *P, int32_t k, double *out, void *status,
                                  void *stream)
{
    coef::Args a;
    int st = coef::fill(a, starts, n_groups, codes, D, n_levels, n, nullptr, 0, k,
                        (unsigned *)status);
    if (st != HDFE_OK) return st;
    if (!n || !P || !out) return hdfe_set_arg_error("hdfe_stream_matvec: bad argument");
    a.U = P;
    a.collect = true;
    a.acc = out;
    cudaStream_t s = (cudaStream_t)stream;
    HDFE_CUDA_TRY(cudaMemsetAsync(out, 0, a.L * k * 8, s));
    return coef::project(a, s);
}
