// The centring pass over Rademacher draws (draws.cuh).
#include "draws.cuh"

namespace hdfe {
namespace rows {

template <int BP, int C, bool W>
__global__ void __launch_bounds__(kPassThreads) k_center_draws(Args a)
{
    extern __shared__ __align__(16) char s_raw[];
    double *s_acc = reinterpret_cast<double *>(s_raw);              // small dimensions
    const Lanes<BP> ln(a.B);
    const int c = C < 0 ? a.c : C;
    constexpr int CM = C < 0 ? kMaxCov : (C > 0 ? C : 1);
    Win<BP> wn(s_raw + (a.n_small * a.B * 8 + 15) / 16 * 16 +
                   (threadIdx.x / BP) * Win<BP>::bytes(c, a.D, W, false),
               c, a.D, W, false);
    for (int64_t k = threadIdx.x; k < a.n_small * a.B; k += kPassThreads) s_acc[k] = 0.0;
    __syncthreads();
    const uint64_t dterm = (uint64_t)(a.first_draw + ln.j) * kDrawMul;
    double ax[CM], sq = 0.0;
#pragma unroll
    for (int k = 0; k < CM; k++) ax[k] = 0.0;
    auto flush = [&](int q, double v) {         // a run's sum to its levels
        if (!ln.on) return;
#pragma unroll
        for (int d = 0; d < HDFE_MAX_DIMS; d++) {
            if (d >= a.D) break;
            const uint32_t code = wn.codes[q * a.D + d];
            if (a.small[d]) atomicAdd(s_acc + (a.soff[d] + code) * a.B + ln.j, v);
            else atomicAdd(a.acc + (a.offs[d] + code) * a.B + ln.j, v);
        }
    };
    // sum over rows [q0, q1) of w r and of w
    auto sums = [&](uint32_t word, int q0, int q1, double &tot, double &sw) {
        if (W) {
            tot = sw = 0.0;
            for (int q = q0; q < q1; q++) {
                tot += flip(wn.wr[q], word, q);
                sw += wn.w[q];
            }
        } else {
            const unsigned m = below(q1) & ~below(q0);
            sw = (double)(q1 - q0);
            tot = (double)(q1 - q0 - 2 * __popc(word & m));
        }
    };
    auto cov_rows = [&](uint32_t word, int n) {     // ax += x w r over the rows
        if (c > 0) {
#pragma unroll 4
            for (int q = 0; q < n; q++) {
                const double r = flip(W ? wn.wr[q] : 1.0, word, q);
#pragma unroll
                for (int k = 0; k < CM; k++) {
                    if (k >= c) break;
                    ax[k] += wn.x[q * c + k] * r;
                }
            }
        }
    };
    // a group without weight adds nothing, whatever its covariates: they are
    // staged as zeros
    auto drop_weightless = [&](unsigned gheads, int ng, int n) {
        if constexpr (W && C != 0) {
            for (int g = ln.j; g < ng; g += BP) {
                double *gx = wn.gx + g * (c + 1);
                if (gx[c] > 0.0) continue;
                const int q0 = nth_bit(gheads, g), q1 = next_bit(gheads, q0, n);
                for (int k = 0; k < c; k++) gx[k] = 0.0;
                for (int t = q0 * c; t < q1 * c; t++) wn.x[t] = 0.0;
            }
            __syncwarp(ln.mask);
        }
    };
    auto window = [&](int64_t, int64_t i0, int n, unsigned gheads, int ng) {
        const unsigned heads = load_window<BP, C, W>(a, ln, wn, i0, n, &sq) | gheads;
        group_sums<BP, C, W>(a, ln, wn, gheads, ng, n);
        drop_weightless(gheads, ng, n);
        const uint32_t word = window_signs(a, i0, n, dterm);
        cov_rows(word, n);
        int q0 = 0;
        for (int g = 0; g < ng; g++) {
            const int q1 = next_bit(gheads, q0, n);
            double tot, sw;
            sums(word, q0, q1, tot, sw);
            const double mean = sw > 0.0 ? tot / sw : 0.0;
#pragma unroll
            for (int k = 0; k < CM; k++) {
                if (k >= c) break;
                ax[k] -= wn.gx[g * (c + 1) + k] * mean;
            }
            for (int p0 = q0; p0 < q1;) {
                const int p1 = next_bit(heads, p0, q1);
                double rt, rw;
                sums(word, p0, p1, rt, rw);
                if (sw > 0.0) flush(p0, rt - rw * mean);
                p0 = p1;
            }
            q0 = q1;
        }
    };
    auto lone = [&](int64_t, int64_t s, int64_t e) {
        double tot = 0.0, sw = 0.0;
        for (int64_t i0 = s; i0 < e; i0 += kWin) {
            const int n = (int)min((int64_t)kWin, e - i0);
            load_window<BP, C, W>(a, ln, wn, i0, n, nullptr);
            double t, w;
            sums(window_signs(a, i0, n, dterm), 0, n, t, w);
            tot += t;
            sw += w;
            __syncwarp(ln.mask);
        }
        const double mean = sw > 0.0 ? tot / sw : 0.0;
        for (int64_t i0 = s; i0 < e; i0 += kWin) {
            const int n = (int)min((int64_t)kWin, e - i0);
            const unsigned heads = load_window<BP, C, W>(a, ln, wn, i0, n, &sq);
            if (W && !(sw > 0.0)) {         // as drop_weightless
                __syncwarp(ln.mask);
                continue;
            }
            group_sums<BP, C, W>(a, ln, wn, 1u, 1, n);
            const uint32_t word = window_signs(a, i0, n, dterm);
            cov_rows(word, n);
#pragma unroll
            for (int k = 0; k < CM; k++) {
                if (k >= c) break;
                ax[k] -= wn.gx[k] * mean;
            }
            for (int p0 = 0; p0 < n;) {
                const int p1 = next_bit(heads, p0, n);
                double rt, rw;
                sums(word, p0, p1, rt, rw);
                if (sw > 0.0) flush(p0, rt - rw * mean);
                p0 = p1;
            }
            __syncwarp(ln.mask);
        }
    };
    walk(a, ln, window, lone);
    // the covariate block and the sums of squares (the same for every draw)
    if (a.acc_x && ln.on) {
#pragma unroll
        for (int k = 0; k < CM; k++) {
            if (k >= c) break;
            atomicAdd(a.acc_x + k * a.B + ln.j, ax[k]);
        }
    }
    if (a.squares) {
#pragma unroll
        for (int o = BP / 2; o > 0; o >>= 1) sq += __shfl_xor_sync(ln.mask, sq, o, BP);
        if (ln.on) atomicAdd(a.squares + ln.j, sq);
    }
    __syncthreads();
    for (int d = 0; d < a.D; d++) {
        if (!a.small[d]) continue;
        for (int64_t q = threadIdx.x; q < a.nlev[d] * a.B; q += kPassThreads) {
            const double v = s_acc[a.soff[d] * a.B + q];
            if (v != 0.0) atomicAdd(a.acc + a.offs[d] * a.B + q, v);
        }
    }
}

template <int BP, int C, bool W>
struct Center {
    static constexpr bool kTile = false;
    static void (*kernel())(Args) { return k_center_draws<BP, C, W>; }
};

int launch_center_draws(Args &a, cudaStream_t s) { return launch_draws<Center>(a, s); }

}  // namespace rows
}  // namespace hdfe
