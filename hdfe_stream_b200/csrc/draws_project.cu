// The projection pass over Rademacher draws and the JLA sink (draws.cuh).
#include "draws.cuh"

namespace hdfe {
namespace rows {

template <int BP, int C, bool W>
__global__ void __launch_bounds__(kPassThreads) k_project_draws(Args a)
{
    extern __shared__ __align__(16) char s_raw[];
    const Lanes<BP> ln(a.B);
    const int c = C < 0 ? a.c : C;
    constexpr int CM = C < 0 ? kMaxCov : (C > 0 ? C : 1);
    constexpr int LD = BP + 1;
    Win<BP> wn(s_raw + (threadIdx.x / BP) * Win<BP>::bytes(c, a.D, W, true), c, a.D, W, true);
    const uint64_t dterm = (uint64_t)(a.first_draw + ln.j) * kDrawMul;
    double Cj[CM];
#pragma unroll
    for (int k = 0; k < CM; k++) Cj[k] = k < c && ln.on ? a.C[k * a.B + ln.j] : 0.0;
    double *col = wn.tile + ln.j;               // this lane's column, stride LD
    auto gather = [&](int q) {                  // sum_d U[level_d, j] of row q's run
        double h = 0.0;
#pragma unroll
        for (int d = 0; d < HDFE_MAX_DIMS; d++) {
            if (d >= a.D) break;
            h += a.U[(a.offs[d] + wn.codes[q * a.D + d]) * a.B + ln.j];
        }
        return h;
    };
    // hU of every run into the tile at its head row; the first eight runs'
    // loads are in flight while the signs are hashed
    auto runs_and_signs = [&](int64_t i0, int n, unsigned heads) -> uint32_t {
        constexpr int F = 8;
        double h[F];
        unsigned m = heads;
#pragma unroll
        for (int f = 0; f < F; f++) {
            h[f] = m && ln.on ? gather(__ffs(m) - 1) : 0.0;
            m &= m - 1;
        }
        const uint32_t word = window_signs(a, i0, n, dterm);
        unsigned m2 = heads;
#pragma unroll
        for (int f = 0; f < F; f++) {
            if (m2) col[(__ffs(m2) - 1) * LD] = h[f];
            m2 &= m2 - 1;
        }
        for (; m; m &= m - 1) {
            const int q = __ffs(m) - 1;
            col[q * LD] = ln.on ? gather(q) : 0.0;
        }
        return word;
    };
    // sum over rows [q0, q1) of w (r - hU), and of w
    auto sums = [&](uint32_t word, unsigned heads, int q0, int q1, double &tot, double &sw) {
        tot = sw = 0.0;
        for (int p0 = q0; p0 < q1;) {
            const int p1 = next_bit(heads, p0, q1);
            const double h = col[p0 * LD];
            if (W) {
                double rw = 0.0;
                for (int q = p0; q < p1; q++) {
                    tot += flip(wn.wr[q], word, q);
                    rw += wn.w[q];
                }
                tot -= rw * h;
                sw += rw;
            } else {
                const unsigned m = below(p1) & ~below(p0);
                tot += (double)(p1 - p0 - 2 * __popc(word & m)) - (double)(p1 - p0) * h;
            }
            p0 = p1;
        }
        if (!W) sw = (double)(q1 - q0);
    };
    // rows [q0, q1) of one group: o = hU + mean + x C, r o into the tile
    auto emit = [&](uint32_t word, unsigned heads, int64_t i0, int q0, int q1, double mean) {
        for (int p0 = q0; p0 < q1;) {
            const int p1 = next_bit(heads, p0, q1);
            const double base = col[p0 * LD] + mean;
#pragma unroll 4
            for (int q = p0; q < p1; q++) {
                double o = base;
#pragma unroll
                for (int k = 0; k < CM; k++) {
                    if (k >= c) break;
                    o += wn.x[q * c + k] * Cj[k];
                }
                if (W && a.sqrt_weights) o *= wn.root[q];
                if (a.out && ln.on) a.out[(i0 + q) * a.B + ln.j] = o;
                col[q * LD] = flip(o, word, q);
            }
            p0 = p1;
        }
    };
    auto flush = [&](int64_t i0, int n) {       // lane t: row t's sums over the draws
        if (!a.moments) return;
        __syncwarp(ln.mask);
        for (int t = ln.j; t < n; t += BP) {
            double *mom = a.moments + i0 + t;
            double m0 = 0.0, m1 = 0.0, m2 = 0.0, m3 = 0.0, m4 = 0.0;
            const double b0 = mom[0], b1 = mom[a.N], b2 = mom[2 * a.N], b3 = mom[3 * a.N],
                         b4 = mom[4 * a.N];
            const double *row = wn.tile + t * LD;
#pragma unroll 8
            for (int k = 0; k < a.B; k++) {
                const double x = row[k], P = x * x, y = 1.0 - x, M = y * y;
                m0 += P;
                m1 += M;
                m2 += P * P;
                m3 += M * M;
                m4 += P * M;
            }
            mom[0] = b0 + m0;
            mom[a.N] = b1 + m1;
            mom[2 * a.N] = b2 + m2;
            mom[3 * a.N] = b3 + m3;
            mom[4 * a.N] = b4 + m4;
        }
    };
    auto window = [&](int64_t, int64_t i0, int n, unsigned gheads, int ng) {
        const unsigned heads = load_window<BP, C, W>(a, ln, wn, i0, n, nullptr) | gheads;
        group_sums<BP, C, W>(a, ln, wn, gheads, ng, n);
        const uint32_t word = runs_and_signs(i0, n, heads);
        int q0 = 0;
        for (int g = 0; g < ng; g++) {
            const int q1 = next_bit(gheads, q0, n);
            double tot, sw;
            sums(word, heads, q0, q1, tot, sw);
#pragma unroll
            for (int k = 0; k < CM; k++) {
                if (k >= c) break;
                tot -= wn.gx[g * (c + 1) + k] * Cj[k];
            }
            emit(word, heads, i0, q0, q1, sw > 0.0 ? tot / sw : 0.0);
            q0 = q1;
        }
        flush(i0, n);
    };
    auto lone = [&](int64_t, int64_t s, int64_t e) {
        double tot = 0.0, sw = 0.0;
        for (int64_t i0 = s; i0 < e; i0 += kWin) {
            const int n = (int)min((int64_t)kWin, e - i0);
            const unsigned heads = load_window<BP, C, W>(a, ln, wn, i0, n, nullptr);
            group_sums<BP, C, W>(a, ln, wn, 1u, 1, n);
            double t, w;
            sums(runs_and_signs(i0, n, heads), heads, 0, n, t, w);
            tot += t;
            sw += w;
#pragma unroll
            for (int k = 0; k < CM; k++) {
                if (k >= c) break;
                tot -= wn.gx[k] * Cj[k];
            }
            __syncwarp(ln.mask);
        }
        const double mean = sw > 0.0 ? tot / sw : 0.0;
        for (int64_t i0 = s; i0 < e; i0 += kWin) {
            const int n = (int)min((int64_t)kWin, e - i0);
            const unsigned heads = load_window<BP, C, W>(a, ln, wn, i0, n, nullptr);
            emit(runs_and_signs(i0, n, heads), heads, i0, 0, n, mean);
            flush(i0, n);
            __syncwarp(ln.mask);
        }
    };
    walk(a, ln, window, lone);
}

template <int BP, int C, bool W>
struct Project {
    static constexpr bool kTile = true;
    static void (*kernel())(Args) { return k_project_draws<BP, C, W>; }
};

int launch_project_draws(Args &a, cudaStream_t s) { return launch_draws<Project>(a, s); }

}  // namespace rows
}  // namespace hdfe
