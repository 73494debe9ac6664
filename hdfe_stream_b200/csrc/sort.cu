// Pass 0 on the device: a stable LSD radix sort of 64-bit keys with int32
// payloads, and factorization (the rank of each id among the distinct ids).
//
// Reference: core/passes.py:285-294 codes each fixed effect by the rank of
// its level among the sorted distinct levels, and :359-373 sorts the rows by
// (streamed code, other codes, variables).  The sort here is the one the
// reference's ordering needs: stable, 8 bits per pass over the key's low
// `key_bits` bits (the bits that can be nonzero), so a multi-key order is a
// sequence of sorts, least significant key first.
//   Per pass, tiles of kTile items:
//     hist      each CTA counts its tile's digits (shared-memory histogram)
//               into counts[digit * tiles + tile] (digit-major);
//     scan      exclusive offsets of counts in that order (per-CTA sums, a
//               one-CTA scan of those, then the offsets applied), so digit d
//               of tile t starts after every smaller digit and every earlier
//               tile's d: the order is stable;
//     scatter   a warp holds kItems rounds of 32 consecutive items in
//               registers; an item's place among its tile's equal digits is
//               the count in earlier warps, in its warp's earlier rounds (a
//               counter per warp and digit in shared memory) and in earlier
//               lanes of its round (__match_any_sync), so equal digits keep
//               their order.  The tile is then put in digit order in shared
//               memory and written from there: runs of consecutive output
//               slots instead of one sector an item, which bounded the pass
//               (142 -> 86 us for 8.5M pairs).
//   The first pass reads the caller's keys and numbers the values itself when
// there are none; the last writes the caller's output.
// Factorize: the (id, position) pairs sorted by id; a run head marks each
// distinct id; an exclusive scan of the heads gives the ranks, scattered back
// to the positions; the distinct ids are written in order.  Ids of a small
// range need no sort: a bitmap of the ids present, its words' exclusive bit
// counts, and the rank of an id is its word's count plus the bits below its
// own (hdfe_factorize_range).
#include <algorithm>
#include <cuda_runtime.h>

#include "common.cuh"

namespace hdfe {
namespace sorting {

constexpr int kThreads = 256;
constexpr int kItems = 16;              // items per thread per tile (the scatter's 48 KB
                                        // tile and 11 KB of counts: three CTAs an SM)
constexpr int kTile = kThreads * kItems;
constexpr int kBins = 256;
constexpr int kWarps = kThreads / 32;

__global__ void __launch_bounds__(kThreads) k_hist(const uint64_t *keys, int64_t n, int shift,
                                                   int64_t tiles, uint32_t *counts)
{
    __shared__ uint32_t s_h[kBins];
    s_h[threadIdx.x] = 0;
    __syncthreads();
    const int64_t t0 = (int64_t)blockIdx.x * kTile;
    const int64_t t1 = min(t0 + kTile, n);
    for (int64_t i = t0 + threadIdx.x; i < t1; i += kThreads)
        atomicAdd(s_h + ((keys[i] >> shift) & 0xFF), 1u);
    __syncthreads();
    counts[(int64_t)threadIdx.x * tiles + blockIdx.x] = s_h[threadIdx.x];
}

// exclusive scan of x (n) into out, 3 kernels: per-CTA sums of kTile-item
// chunks, a scan of those (one CTA), then each chunk's scan with its offset
__global__ void __launch_bounds__(kThreads) k_scan_sums(const uint32_t *x, int64_t n,
                                                        int64_t *sums)
{
    __shared__ int64_t s_w[kWarps];
    const int64_t t0 = (int64_t)blockIdx.x * kTile;
    int64_t v = 0;
    for (int64_t i = t0 + threadIdx.x; i < min(t0 + kTile, n); i += kThreads) v += x[i];
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        int64_t t = 0;
        for (int w = 0; w < kWarps; w++) t += s_w[w];
        sums[blockIdx.x] = t;
    }
}

__global__ void __launch_bounds__(1024) k_scan_top(int64_t *sums, int64_t m, int64_t *total)
{
    cta_exclusive_scan<1024>(sums, m, total);
}

__global__ void __launch_bounds__(kThreads) k_scan_apply(const uint32_t *x, int64_t n,
                                                         const int64_t *sums, int64_t *out)
{
    __shared__ int64_t s_w[kWarps + 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t t0 = (int64_t)blockIdx.x * kTile;
    int64_t run = sums[blockIdx.x];
    for (int64_t b = t0; b < min(t0 + kTile, n); b += kThreads) {
        const int64_t i = b + threadIdx.x;
        const int64_t v = i < n ? x[i] : 0;
        int64_t inc = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += y;
        }
        if (lane == 31) s_w[warp] = inc;
        __syncthreads();
        if (threadIdx.x == 0) {
            int64_t r = 0;
            for (int w = 0; w < kWarps; w++) { const int64_t t = s_w[w]; s_w[w] = r; r += t; }
            s_w[kWarps] = r;
        }
        __syncthreads();
        if (i < n) out[i] = run + s_w[warp] + inc - v;
        run += s_w[kWarps];
        __syncthreads();
    }
}

// vals null: the items' positions
__global__ void __launch_bounds__(kThreads) k_scatter(const uint64_t *keys, const int32_t *vals,
                                                      int64_t n, int shift, int64_t tiles,
                                                      const int64_t *offsets, uint64_t *keys_out,
                                                      int32_t *vals_out)
{
    extern __shared__ __align__(16) char s_raw[];
    uint64_t *s_key = reinterpret_cast<uint64_t *>(s_raw);              // the tile in digit order
    int32_t *s_val = reinterpret_cast<int32_t *>(s_key + kTile);
    __shared__ uint32_t s_warp[kWarps][kBins];      // items of the digit per warp, then before it
    __shared__ uint32_t s_total[kWarps];
    __shared__ uint32_t s_start[kBins];             // the digit's first place in the tile
    __shared__ int64_t s_off[kBins];                // and its output slot less that place
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t t0 = (int64_t)blockIdx.x * kTile;
    const int m = (int)min((int64_t)kTile, n - t0);
    for (int w = 0; w < kWarps; w++) s_warp[w][threadIdx.x] = 0;
    uint64_t k[kItems];
    int32_t v[kItems];
    uint16_t place[kItems];             // among the warp's items of the digit
#pragma unroll
    for (int r = 0; r < kItems; r++) {
        const int q = warp * (32 * kItems) + r * 32 + lane;
        k[r] = q < m ? keys[t0 + q] : 0;
        v[r] = vals ? (q < m ? vals[t0 + q] : 0) : (int32_t)(t0 + q);
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kItems; r++) {
        const bool valid = warp * (32 * kItems) + r * 32 + lane < m;
        const unsigned d = valid ? (unsigned)((k[r] >> shift) & 0xFF) : kBins;  // kBins: none
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        const int below = __popc(peers & ((1u << lane) - 1));
        uint32_t before = 0;
        if (valid) before = s_warp[warp][d];
        place[r] = (uint16_t)(before + below);
        __syncwarp();
        if (valid && below == 0) s_warp[warp][d] = before + __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    // thread d: the digit's counts made exclusive over the warps, its total
    // scanned over the digits
    uint32_t total = 0;
    for (int w = 0; w < kWarps; w++) {
        const uint32_t c = s_warp[w][threadIdx.x];
        s_warp[w][threadIdx.x] = total;
        total += c;
    }
    uint32_t inc = total;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    if (lane == 31) s_total[warp] = inc;
    __syncthreads();
    uint32_t start = inc - total;
    for (int w = 0; w < warp; w++) start += s_total[w];
    s_start[threadIdx.x] = start;
    s_off[threadIdx.x] = offsets[(int64_t)threadIdx.x * tiles + blockIdx.x] - start;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kItems; r++) {
        if (warp * (32 * kItems) + r * 32 + lane >= m) continue;
        const unsigned d = (unsigned)((k[r] >> shift) & 0xFF);
        const uint32_t at = s_start[d] + s_warp[warp][d] + place[r];
        s_key[at] = k[r];
        s_val[at] = v[r];
    }
    __syncthreads();
    for (int q = threadIdx.x; q < m; q += kThreads) {
        const uint64_t x = s_key[q];
        const int64_t at = s_off[(x >> shift) & 0xFF] + q;
        keys_out[at] = x;
        vals_out[at] = s_val[q];
    }
}

// heads[i] = 1 where the sorted ids change (and at 0)
__global__ void __launch_bounds__(kThreads) k_heads(const uint64_t *ids, int64_t n,
                                                    uint32_t *heads)
{
    for (int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * kThreads)
        heads[i] = (i == 0 || ids[i] != ids[i - 1]) ? 1u : 0u;
}

// the rank of sorted item i is (exclusive scan of heads)[i] + heads[i] - 1
__global__ void __launch_bounds__(kThreads) k_ranks(const uint64_t *ids, const int32_t *pos,
                                                    const uint32_t *heads, const int64_t *excl,
                                                    int64_t n, int32_t *codes, uint64_t *levels,
                                                    int64_t *n_levels)
{
    for (int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * kThreads) {
        const int64_t r = excl[i] + heads[i] - 1;
        codes[pos[i]] = (int32_t)r;
        if (heads[i] && levels) levels[r] = ids[i];
        if (i == n - 1) *n_levels = r + 1;
    }
}

__global__ void __launch_bounds__(kThreads) k_iota(int32_t *v, int64_t n)
{
    for (int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * kThreads)
        v[i] = (int32_t)i;
}

struct Work {       // workspace layout
    uint64_t *keys[2];
    int32_t *vals[2];
    uint32_t *counts;
    int64_t *offsets;
    int64_t *sums;
    int64_t tiles, ncounts, nsums;
};

inline int64_t align256(int64_t b) { return (b + 255) / 256 * 256; }

inline Work layout(void *ws, int64_t n)
{
    Work w;
    w.tiles = (n + kTile - 1) / kTile;
    w.ncounts = w.tiles * kBins;
    // chunk sums for either scan: the counts (ncounts entries) or n heads
    w.nsums = std::max((w.ncounts + kTile - 1) / kTile, w.tiles);
    char *p = (char *)ws;
    auto take = [&](int64_t bytes) { char *at = p; p += align256(bytes); return at; };
    w.keys[0] = (uint64_t *)take(n * 8);
    w.keys[1] = (uint64_t *)take(n * 8);
    w.vals[0] = (int32_t *)take(n * 4);
    w.vals[1] = (int32_t *)take(n * 4);
    w.counts = (uint32_t *)take(w.ncounts * 4);
    w.offsets = (int64_t *)take(std::max(w.ncounts, n) * 8);
    w.sums = (int64_t *)take(w.nsums * 8 + 8);      // and the total
    return w;
}

inline int64_t layout_bytes(int64_t n)
{
    const int64_t tiles = (n + kTile - 1) / kTile, nc = tiles * kBins;
    const int64_t ns = std::max((nc + kTile - 1) / kTile, tiles);
    return 2 * align256(n * 8) + 2 * align256(n * 4) + align256(nc * 4) +
           align256(std::max(nc, n) * 8) + align256(ns * 8 + 8);
}

// exclusive scan of x (m entries) into out
inline void scan(const uint32_t *x, int64_t m, int64_t *sums, int64_t *out, cudaStream_t s)
{
    const int64_t chunks = (m + kTile - 1) / kTile;
    k_scan_sums<<<(unsigned)chunks, kThreads, 0, s>>>(x, m, sums);
    k_scan_top<<<1, 1024, 0, s>>>(sums, chunks, sums + chunks);
    k_scan_apply<<<(unsigned)chunks, kThreads, 0, s>>>(x, m, sums, out);
}

constexpr int kScatterSmem = kTile * 12;

// sort (keys, vals) -- vals null: the positions -- by the low key_bits bits into
// keys_out, vals_out (not the inputs)
int radix_sort(Work &w, const uint64_t *keys, const int32_t *vals, int64_t n, int key_bits,
               uint64_t *keys_out, int32_t *vals_out, cudaStream_t s)
{
    const unsigned tiles = (unsigned)w.tiles;
    const int passes = (key_bits + 7) / 8;
    if (passes == 0) {
        HDFE_CUDA_TRY(cudaMemcpyAsync(keys_out, keys, n * 8, cudaMemcpyDeviceToDevice, s));
        if (vals) {
            HDFE_CUDA_TRY(cudaMemcpyAsync(vals_out, vals, n * 4, cudaMemcpyDeviceToDevice, s));
        } else {
            k_iota<<<(unsigned)std::min<int64_t>((n + kThreads - 1) / kThreads, 148 * 32),
                     kThreads, 0, s>>>(vals_out, n);
            hdfe_add_launches(1);
        }
        return HDFE_OK;
    }
    HDFE_CUDA_TRY(cudaFuncSetAttribute(k_scatter, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       kScatterSmem));
    for (int p = 0; p < passes; p++) {
        uint64_t *ko = p == passes - 1 ? keys_out : w.keys[p & 1];
        int32_t *vo = p == passes - 1 ? vals_out : w.vals[p & 1];
        k_hist<<<tiles, kThreads, 0, s>>>(keys, n, 8 * p, w.tiles, w.counts);
        scan(w.counts, w.ncounts, w.sums, w.offsets, s);
        k_scatter<<<tiles, kThreads, kScatterSmem, s>>>(keys, vals, n, 8 * p, w.tiles, w.offsets,
                                                        ko, vo);
        keys = ko;
        vals = vo;
        hdfe_add_launches(5);
    }
    return HDFE_OK;
}

// ------------------------------------------- factorize by a bitmap of the ids

template <typename T>
__global__ void __launch_bounds__(kThreads) k_mark(const T *ids, int64_t n, int64_t lo,
                                                   int64_t range, uint32_t *bits,
                                                   unsigned *status)
{
#pragma unroll 4
    for (int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * kThreads) {
        const int64_t x = (int64_t)ids[i] - lo;
        if (x < 0 || x >= range) { atomicCAS(status, 0u, (unsigned)HDFE_ERR_BAD_CODE); continue; }
        const uint32_t b = 1u << (x & 31);
        if (!(bits[x >> 5] & b)) atomicOr(bits + (x >> 5), b);
    }
}

__global__ void __launch_bounds__(kThreads) k_popc(const uint32_t *bits, int64_t words,
                                                   uint32_t *count)
{
    for (int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x; i < words;
         i += (int64_t)gridDim.x * kThreads)
        count[i] = __popc(bits[i]);
}

// the distinct ids in order, and their number
__global__ void __launch_bounds__(kThreads) k_present(const uint32_t *bits, const int64_t *rank,
                                                      int64_t words, int64_t lo, int64_t *levels,
                                                      int64_t *n_levels)
{
    for (int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x; i < words;
         i += (int64_t)gridDim.x * kThreads) {
        int64_t r = rank[i];
        for (uint32_t m = bits[i]; m; m &= m - 1) levels[r++] = lo + i * 32 + __ffs(m) - 1;
        if (i == words - 1) *n_levels = r;
    }
}

template <typename T>
__global__ void __launch_bounds__(kThreads) k_rank_of(const T *ids, int64_t n, int64_t lo,
                                                      int64_t range, const uint32_t *bits,
                                                      const int64_t *rank, int32_t *codes)
{
#pragma unroll 4
    for (int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * kThreads) {
        const int64_t x = (int64_t)ids[i] - lo;
        if (x < 0 || x >= range) continue;
        const int64_t w = x >> 5;
        codes[i] = (int32_t)(rank[w] + __popc(bits[w] & ((1u << (x & 31)) - 1u)));
    }
}

// ------------------------------------------------------- rows from the order

constexpr int kMaxCols = 8;

struct PackArgs {
    const int32_t *cols[kMaxCols];
    int shift[kMaxCols], bits[kMaxCols];
    int n_cols;
    int64_t n;
};

__global__ void __launch_bounds__(kThreads) k_pack(PackArgs a, uint64_t *keys)
{
    for (int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x; i < a.n;
         i += (int64_t)gridDim.x * kThreads) {
        uint64_t k = 0;
#pragma unroll
        for (int c = 0; c < kMaxCols; c++) {
            if (c >= a.n_cols) break;
            k |= (uint64_t)(uint32_t)a.cols[c][i] << a.shift[c];
        }
        keys[i] = k;
    }
}

// The sorted rows: group codes and the D codes after it out of the sorted
// keys, the variables (N, m) and weights gathered in the order, one variable
// contiguous; *ties = 1 when two neighbours have one key.
__global__ void __launch_bounds__(kThreads) k_rows(PackArgs a, int D, const uint64_t *keys,
                                                   const int32_t *order, const double *V, int m,
                                                   const double *w, int32_t *gcode,
                                                   int32_t *codes, double *V_out, double *w_out,
                                                   int32_t *ties)
{
    for (int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x; i < a.n;
         i += (int64_t)gridDim.x * kThreads) {
        const uint64_t k = keys[i];
        if (i > 0 && keys[i - 1] == k) *ties = 1;
        const int64_t o = order[i];
        gcode[i] = (int32_t)((k >> a.shift[0]) & ((1ull << a.bits[0]) - 1));
        for (int d = 0; d < D; d++)
            codes[i * D + d] = (int32_t)((k >> a.shift[1 + d]) & ((1ull << a.bits[1 + d]) - 1));
#pragma unroll 4
        for (int j = 0; j < m; j++) V_out[(int64_t)j * a.n + i] = V[o * m + j];
        if (w) w_out[i] = w[o];
    }
}

inline unsigned grid_for(int64_t n)
{
    return (unsigned)std::min<int64_t>((n + kThreads - 1) / kThreads, 148 * 32);
}

}  // namespace sorting
}  // namespace hdfe

using namespace hdfe;

extern "C" int64_t hdfe_sort_workspace_bytes(int64_t n)
{
    return n < 0 ? -1 : sorting::layout_bytes(n > 0 ? n : 1);
}

extern "C" int hdfe_sort_pairs(const uint64_t *keys, const int32_t *vals, int64_t n,
                               int32_t key_bits, uint64_t *keys_out, int32_t *vals_out,
                               void *workspace, int64_t workspace_bytes, void *stream)
{
    if (!keys || !keys_out || !vals_out || !workspace || n < 0 || key_bits < 0 || key_bits > 64 ||
        n > INT32_MAX)
        return hdfe_set_arg_error("hdfe_sort_pairs: bad argument");
    if (workspace_bytes < hdfe_sort_workspace_bytes(n))
        return hdfe_set_error(HDFE_ERR_WORKSPACE, "hdfe_sort_pairs: workspace too small");
    if (n == 0) return HDFE_OK;
    cudaStream_t s = (cudaStream_t)stream;
    sorting::Work w = sorting::layout(workspace, n);
    // an output over an input: one pass (or none) would write what it still reads
    auto meet = [](const void *a, int64_t a_bytes, const void *b, int64_t b_bytes) {
        const char *x = (const char *)a, *y = (const char *)b;
        return a && x < y + b_bytes && y < x + a_bytes;
    };
    auto over = [&](const void *out, int64_t out_bytes) {
        return meet(keys, n * 8, out, out_bytes) || meet(vals, n * 4, out, out_bytes);
    };
    if (key_bits <= 8 && (over(keys_out, n * 8) || over(vals_out, n * 4))) {
        HDFE_CUDA_TRY(cudaMemcpyAsync(w.keys[1], keys, n * 8, cudaMemcpyDeviceToDevice, s));
        keys = w.keys[1];
        if (vals) {
            HDFE_CUDA_TRY(cudaMemcpyAsync(w.vals[1], vals, n * 4, cudaMemcpyDeviceToDevice, s));
            vals = w.vals[1];
        }
    }
    const int st = sorting::radix_sort(w, keys, vals, n, key_bits, keys_out, vals_out, s);
    if (st != HDFE_OK) return st;
    HDFE_CUDA_TRY(cudaGetLastError());
    return HDFE_OK;
}

extern "C" int hdfe_factorize(const uint64_t *ids, int64_t n, int32_t key_bits, int32_t *codes,
                              uint64_t *levels, int64_t *n_levels, void *workspace,
                              int64_t workspace_bytes, void *stream)
{
    if (!ids || !codes || !n_levels || !workspace || n < 1 || key_bits < 0 || key_bits > 64 ||
        n > INT32_MAX)
        return hdfe_set_arg_error("hdfe_factorize: bad argument");
    if (workspace_bytes < hdfe_sort_workspace_bytes(n))
        return hdfe_set_error(HDFE_ERR_WORKSPACE, "hdfe_factorize: workspace too small");
    cudaStream_t s = (cudaStream_t)stream;
    sorting::Work w = sorting::layout(workspace, n);
    const unsigned grid = sorting::grid_for(n);
    // the passes end in the buffers that the last of them does not read
    const int last = ((key_bits + 7) / 8 + 1) & 1;
    const int st = sorting::radix_sort(w, ids, nullptr, n, key_bits, w.keys[last], w.vals[last], s);
    if (st != HDFE_OK) return st;
    // the heads in the spare key buffer (n x 8 bytes), their scan in offsets
    uint32_t *heads = reinterpret_cast<uint32_t *>(w.keys[1 - last]);
    sorting::k_heads<<<grid, sorting::kThreads, 0, s>>>(w.keys[last], n, heads);
    sorting::scan(heads, n, w.sums, w.offsets, s);
    sorting::k_ranks<<<grid, sorting::kThreads, 0, s>>>(w.keys[last], w.vals[last], heads,
                                                        w.offsets, n, codes, levels, n_levels);
    HDFE_CUDA_TRY(cudaGetLastError());
    hdfe_add_launches(5);
    return HDFE_OK;
}

// ids of a small range: bitmap, word counts, their scan
extern "C" int64_t hdfe_factorize_range_workspace_bytes(int64_t range)
{
    if (range < 1 || range >= (int64_t)1 << 40) return -1;
    const int64_t words = (range + 31) / 32;
    return 256 + 2 * sorting::align256(words * 4) + sorting::align256(words * 8) +
           sorting::align256(((words + sorting::kTile - 1) / sorting::kTile + 1) * 8);
}

extern "C" int hdfe_factorize_range(const void *ids, int32_t id_bytes, int64_t n, int64_t lo,
                                    int64_t range, int32_t *codes, int64_t *levels,
                                    int64_t *n_levels, void *workspace, int64_t workspace_bytes,
                                    void *stream)
{
    if (!ids || (id_bytes != 4 && id_bytes != 8) || n < 1 || n > INT32_MAX || range < 1 ||
        !codes || !levels || !n_levels || !workspace)
        return hdfe_set_arg_error("hdfe_factorize_range: bad argument");
    const int64_t need = hdfe_factorize_range_workspace_bytes(range);
    if (need < 0) return hdfe_set_arg_error("hdfe_factorize_range: range must be below 2^40");
    if (workspace_bytes < need)
        return hdfe_set_error(HDFE_ERR_WORKSPACE, "hdfe_factorize_range: workspace too small");
    cudaStream_t s = (cudaStream_t)stream;
    using namespace sorting;
    const int64_t words = (range + 31) / 32;
    char *p = (char *)workspace;
    unsigned *status = (unsigned *)p;       // an id outside [lo, lo + range)
    uint32_t *bits = (uint32_t *)(p + 256);
    uint32_t *count = (uint32_t *)((char *)bits + align256(words * 4));
    int64_t *rank = (int64_t *)((char *)count + align256(words * 4));
    int64_t *sums = (int64_t *)((char *)rank + align256(words * 8));
    HDFE_CUDA_TRY(cudaMemsetAsync(workspace, 0, 256 + words * 4, s));
    const unsigned gi = grid_for(n), gw = grid_for(words);
    if (id_bytes == 4) k_mark<<<gi, kThreads, 0, s>>>((const int32_t *)ids, n, lo, range, bits, status);
    else k_mark<<<gi, kThreads, 0, s>>>((const int64_t *)ids, n, lo, range, bits, status);
    k_popc<<<gw, kThreads, 0, s>>>(bits, words, count);
    scan(count, words, sums, rank, s);
    k_present<<<gw, kThreads, 0, s>>>(bits, rank, words, lo, levels, n_levels);
    if (id_bytes == 4) k_rank_of<<<gi, kThreads, 0, s>>>((const int32_t *)ids, n, lo, range, bits, rank, codes);
    else k_rank_of<<<gi, kThreads, 0, s>>>((const int64_t *)ids, n, lo, range, bits, rank, codes);
    HDFE_CUDA_TRY(cudaGetLastError());
    hdfe_add_launches(7);
    return HDFE_OK;
}

namespace {

// columns packed most significant first; false when they are not 64 bits or less
bool pack_args(sorting::PackArgs &a, const int32_t *const *cols, const int32_t *bits,
               int32_t n_cols, int64_t n)
{
    a = sorting::PackArgs{};
    int total = 0;
    for (int c = n_cols - 1; c >= 0; c--) {
        if (bits[c] < 1 || bits[c] > 31 || (cols && !cols[c])) return false;
        a.cols[c] = cols ? cols[c] : nullptr;
        a.shift[c] = total;
        a.bits[c] = bits[c];
        total += bits[c];
    }
    a.n_cols = n_cols;
    a.n = n;
    return total <= 64;
}

}  // namespace

extern "C" int hdfe_pack_codes(const int32_t *const *cols, const int32_t *bits, int32_t n_cols,
                               int64_t n, uint64_t *keys, void *stream)
{
    sorting::PackArgs a;
    if (!cols || !bits || n_cols < 1 || n_cols > sorting::kMaxCols || n < 0 || !keys ||
        !pack_args(a, cols, bits, n_cols, n))
        return hdfe_set_arg_error("hdfe_pack_codes: bad argument");
    if (n == 0) return HDFE_OK;
    sorting::k_pack<<<sorting::grid_for(n), sorting::kThreads, 0, (cudaStream_t)stream>>>(a, keys);
    HDFE_CUDA_TRY(cudaGetLastError());
    hdfe_add_launches(1);
    return HDFE_OK;
}

extern "C" int hdfe_rows_from_order(const int32_t *bits, int32_t n_cols, int32_t D, int64_t n,
                                    const uint64_t *keys, const int32_t *order, const double *V,
                                    int32_t m, const double *w, int32_t *gcode, int32_t *codes,
                                    double *V_out, double *w_out, int32_t *ties, void *stream)
{
    sorting::PackArgs a;
    if (!bits || n_cols < 1 || n_cols > sorting::kMaxCols || D < 0 || D >= n_cols || n < 0 ||
        m < 0 || !keys || !order || (m > 0 && (!V || !V_out)) || !gcode || (D > 0 && !codes) ||
        (w && !w_out) || !ties || !pack_args(a, nullptr, bits, n_cols, n))
        return hdfe_set_arg_error("hdfe_rows_from_order: bad argument");
    cudaStream_t s = (cudaStream_t)stream;
    HDFE_CUDA_TRY(cudaMemsetAsync(ties, 0, 4, s));
    if (n == 0) return HDFE_OK;
    sorting::k_rows<<<sorting::grid_for(n), sorting::kThreads, 0, s>>>(
        a, D, keys, order, V, m, w, gcode, codes, V_out, w_out, ties);
    HDFE_CUDA_TRY(cudaGetLastError());
    hdfe_add_launches(1);
    return HDFE_OK;
}
