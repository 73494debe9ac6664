// Connected components of the bipartite network of two fixed effects, with
// the min_degree core: core/connected.py:378-493 `_find_components` on coded
// rows, with core/kernels_graph.py:188-221 `_nb_peel`, :225-241
// `_nb_union_keys`, :244-266 `_nb_dense_labels` and :277-289 `_nb_pair_rows`
// (and `_DistinctPairs`, core/connected.py:656-687).
//
// Rows come in pass 0's order, sorted by the first dimension and then the
// second, so the distinct (a, b) pairs are runs of rows:
//   pair_heads / pair_write   tile counts of run heads, one scan, the heads'
//                             rows -> pairs a[P], b[P], count[P] in key order
//   peel rounds               per round, the degrees of every level over the
//                             pairs whose two levels are alive, then every
//                             level under its threshold removed at once; the
//                             host repeats until a round removes nothing
//                             (`_nb_peel`'s rounds, same core)
//   k_join                    alive pairs joined, larger root under smaller
//   labels                    roots numbered in vertex order (a scan of root
//                             flags), -1 for removed levels; rows per label
//
// The leave-one-out connected set (core/connected.py:503-557 `_leave_one_out`)
// adds a CSR adjacency of the alive pairs and, per round, the articulation
// points of what is alive.  The reference finds them by Tarjan's depth-first
// search (core/kernels_graph.py:23-86), which is sequential; here they come
// from a breadth-first spanning tree and the Tarjan-Vishkin rules, which are
// data-parallel (k_cut_round, one cooperative launch a round; k_largest keeps
// the largest component before and after it):
//   BFS tree                  level-synchronous, from the smallest alive
//                             vertex; depth and tree parent per vertex, the
//                             vertices queued by depth
//   subtree sizes, preorder   bottom-up sums per level, then each vertex's
//                             number from its parent's, top-down
//   low / high                min / max preorder number over every neighbour
//                             of the subtree (bottom-up per level)
//   tree-edge classes         union-find over tree edges (named by their
//                             child): a non-tree edge (x, y) joins x's and
//                             y's; a tree edge (u, v), u not the root, joins
//                             u's when v's subtree reaches outside u's
//                             (low(v) < pre(u) or high(v) >= pre(u)+size(u))
//   cut vertices              u whose children's edges are not all in u's own
//                             edge's class; the root when its children's
//                             edges fall in two classes or more
// A spanning tree by breadth has no edge between vertices of equal depth in a
// bipartite graph and every non-tree edge joins two vertices of which neither
// is an ancestor of the other, which is the case the rules cover.  The set of
// cut vertices is a property of the graph, so it does not depend on the tree
// the race between parents picks.
#include <climits>
#include <cuda_runtime.h>

#include "unionfind.cuh"

namespace hdfe {
namespace pairs {

constexpr int kThreads = 256;
constexpr int kTile = 4096;

inline unsigned grid_for(int64_t n, int64_t cap = 148 * 32)
{
    int64_t b = (n + kThreads - 1) / kThreads;
    if (b > cap) b = cap;
    return (unsigned)(b > 0 ? b : 1);
}

__device__ __forceinline__ bool head(const uint32_t *a, const uint32_t *b, int64_t i)
{
    return i == 0 || a[i] != a[i - 1] || b[i] != b[i - 1];
}

// heads per tile of rows; rows out of (a, b) order are reported
__global__ void __launch_bounds__(kThreads) k_heads(const uint32_t *a, const uint32_t *b,
                                                    int64_t N, int64_t *tiles, unsigned *status)
{
    __shared__ double s_red[kThreads / 32];
    const int64_t t0 = (int64_t)blockIdx.x * kTile, t1 = min(t0 + kTile, N);
    int c = 0;
    for (int64_t i = t0 + threadIdx.x; i < t1; i += kThreads) {
        c += head(a, b, i);
        if (i > 0 && (a[i] < a[i - 1] || (a[i] == a[i - 1] && b[i] < b[i - 1])))
            atomicCAS(status, 0u, (unsigned)HDFE_ERR_ARG);
    }
    const double t = block_sum((double)c, s_red);
    if (threadIdx.x == 0) tiles[blockIdx.x] = (int64_t)t;
}

// exclusive scan of the tile counts, one CTA (one thread took 37 us for the 2,075
// tiles of 8.5M rows)
__global__ void __launch_bounds__(1024) k_scan(int64_t *tiles, int64_t nt, int64_t *total)
{
    cta_exclusive_scan<1024>(tiles, nt, total);
}

// each pair's first row, in row order
__global__ void __launch_bounds__(kThreads) k_write(const uint32_t *a, const uint32_t *b,
                                                    int64_t N, const int64_t *tiles,
                                                    int64_t *first)
{
    __shared__ int s_w[kThreads / 32 + 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t t0 = (int64_t)blockIdx.x * kTile, t1 = min(t0 + kTile, N);
    int64_t run = tiles[blockIdx.x];
    for (int64_t base = t0; base < t1; base += kThreads) {
        const int64_t i = base + threadIdx.x;
        const bool f = i < t1 && head(a, b, i);
        const unsigned m = __ballot_sync(0xffffffffu, f);
        if (lane == 0) s_w[warp] = __popc(m);
        __syncthreads();
        if (threadIdx.x == 0) {
            int r = 0;
            for (int k = 0; k < kThreads / 32; k++) { const int t = s_w[k]; s_w[k] = r; r += t; }
            s_w[kThreads / 32] = r;
        }
        __syncthreads();
        if (f) first[run + s_w[warp] + __popc(m & ((1u << lane) - 1))] = i;
        run += s_w[kThreads / 32];
        __syncthreads();
    }
}

// the pairs: levels and rows behind each (first[P] = N)
__global__ void __launch_bounds__(kThreads) k_pairs(const uint32_t *a, const uint32_t *b,
                                                    const int64_t *first, const int64_t *P,
                                                    int64_t N, int64_t n0, int64_t n1,
                                                    uint32_t *pa, uint32_t *pb, int64_t *count,
                                                    unsigned *status)
{
    const int64_t np = *P;
    for (int64_t p = (int64_t)blockIdx.x * kThreads + threadIdx.x; p < np;
         p += (int64_t)gridDim.x * kThreads) {
        const int64_t i = first[p];
        const int64_t e = p + 1 < np ? first[p + 1] : N;
        uint32_t x = a[i], y = b[i];
        if ((int64_t)x >= n0 || (int64_t)y >= n1) {
            atomicCAS(status, 0u, (unsigned)HDFE_ERR_BAD_CODE);
            x = 0;
            y = 0;
        }
        pa[p] = x;
        pb[p] = y;
        count[p] = e - i;
    }
}

// one peel round, part 1: degrees over the pairs whose levels are both alive
__global__ void __launch_bounds__(kThreads) k_degrees(const uint32_t *pa, const uint32_t *pb,
                                                      const int64_t *P, int64_t n0,
                                                      const uint8_t *alive, int64_t *deg)
{
    const int64_t np = *P;
    for (int64_t p = (int64_t)blockIdx.x * kThreads + threadIdx.x; p < np;
         p += (int64_t)gridDim.x * kThreads) {
        const int64_t x = pa[p], y = n0 + pb[p];
        if (alive[x] && alive[y]) {
            atomicAdd(reinterpret_cast<unsigned long long *>(deg) + x, 1ull);
            atomicAdd(reinterpret_cast<unsigned long long *>(deg) + y, 1ull);
        }
    }
}

// part 2: every alive level under its threshold removed; degrees cleared
__global__ void __launch_bounds__(kThreads) k_mark(int64_t n0, int64_t n, int64_t k0, int64_t k1,
                                                   uint8_t *alive, int64_t *deg,
                                                   unsigned *changed)
{
    for (int64_t v = (int64_t)blockIdx.x * kThreads + threadIdx.x; v < n;
         v += (int64_t)gridDim.x * kThreads) {
        const int64_t k = v < n0 ? k0 : k1;
        if (alive[v] && deg[v] < k) {
            alive[v] = 0;
            *changed = 1;
        }
        deg[v] = 0;
    }
}

// ---- cooperative kernels (k_join, k_largest, k_cut_round)
//
// One CTA of 1024 threads an SM; the phases of an algorithm are separated by
// grid barriers (2.5-3 us) instead of launches and host reads (a launch over
// every vertex per BFS level and phase, with a read per level: 60% of the
// leave-one-out set's 3.7 ms on 8.5M rows).
constexpr int kCoop = 1024;

struct Graph {
    const uint32_t *pa, *pb;    // the pairs, *P of them
    const int64_t *count, *P;
    int64_t n0, n;              // first-dimension vertices, all vertices
    uint8_t *alive;
    unsigned *status;
    GridBarrier bar;

    __device__ bool sync() const
    {
        if (bar.sync()) return true;
        if (threadIdx.x == 0) atomicCAS(status, 0u, (unsigned)HDFE_ERR_SPIN_LIMIT);
        return false;
    }
};

// The components of the vertices lo .. n over the edges that edges(join) gives:
// rounds of hooking every edge's larger parent under the smaller and
// flattening, which leave nearly every edge inside one tree, then unions of
// what is left (unions alone contend for the giant component's root).  parent
// must be the identity, visible to all; every root is its component's smallest
// vertex, and the caller flattens after a further barrier.
template <int ROUNDS, typename F>
__device__ __forceinline__ bool join_edges(const Graph &g, int64_t lo, int32_t *parent, F edges)
{
    const int64_t t0 = (int64_t)blockIdx.x * kCoop + threadIdx.x;
    const int64_t step = (int64_t)gridDim.x * kCoop;
    for (int r = 0; r < ROUNDS; r++) {
        edges([&](int32_t x, int32_t y) {
            const int32_t px = parent[x], py = parent[y];
            if (px != py) hook(parent, px, py);
        });
        if (!g.sync()) return false;
        for (int64_t v = lo + t0; v < g.n; v += step) parent[v] = root_of(parent, (int32_t)v);
        if (!g.sync()) return false;
    }
    edges([&](int32_t x, int32_t y) {
        if (parent[x] != parent[y]) unite(parent, x, y, g.status);
    });
    return true;
}

// f(x, y) for every pair whose levels are both alive
template <typename F>
__device__ __forceinline__ void alive_pairs(const Graph &g, int64_t np, F f)
{
    const int64_t t0 = (int64_t)blockIdx.x * kCoop + threadIdx.x;
    const int64_t step = (int64_t)gridDim.x * kCoop;
#pragma unroll 4
    for (int64_t p = t0; p < np; p += step) {
        const int32_t x = (int32_t)g.pa[p], y = (int32_t)(g.n0 + g.pb[p]);
        if (g.alive[x] && g.alive[y]) f(x, y);
    }
}

// The components of the alive pairs: parent[v] = the component's smallest
// second-dimension vertex, v itself for a vertex without alive pairs.  Each
// first-dimension level picks one of its alive neighbours as its anchor (any:
// a plain store) and its pairs join the anchor with the others, so that the
// trees are over the second dimension alone: 100,000 firms instead of 1.1M
// vertices, whose unions took 220 us of 310 (1.75M pairs) because a worker is
// always the smaller end and the rounds' hooks found few of them.
__device__ __forceinline__ bool components(const Graph &g, int32_t *parent)
{
    const int64_t t0 = (int64_t)blockIdx.x * kCoop + threadIdx.x;
    const int64_t step = (int64_t)gridDim.x * kCoop;
    const int64_t np = *g.P;
    for (int64_t v = t0; v < g.n; v += step) parent[v] = (int32_t)v;
    if (!g.sync()) return false;
    alive_pairs(g, np, [&](int32_t x, int32_t y) { parent[x] = y; });
    if (!g.sync()) return false;
    const bool ok = join_edges<3>(g, g.n0, parent, [&](auto join) {
        alive_pairs(g, np, [&](int32_t x, int32_t y) {
            const int32_t z = parent[x];
            if (z != y) join(z, y);
        });
    });
    if (!ok || !g.sync()) return false;
    for (int64_t v = t0; v < g.n; v += step) {
        const int32_t r = parent[v];
        parent[v] = v < g.n0 ? (r == (int32_t)v ? r : root_of(parent, r))
                             : root_of(parent, (int32_t)v);
    }
    return g.sync();
}

// least[r] = the smallest vertex of the component with root r (INT_MAX where no
// first-dimension level has that root; those come first in vertex order), by a
// warp's lanes of one root together: all warps meet at the giant's
__device__ __forceinline__ void smallest(const Graph &g, const int32_t *parent, int32_t *least)
{
    const int64_t t0 = (int64_t)blockIdx.x * kCoop + threadIdx.x;
    const int64_t step = (int64_t)gridDim.x * kCoop;
    const int lane = threadIdx.x & 31;
    for (int64_t base = t0 - lane; base < g.n0; base += step) {
        const int64_t x = base + lane;
        const int32_t r = x < g.n0 ? parent[x] : -1;
        const unsigned peers = __match_any_sync(0xffffffffu, r);
        if (r >= g.n0 && lane == __ffs(peers) - 1 && (int32_t)x < least[r])
            atomicMin(least + r, (int32_t)x);
    }
}

// the alive pairs' components with their smallest vertices as roots
__global__ void __launch_bounds__(kCoop, 1) k_join(Graph g, int32_t *parent, int32_t *least)
{
    const int64_t t0 = (int64_t)blockIdx.x * kCoop + threadIdx.x;
    const int64_t step = (int64_t)gridDim.x * kCoop;
    for (int64_t v = t0; v < g.n; v += step) least[v] = INT_MAX;
    if (!components(g, parent)) return;
    smallest(g, parent, least);
    if (!g.sync()) return;
    for (int64_t v = t0; v < g.n; v += step) {
        const int32_t r = parent[v];
        if (r >= g.n0 && least[r] != INT_MAX) parent[v] = least[r];
    }
}

// Rows per root: a thread carries the count of its current root along its
// pairs; at the end the lanes of a warp that hold the same one add theirs
// together (nearly every pair is in the giant component, and an atomic a pair
// on its address took 1.14 ms for 1.75M pairs).
struct Carry {
    unsigned long long *rows;
    int32_t at = -1;
    unsigned long long sum = 0;

    __device__ void add(int32_t label, int64_t count)
    {
        if (label != at) {
            if (sum) atomicAdd(rows + at, sum);
            at = label;
            sum = 0;
        }
        sum += (unsigned long long)count;
    }

    __device__ void flush()         // by whole warps
    {
        const unsigned peers = __match_any_sync(0xffffffffu, at);
        const int lane = threadIdx.x & 31, leader = __ffs(peers) - 1;
        unsigned long long total = 0;
        for (int q = 0; q < 32; q++) {
            const unsigned long long v = __shfl_sync(0xffffffffu, sum, q);
            if ((peers >> q) & 1u) total += v;
        }
        if (lane == leader && at >= 0 && total) atomicAdd(rows + at, total);
    }
};

// roots of every vertex, and the alive roots' flags per tile
__global__ void __launch_bounds__(kThreads) k_roots(int32_t *parent, const uint8_t *alive,
                                                    int64_t n, int64_t *tiles)
{
    __shared__ double s_red[kThreads / 32];
    const int64_t t0 = (int64_t)blockIdx.x * kTile, t1 = min(t0 + kTile, n);
    int c = 0;
    for (int64_t v = t0 + threadIdx.x; v < t1; v += kThreads) {
        const int32_t r = root_of(parent, (int32_t)v);
        parent[v] = r;
        c += alive[v] && r == (int32_t)v;
    }
    const double t = block_sum((double)c, s_red);
    if (threadIdx.x == 0) tiles[blockIdx.x] = (int64_t)t;
}

// number the alive roots in vertex order (labels[root] = its number)
__global__ void __launch_bounds__(kThreads) k_number(const int32_t *parent, const uint8_t *alive,
                                                     int64_t n, const int64_t *tiles,
                                                     int32_t *labels)
{
    __shared__ int s_w[kThreads / 32 + 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t t0 = (int64_t)blockIdx.x * kTile, t1 = min(t0 + kTile, n);
    int64_t run = tiles[blockIdx.x];
    for (int64_t base = t0; base < t1; base += kThreads) {
        const int64_t v = base + threadIdx.x;
        const bool f = v < t1 && alive[v] && parent[v] == (int32_t)v;
        const unsigned m = __ballot_sync(0xffffffffu, f);
        if (lane == 0) s_w[warp] = __popc(m);
        __syncthreads();
        if (threadIdx.x == 0) {
            int r = 0;
            for (int k = 0; k < kThreads / 32; k++) { const int t = s_w[k]; s_w[k] = r; r += t; }
            s_w[kThreads / 32] = r;
        }
        __syncthreads();
        if (f) labels[v] = (int32_t)(run + s_w[warp] + __popc(m & ((1u << lane) - 1)));
        run += s_w[kThreads / 32];
        __syncthreads();
    }
}

// every vertex's label from its root's (-1 where removed)
__global__ void __launch_bounds__(kThreads) k_label(const int32_t *parent, const uint8_t *alive,
                                                    int64_t n, int32_t *labels)
{
    for (int64_t v = (int64_t)blockIdx.x * kThreads + threadIdx.x; v < n;
         v += (int64_t)gridDim.x * kThreads) {
        const int32_t r = parent[v];
        if (!alive[v]) labels[v] = -1;
        else if (r != (int32_t)v) labels[v] = -2 - r;     // resolved by k_resolve
    }
}

__global__ void __launch_bounds__(kThreads) k_resolve(int32_t *labels, int64_t n)
{
    for (int64_t v = (int64_t)blockIdx.x * kThreads + threadIdx.x; v < n;
         v += (int64_t)gridDim.x * kThreads) {
        const int32_t l = labels[v];
        if (l <= -2) labels[v] = labels[-2 - l];     // the root's number
    }
}

// rows per component: each pair's count where both levels are labeled
__global__ void __launch_bounds__(kThreads) k_pair_rows(const uint32_t *pa, const uint32_t *pb,
                                                        const int64_t *count, const int64_t *P,
                                                        int64_t n0, const int32_t *labels,
                                                        int64_t *rows)
{
    const int64_t np = *P;
    Carry c{reinterpret_cast<unsigned long long *>(rows)};
    for (int64_t p = (int64_t)blockIdx.x * kThreads + threadIdx.x; p < np;
         p += (int64_t)gridDim.x * kThreads) {
        const int32_t la = labels[pa[p]], lb = labels[n0 + pb[p]];
        if (la >= 0 && lb >= 0) c.add(la, count[p]);
    }
    c.flush();
}

// ------------------------------------------------ leave-one-out connected set

// tile sums of v (n int64), for an exclusive scan
__global__ void __launch_bounds__(kThreads) k_tile_sums(const int64_t *v, int64_t n,
                                                        int64_t *tiles)
{
    __shared__ double s_red[kThreads / 32];
    const int64_t t0 = (int64_t)blockIdx.x * kTile, t1 = min(t0 + kTile, n);
    int64_t c = 0;
    for (int64_t i = t0 + threadIdx.x; i < t1; i += kThreads) c += v[i];
    const double t = block_sum((double)c, s_red);
    if (threadIdx.x == 0) tiles[blockIdx.x] = (int64_t)t;
}

// out[i] = tiles[tile of i] + sum of v over the tile before i; out[n] = total
__global__ void __launch_bounds__(kThreads) k_tile_scan(const int64_t *v, int64_t n,
                                                        const int64_t *tiles,
                                                        const int64_t *total, int64_t *out)
{
    constexpr int kPer = kTile / kThreads;
    __shared__ int64_t s_w[kThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t t0 = (int64_t)blockIdx.x * kTile + (int64_t)threadIdx.x * kPer;
    int64_t x[kPer], sum = 0;
#pragma unroll
    for (int k = 0; k < kPer; k++) {
        x[k] = t0 + k < n ? v[t0 + k] : 0;
        sum += x[k];
    }
    int64_t inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int64_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    if (lane == 31) s_w[warp] = inc;
    __syncthreads();
    int64_t before = tiles[blockIdx.x];
    for (int k = 0; k < warp; k++) before += s_w[k];
    before += inc - sum;
#pragma unroll
    for (int k = 0; k < kPer; k++) {
        if (t0 + k < n) out[t0 + k] = before;
        before += x[k];
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) out[n] = *total;
}

// degrees of the alive pairs' levels, both directions
__global__ void __launch_bounds__(kThreads) k_adj_degree(const uint32_t *pa, const uint32_t *pb,
                                                         const int64_t *P, int64_t n0,
                                                         const uint8_t *alive, int64_t *deg)
{
    const int64_t np = *P;
    for (int64_t p = (int64_t)blockIdx.x * kThreads + threadIdx.x; p < np;
         p += (int64_t)gridDim.x * kThreads) {
        const int64_t x = pa[p], y = n0 + pb[p];
        if (alive[x] && alive[y]) {
            atomicAdd(reinterpret_cast<unsigned long long *>(deg) + x, 1ull);
            atomicAdd(reinterpret_cast<unsigned long long *>(deg) + y, 1ull);
        }
    }
}

__global__ void __launch_bounds__(kThreads) k_adj_fill(const uint32_t *pa, const uint32_t *pb,
                                                       const int64_t *P, int64_t n0,
                                                       const uint8_t *alive,
                                                       const int64_t *indptr, int64_t *cursor,
                                                       int32_t *indices)
{
    const int64_t np = *P;
    for (int64_t p = (int64_t)blockIdx.x * kThreads + threadIdx.x; p < np;
         p += (int64_t)gridDim.x * kThreads) {
        const int64_t x = pa[p], y = n0 + pb[p];
        if (alive[x] && alive[y]) {
            const int64_t i = (int64_t)atomicAdd(
                reinterpret_cast<unsigned long long *>(cursor) + x, 1ull);
            const int64_t j = (int64_t)atomicAdd(
                reinterpret_cast<unsigned long long *>(cursor) + y, 1ull);
            indices[indptr[x] + i] = (int32_t)y;
            indices[indptr[y] + j] = (int32_t)x;
        }
    }
}

// Everything but the largest component by rows removed (the first of equals,
// i.e. the one whose smallest vertex comes first); the number of components
// into *ncomp.  Scratch: least and crow (n), smallest vertex and rows by root;
// cbest, two words a CTA.
__global__ void __launch_bounds__(kCoop, 1) k_largest(Graph g, int32_t *parent, int32_t *least,
                                                      int64_t *crow, int64_t *cbest,
                                                      int64_t *ncomp)
{
    __shared__ int64_t s_r[kCoop / 32], s_i[kCoop / 32];
    const int64_t t0 = (int64_t)blockIdx.x * kCoop + threadIdx.x;
    const int64_t step = (int64_t)gridDim.x * kCoop;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t np = *g.P;
    for (int64_t v = t0; v < g.n; v += step) {
        crow[v] = 0;
        least[v] = INT_MAX;
    }
    if (t0 == 0) *ncomp = 0;
    if (!components(g, parent)) return;
    unsigned long long roots = 0;
    for (int64_t v = t0; v < g.n; v += step) roots += parent[v] == (int32_t)v && g.alive[v];
    roots = warp_sum(roots);
    if (lane == 0 && roots) atomicAdd(reinterpret_cast<unsigned long long *>(ncomp), roots);
    smallest(g, parent, least);
    Carry c{reinterpret_cast<unsigned long long *>(crow)};
    for (int64_t p = t0; p < np; p += step) {
        const int64_t y = g.n0 + g.pb[p];
        if (g.alive[g.pa[p]] && g.alive[y]) c.add(parent[y], g.count[p]);
    }
    __syncwarp();
    c.flush();
    if (!g.sync()) return;
    // the most rows, ties to the smallest vertex: per lane, warp, CTA, then
    // every CTA over the CTAs' bests
    int64_t br = -1, bi = -1;
    auto take = [&](int64_t r, int64_t i) {
        if (i >= 0 && (r > br || (r == br && (bi < 0 || i < bi)))) { br = r; bi = i; }
    };
    auto warp_take = [&]() {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const int64_t r = __shfl_xor_sync(0xffffffffu, br, o);
            const int64_t i = __shfl_xor_sync(0xffffffffu, bi, o);
            take(r, i);
        }
    };
    for (int64_t v = t0; v < g.n; v += step)
        if (g.alive[v] && parent[v] == (int32_t)v)
            take(crow[v], least[v] != INT_MAX ? least[v] : v);
    warp_take();
    if (lane == 0) { s_r[warp] = br; s_i[warp] = bi; }
    __syncthreads();
    if (warp == 0) {
        take(s_r[lane], s_i[lane]);
        warp_take();
        if (lane == 0) { cbest[2 * blockIdx.x] = br; cbest[2 * blockIdx.x + 1] = bi; }
    }
    if (!g.sync()) return;
    br = bi = -1;
    for (unsigned b = lane; b < gridDim.x; b += 32) take(cbest[2 * b], cbest[2 * b + 1]);
    warp_take();
    if (bi < 0) return;
    const int32_t keep = parent[bi];
    for (int64_t v = t0; v < g.n; v += step)
        if (g.alive[v] && parent[v] != keep) g.alive[v] = 0;
}

// rows per first-dimension level over the alive pairs (`_nb_level_rows`)
__global__ void __launch_bounds__(kThreads) k_level_rows(const uint32_t *pa, const uint32_t *pb,
                                                         const int64_t *count, const int64_t *P,
                                                         int64_t n0, const uint8_t *alive,
                                                         int64_t *lrows, int64_t *total)
{
    const int64_t np = *P;
    unsigned long long t = 0;
    for (int64_t p = (int64_t)blockIdx.x * kThreads + threadIdx.x; p < np;
         p += (int64_t)gridDim.x * kThreads) {
        const int64_t x = pa[p];
        if (alive[x] && alive[n0 + pb[p]]) {
            if (lrows) atomicAdd(reinterpret_cast<unsigned long long *>(lrows) + x,
                                 (unsigned long long)count[p]);
            t += (unsigned long long)count[p];
        }
    }
    if (total) {
        t = warp_sum(t);
        if ((threadIdx.x & 31) == 0 && t)
            atomicAdd(reinterpret_cast<unsigned long long *>(total), t);
    }
}

// workers seen once removed; their number added to *removed
__global__ void __launch_bounds__(kThreads) k_single(uint8_t *alive, const int64_t *lrows,
                                                     int64_t n0, int64_t *removed)
{
    for (int64_t v = (int64_t)blockIdx.x * kThreads + threadIdx.x; v < n0;
         v += (int64_t)gridDim.x * kThreads)
        if (alive[v] && lrows[v] == 1) {
            alive[v] = 0;
            atomicAdd(reinterpret_cast<unsigned long long *>(removed), 1ull);
        }
}

// Vertices of this many neighbours or more are dealt to the whole grid, one
// after the other, instead of to one warp: a warp takes some 1.5 us per 32
// edges, so a vertex of tens of millions would hold the grid at a barrier for
// longer than the barrier's limit.  A hub costs a barrier a level; below the
// bound a warp's 32 vertices take 0.1 s at most.
constexpr int64_t kHub = 1 << 16;

struct CutArgs {
    Graph g;
    const int64_t *indptr;
    const int32_t *indices;
    int32_t *depth, *tpar, *size, *pre, *low, *high, *aux, *cut;
    int32_t *order;         // (n) reached vertices by depth
    int32_t *lvl;           // (n + 1) where each depth begins in order
    int32_t *hubs;          // (n + 1) reached vertices of kHub neighbours or more
    // zeroed before the launch: three levels' counters of queued vertices and of
    // hubs, side by side (every warp reads both after a level's barrier; at two
    // addresses that cost 2 us a level: 1.16 ms for two rounds, 1.11 at one), and
    // the root's key
    unsigned *queue;
    int *root_key;          // n - the smallest alive vertex
    unsigned long long *removed;
    int64_t *levels;
};

// f(u, v) for every neighbour u of the vertices v in list[0 .. count), the
// edges of up to 32 vertices dealt to the lanes one by one (a hub's neighbours
// to one thread would be a serial chain); all lanes reach every f together,
// with u < 0 where a lane has no edge.  Few vertices are dealt to more warps.
// Hubs are left out: put into hubs, counted by *n_hubs (walk_hubs).
template <typename F>
__device__ __forceinline__ void walk_edges(const CutArgs &a, const int32_t *list, int64_t count,
                                           int32_t *hubs, unsigned *n_hubs, F f)
{
    const int lane = threadIdx.x & 31;
    const int64_t wid = ((int64_t)blockIdx.x * kCoop + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * kCoop) >> 5;
    int64_t per = (count + nw - 1) / nw;
    per = per > 32 ? 32 : (per < 1 ? 1 : per);
    for (int64_t base = wid * per; base < count; base += nw * per) {
        const bool have = lane < per && base + lane < count;
        const int32_t v = have ? list[base + lane] : 0;
        const int64_t beg = have ? a.indptr[v] : 0;
        int64_t deg = have ? a.indptr[v + 1] - beg : 0;
        if (deg >= kHub) {
            hubs[atomicAdd(n_hubs, 1u)] = v;
            deg = 0;
        }
        int64_t inc = deg;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += y;
        }
        const int64_t total = __shfl_sync(0xffffffffu, inc, 31);
        const int64_t shift = beg - (inc - deg);        // edge e of the 32 is at e + shift
        for (int64_t e0 = 0; e0 < total; e0 += 32) {
            const int64_t e = e0 + lane;
            int own = 0;                // the first lane whose edges end after e
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const int64_t y = __shfl_sync(0xffffffffu, inc, own + o - 1);
                if (y <= e) own += o;
            }
            const int64_t sh = __shfl_sync(0xffffffffu, shift, own);
            const int32_t w = __shfl_sync(0xffffffffu, v, own);
            f(e < total ? a.indices[e + sh] : -1, w);
        }
    }
}

// f(u, v) for every neighbour u of the hubs v in list[0 .. count), each hub's
// edges dealt to the grid's warps 32 at a time; the lanes of a warp together, u
// < 0 where a lane has no edge.
template <typename F>
__device__ __forceinline__ void walk_hubs(const CutArgs &a, const int32_t *list, unsigned count,
                                          F f)
{
    const int lane = threadIdx.x & 31;
    const int64_t wid = ((int64_t)blockIdx.x * kCoop + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * kCoop) >> 5;
    for (unsigned i = 0; i < count; i++) {
        const int32_t v = list[i];
        const int64_t end = a.indptr[v + 1];
        for (int64_t e = a.indptr[v] + wid * 32; e < end; e += nw * 32)
            f(e + lane < end ? a.indices[e + lane] : -1, v);
    }
}

// One round of the articulation points (the rules above): every alive worker
// that is a cut vertex of the alive graph, which is connected, is removed.
// The levels of the breadth-first tree are stretches of `order`, so the passes
// up and down the tree touch each vertex once.  A vertex's preorder number is
// its parent's plus what the sizes' pass up the tree returned when it added the
// vertex's size to its parent's (one plus the siblings added before).
__global__ void __launch_bounds__(kCoop, 1) k_cut_round(CutArgs a)
{
    constexpr int kBuf = 128, kFull = kBuf - 32;
    __shared__ int32_t s_buf[kCoop / 32][kBuf];
    const Graph &g = a.g;
    const int64_t t0 = (int64_t)blockIdx.x * kCoop + threadIdx.x;
    const int64_t step = (int64_t)gridDim.x * kCoop;
    const int lane = threadIdx.x & 31;
    const int64_t np = *g.P;
    int key = 0;
    for (int64_t v = t0; v < g.n; v += step) {
        const bool up = g.alive[v];
        a.depth[v] = up ? -1 : -2;
        a.tpar[v] = -1;
        a.size[v] = 1;
        a.aux[v] = (int32_t)v;
        a.cut[v] = 0;
        if (up && key == 0) key = (int)(g.n - v);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) key = max(key, __shfl_xor_sync(0xffffffffu, key, o));
    if (lane == 0 && key) atomicMax(a.root_key, key);
    if (!g.sync()) return;
    key = *(volatile int *)a.root_key;
    if (key == 0) return;                       // nothing is alive
    const int32_t root = (int32_t)(g.n - key);
    if (t0 == 0) {
        a.order[0] = root;
        a.depth[root] = 0;
        a.pre[root] = 0;
    }
    __syncwarp();                               // the root's warp is thread 0's
    // the tree, level by level; claimed vertices leave a warp's buffer 96 or
    // more at a time
    int32_t *buf = s_buf[threadIdx.x >> 5];
    int64_t start = 0, count = 1;
    unsigned n_hubs = 0;                        // on the levels so far
    int level = 0;
    for (;; level++) {
        unsigned *tail = a.queue + 2 * ((level + 1) % 3);
        int32_t *next = a.order + start + count;
        if (t0 == 0) {
            a.lvl[level] = (int32_t)start;
            // (last read before the previous barrier)
            *reinterpret_cast<unsigned long long *>(a.queue + 2 * ((level + 2) % 3)) = 0;
        }
        int held = 0;
        auto flush = [&]() {
            unsigned at = 0;
            if (lane == 0) at = atomicAdd(tail, (unsigned)held);
            at = __shfl_sync(0xffffffffu, at, 0);
            __syncwarp();
            for (int i = lane; i < held; i += 32) next[at + i] = buf[i];
            __syncwarp();
            held = 0;
        };
        auto claim = [&](int32_t u, int32_t v) {
            const bool mine = u >= 0 && a.depth[u] == -1 &&
                              atomicCAS(a.depth + u, -1, level + 1) == -1;
            const unsigned m = __ballot_sync(0xffffffffu, mine);
            if (mine) {
                a.tpar[u] = v;
                buf[held + __popc(m & ((1u << lane) - 1))] = u;
            }
            held += __popc(m);
            if (held >= kFull) flush();
        };
        walk_edges(a, a.order + start, count, a.hubs + n_hubs, tail + 1, claim);
        if (held) flush();
        if (!g.sync()) return;
        const unsigned long long counts = *(volatile unsigned long long *)tail;
        const unsigned found = (unsigned)(counts >> 32);
        unsigned reached = (unsigned)counts;
        if (found) {                            // the same in every CTA
            walk_hubs(a, a.hubs + n_hubs, found, claim);
            if (held) flush();
            n_hubs += found;
            if (!g.sync()) return;
            reached = *(volatile unsigned *)tail;
        }
        start += count;
        count = reached;
        if (count == 0) break;
    }
    if (t0 == 0) a.lvl[level + 1] = (int32_t)start;
    if (!g.sync()) return;
    // subtree sizes up, preorder numbers down
    for (int l = level; l >= 1; l--) {
        const int64_t e = a.lvl[l + 1];
        for (int64_t i = a.lvl[l] + t0; i < e; i += step) {
            const int32_t v = a.order[i];
            a.pre[v] = atomicAdd(a.size + a.tpar[v], a.size[v]);
        }
        if (!g.sync()) return;
    }
    for (int l = 1; l <= level; l++) {
        const int64_t e = a.lvl[l + 1];
        for (int64_t i = a.lvl[l] + t0; i < e; i += step) {
            const int32_t v = a.order[i];
            a.pre[v] += a.pre[a.tpar[v]];
        }
        if (!g.sync()) return;
    }
    // least and greatest number over each vertex and its neighbours: a thread a
    // vertex, a warp for one of 32 neighbours or more, the grid for hubs
    for (int64_t base = t0 - lane; base < g.n; base += step) {
        const int64_t v = base + lane;
        const bool have = v < g.n && a.depth[v] >= 0;
        const int64_t beg = have ? a.indptr[v] : 0, end = have ? a.indptr[v + 1] : 0;
        int32_t lo = have ? a.pre[v] : 0, hi = lo;
        if (end - beg < 32) {
#pragma unroll 4
            for (int64_t k = beg; k < end; k++) {
                const int32_t w = a.indices[k];
                if (a.depth[w] < 0) continue;
                const int32_t p = a.pre[w];
                lo = min(lo, p);
                hi = max(hi, p);
            }
        }
        for (unsigned big = __ballot_sync(0xffffffffu, end - beg >= 32 && end - beg < kHub); big;
             big &= big - 1) {
            const int q = __ffs(big) - 1;
            const int64_t b = __shfl_sync(0xffffffffu, beg, q), e = __shfl_sync(0xffffffffu, end, q);
            int32_t l = INT_MAX, h = -1;
#pragma unroll 4
            for (int64_t k = b + lane; k < e; k += 32) {
                const int32_t w = a.indices[k];
                if (a.depth[w] < 0) continue;
                const int32_t p = a.pre[w];
                l = min(l, p);
                h = max(h, p);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                l = min(l, __shfl_xor_sync(0xffffffffu, l, o));
                h = max(h, __shfl_xor_sync(0xffffffffu, h, o));
            }
            if (lane == q) {
                lo = min(lo, l);
                hi = max(hi, h);
            }
        }
        if (have) {
            a.low[v] = lo;
            a.high[v] = hi;
        }
    }
    if (!g.sync()) return;
    if (n_hubs) {
        walk_hubs(a, a.hubs, n_hubs, [&](int32_t w, int32_t v) {
            const bool in = w >= 0 && a.depth[w] >= 0;
            const int32_t p = in ? a.pre[w] : 0;
            const int32_t l = __reduce_min_sync(0xffffffffu, in ? p : INT_MAX);
            const int32_t h = __reduce_max_sync(0xffffffffu, in ? p : -1);
            if (lane == 0 && l < a.low[v]) atomicMin(a.low + v, l);
            if (lane == 0 && h > a.high[v]) atomicMax(a.high + v, h);
        });
        if (!g.sync()) return;
    }
    for (int l = level; l >= 3; l--) {          // the rules read them from depth 2 on
        const int64_t e = a.lvl[l + 1];
        for (int64_t i = a.lvl[l] + t0; i < e; i += step) {
            const int32_t v = a.order[i], u = a.tpar[v];
            const int32_t lo = a.low[v], hi = a.high[v];
            if (lo < a.low[u]) atomicMin(a.low + u, lo);
            if (hi > a.high[u]) atomicMax(a.high + u, hi);
        }
        if (!g.sync()) return;
    }
    // tree-edge classes: rule 1 over the non-tree pairs, rule 2 over the tree
    // edges (u, v) with u not the root
    const bool ok = join_edges<2>(g, 0, a.aux, [&](auto join) {
#pragma unroll 4
        for (int64_t p = t0; p < np; p += step) {
            const int32_t x = (int32_t)g.pa[p], y = (int32_t)(g.n0 + g.pb[p]);
            if (a.depth[x] >= 0 && a.depth[y] >= 0 && a.tpar[x] != y && a.tpar[y] != x)
                join(x, y);
        }
        for (int64_t v = t0; v < g.n; v += step) {
            if (a.depth[v] < 2) continue;
            const int32_t u = a.tpar[v], pu = a.pre[u];
            if (a.low[v] < pu || a.high[v] >= pu + a.size[u]) join(u, (int32_t)v);
        }
    });
    if (!ok || !g.sync()) return;
    for (int64_t v = t0; v < g.n; v += step) a.aux[v] = root_of(a.aux, (int32_t)v);
    if (!g.sync()) return;
    // cut vertices: u with a child's edge outside u's own edge's class, the root
    // with children's edges in two classes
    const int32_t first = level > 0 ? a.aux[a.order[1]] : 0;
    unsigned long long gone = 0;
    for (int64_t v = t0; v < g.n; v += step) {
        if (a.depth[v] < 1) continue;
        const int32_t u = a.tpar[v];
        if (a.aux[v] != (u == root ? first : a.aux[u]) && u < g.n0 &&
            atomicExch(a.cut + u, 1) == 0) {
            g.alive[u] = 0;
            gone++;
        }
    }
    gone = warp_sum(gone);
    if (lane == 0 && gone) atomicAdd(a.removed, gone);
    if (t0 == 0) *a.levels = level;
}

struct Layout {
    int64_t tiles, first, pa, pb, count, deg, parent, scalars, total;
    // leave-one-out only
    int64_t indptr, indices, depth, tpar, size, pre, low, high, aux, cut, order, crow, cbest, lrows;
};

inline Layout layout(int64_t N, int64_t n, bool loo = false)
{
    Layout o = {};
    int64_t p = 0;
    auto take = [&](int64_t bytes) { int64_t at = p; p += (bytes + 255) / 256 * 256; return at; };
    const int64_t nt = ((N > n ? N : n) + kTile - 1) / kTile + 1;
    o.tiles = take(nt * 8);
    o.first = take((N + 1) * 8);
    o.pa = take(N * 4);
    o.pb = take(N * 4);
    o.count = take(N * 8);
    o.deg = take(n * 8);
    o.parent = take(n * 4);
    o.scalars = take(256);
    if (loo) {
        o.indptr = take((n + 1) * 8);
        o.indices = take(2 * N * 4);
        o.depth = take(n * 4);
        o.tpar = take(n * 4);
        o.size = take(n * 4);
        o.pre = take(n * 4);
        o.low = take(n * 4);
        o.high = take(n * 4);
        o.aux = take(n * 4);
        o.cut = take(n * 4);
        o.order = take(n * 4);
        o.crow = take((n + 1) * 8);
        o.cbest = take(1024 * 16);
        o.lrows = take(n * 8);
    }
    o.total = p;
    return o;
}

}  // namespace pairs
}  // namespace hdfe

using namespace hdfe;

namespace {

// Pointers into the workspace, and the steps both entry points share.
struct Ctx {
    const uint32_t *a, *b;
    int64_t N, n0, n1, n;
    cudaStream_t s;
    pairs::Layout lay;
    int64_t *tiles, *first, *count, *deg;
    uint32_t *pa, *pb;
    int32_t *parent;
    pairs::Graph g;
    // scalars (8 bytes each): P, ncomp, status, changed, rows kept, components before,
    // single observations; from 8 a round's own (root key, at 10 workers removed, the
    // tree's depth, the queue's counters); at 16 the grid barrier
    int64_t *P, *ncomp, *removed, *levels, *kept, *before, *single;
    unsigned *status, *changed, *queue;
    int *root_key;
    int launches = 0;

    Ctx(const uint32_t *a_, const uint32_t *b_, int64_t N_, int64_t n0_, int64_t n1_, bool loo,
        void *workspace, cudaStream_t s_)
        : a(a_), b(b_), N(N_), n0(n0_), n1(n1_), n(n0_ + n1_), s(s_),
          lay(pairs::layout(N_, n0_ + n1_, loo))
    {
        char *ws = (char *)workspace;
        tiles = (int64_t *)(ws + lay.tiles);
        first = (int64_t *)(ws + lay.first);
        pa = (uint32_t *)(ws + lay.pa);
        pb = (uint32_t *)(ws + lay.pb);
        count = (int64_t *)(ws + lay.count);
        deg = (int64_t *)(ws + lay.deg);
        parent = (int32_t *)(ws + lay.parent);
        int64_t *sc = (int64_t *)(ws + lay.scalars);
        P = sc;
        ncomp = sc + 1;
        status = (unsigned *)(sc + 2);
        changed = (unsigned *)(sc + 3);
        kept = sc + 4;
        before = sc + 5;
        single = sc + 6;
        root_key = (int *)(sc + 8);
        removed = sc + 10;
        levels = sc + 11;
        queue = (unsigned *)(sc + 12);
        g.pa = pa;
        g.pb = pb;
        g.count = count;
        g.P = P;
        g.n0 = n0;
        g.n = n;
        g.status = status;
        g.bar = GridBarrier{(unsigned *)(sc + 16)};
    }

    // the distinct pairs and the (k0, k1)-core; returns the peel rounds
    int pairs_and_core(uint8_t *alive, int64_t k0, int64_t k1, int64_t *rounds)
    {
        using namespace pairs;
        HDFE_CUDA_TRY(cudaMemsetAsync(P, 0, 256, s));
        const int64_t rt = (N + kTile - 1) / kTile;
        k_heads<<<(unsigned)rt, kThreads, 0, s>>>(a, b, N, tiles, status);
        k_scan<<<1, 1024, 0, s>>>(tiles, rt, P);
        k_write<<<(unsigned)rt, kThreads, 0, s>>>(a, b, N, tiles, first);
        k_pairs<<<grid_for(N), kThreads, 0, s>>>(a, b, first, P, N, n0, n1, pa, pb, count,
                                                 status);
        launches += 4;
        HDFE_CUDA_TRY(cudaMemsetAsync(alive, 1, n, s));
        HDFE_CUDA_TRY(cudaMemsetAsync(deg, 0, n * 8, s));
        *rounds = 0;
        if (k0 > 1 || k1 > 1) {
            for (;; (*rounds)++) {
                HDFE_CUDA_TRY(cudaMemsetAsync(changed, 0, 4, s));
                k_degrees<<<grid_for(N), kThreads, 0, s>>>(pa, pb, P, n0, alive, deg);
                k_mark<<<grid_for(n), kThreads, 0, s>>>(n0, n, k0, k1, alive, deg, changed);
                launches += 2;
                unsigned h = 0;
                HDFE_CUDA_TRY(cudaMemcpyAsync(&h, changed, 4, cudaMemcpyDeviceToHost, s));
                HDFE_CUDA_TRY(cudaStreamSynchronize(s));
                if (!h || *rounds > n) break;
            }
        }
        return HDFE_OK;
    }

    // a cooperative launch of one CTA an SM, fewer where the graph is small
    int coop(const void *kernel, void **args)
    {
        using namespace pairs;
        int dev = 0, sms = 0;
        HDFE_CUDA_TRY(cudaGetDevice(&dev));
        HDFE_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        int64_t need = ((N > n ? N : n) + 4 * kCoop - 1) / (4 * kCoop);
        need = need < 1 ? 1 : (need > sms ? sms : need);
        HDFE_CUDA_TRY(cudaLaunchCooperativeKernel(kernel, dim3((unsigned)need), dim3(kCoop), args,
                                                  0, s));
        launches++;
        return HDFE_OK;
    }

    // components of the alive pairs numbered by their roots into labels, rows
    // per label into rows (n), their number into *ncomp
    int components(uint8_t *alive, int32_t *labels, int64_t *rows)
    {
        using namespace pairs;
        const int64_t vt = (n + kTile - 1) / kTile;
        g.alive = alive;
        int32_t *least = (int32_t *)deg;        // (the degrees are done with)
        void *args[] = {&g, &parent, &least};
        const int st = coop((const void *)k_join, args);
        if (st != HDFE_OK) return st;
        k_roots<<<(unsigned)vt, kThreads, 0, s>>>(parent, alive, n, tiles);
        k_scan<<<1, 1024, 0, s>>>(tiles, vt, ncomp);
        k_number<<<(unsigned)vt, kThreads, 0, s>>>(parent, alive, n, tiles, labels);
        k_label<<<grid_for(n), kThreads, 0, s>>>(parent, alive, n, labels);
        k_resolve<<<grid_for(n), kThreads, 0, s>>>(labels, n);
        HDFE_CUDA_TRY(cudaMemsetAsync(rows, 0, n * 8, s));
        k_pair_rows<<<grid_for(N, 148 * 4), kThreads, 0, s>>>(pa, pb, count, P, n0, labels, rows);
        launches += 6;
        return HDFE_OK;
    }
};

}  // namespace

extern "C" int64_t hdfe_pair_components_workspace_bytes(int64_t n_rows, int64_t n0, int64_t n1)
{
    if (n_rows < 0 || n0 < 1 || n1 < 1) return -1;
    return pairs::layout(n_rows, n0 + n1).total;
}

extern "C" int hdfe_pair_components(const uint32_t *a, const uint32_t *b, int64_t n_rows,
                                    int64_t n0, int64_t n1, int64_t k0, int64_t k1,
                                    uint8_t *alive, int32_t *labels, int64_t *rows,
                                    int64_t *counts, void *workspace, int64_t workspace_bytes,
                                    void *stream)
{
    if (!a || !b || n_rows < 1 || n0 < 1 || n1 < 1 || n0 + n1 >= INT32_MAX || k0 < 1 || k1 < 1 ||
        !alive || !labels || !rows || !counts || !workspace)
        return hdfe_set_arg_error("hdfe_pair_components: bad argument");
    Ctx c(a, b, n_rows, n0, n1, false, workspace, (cudaStream_t)stream);
    if (workspace_bytes < c.lay.total)
        return hdfe_set_error(HDFE_ERR_WORKSPACE, "hdfe_pair_components: workspace too small");
    int64_t rounds = 0;
    int st = c.pairs_and_core(alive, k0, k1, &rounds);
    if (st != HDFE_OK) return st;
    if ((st = c.components(alive, labels, rows)) != HDFE_OK) return st;
    HDFE_CUDA_TRY(cudaGetLastError());
    hdfe_add_launches(c.launches);
    // counts: pairs, components, status, peel rounds
    cudaStream_t s = c.s;
    HDFE_CUDA_TRY(cudaMemcpyAsync(counts, c.P, 16, cudaMemcpyDeviceToDevice, s));
    HDFE_CUDA_TRY(cudaMemsetAsync(counts + 2, 0, 8, s));
    HDFE_CUDA_TRY(cudaMemcpyAsync(counts + 2, c.status, 4, cudaMemcpyDeviceToDevice, s));
    HDFE_CUDA_TRY(cudaMemcpyAsync(counts + 3, &rounds, 8, cudaMemcpyHostToDevice, s));
    HDFE_CUDA_TRY(cudaStreamSynchronize(s));
    return HDFE_OK;
}

extern "C" int64_t hdfe_leave_one_out_workspace_bytes(int64_t n_rows, int64_t n0, int64_t n1)
{
    if (n_rows < 0 || n0 < 1 || n1 < 1) return -1;
    return pairs::layout(n_rows, n0 + n1, true).total;
}

extern "C" int hdfe_leave_one_out(const uint32_t *a, const uint32_t *b, int64_t n_rows,
                                  int64_t n0, int64_t n1, int64_t k0, int64_t k1,
                                  uint8_t *alive, int64_t *counts, void *workspace,
                                  int64_t workspace_bytes, void *stream)
{
    using namespace pairs;
    if (!a || !b || n_rows < 1 || n0 < 1 || n1 < 1 || n0 + n1 >= INT32_MAX || k0 < 1 ||
        k1 < 1 || !alive || !counts || !workspace)
        return hdfe_set_arg_error("hdfe_leave_one_out: bad argument");
    Ctx c(a, b, n_rows, n0, n1, true, workspace, (cudaStream_t)stream);
    if (workspace_bytes < c.lay.total)
        return hdfe_set_error(HDFE_ERR_WORKSPACE, "hdfe_leave_one_out: workspace too small");
    cudaStream_t s = c.s;
    const int64_t n = c.n, N = n_rows;
    char *ws = (char *)workspace;
    const Layout &L = c.lay;
    int64_t *indptr = (int64_t *)(ws + L.indptr);
    int32_t *indices = (int32_t *)(ws + L.indices);
    int32_t *depth = (int32_t *)(ws + L.depth), *tpar = (int32_t *)(ws + L.tpar);
    int32_t *size = (int32_t *)(ws + L.size), *pre = (int32_t *)(ws + L.pre);
    int32_t *low = (int32_t *)(ws + L.low), *high = (int32_t *)(ws + L.high);
    int32_t *aux = (int32_t *)(ws + L.aux), *cut = (int32_t *)(ws + L.cut);
    int32_t *order = (int32_t *)(ws + L.order);
    int64_t *crow = (int64_t *)(ws + L.crow), *lrows = (int64_t *)(ws + L.lrows);
    int64_t peel_rounds = 0;
    int st = c.pairs_and_core(alive, k0, k1, &peel_rounds);
    if (st != HDFE_OK) return st;

    // CSR adjacency of the pairs alive now (later removals only clear `alive`)
    const int64_t vt = (n + kTile - 1) / kTile;
    HDFE_CUDA_TRY(cudaMemsetAsync(c.deg, 0, n * 8, s));
    k_adj_degree<<<grid_for(N), kThreads, 0, s>>>(c.pa, c.pb, c.P, n0, alive, c.deg);
    k_tile_sums<<<(unsigned)vt, kThreads, 0, s>>>(c.deg, n, c.tiles);
    k_scan<<<1, 1024, 0, s>>>(c.tiles, vt, c.removed);
    k_tile_scan<<<(unsigned)vt, kThreads, 0, s>>>(c.deg, n, c.tiles, c.removed, indptr);
    HDFE_CUDA_TRY(cudaMemsetAsync(c.deg, 0, n * 8, s));
    k_adj_fill<<<grid_for(N), kThreads, 0, s>>>(c.pa, c.pb, c.P, n0, alive, indptr, c.deg,
                                                indices);
    c.launches += 5;

    c.g.alive = alive;
    int64_t *cbest = (int64_t *)(ws + L.cbest);
    auto keep_largest = [&]() -> int {
        int32_t *least = (int32_t *)c.deg;      // (the adjacency's degrees are done with)
        void *args[] = {&c.g, &c.parent, &least, &crow, &cbest, &c.ncomp};
        return c.coop((const void *)k_largest, args);
    };
    auto read = [&](const void *dev, size_t bytes, void *host) -> int {
        HDFE_CUDA_TRY(cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, s));
        HDFE_CUDA_TRY(cudaStreamSynchronize(s));
        return HDFE_OK;
    };

    // 1. the largest component
    if ((st = keep_largest()) != HDFE_OK) return st;
    HDFE_CUDA_TRY(cudaMemcpyAsync(c.before, c.ncomp, 8, cudaMemcpyDeviceToDevice, s));
    // 2. workers seen once (their leverage is 1), then the largest piece left
    HDFE_CUDA_TRY(cudaMemsetAsync(lrows, 0, n0 * 8, s));
    k_level_rows<<<grid_for(N), kThreads, 0, s>>>(c.pa, c.pb, c.count, c.P, n0, alive, lrows,
                                                  nullptr);
    k_single<<<grid_for(n0), kThreads, 0, s>>>(alive, lrows, n0, c.single);
    c.launches += 2;
    if ((st = keep_largest()) != HDFE_OK) return st;
    // 3-4. workers that are articulation points, until there are none
    int64_t cut_total = 0, rounds = 0, max_levels = 0;
    // (the levels' stretches and the hubs, n + 1 each, lie in the rows by root,
    // done with by then)
    CutArgs ca{c.g,  indptr, indices, depth,   tpar,    size,       pre,       low,
               high, aux,    cut,     order, (int32_t *)crow, (int32_t *)crow + n + 1, c.queue,
               c.root_key, reinterpret_cast<unsigned long long *>(c.removed),
               c.levels};
    for (;;) {
        HDFE_CUDA_TRY(cudaMemsetAsync(c.root_key, 0, 56, s));   // through the queue's counters
        void *args[] = {&ca};
        if ((st = c.coop((const void *)k_cut_round, args)) != HDFE_OK) return st;
        int64_t h[2];                       // workers removed, the tree's depth
        if ((st = read(c.removed, 16, h)) != HDFE_OK) return st;
        if (h[1] > max_levels) max_levels = h[1];
        if (!h[0] || rounds > n) break;
        cut_total += h[0];
        rounds++;
        if ((st = keep_largest()) != HDFE_OK) return st;
    }
    // rows kept
    HDFE_CUDA_TRY(cudaMemsetAsync(c.kept, 0, 8, s));
    k_level_rows<<<grid_for(N), kThreads, 0, s>>>(c.pa, c.pb, c.count, c.P, n0, alive, nullptr,
                                                  c.kept);
    c.launches++;
    HDFE_CUDA_TRY(cudaGetLastError());
    hdfe_add_launches(c.launches);
    // counts: pairs, components before, single observations, workers cut, rounds, rows
    // kept, status, BFS depth (largest over rounds)
    int64_t h[8];
    int64_t dev_sc[7];
    if ((st = read(c.P, sizeof(dev_sc), dev_sc)) != HDFE_OK) return st;
    h[0] = dev_sc[0];
    h[1] = dev_sc[5];
    h[2] = dev_sc[6];
    h[3] = cut_total;
    h[4] = rounds;
    h[5] = dev_sc[4];
    h[6] = (int64_t)(unsigned)(dev_sc[2] & 0xffffffff);
    h[7] = max_levels;
    HDFE_CUDA_TRY(cudaMemcpyAsync(counts, h, sizeof(h), cudaMemcpyHostToDevice, s));
    HDFE_CUDA_TRY(cudaStreamSynchronize(s));
    return HDFE_OK;
}
