// Union-find over int32 vertices whose roots are their components' smallest
// vertices: what the component kernels of graph.cu and pairs.cu share.
#pragma once

#include "common.cuh"

namespace hdfe {

constexpr int kMaxSteps = 1 << 22;     // retries of one union before giving up

__device__ __forceinline__ int32_t find_root(int32_t *parent, int32_t x)
{
    // path halving with relaxed writes: parent pointers only ever decrease
    int32_t p = parent[x];
    int steps = 0;
    while (p != x && steps < kMaxSteps) {
        const int32_t gp = parent[p];
        if (gp != p) parent[x] = gp;    // a benign race: gp is an ancestor of x
        x = p;
        p = gp;
        steps++;
    }
    return x;
}

// The root of x without writing: for the flattening passes, where each thread
// writes only its own vertex's entry (a compressing find could overwrite a
// vertex another thread has just set to its root with a non-root ancestor).
__device__ __forceinline__ int32_t root_of(const int32_t *parent, int32_t x)
{
    int steps = 0;
    for (int32_t p = parent[x]; p != x && steps < kMaxSteps; p = parent[x], steps++) x = p;
    return x;
}

// link a and b: the larger root under the smaller (bounded retries)
__device__ __forceinline__ void unite(int32_t *parent, int32_t a, int32_t b, unsigned *status)
{
    for (int step = 0;; step++) {
        if (step >= kMaxSteps) { atomicCAS(status, 0u, (unsigned)HDFE_ERR_SPIN_LIMIT); return; }
        a = find_root(parent, a);
        b = find_root(parent, b);
        if (a == b) return;
        const int32_t hi = a > b ? a : b, lo = a > b ? b : a;
        const int32_t old = atomicCAS(parent + hi, hi, lo);
        if (old == hi) return;
        a = old;        // hi gained this parent meanwhile: retry from there
        b = lo;
    }
}

// hook the larger vertex under the smaller where that lowers its parent
__device__ __forceinline__ void hook(int32_t *parent, int32_t a, int32_t b)
{
    const int32_t hi = a > b ? a : b, lo = a > b ? b : a;
    if (parent[hi] > lo) atomicMin(parent + hi, lo);
}

}  // namespace hdfe
