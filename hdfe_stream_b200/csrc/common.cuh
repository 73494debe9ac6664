// Shared device helpers of libhdfe_b200: status codes, a bounded grid-wide
// barrier for the persistent (cooperatively launched) kernels, and warp/block
// reductions whose order is fixed, so sums do not depend on scheduling.
#pragma once

#include <atomic>
#include <cstdint>
#include <cuda_runtime.h>

#include "hdfe_b200.h"

namespace hdfe {

// Upper bound on one wait in a grid barrier.  Every CTA of a cooperative
// launch is resident, so a barrier completes in microseconds; if one does not
// complete within this many nanoseconds the kernel records
// HDFE_ERR_SPIN_LIMIT and every CTA returns instead of waiting on.
constexpr unsigned long long kSpinLimitNs = 1000000000ull;   // 1 s

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ unsigned ld_acquire(const unsigned *p)
{
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st_release(unsigned *p, unsigned v)
{
    asm volatile("st.release.gpu.global.u32 [%0], %1;" :: "l"(p), "r"(v) : "memory");
}

// fetch-and-add with release semantics at GPU scope: the writes this thread
// has made or observed (the CTA's, after its __syncthreads) are visible to
// whoever acquires the result
__device__ __forceinline__ unsigned atom_add_release(unsigned *p, unsigned v)
{
    unsigned old;
    asm volatile("atom.add.release.gpu.global.u32 %0, [%1], %2;"
                 : "=r"(old) : "l"(p), "r"(v) : "memory");
    return old;
}

// Grid barrier state: bar[0] arrivals, bar[1] generation, bar[2] error code.
// Zeroed by the host (or a set-up kernel) before the launch that uses it.
struct GridBarrier {
    unsigned *bar;

    // Returns false when the kernel must stop (an error was recorded, by this
    // CTA on a timeout or by another one).  All threads of the CTA return the
    // same value.
    //   Arrival is one release fetch-and-add (it orders the CTA's writes,
    // made visible to thread 0 by the __syncthreads, before it); the last CTA
    // resets the count and publishes the next generation with a release
    // store; the others spin on the generation alone with acquire loads,
    // looking at the error word and the clock every 32 polls (the wait stays
    // bounded by kSpinLimitNs, give or take 32 polls).
    __device__ bool sync() const
    {
        __shared__ int s_ok;
        __syncthreads();
        if (threadIdx.x == 0) {
            int ok = 1;
            const unsigned gen = ld_acquire(bar + 1);
            const unsigned arrived = atom_add_release(bar, 1u);
            if (arrived == gridDim.x - 1) {
                bar[0] = 0;                 // ordered before the release below
                st_release(bar + 1, gen + 1);
            } else {
                const unsigned long long t0 = global_ns();
                for (unsigned polls = 1; ld_acquire(bar + 1) == gen; polls++) {
                    if ((polls & 31u) == 0) {
                        if (ld_acquire(bar + 2) != 0) { ok = 0; break; }
                        if (global_ns() - t0 > kSpinLimitNs) {
                            atomicCAS(bar + 2, 0u, (unsigned)HDFE_ERR_SPIN_LIMIT);
                            ok = 0;
                            break;
                        }
                    }
                }
            }
            if (ok && ld_acquire(bar + 2) != 0) ok = 0;
            s_ok = ok;
        }
        __syncthreads();
        return s_ok != 0;
    }

    __device__ void fail(int code) const { atomicCAS(bar + 2, 0u, (unsigned)code); }
};

template <typename T>
__device__ __forceinline__ T warp_sum(T v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Fixed-order sum over the CTA of one value per thread; result valid in
// thread 0.  `scratch` holds one slot per warp.
template <typename T>
__device__ __forceinline__ T block_sum(T v, T *scratch)
{
    v = warp_sum(v);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    T total = T(0);
    if (threadIdx.x == 0) {
        const int nw = (blockDim.x + 31) >> 5;
        for (int w = 0; w < nw; w++) total += scratch[w];
    }
    __syncthreads();
    return total;
}

// Exclusive scan of v[0 .. n) in place by one CTA of T threads, *total = the
// sum: each thread takes a consecutive stretch, the stretches' sums are scanned
// by warps and then over warps.
template <int T>
__device__ __forceinline__ void cta_exclusive_scan(int64_t *v, int64_t n, int64_t *total)
{
    __shared__ int64_t s_warp[T / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t per = (n + T - 1) / T;
    const int64_t lo = min((int64_t)threadIdx.x * per, n), hi = min(lo + per, n);
    int64_t sum = 0;
    for (int64_t i = lo; i < hi; i++) sum += v[i];
    int64_t inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int64_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    if (lane == 31) s_warp[warp] = inc;
    __syncthreads();
    int64_t run = inc - sum;
    for (int k = 0; k < warp; k++) run += s_warp[k];
    for (int64_t i = lo; i < hi; i++) {
        const int64_t x = v[i];
        v[i] = run;
        run += x;
    }
    if (threadIdx.x == T - 1) *total = run;
}

}  // namespace hdfe

int hdfe_set_cuda_error(cudaError_t e);
int hdfe_set_error(int code, const char *msg);
int hdfe_set_arg_error(const char *msg);

#define HDFE_CUDA_TRY(expr)                                            \
    do {                                                               \
        cudaError_t _e = (expr);                                       \
        if (_e != cudaSuccess) return hdfe_set_cuda_error(_e);         \
    } while (0)

// Up to eight ranges zeroed by one launch (a fill each costs the host and the
// stream about 2 us; a small fit had twenty).
struct hdfe_zero_list {
    void *ptr[8];
    int64_t bytes[8];       // multiples of 4, 4-byte aligned
    int n = 0;
    void add(void *p, int64_t b)
    {
        if (b <= 0) return;
        ptr[n] = p;
        bytes[n++] = b;
    }
};
int hdfe_zero(const hdfe_zero_list &list, cudaStream_t s);

// A kernel's dynamic shared memory limit, raised once per device to the most
// that any of its launches asks for.  The limit belongs to the kernel, not to
// the launch: set to each launch's own size, another host thread could lower it
// between this thread's set and its launch; and compared with 48 KB it would
// leave out the kernel's static shared memory, which counts against them too.
// One object per kernel (a static of the template that launches it).
struct hdfe_shared_limit {
    std::atomic<bool> done[64];
    int raise(const void *kernel, size_t most)
    {
        int dev = 0;
        HDFE_CUDA_TRY(cudaGetDevice(&dev));
        const bool known = dev >= 0 && dev < 64;
        if (known && done[dev].load()) return HDFE_OK;
        HDFE_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)most));
        if (known) done[dev].store(true);
        return HDFE_OK;
    }
};

// counts kernels launched by the library (hdfe_kernel_launches)
void hdfe_add_launches(int n);
