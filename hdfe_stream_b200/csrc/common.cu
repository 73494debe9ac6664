// Error reporting and version of libhdfe_b200.
#include <cstdio>
#include <atomic>
#include <cstring>
#include <cuda_runtime.h>

#include "common.cuh"

namespace {
thread_local char g_msg[512] = "no error";
std::atomic<long long> g_launches{0};
}

void hdfe_add_launches(int n) { g_launches.fetch_add(n, std::memory_order_relaxed); }

extern "C" int64_t hdfe_kernel_launches(void) { return g_launches.load(); }

int hdfe_set_cuda_error(cudaError_t e)
{
    std::snprintf(g_msg, sizeof g_msg, "CUDA error %d: %s", (int)e, cudaGetErrorString(e));
    return HDFE_ERR_CUDA;
}

int hdfe_set_error(int code, const char *msg)
{
    std::snprintf(g_msg, sizeof g_msg, "%s", msg);
    return code;
}

int hdfe_set_arg_error(const char *msg) { return hdfe_set_error(HDFE_ERR_ARG, msg); }

namespace {

__global__ void __launch_bounds__(256) k_zero(hdfe_zero_list list)
{
    for (int r = 0; r < list.n; r++) {
        // 16 bytes a thread between the 16-byte boundaries, words at the ends
        char *p = (char *)list.ptr[r], *e = p + list.bytes[r];
        char *a = (char *)(((uintptr_t)p + 15) & ~(uintptr_t)15);
        char *b = (char *)((uintptr_t)e & ~(uintptr_t)15);
        if (a > b) a = b = e;
        const int64_t t = (int64_t)blockIdx.x * 256 + threadIdx.x, step = (int64_t)gridDim.x * 256;
        for (char *q = a + 16 * t; q < b; q += 16 * step) *(int4 *)q = make_int4(0, 0, 0, 0);
        if (blockIdx.x == 0) {
            for (char *q = p + 4 * threadIdx.x; q < a; q += 4 * 256) *(int *)q = 0;
            for (char *q = b + 4 * threadIdx.x; q < e; q += 4 * 256) *(int *)q = 0;
        }
    }
}

}  // namespace

int hdfe_zero(const hdfe_zero_list &list, cudaStream_t s)
{
    if (list.n == 0) return HDFE_OK;
    int64_t most = 0;
    for (int r = 0; r < list.n; r++) most = list.bytes[r] > most ? list.bytes[r] : most;
    int64_t blocks = (most / 16 + 255) / 256;
    blocks = blocks < 1 ? 1 : (blocks > 148 * 8 ? 148 * 8 : blocks);
    k_zero<<<(unsigned)blocks, 256, 0, s>>>(list);
    HDFE_CUDA_TRY(cudaGetLastError());
    hdfe_add_launches(1);
    return HDFE_OK;
}

extern "C" const char *hdfe_error_string(void) { return g_msg; }

extern "C" const char *hdfe_version(void) { return "hdfe_b200 0.1.0 (sm_100a)"; }
