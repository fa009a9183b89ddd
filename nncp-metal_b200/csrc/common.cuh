// common.cuh -- status/error plumbing and dtype helpers shared by every kernel file.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>

#include "device_once.h"
#include "nncu.h"

typedef __nv_bfloat16 bf16;

// last error message of the calling thread (nncu_last_error)
extern thread_local char g_nncu_err[512];
int nncu_fail(int code, const char *fmt, ...);

#define CUDA_TRY(expr)                                                                     \
    do {                                                                                   \
        cudaError_t e_ = (expr);                                                           \
        if (e_ != cudaSuccess)                                                             \
            return nncu_fail(e_ == cudaErrorMemoryAllocation ? NNCU_ERR_NOMEM : NNCU_ERR_CUDA, \
                             "%s:%d: %s -> %s", __FILE__, __LINE__, #expr,                 \
                             cudaGetErrorString(e_));                                      \
    } while (0)

#define NNCU_TRY(expr)       \
    do {                     \
        int rc_ = (expr);    \
        if (rc_ != NNCU_OK)  \
            return rc_;      \
    } while (0)

constexpr int SMEM_MOST = 227 * 1024; // shared memory a block can have

// Lets a kernel take up to `bytes` of dynamic shared memory on the current device; `once` is the kernel's own.
// The limit is the most that any shape asks for, so models of different shapes do not lower one another's.
template <typename K> static int smem_limit(DeviceOnce &once, K kernel, int bytes)
{
    int dev = -1;
    CUDA_TRY(cudaGetDevice(&dev));
    return once.run(dev, [&]() -> int {
        CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
        return NNCU_OK;
    });
}

// Programmatic dependent launch.  A kernel started through launch_k may begin while the kernel
// before it on the stream is still draining: its CTAs become resident, run whatever comes before
// pdl_wait() (barrier set-up, TMEM allocation, index arithmetic) and block there until the
// predecessor has completed and its writes are visible.  Rules for a kernel launched this way:
// every thread executes pdl_wait() before its first global-memory access and before any early
// return, so that the kernel cannot complete before its predecessor has.  Both calls are no-ops in
// a kernel launched the ordinary way.  On in the one-symbol steps of a decoder, a single chain of short
// kernels (128 streams, 12 layers of 512: 80.4 -> 76.2 ms a segment of 64 steps; pdl_trigger() lets the
// successor start as soon as all CTAs of a kernel are resident), and in the isolated attention op
// (forward, backward and reduction of 16 x 8 heads 36.4 -> 28.0 us); off in whole-segment passes unless
// NNCU_PDL=1: there a side stream's kernels fill the gaps, and the resident successors take SM resources
// from them (train steps of the bf16 models between 4 % faster and 2 % slower).
__device__ __forceinline__ void pdl_wait()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
__device__ __forceinline__ void pdl_trigger()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
// set while the launches of a chain are queued by this thread
extern thread_local bool g_nncu_step_chain;
struct ChainScope {
    const bool before = g_nncu_step_chain;
    ChainScope() { g_nncu_step_chain = true; }
    ~ChainScope() { g_nncu_step_chain = before; }
};
inline bool nncu_pdl_enabled()
{
    if (g_nncu_step_chain)
        return true;
    static int on = -1;
    if (on < 0) {
        const char *e = getenv("NNCU_PDL");
        on = (e && e[0] == '1') ? 1 : 0;
    }
    return on != 0;
}
template <typename... KArgs, typename... Args>
static cudaError_t launch_k(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                            Args &&...args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = nncu_pdl_enabled() ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

// every kernel launch in the library is followed by exactly one KERNEL_CHECK
extern unsigned long long g_nncu_launches;
#define KERNEL_CHECK()                 \
    do {                               \
        g_nncu_launches++;             \
        CUDA_TRY(cudaGetLastError());  \
    } while (0)

// optional per-launch timing of the tensor-core GEMM (nncu_profile_begin/end)
struct GemmProfiler {
    static const int MAX_EV = 8192;
    cudaEvent_t ev[2 * MAX_EV];
    double flops[MAX_EV];
    int n;
    bool ready;
};
extern GemmProfiler *g_nncu_prof;

__device__ __forceinline__ float to_f(float x) { return x; }
__device__ __forceinline__ float to_f(bf16 x) { return __bfloat162float(x); }
template <typename T> __device__ __forceinline__ T from_f(float x);
template <> __device__ __forceinline__ float from_f<float>(float x) { return x; }
template <> __device__ __forceinline__ bf16 from_f<bf16>(float x) { return __float2bfloat16_rn(x); }
// value after a round trip through the storage type
template <typename T> __device__ __forceinline__ float round_to(float x) { return to_f(from_f<T>(x)); }

static inline int ceil_div(long long a, long long b) { return (int)((a + b - 1) / b); }

// fixed-order warp reductions (xor butterfly: every lane ends with the same value,
// and the association depends on nothing but the lane count)
__device__ __forceinline__ float warp_sum(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_max(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
