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
// every thread executes pdl_wait() before its first access to memory that a kernel of the same pass or step
// touches and before any early return, so that the kernel cannot complete before its predecessor has.  (What
// stands since before the pass may be read earlier -- parameters, keys of other steps, the decoder's state -- because the
// pass's first kernel triggers only behind its own wait.)  Both calls are no-ops in
// a kernel launched the ordinary way.
//
// Which launches get such an edge (g_nncu_edges):
//   all      the one-symbol steps of a decoder, a single chain of short kernels (128 streams, 12 layers of 512: 80.4 ->
//            76.2 ms a segment of 64 steps; pdl_trigger() lets the successor start as soon as all CTAs of a kernel
//            are resident), and the isolated attention op (16 x 8 heads 36.4 -> 28.0 us)
//   GEMMs    whole-segment passes of bf16 models: a tensor-core GEMM sets up barriers, tensor memory and tensor maps
//            before it needs its operands, a microsecond that passes under its predecessor (6 layers of 512, 1024
//            rows: 790 -> 756 us; 12 layers, 2048 rows: 2489 -> 2345; 8 layers, 650 rows: 1307 -> 1216).  Edges on the
//            short kernels beside them take SM resources from the side stream's (1 to 2 % slower with them)
//   others   whole-segment passes of fp32 models, whose GEMMs have nothing to set up (4 layers of 256, 512 rows:
//            737 -> 699 us, with edges on the GEMMs too 759), but for the attention kernels
__device__ __forceinline__ void pdl_wait()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
__device__ __forceinline__ void pdl_trigger()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
enum { EDGE_GEMM = 1, EDGE_OTHER = 2, EDGE_ATTN = 4 };
// the kinds of launches of this thread that get an edge
extern thread_local int g_nncu_edges;
struct EdgeScope {
    const int before = g_nncu_edges;
    explicit EdgeScope(int kinds) { g_nncu_edges |= kinds; }
    ~EdgeScope() { g_nncu_edges = before; }
};
struct ChainScope : EdgeScope {
    ChainScope() : EdgeScope(EDGE_GEMM | EDGE_OTHER | EDGE_ATTN) {}
};
template <typename... KArgs, typename... Args>
static cudaError_t launch_kind(int kind, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
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
    cfg.numAttrs = (g_nncu_edges & kind) ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}
template <typename... KArgs, typename... Args>
static cudaError_t launch_k(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args &&...args)
{
    return launch_kind(EDGE_OTHER, kernel, grid, block, smem, st, static_cast<Args &&>(args)...);
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
