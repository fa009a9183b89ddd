// gemm_simt.cuh -- CUDA-core GEMM with fp32 accumulation.
//
// The fp32 engine of the library (fp32 models must not lose mantissa bits to
// tensor-core input formats) and the reference every tensor-core kernel is
// checked against.  Replaces nc_matmul / nc_matmul_add (libnc.h:270-276).
//
// Association, the same for every tile shape and launch: the contraction is cut into
// 16-wide slices, slice s belongs to chain s mod 4, every chain is one fp32 accumulator that
// receives fmaf(a, b, acc) in k order, and the result is (c0 + c1) + (c2 + c3).  It depends on
// K alone, so a row computed alone (one-symbol step) is bit-identical to the same row computed
// inside a whole segment.
//
// Why this split: fp32 models are small (128..512 rows and columns, K 128..1024), so what
// bounds a launch is latency, not the FMA pipe.  The four chains are four groups of 64 threads
// of one block: they give a 32 x 32 tile eight warps instead of two, so that a 512 x 256 output
// fills the chip with one wave.  Operands arrive by cp.async, three or four 64-wide stages in
// flight, so a K of 256 pays one memory latency instead of sixteen (one per 16-wide slice, which
// is what the loop of load - barrier - multiply - barrier before it paid).
#pragma once
#include "common.cuh"

enum { GEMM_NT = 0, GEMM_NN = 1, GEMM_TN = 2 };
// NT: C[m][n] = sum_k A[m][k] * B[n][k]      (y = x W^T)
// NN: C[m][n] = sum_k A[m][k] * B[k][n]      (dx = dy W)
// TN: C[m][n] = sum_k A[k][m] * B[k][n]      (dW = dy^T x; k runs over rows)

namespace simt {

constexpr int BKS = 64;         // k per stage: one 16-wide slice for each of the four chains
constexpr int KPITCH = BKS + 4; // row pitch of a K-contiguous tile (floats): eight consecutive rows fall on
                                // different 16-byte bank groups

// floats of one operand tile of R rows (or columns)
template <int R, bool KC> __host__ __device__ constexpr int tile_floats() { return KC ? R * KPITCH : BKS * (R + 4); }

__device__ __forceinline__ void cp16(float *dst, const float *src, int valid)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
                 "r"(valid * 4)
                 : "memory");
}
__device__ __forceinline__ void cp4(float *dst, const float *src, int valid)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
                 "r"(valid * 4)
                 : "memory");
}

// four consecutive elements from src (`valid` of them inside the matrix) to dst; base: any valid address
__device__ __forceinline__ void load4(float *dst, const float *src, const float *base, int valid, bool vec)
{
    if (vec) {
        cp16(dst, valid > 0 ? src : base, valid);
    } else {
#pragma unroll
        for (int e = 0; e < 4; e++)
            cp4(dst + e, e < valid ? src + e : base, e < valid ? 1 : 0);
    }
}
__device__ __forceinline__ void load4(float *dst, const bf16 *src, const bf16 *, int valid, bool)
{
    float4 v;
    v.x = valid > 0 ? to_f(src[0]) : 0.0f;
    v.y = valid > 1 ? to_f(src[1]) : 0.0f;
    v.z = valid > 2 ? to_f(src[2]) : 0.0f;
    v.w = valid > 3 ? to_f(src[3]) : 0.0f;
    *reinterpret_cast<float4 *>(dst) = v;
}

// one stage of an operand: rows [r0, r0 + R) x k [k0, k0 + 64), zero outside the matrix
template <int R, bool KC, typename T>
__device__ __forceinline__ void load_tile(float *s, const T *P, long ld, int r0, int rows, int k0, int K, bool vec)
{
    constexpr int CHUNKS = R * BKS / 4;
#pragma unroll
    for (int c0 = 0; c0 < CHUNKS; c0 += 256) {
        const int c = c0 + threadIdx.x;
        if (CHUNKS % 256 != 0 && c >= CHUNKS)
            break;
        if (KC) {
            const int r = c / (BKS / 4), k = (c % (BKS / 4)) * 4;
            const int valid = r0 + r < rows ? max(0, min(4, K - (k0 + k))) : 0;
            load4(s + r * KPITCH + k, P + (long)(r0 + r) * ld + k0 + k, P, valid, vec);
        } else {
            const int k = c / (R / 4), r = (c % (R / 4)) * 4;
            const int valid = k0 + k < K ? max(0, min(4, rows - (r0 + r))) : 0;
            load4(s + k * (R + 4) + r, P + (long)(k0 + k) * ld + r0 + r, P, valid, vec);
        }
    }
}

// row (or column) of the tile that element i of a thread's T-long run stands for; t: the thread's
// place along that side, N: threads along it.  K-contiguous tiles deal rows out one by one (eight
// neighbours read eight consecutive rows), the others in runs of up to four (one vector load).
template <int R, int T, bool KC> __device__ __forceinline__ int place(int t, int i)
{
    constexpr int N = R / T;
    if (KC)
        return t + N * i;
    return T == 8 ? (i >> 2) * (R / 2) + t * 4 + (i & 3) : t * T + i;
}

// elements of k slot kk (0..3 of a group of four) of a thread's run, from a tile that is not K-contiguous
template <int R, int T> __device__ __forceinline__ void run_load(const float *s, int k, int t, float (&v)[T])
{
    const float *p = s + k * (R + 4);
    if (T == 2) {
        const float2 x = *reinterpret_cast<const float2 *>(p + t * 2);
        v[0] = x.x; v[1] = x.y;
    } else {
#pragma unroll
        for (int c = 0; c < T / 4; c++) {
            const float4 x = *reinterpret_cast<const float4 *>(p + c * (R / 2) + t * 4);
            v[c * 4] = x.x; v[c * 4 + 1] = x.y; v[c * 4 + 2] = x.z; v[c * 4 + 3] = x.w;
        }
    }
}

template <int BM, int BN, bool AKC, bool BKC> __host__ __device__ constexpr int stages() { return BM >= 64 ? 3 : 4; }
template <int BM, int BN, bool AKC, bool BKC> __host__ __device__ constexpr size_t smem_bytes()
{
    constexpr size_t ring = (size_t)stages<BM, BN, AKC, BKC>() * (tile_floats<BM, AKC>() + tile_floats<BN, BKC>()) * 4;
    constexpr size_t sums = (size_t)4 * BM * BN * 4;
    return ring > sums ? ring : sums;
}

// a stage of one chain: 16 k
template <int BM, int BN, int TM, int TN, bool AKC, bool BKC>
__device__ __forceinline__ void slice(const float *As, const float *Bs, int kbase, int ty, int tx, float (&acc)[TM][TN])
{
#pragma unroll
    for (int k4 = 0; k4 < 4; k4++) {
        const int k = kbase + k4 * 4;
        float a[4][TM], b[4][TN];
        if (AKC) {
#pragma unroll
            for (int i = 0; i < TM; i++) {
                const float4 v = *reinterpret_cast<const float4 *>(As + place<BM, TM, true>(ty, i) * KPITCH + k);
                a[0][i] = v.x; a[1][i] = v.y; a[2][i] = v.z; a[3][i] = v.w;
            }
        } else {
#pragma unroll
            for (int kk = 0; kk < 4; kk++)
                run_load<BM, TM>(As, k + kk, ty, a[kk]);
        }
        if (BKC) {
#pragma unroll
            for (int j = 0; j < TN; j++) {
                const float4 v = *reinterpret_cast<const float4 *>(Bs + place<BN, TN, true>(tx, j) * KPITCH + k);
                b[0][j] = v.x; b[1][j] = v.y; b[2][j] = v.z; b[3][j] = v.w;
            }
        } else {
#pragma unroll
            for (int kk = 0; kk < 4; kk++)
                run_load<BN, TN>(Bs, k + kk, tx, b[kk]);
        }
#pragma unroll
        for (int kk = 0; kk < 4; kk++)
#pragma unroll
            for (int i = 0; i < TM; i++)
#pragma unroll
                for (int j = 0; j < TN; j++)
                    acc[i][j] = fmaf(a[kk][i], b[kk][j], acc[i][j]);
    }
}

template <int BM, int BN, int TM, int TN, int MODE, typename TA, typename TB, typename TC>
__global__ void __launch_bounds__(256, 2)
gemm_simt_kernel(int M, int N, int K, const TA *__restrict__ A, long lda, const TB *__restrict__ B, long ldb, TC *C, long ldc,
                 const float *__restrict__ bias, const TC *addsrc, int bias_n, int vec_a, int vec_b)
{
    constexpr bool AKC = MODE != GEMM_TN, BKC = MODE == GEMM_NT;
    constexpr int NST = stages<BM, BN, AKC, BKC>(), AF = tile_floats<BM, AKC>(), SF = AF + tile_floats<BN, BKC>();
    static_assert((BM / TM) * (BN / TN) == 64, "64 threads per chain");
    extern __shared__ __align__(16) float ring[];
    const int group = threadIdx.x >> 6, tid = threadIdx.x & 63;
    const int tx = tid % (BN / TN), ty = tid / (BN / TN);
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN; j++)
            acc[i][j] = 0.0f;
    pdl_trigger();
    pdl_wait();

    const int nst = (K + BKS - 1) / BKS;
    auto fetch = [&](int st) {
        float *s = ring + (st % NST) * SF;
        load_tile<BM, AKC>(s, A, lda, m0, M, st * BKS, K, vec_a != 0);
        load_tile<BN, BKC>(s + AF, B, ldb, n0, N, st * BKS, K, vec_b != 0);
    };
#pragma unroll
    for (int st = 0; st < NST - 1; st++) {
        if (st < nst)
            fetch(st);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    for (int st = 0; st < nst; st++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(NST - 2) : "memory");
        __syncthreads();
        if (st + NST - 1 < nst)
            fetch(st + NST - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float *s = ring + (st % NST) * SF;
        slice<BM, BN, TM, TN, AKC, BKC>(s, s + AF, group * 16, ty, tx, acc);
    }
    __syncthreads(); // the ring is idle: it takes the chains' sums, [chain][BM][BN]
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN; j++)
            ring[(group * BM + place<BM, TM, AKC>(ty, i)) * BN + place<BN, TN, BKC>(tx, j)] = acc[i][j];
    __syncthreads();
    for (int e = threadIdx.x; e < BM * BN; e += 256) {
        const int gm = m0 + e / BN, gn = n0 + e % BN;
        if (gm >= M || gn >= N)
            continue;
        float v = (ring[e] + ring[BM * BN + e]) + (ring[2 * BM * BN + e] + ring[3 * BM * BN + e]);
        if (bias && gn < bias_n)
            v += bias[gn];
        if (addsrc)
            v += to_f(addsrc[(long)gm * ldc + gn]);
        C[(long)gm * ldc + gn] = from_f<TC>(v);
    }
}

template <int BM, int BN, int TM, int TN, int MODE, typename TA, typename TB, typename TC>
static int launch(cudaStream_t st, int M, int N, int K, const TA *A, long lda, const TB *B, long ldb, TC *C, long ldc,
                  const float *bias, const TC *addsrc, int bias_n)
{
    constexpr size_t smem = smem_bytes<BM, BN, MODE != GEMM_TN, MODE == GEMM_NT>();
    static DeviceOnce once;
    NNCU_TRY(smem_limit(once, gemm_simt_kernel<BM, BN, TM, TN, MODE, TA, TB, TC>, (int)smem));
    const int vec_a = (reinterpret_cast<uintptr_t>(A) & 15) == 0 && lda % 4 == 0;
    const int vec_b = (reinterpret_cast<uintptr_t>(B) & 15) == 0 && ldb % 4 == 0;
    launch_kind(EDGE_GEMM, gemm_simt_kernel<BM, BN, TM, TN, MODE, TA, TB, TC>, dim3(ceil_div(N, BN), ceil_div(M, BM)), dim3(256), smem, st,
             M, N, K, A, lda, B, ldb, C, ldc, bias, addsrc, bias_n, vec_a, vec_b);
    KERNEL_CHECK();
    return NNCU_OK;
}

// The widest tile that still gives every SM a block: a wide tile reads shared memory least per FMA
// (64 x 32: 12 vector loads per 128, 32 x 32: 8 per 64), a narrow one spreads a small output over the chip.
// (64 x 64 reads less still, but its 192 blocks of a 1024 x 768 output load 44 SMs twice: 25 us at K 256 against 20.)
template <int MODE, typename TA, typename TB, typename TC>
static int gemm_mode(cudaStream_t st, int M, int N, int K, const TA *A, long lda, const TB *B, long ldb, TC *C, long ldc,
                     const float *bias, const TC *addsrc, int bias_n)
{
    if ((long)ceil_div(M, 64) * ceil_div(N, 32) >= 148)
        return launch<64, 32, 8, 4, MODE>(st, M, N, K, A, lda, B, ldb, C, ldc, bias, addsrc, bias_n);
    if ((long)ceil_div(M, 32) * ceil_div(N, 32) >= 100)
        return launch<32, 32, 4, 4, MODE>(st, M, N, K, A, lda, B, ldb, C, ldc, bias, addsrc, bias_n);
    return launch<16, 16, 2, 2, MODE>(st, M, N, K, A, lda, B, ldb, C, ldc, bias, addsrc, bias_n);
}

} // namespace simt

// addsrc (may be NULL, may alias C) is added to the product and has C's layout; bias goes to the
// output columns n < bias_n only
template <typename TA, typename TB, typename TC>
static int gemm_simt(cudaStream_t st, int mode, int M, int N, int K, const TA *A, long lda,
                     const TB *B, long ldb, TC *C, long ldc, const float *bias, const TC *addsrc, int bias_n = 1 << 30)
{
    if (M <= 0 || N <= 0)
        return NNCU_OK;
    switch (mode) {
    case GEMM_NT: return simt::gemm_mode<GEMM_NT>(st, M, N, K, A, lda, B, ldb, C, ldc, bias, addsrc, bias_n);
    case GEMM_NN: return simt::gemm_mode<GEMM_NN>(st, M, N, K, A, lda, B, ldb, C, ldc, bias, addsrc, bias_n);
    case GEMM_TN: return simt::gemm_mode<GEMM_TN>(st, M, N, K, A, lda, B, ldb, C, ldc, bias, addsrc, bias_n);
    }
    return nncu_fail(NNCU_ERR_INVALID, "gemm_simt: bad mode %d", mode);
}
