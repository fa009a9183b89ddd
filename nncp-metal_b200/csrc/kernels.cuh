// kernels.cuh -- the HBM-bound kernels of the train step: embedding, LayerNorm /
// RMSNorm with residual, activations, output softmax, loss gradient, column
// sums for bias gradients, the optimizer, the embedding gradient, transposes.
//
// Every reduction has a fixed association (warp butterflies, block trees and
// ordered loops; no atomics on floats), so a step is reproducible run to run
// and each forward row is independent of how many rows share the launch.
#pragma once
#include "common.cuh"

// ------------------------------------------------------------------
// embedding gather: x[r][:] = embed[id[r]][:] * mult        (nc_get_col, nncp.c:625-630)
template <typename T>
__global__ void embed_kernel(const int32_t *__restrict__ ids, const float *__restrict__ embed,
                             T *__restrict__ x, int rows, int D, float mult, int V)
{
    pdl_wait();
    pdl_trigger(); // behind the wait: the GEMM that follows reads weights before its own, and an update may precede this kernel
    int r = blockIdx.x;
    if (r >= rows)
        return;
    int id = ids[r];
    id = id < 0 ? 0 : (id >= V ? V - 1 : id);
    const float *e = embed + (size_t)id * D;
    T *o = x + (size_t)r * D;
    for (int i = threadIdx.x; i < D; i += blockDim.x)
        o[i] = from_f<T>(e[i] * mult);
}

// ------------------------------------------------------------------
// s = a (+ res); y = norm(s) * g + b.  One warp per row.     (layer_norm, nncp.c:279-288)
// mode: 0 = copy only (y = s), 1 = LayerNorm, 2 = RMSNorm.  s_out / stats may be NULL.
// The statistics are taken from s after rounding to the storage type, so that the
// backward pass, which reads the stored s, sees exactly the normalised values.
template <typename T>
__global__ void __launch_bounds__(128)
residual_norm_kernel(const T *__restrict__ a, const T *__restrict__ res, T *__restrict__ s_out,
                     T *__restrict__ y, const float *__restrict__ g, const float *__restrict__ b,
                     float *__restrict__ stats, int rows, int D, int mode)
{
    pdl_trigger();
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r = blockIdx.x * 4 + warp;
    if (r >= rows)
        return;
    const T *ar = a + (size_t)r * D;
    const T *rr = res ? res + (size_t)r * D : nullptr;
    float sum = 0.0f;
    for (int i = lane; i < D; i += 32) {
        float v = to_f(ar[i]);
        if (rr)
            v = round_to<T>(v + to_f(rr[i]));
        sum += v;
    }
    float mu = 0.0f, rstd = 1.0f;
    if (mode != 0) {
        if (mode == 1)
            mu = warp_sum(sum) / (float)D;
        float var = 0.0f;
        for (int i = lane; i < D; i += 32) {
            float v = to_f(ar[i]);
            if (rr)
                v = round_to<T>(v + to_f(rr[i]));
            var += (v - mu) * (v - mu);
        }
        var = warp_sum(var) / (float)D;
        rstd = 1.0f / sqrtf(var + 1e-5f);
        if (stats && lane == 0) {
            stats[2 * r] = mu;
            stats[2 * r + 1] = rstd;
        }
    }
    for (int i = lane; i < D; i += 32) {
        float v = to_f(ar[i]);
        if (rr)
            v = round_to<T>(v + to_f(rr[i]));
        if (s_out)
            s_out[(size_t)r * D + i] = from_f<T>(v);
        float o = (mode != 0) ? (v - mu) * rstd * g[i] + b[i] : v;
        y[(size_t)r * D + i] = from_f<T>(o);
    }
}

// Adjoint of y = norm(x)*g + b:  dx = (base ? base : 0) + J^T dy ; per-block partial column
// sums in part[blockIdx][3][D]: dg, db and (if want_sum) the column sums of the dx just
// written (the bias gradient of the projection that produced x).  Block = 8 warps, each warp
// walks rows blockIdx*RPB + warp, +8, ... inside the block's RPB-row chunk.
template <typename T>
__global__ void __launch_bounds__(256)
norm_bwd_kernel(const T *__restrict__ dy, const T *__restrict__ x, const float *__restrict__ g,
                const float *__restrict__ stats, const T *__restrict__ base, T *__restrict__ dx,
                float *__restrict__ part, int rows, int D, int mode, int rpb, int want_sum)
{
    pdl_trigger();
    pdl_wait();
    extern __shared__ float sm[]; // [8][3][D]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float *mydg = sm + (size_t)warp * 3 * D, *mydb = mydg + D, *mydx = mydb + D;
    for (int i = lane; i < 3 * D; i += 32)
        mydg[i] = 0.0f;
    const int r_end = min(rows, (blockIdx.x + 1) * rpb);
    for (int r = blockIdx.x * rpb + warp; r < r_end; r += 8) {
        const T *xr = x + (size_t)r * D, *dyr = dy + (size_t)r * D;
        const float mu = stats[2 * r], rstd = stats[2 * r + 1];
        float s1 = 0.0f, s2 = 0.0f;
        for (int i = lane; i < D; i += 32) {
            float xh = (to_f(xr[i]) - mu) * rstd;
            float d = to_f(dyr[i]);
            float dxh = d * g[i];
            s1 += dxh;
            s2 += dxh * xh;
            mydg[i] += d * xh;
            mydb[i] += d;
        }
        s1 = warp_sum(s1) / (float)D;
        s2 = warp_sum(s2) / (float)D;
        if (mode == 2)
            s1 = 0.0f;
        for (int i = lane; i < D; i += 32) {
            float xh = (to_f(xr[i]) - mu) * rstd;
            float dxh = to_f(dyr[i]) * g[i];
            float v = rstd * (dxh - s1 - xh * s2);
            if (base)
                v += to_f(base[(size_t)r * D + i]);
            T o = from_f<T>(v);
            dx[(size_t)r * D + i] = o;
            if (want_sum)
                mydx[i] += to_f(o);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 3 * D; i += blockDim.x) {
        float s = 0.0f;
#pragma unroll
        for (int w = 0; w < 8; w++)
            s += sm[(size_t)w * 3 * D + i];
        part[(size_t)blockIdx.x * 3 * D + i] = s;
    }
}

// ---- rows held in registers: 16-byte accesses, one pass over memory, one warp per row.  Lane l owns
// the W = 16 / sizeof(T) elements from c * 32 * W + l * W of every chunk c; D is a multiple of W and at
// most NC * 32 * W, what lies past D reads as zero and is not written.
template <typename T> struct RowVec {
    static constexpr int W = 16 / (int)sizeof(T), CHUNK = 32 * W;
};
template <typename T, int NC, int W>
__device__ __forceinline__ void row_load(const T *row, int lane, int D, float (&v)[NC][W])
{
#pragma unroll
    for (int c = 0; c < NC; c++) {
        const int at = c * 32 * W + lane * W;
        uint4 u = make_uint4(0u, 0u, 0u, 0u);
        if (at < D)
            u = *reinterpret_cast<const uint4 *>(row + at);
        const T *h = reinterpret_cast<const T *>(&u);
#pragma unroll
        for (int e = 0; e < W; e++)
            v[c][e] = to_f(h[e]);
    }
}
template <typename T, int NC, int W>
__device__ __forceinline__ void row_store(T *row, int lane, int D, const float (&v)[NC][W])
{
#pragma unroll
    for (int c = 0; c < NC; c++) {
        const int at = c * 32 * W + lane * W;
        uint4 u;
        T *h = reinterpret_cast<T *>(&u);
#pragma unroll
        for (int e = 0; e < W; e++)
            h[e] = from_f<T>(v[c][e]);
        if (at < D)
            *reinterpret_cast<uint4 *>(row + at) = u;
    }
}
template <int NC, int W>
__device__ __forceinline__ void vec_load_f32(const float *p, int lane, int D, float (&v)[NC][W])
{
#pragma unroll
    for (int c = 0; c < NC; c++) {
        const int at = c * 32 * W + lane * W;
#pragma unroll
        for (int e = 0; e < W; e += 4) {
            const float4 a = at < D ? *reinterpret_cast<const float4 *>(p + at + e) : make_float4(0.f, 0.f, 0.f, 0.f);
            v[c][e] = a.x; v[c][e + 1] = a.y; v[c][e + 2] = a.z; v[c][e + 3] = a.w;
        }
    }
}

// v <- norm(v) * g + b for a row over a warp's registers (mode 1 LayerNorm, 2 RMSNorm); lane 0 leaves the
// statistics in stats[0], stats[1] when wanted
template <int NC, int W>
__device__ __forceinline__ void norm_row(float (&v)[NC][W], const float (&gv)[NC][W], const float (&bv)[NC][W], int lane, int D, int mode,
                                         float *stats)
{
    float mu = 0.0f;
    if (mode == 1) {
        float sum = 0.0f;
#pragma unroll
        for (int c = 0; c < NC; c++)
#pragma unroll
            for (int e = 0; e < W; e++)
                sum += v[c][e];
        mu = warp_sum(sum) / (float)D;
    }
    float var = 0.0f;
#pragma unroll
    for (int c = 0; c < NC; c++)
        if (c * 32 * W + lane * W < D)
#pragma unroll
            for (int e = 0; e < W; e++)
                var += (v[c][e] - mu) * (v[c][e] - mu);
    var = warp_sum(var) / (float)D;
    const float rstd = 1.0f / sqrtf(var + 1e-5f);
    if (stats && lane == 0) {
        stats[0] = mu;
        stats[1] = rstd;
    }
#pragma unroll
    for (int c = 0; c < NC; c++)
#pragma unroll
        for (int e = 0; e < W; e++)
            v[c][e] = (v[c][e] - mu) * rstd * gv[c][e] + bv[c][e];
}

// residual_norm_kernel with the row in registers; same arguments and rounding points (s is rounded
// to the storage type before the statistics), sums taken per lane, then over the warp.
template <typename T, int NC>
__global__ void __launch_bounds__(128)
residual_norm_vec_kernel(const T *__restrict__ a, const T *__restrict__ res, T *__restrict__ s_out,
                         T *__restrict__ y, const float *__restrict__ g, const float *__restrict__ b,
                         float *__restrict__ stats, int rows, int D, int mode)
{
    pdl_trigger();
    constexpr int W = RowVec<T>::W;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r = blockIdx.x * 4 + warp;
    // gain and bias are parameters, which no kernel of a pass writes (see gemm_tc_kernel's weights): on their way before the wait
    float gv[NC][W], bv[NC][W];
    if (mode != 0) {
        vec_load_f32<NC, W>(g, lane, D, gv);
        vec_load_f32<NC, W>(b, lane, D, bv);
    }
    pdl_wait();
    if (r >= rows)
        return;
    float v[NC][W];
    row_load<T, NC, W>(a + (size_t)r * D, lane, D, v);
    if (res) {
        float w[NC][W];
        row_load<T, NC, W>(res + (size_t)r * D, lane, D, w);
#pragma unroll
        for (int c = 0; c < NC; c++)
#pragma unroll
            for (int e = 0; e < W; e++)
                v[c][e] = round_to<T>(v[c][e] + w[c][e]);
    }
    if (s_out)
        row_store<T, NC, W>(s_out + (size_t)r * D, lane, D, v);
    if (mode == 0) {
        row_store<T, NC, W>(y + (size_t)r * D, lane, D, v);
        return;
    }
    norm_row<NC, W>(v, gv, bv, lane, D, mode, stats ? stats + 2 * r : nullptr);
    row_store<T, NC, W>(y + (size_t)r * D, lane, D, v);
}

// norm_bwd_kernel with the row in registers: every warp walks rpb / 8 rows and keeps its lanes'
// column sums (dg, db and, if asked, the sums of the dx just written) in registers; the block's
// sums go to part[block][3][D].  Several rows per warp keep the number of partial rows that the
// reduction launch has to read near two per SM.
template <typename T, int NC>
__global__ void __launch_bounds__(256)
norm_bwd_vec_kernel(const T *__restrict__ dy, const T *__restrict__ x, const float *__restrict__ g,
                    const float *__restrict__ stats, const T *__restrict__ base, T *__restrict__ dx,
                    float *__restrict__ part, int rows, int D, int mode, int rpb, int want_sum)
{
    pdl_trigger();
    pdl_wait();
    constexpr int W = RowVec<T>::W;
    extern __shared__ float sm[]; // [8][D]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // The row's operands stay packed as they came (NC 16-byte pieces each) and are unpacked at each use,
    // and the gains are read again from the L1 cache: the sums alone are 3 * NC * W registers.
    float dg[NC][W], db[NC][W], ds[NC][W];
#pragma unroll
    for (int c = 0; c < NC; c++)
#pragma unroll
        for (int e = 0; e < W; e++)
            dg[c][e] = db[c][e] = ds[c][e] = 0.0f;
    auto gain = [&](int c, int e4) {
        const int at = c * 32 * W + lane * W + e4;
        return at < D ? __ldg(reinterpret_cast<const float4 *>(g + at)) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    const int r_end = min(rows, (int)(blockIdx.x + 1) * rpb);
    for (int r = blockIdx.x * rpb + warp; r < r_end; r += 8) {
        uint4 xu[NC], du[NC], bu[NC];
        const float mu = stats[2 * r], rstd = stats[2 * r + 1];
#pragma unroll
        for (int c = 0; c < NC; c++) {
            const int at = c * 32 * W + lane * W;
            xu[c] = du[c] = bu[c] = make_uint4(0u, 0u, 0u, 0u);
            if (at < D) {
                xu[c] = *reinterpret_cast<const uint4 *>(x + (size_t)r * D + at);
                du[c] = *reinterpret_cast<const uint4 *>(dy + (size_t)r * D + at);
                if (base)
                    bu[c] = *reinterpret_cast<const uint4 *>(base + (size_t)r * D + at);
            }
        }
        float s1 = 0.0f, s2 = 0.0f;
#pragma unroll
        for (int c = 0; c < NC; c++) {
            const T *xp = reinterpret_cast<const T *>(&xu[c]), *dp = reinterpret_cast<const T *>(&du[c]);
#pragma unroll
            for (int e4 = 0; e4 < W; e4 += 4) {
                const float4 g4 = gain(c, e4);
                const float gg[4] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const int e = e4 + k;
                    const float xh = (to_f(xp[e]) - mu) * rstd, d = to_f(dp[e]), dxh = gg[k] * d;
                    s1 += dxh;
                    s2 += dxh * xh;
                    dg[c][e] += xh * d;
                    db[c][e] += d;
                }
            }
        }
        s1 = warp_sum(s1) / (float)D;
        s2 = warp_sum(s2) / (float)D;
        if (mode == 2)
            s1 = 0.0f;
#pragma unroll
        for (int c = 0; c < NC; c++) {
            const T *xp = reinterpret_cast<const T *>(&xu[c]), *dp = reinterpret_cast<const T *>(&du[c]),
                    *bp = reinterpret_cast<const T *>(&bu[c]);
            uint4 ou;
            T *op = reinterpret_cast<T *>(&ou);
#pragma unroll
            for (int e4 = 0; e4 < W; e4 += 4) {
                const float4 g4 = gain(c, e4);
                const float gg[4] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const int e = e4 + k;
                    const float xh = (to_f(xp[e]) - mu) * rstd;
                    const float vv = rstd * (gg[k] * to_f(dp[e]) - s1 - xh * s2);
                    op[e] = from_f<T>(base ? vv + to_f(bp[e]) : vv);
                    ds[c][e] += to_f(op[e]);
                }
            }
            if (c * 32 * W + lane * W < D)
                *reinterpret_cast<uint4 *>(dx + (size_t)r * D + c * 32 * W + lane * W) = ou;
        }
    }
    // the eight warps' sums, one quantity after the other through one buffer
    float *mine = sm + (size_t)warp * D;
    auto fold = [&](const float (&v)[NC][W], int q) {
        if (q)
            __syncthreads();
#pragma unroll
        for (int c = 0; c < NC; c++) {
            const int at = c * 32 * W + lane * W;
            if (at < D)
#pragma unroll
                for (int e = 0; e < W; e += 4)
                    *reinterpret_cast<float4 *>(mine + at + e) = make_float4(v[c][e], v[c][e + 1], v[c][e + 2], v[c][e + 3]);
        }
        __syncthreads();
        for (int i = threadIdx.x; i < D; i += 256) {
            float s = 0.0f;
#pragma unroll
            for (int w = 0; w < 8; w++)
                s += sm[(size_t)w * D + i];
            part[((size_t)blockIdx.x * 3 + q) * D + i] = s;
        }
    };
    fold(dg, 0);
    fold(db, 1);
    if (want_sum)
        fold(ds, 2);
}

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi)
{
    __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t *>(&h);
}

// out[i] = ws[0][i] + ws[1][i] + ... (in that order) for the partial products of a split-K GEMM;
// n a multiple of 4.
template <typename TO>
__global__ void splitk_reduce_kernel(const float *__restrict__ ws, int ksplit, size_t n, TO *__restrict__ out)
{
    pdl_trigger();
    pdl_wait();
    const size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (i >= n)
        return;
    float4 acc = *reinterpret_cast<const float4 *>(ws + i);
    for (int z = 1; z < ksplit; z++) {
        const float4 v = *reinterpret_cast<const float4 *>(ws + (size_t)z * n + i);
        acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
    }
    if constexpr (sizeof(TO) == 4) {
        *reinterpret_cast<float4 *>(out + i) = acc;
    } else {
        const uint2 pk = make_uint2(pack_bf16x2(acc.x, acc.y), pack_bf16x2(acc.z, acc.w));
        *reinterpret_cast<uint2 *>(out + i) = pk;
    }
}

// Every column / stream reduction of one layer's backward pass in one launch.  Job kinds:
//   0  out[c] = sum over parts p of part[p*stride + off + c], the parts dealt to 8 groups of
//      consecutive parts whose sums are added in group order
//   1  out[i] (+)= sum over parts (streams) in order of part[p*stride + i]
//   2  the same for the position table, [n_parts streams] x [heads][off] values, whose heads are each summed over streams
//      into fab::slots_of parts already
// blk0 is the job's first block; a block finds its job by a short scan (the table is a kernel
// argument, so the launch can sit in a captured graph).
struct ReduceJob {
    const float *part;
    float *out;
    int n_parts, stride, n, off, kind, accumulate, blk0;
};
constexpr int MAX_REDUCE_JOBS = 16;
struct ReduceJobs {
    int n_jobs;
    ReduceJob job[MAX_REDUCE_JOBS];
};
__global__ void __launch_bounds__(256) reduce_jobs_kernel(const __grid_constant__ ReduceJobs jobs)
{
    pdl_wait();
    __shared__ float sm[8][33];
    int j = 0;
    while (j + 1 < jobs.n_jobs && (int)blockIdx.x >= jobs.job[j + 1].blk0)
        j++;
    const ReduceJob &jb = jobs.job[j];
    const int blk = blockIdx.x - jb.blk0;
    if (jb.kind >= 1) {
        const int i = blk * 256 + threadIdx.x;
        if (i < jb.n) {
            // a loop for each kind: one over a number that either may have set is 5 to 35 % slower (148 parts of 8192 values
            // 5.8 -> 7.7 us, 32 of 65536 2.4 -> 2.8)
            float s = 0.0f;
            if (jb.kind == 1) {
#pragma unroll 8 // eight parts' loads in flight
                for (int p = 0; p < jb.n_parts; p++)
                    s += jb.part[(size_t)p * jb.stride + i];
            } else {
                const int parts = fab::slots_of(jb.n_parts, jb.n / jb.off, i / jb.off);
#pragma unroll 8
                for (int p = 0; p < parts; p++)
                    s += jb.part[(size_t)p * jb.stride + i];
            }
            jb.out[i] = jb.accumulate ? jb.out[i] + s : s;
        }
        return;
    }
    const int c = blk * 32 + (threadIdx.x & 31), grp = threadIdx.x >> 5;
    const int per = (jb.n_parts + 7) / 8;
    float s = 0.0f;
    if (c < jb.n) {
        const float *src = jb.part + jb.off + c;
        const int p1 = min(jb.n_parts, (grp + 1) * per);
#pragma unroll 8
        for (int p = grp * per; p < p1; p++)
            s += src[(size_t)p * jb.stride];
    }
    sm[grp][threadIdx.x & 31] = s;
    __syncthreads();
    if (grp == 0 && c < jb.n) {
        float t = 0.0f;
#pragma unroll
        for (int w = 0; w < 8; w++)
            t += sm[w][threadIdx.x];
        jb.out[c] = t;
    }
}

// dst = a + b (elementwise), used where a residual joins without a norm
template <typename T>
__global__ void add_kernel(const T *__restrict__ a, const T *__restrict__ b, T *__restrict__ dst,
                           size_t n)
{
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n)
        dst[i] = from_f<T>(to_f(a[i]) + to_f(b[i]));
}

// ------------------------------------------------------------------
// LN_COEF (nncp.c:892-894, 975-977): a sub-layer's output is multiplied by the layer's learned
// scalar alpha before the residual sum.  Forward: dst = alpha * src.  Backward, one block per row:
// dt = alpha * ds for the branch, and part[r] = sum_c ds[r][c] * a[r][c] (the row's share of
// d alpha, columns added in a fixed order); the rows are summed later by one ordered job.
template <typename T>
__global__ void scale_rows_kernel(const T *__restrict__ src, const float *__restrict__ alpha, T *__restrict__ dst, size_t n)
{
    pdl_trigger();
    pdl_wait();
    const float al = alpha[0];
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        dst[i] = from_f<T>(al * to_f(src[i]));
}

template <typename T>
__global__ void __launch_bounds__(128)
scale_dot_kernel(const T *__restrict__ ds, const T *__restrict__ a, const float *__restrict__ alpha, T *__restrict__ dt,
                 float *__restrict__ part, int rows, int D)
{
    pdl_trigger();
    pdl_wait();
    __shared__ float red[4];
    const int r = blockIdx.x;
    if (r >= rows)
        return;
    const float al = alpha[0];
    float s = 0.0f;
    for (int c = threadIdx.x; c < D; c += 128) {
        const float d = to_f(ds[(size_t)r * D + c]);
        s += d * to_f(a[(size_t)r * D + c]);
        dt[(size_t)r * D + c] = from_f<T>(al * d);
    }
    s = warp_sum(s);
    if ((threadIdx.x & 31) == 0)
        red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0)
        part[r] = (red[0] + red[1]) + (red[2] + red[3]);
}

// ------------------------------------------------------------------
// feed-forward activation (nncp.c:938-966).  hpre [rows][F1], hact [rows][F].
__device__ __forceinline__ float gelu_f(float x)
{
    return 0.5f * x * (1.0f + tanhf(0.7978845608028654f * (x + 0.044715f * x * x * x)));
}
__device__ __forceinline__ float gelu_grad_f(float x)
{
    float u = 0.7978845608028654f * (x + 0.044715f * x * x * x);
    float t = tanhf(u);
    float du = 0.7978845608028654f * (1.0f + 3.0f * 0.044715f * x * x);
    return 0.5f * (1.0f + t) + 0.5f * x * (1.0f - t * t) * du;
}

// The same two functions on the hardware tanh (one MUFU instruction, absolute error about 5e-4,
// below the rounding step of the bf16 values they feed): the bf16 activation kernels are bound
// by their instruction count, and tanhf is most of it.
__device__ __forceinline__ float tanh_hw(float x)
{
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float gelu_hw(float x)
{
    return 0.5f * x * (1.0f + tanh_hw(0.7978845608028654f * (x + 0.044715f * x * x * x)));
}
__device__ __forceinline__ float gelu_grad_hw(float x)
{
    float u = 0.7978845608028654f * (x + 0.044715f * x * x * x);
    float t = tanh_hw(u);
    float du = 0.7978845608028654f * (1.0f + 3.0f * 0.044715f * x * x);
    return 0.5f * (1.0f + t) + 0.5f * x * (1.0f - t * t) * du;
}

// x * sigmoid(x), the gate function of FF_ACT_GATED_SILU (nc_gated_swish with beta 1, nncp.c:957-962),
// and its derivative; the _hw forms take the sigmoid from the hardware tanh.
__device__ __forceinline__ float silu_f(float x) { return x / (1.0f + expf(-x)); }
__device__ __forceinline__ float silu_grad_f(float x)
{
    const float s = 1.0f / (1.0f + expf(-x));
    return s * (1.0f + x * (1.0f - s));
}
__device__ __forceinline__ float silu_hw(float x) { return x * (0.5f + 0.5f * tanh_hw(0.5f * x)); }
__device__ __forceinline__ float silu_grad_hw(float x)
{
    const float s = 0.5f + 0.5f * tanh_hw(0.5f * x);
    return s * (1.0f + x * (1.0f - s));
}
// the gated activations: value and derivative of the function applied to the first half
__device__ __forceinline__ float gate_f(float x, int act) { return act == NNCU_FF_GATED_SILU ? silu_f(x) : gelu_f(x); }
__device__ __forceinline__ float gate_grad_f(float x, int act) { return act == NNCU_FF_GATED_SILU ? silu_grad_f(x) : gelu_grad_f(x); }
__device__ __forceinline__ float gate_hw(float x, int act) { return act == NNCU_FF_GATED_SILU ? silu_hw(x) : gelu_hw(x); }
__device__ __forceinline__ float gate_grad_hw(float x, int act) { return act == NNCU_FF_GATED_SILU ? silu_grad_hw(x) : gelu_grad_hw(x); }

template <typename T>
__global__ void act_fwd_kernel(const T *__restrict__ hpre, T *__restrict__ hact, int rows, int F,
                               int F1, int act)
{
    pdl_trigger();
    pdl_wait();
    size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (size_t)rows * F)
        return;
    int r = (int)(idx / F), i = (int)(idx % F);
    float a = to_f(hpre[(size_t)r * F1 + i]), o;
    if (act == NNCU_FF_RELU)
        o = a > 0.0f ? a : 0.0f;
    else if (act == NNCU_FF_GELU)
        o = gelu_f(a);
    else
        o = gate_f(a, act) * to_f(hpre[(size_t)r * F1 + F + i]);
    hact[idx] = from_f<T>(o);
}

// Eight columns per thread (16-byte accesses); same arithmetic per element as act_fwd_kernel.
// Needs F and F1 to be multiples of 8 and 16-byte aligned rows.
__global__ void act_fwd_vec_kernel(const bf16 *__restrict__ hpre, bf16 *__restrict__ hact, int rows, int F,
                                   int F1, int act)
{
    pdl_trigger();
    pdl_wait();
    const int cpr = F / 8;
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (size_t)rows * cpr)
        return;
    const int r = (int)(idx / cpr), i = (int)(idx % cpr) * 8;
    const uint4 va = *reinterpret_cast<const uint4 *>(hpre + (size_t)r * F1 + i);
    const bf16 *a = reinterpret_cast<const bf16 *>(&va);
    uint4 vo;
    bf16 *o = reinterpret_cast<bf16 *>(&vo);
    if (act == NNCU_FF_RELU) {
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const float x = to_f(a[j]);
            o[j] = from_f<bf16>(x > 0.0f ? x : 0.0f);
        }
    } else if (act == NNCU_FF_GELU) {
#pragma unroll
        for (int j = 0; j < 8; j++)
            o[j] = from_f<bf16>(gelu_hw(to_f(a[j])));
    } else {
        const uint4 vg = *reinterpret_cast<const uint4 *>(hpre + (size_t)r * F1 + F + i);
        const bf16 *g = reinterpret_cast<const bf16 *>(&vg);
#pragma unroll
        for (int j = 0; j < 8; j++)
            o[j] = from_f<bf16>(gate_hw(to_f(a[j]), act) * to_f(g[j]));
    }
    *reinterpret_cast<uint4 *>(hact + (size_t)r * F + i) = vo;
}

// Adjoint of the activation, and (part != NULL) per-chunk column sums of the result for the
// ff_bias1 gradient: part[chunk][F1].  grid (ceil(F/128), ceil(rows/ACT_BWD_ROWS)); one column per
// thread, short chains of rows (see act_bwd_vec_kernel).
constexpr int ACT_BWD_ROWS = 8;
template <typename T>
__global__ void __launch_bounds__(128)
act_bwd_kernel(const T *__restrict__ hpre, const T *__restrict__ dhact, T *__restrict__ dhpre,
               float *__restrict__ part, int rows, int F, int F1, int act)
{
    pdl_trigger();
    pdl_wait();
    const int i = blockIdx.x * 128 + threadIdx.x;
    if (i >= F)
        return;
    const int r0 = blockIdx.y * ACT_BWD_ROWS;
    float s0 = 0.0f, s1 = 0.0f;
#pragma unroll
    for (int rr = 0; rr < ACT_BWD_ROWS; rr++) {
        const int r = r0 + rr;
        if (r >= rows)
            break;
        float a = to_f(hpre[(size_t)r * F1 + i]), d = to_f(dhact[(size_t)r * F + i]);
        if (act == NNCU_FF_RELU || act == NNCU_FF_GELU) {
            T o = from_f<T>(act == NNCU_FF_RELU ? (a > 0.0f ? d : 0.0f) : d * gelu_grad_f(a));
            dhpre[(size_t)r * F1 + i] = o;
            s0 += to_f(o);
        } else {
            float gate = to_f(hpre[(size_t)r * F1 + F + i]);
            T o0 = from_f<T>(d * gate * gate_grad_f(a, act)), o1 = from_f<T>(d * gate_f(a, act));
            dhpre[(size_t)r * F1 + i] = o0;
            dhpre[(size_t)r * F1 + F + i] = o1;
            s0 += to_f(o0);
            s1 += to_f(o1);
        }
    }
    if (part) {
        part[(size_t)blockIdx.y * F1 + i] = s0;
        if (F1 > F)
            part[(size_t)blockIdx.y * F1 + F + i] = s1;
    }
}

// W = 2 or 4 columns per thread, ACT_BWD_ROWS rows per block; element arithmetic as in act_bwd_kernel.
// Bound by its instructions (some 20 an element) and, before that, by latency: all of a thread's loads go
// out before the first is used (8192 rows of 2048: 27 -> 22 us, their bytes need 15).  F a multiple of W; grid (ceil(F / (128 W)), ceil(rows/ACT_BWD_ROWS)).
template <int W>
__global__ void __launch_bounds__(128)
act_bwd_vec_kernel(const bf16 *__restrict__ hpre, const bf16 *__restrict__ dhact, bf16 *__restrict__ dhpre,
                   float *__restrict__ part, int rows, int F, int F1, int act)
{
    pdl_trigger();
    pdl_wait();
    constexpr int N = W / 2; // words of two columns
    struct alignas(4 * N) Pack {
        __nv_bfloat162 v[N];
    };
    const int i = (blockIdx.x * 128 + threadIdx.x) * W;
    if (i >= F)
        return;
    const int r0 = blockIdx.y * ACT_BWD_ROWS, n = min(rows - r0, ACT_BWD_ROWS);
    const bool gated = !(act == NNCU_FF_RELU || act == NNCU_FF_GELU);
    Pack pa[ACT_BWD_ROWS], pd[ACT_BWD_ROWS], pg[ACT_BWD_ROWS];
#pragma unroll
    for (int rr = 0; rr < ACT_BWD_ROWS; rr++)
        if (rr < n) {
            const size_t r = r0 + rr;
            pa[rr] = *reinterpret_cast<const Pack *>(hpre + r * F1 + i);
            pd[rr] = *reinterpret_cast<const Pack *>(dhact + r * F + i);
            if (gated)
                pg[rr] = *reinterpret_cast<const Pack *>(hpre + r * F1 + F + i);
        }
    float s0[W], s1[W];
#pragma unroll
    for (int j = 0; j < W; j++)
        s0[j] = s1[j] = 0.0f;
#pragma unroll
    for (int rr = 0; rr < ACT_BWD_ROWS; rr++) {
        if (rr >= n)
            break;
        const size_t r = r0 + rr;
        Pack o0, o1;
#pragma unroll
        for (int k = 0; k < N; k++) {
            const float a[2] = {__low2float(pa[rr].v[k]), __high2float(pa[rr].v[k])}, d[2] = {__low2float(pd[rr].v[k]), __high2float(pd[rr].v[k])};
            bf16 x[2], y[2];
            if (!gated) {
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    x[j] = from_f<bf16>(act == NNCU_FF_RELU ? (a[j] > 0.0f ? d[j] : 0.0f) : d[j] * gelu_grad_hw(a[j]));
                    s0[2 * k + j] += to_f(x[j]);
                }
            } else {
                const float gate[2] = {__low2float(pg[rr].v[k]), __high2float(pg[rr].v[k])};
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    x[j] = from_f<bf16>(d[j] * gate[j] * gate_grad_hw(a[j], act));
                    y[j] = from_f<bf16>(d[j] * gate_hw(a[j], act));
                    s0[2 * k + j] += to_f(x[j]);
                    s1[2 * k + j] += to_f(y[j]);
                }
                o1.v[k] = __halves2bfloat162(y[0], y[1]);
            }
            o0.v[k] = __halves2bfloat162(x[0], x[1]);
        }
        *reinterpret_cast<Pack *>(dhpre + r * F1 + i) = o0;
        if (gated)
            *reinterpret_cast<Pack *>(dhpre + r * F1 + F + i) = o1;
    }
    if (part) {
        float *row = part + (size_t)blockIdx.y * F1;
#pragma unroll
        for (int j = 0; j < W; j++) {
            row[i + j] = s0[j];
            if (gated)
                row[F + i + j] = s1[j];
        }
    }
}

// ------------------------------------------------------------------
// block-wide fixed-order reductions for 256-thread blocks
__device__ __forceinline__ float block_sum_256(float v, float *red)
{
    v = warp_sum(v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0)
        red[threadIdx.x >> 5] = v;
    __syncthreads();
    float s = 0.0f;
#pragma unroll
    for (int w = 0; w < 8; w++)
        s += red[w];
    return s;
}
__device__ __forceinline__ float block_max_256(float v, float *red)
{
    v = warp_max(v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0)
        red[threadIdx.x >> 5] = v;
    __syncthreads();
    float s = red[0];
#pragma unroll
    for (int w = 1; w < 8; w++)
        s = fmaxf(s, red[w]);
    return s;
}

// one row of softmax_rows_kernel, in place, by a block of 256 threads
template <typename T> __device__ __forceinline__ void softmax_row(float *zr, int V, T *d, float scale, float *red)
{
    float mx = -INFINITY;
    for (int i = threadIdx.x; i < V; i += 256)
        mx = fmaxf(mx, zr[i]);
    mx = block_max_256(mx, red);
    float s = 0.0f;
    for (int i = threadIdx.x; i < V; i += 256) {
        float e = expf(zr[i] - mx);
        zr[i] = e;
        s += e;
    }
    s = block_sum_256(s, red);
    float rs = 1.0f / s;
    for (int i = threadIdx.x; i < V; i += 256) {
        const float pv = zr[i] * rs;
        zr[i] = pv;
        d[i] = from_f<T>(pv * scale);
    }
}

// Rows whose sum softmax_rows_reg_kernel takes, in an order of its own: whoever computes such a row alone
// keeps to that order, so that a symbol step has the bits of the whole segment.
__host__ __device__ inline bool softmax_by_fours(int V) { return V % 1024 == 0 && V <= 16384; }

// one row as softmax_rows_reg_kernel computes it (four neighbouring logits at a time), in place
template <typename T> __device__ __forceinline__ void softmax_row_by_fours(float *zr, int V, T *d, float scale, float *red)
{
    float4 *z4 = reinterpret_cast<float4 *>(zr);
    float mx = -INFINITY;
    for (int i = threadIdx.x; i < V / 4; i += 256) {
        const float4 v = z4[i];
        mx = fmaxf(mx, fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w)));
    }
    mx = block_max_256(mx, red);
    float s = 0.0f;
    for (int i = threadIdx.x; i < V / 4; i += 256) {
        float4 v = z4[i];
        v.x = expf(v.x - mx);
        v.y = expf(v.y - mx);
        v.z = expf(v.z - mx);
        v.w = expf(v.w - mx);
        z4[i] = v;
        s += (v.x + v.y) + (v.z + v.w);
    }
    s = block_sum_256(s, red);
    const float rs = 1.0f / s;
    for (int i = threadIdx.x; i < V / 4; i += 256) {
        float4 v = z4[i];
        v.x *= rs;
        v.y *= rs;
        v.z *= rs;
        v.w *= rs;
        z4[i] = v;
        d[4 * i] = from_f<T>(v.x * scale);
        d[4 * i + 1] = from_f<T>(v.y * scale);
        d[4 * i + 2] = from_f<T>(v.z * scale);
        d[4 * i + 3] = from_f<T>(v.w * scale);
    }
}

// in-place softmax over the V symbols of each row of fp32 logits (nc_soft_max, nncp.c:1008).
// The output kernel of the forward pass: besides the probabilities it leaves dz = p * scale, the
// gradient of the loss with respect to the logits of every symbol but the target (which
// loss_fix_kernel corrects once the targets are known), so that the backward pass does not read
// the probability tables again.  *dz_fixed = 0 says that dz holds no target correction.
template <typename T>
__global__ void __launch_bounds__(256) softmax_rows_kernel(float *__restrict__ z, int rows, int V, T *__restrict__ dz, float scale,
                                                           int *__restrict__ dz_fixed)
{
    pdl_trigger();
    pdl_wait();
    __shared__ float red[8];
    int r = blockIdx.x;
    if (r >= rows)
        return;
    if (r == 0 && threadIdx.x == 0)
        *dz_fixed = 0;
    softmax_row(z + (size_t)r * V, V, dz + (size_t)r * V, scale, red);
}

// The same for rows of up to 16384 logits, V a multiple of 1024: the row stays in registers
// (one read and one write of memory, 16-byte accesses).  Thread t owns logits (k*256 + t)*4 .. +3.
template <typename T>
__global__ void __launch_bounds__(256) softmax_rows_reg_kernel(float *__restrict__ z, int rows, int V, T *__restrict__ dz,
                                                               float scale, int *__restrict__ dz_fixed)
{
    pdl_trigger();
    pdl_wait();
    __shared__ float red[8];
    const int r = blockIdx.x;
    if (r >= rows)
        return;
    if (r == 0 && threadIdx.x == 0)
        *dz_fixed = 0;
    float4 *zr = reinterpret_cast<float4 *>(z + (size_t)r * V);
    const int nv = V / 1024;
    float4 v[16];
    float mx = -INFINITY;
#pragma unroll
    for (int k = 0; k < 16; k++)
        if (k < nv) {
            v[k] = zr[k * 256 + threadIdx.x];
            mx = fmaxf(mx, fmaxf(fmaxf(v[k].x, v[k].y), fmaxf(v[k].z, v[k].w)));
        }
    mx = block_max_256(mx, red);
    float s = 0.0f;
#pragma unroll
    for (int k = 0; k < 16; k++)
        if (k < nv) {
            v[k].x = expf(v[k].x - mx);
            v[k].y = expf(v[k].y - mx);
            v[k].z = expf(v[k].z - mx);
            v[k].w = expf(v[k].w - mx);
            s += (v[k].x + v[k].y) + (v[k].z + v[k].w);
        }
    s = block_sum_256(s, red);
    const float rs = 1.0f / s;
#pragma unroll
    for (int k = 0; k < 16; k++)
        if (k < nv) {
            v[k].x *= rs;
            v[k].y *= rs;
            v[k].z *= rs;
            v[k].w *= rs;
            zr[k * 256 + threadIdx.x] = v[k];
            T *d = dz + (size_t)r * V + (size_t)(k * 256 + threadIdx.x) * 4;
            if (sizeof(T) == 2) {
                uint2 pk;
                pk.x = pack_bf16x2(v[k].x * scale, v[k].y * scale);
                pk.y = pack_bf16x2(v[k].z * scale, v[k].w * scale);
                *reinterpret_cast<uint2 *>(d) = pk;
            } else {
                *reinterpret_cast<float4 *>(d) = make_float4(v[k].x * scale, v[k].y * scale, v[k].z * scale, v[k].w * scale);
            }
        }
}

// The target correction of dz: for every row r, dz[r][t_r] = (p[r][t_r] - 1) * scale and
// logp[r] = ln p[r][t_r] (nc_indexed_log and the adjoint of the softmax, nncp.c:1170-1175).  A
// second call for the same forward pass (*dz_fixed != 0) first puts the old targets' entries back
// to p * scale.  loss_sum_kernel, queued behind it, adds the logp in a fixed order (thread i adds
// rows i, i + 256, ...; then the block sum) and raises the flag.
template <typename T>
__global__ void __launch_bounds__(256)
loss_fix_kernel(const float *__restrict__ probs, const int32_t *__restrict__ targets, int32_t *__restrict__ fixed_targets,
                const int *__restrict__ dz_fixed, T *__restrict__ dz, float *__restrict__ logp, int rows, int V, float scale)
{
    pdl_trigger();
    pdl_wait();
    const int r = blockIdx.x * 256 + threadIdx.x;
    if (r >= rows)
        return;
    const float *pr = probs + (size_t)r * V;
    T *d = dz + (size_t)r * V;
    if (*dz_fixed != 0) {
        const int old = fixed_targets[r];
        d[old] = from_f<T>(pr[old] * scale);
    }
    int t = targets[r];
    t = t < 0 ? 0 : (t >= V ? V - 1 : t);
    const float pt = pr[t];
    d[t] = from_f<T>((pt - 1.0f) * scale);
    fixed_targets[r] = t;
    logp[r] = logf(pt);
}

__global__ void __launch_bounds__(256) loss_sum_kernel(const float *__restrict__ v, int n, float *__restrict__ out,
                                                       int *__restrict__ dz_fixed)
{
    pdl_trigger();
    pdl_wait();
    __shared__ float red[8];
    float s = 0.0f;
    for (int i = threadIdx.x; i < n; i += 256)
        s += v[i];
    s = block_sum_256(s, red);
    if (threadIdx.x == 0) {
        *out = s;
        *dz_fixed = 1;
    }
}

// column sums of A [R][N] over row chunks: part[chunk][n]   (bias gradients)
template <typename T>
__global__ void colsum_part_kernel(const T *__restrict__ A, long lda, int R, int N, int rows_per,
                                   float *__restrict__ part)
{
    pdl_trigger();
    pdl_wait();
    int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= N)
        return;
    int r0 = blockIdx.y * rows_per, r1 = min(R, r0 + rows_per);
    float s = 0.0f;
#pragma unroll 16 // the loads of sixteen rows are in flight together
    for (int r = r0; r < r1; r++)
        s += to_f(A[(long)r * lda + n]);
    part[(size_t)blockIdx.y * N + n] = s;
}

// ------------------------------------------------------------------
// optimizer (nc_sgd_opt_update, nncp.c:1229; constants libnc.h:547-561):
//   g' = clamp(g) ; v = b2*v + (1-b2)*g'^2 ; w -= lr*g'/(sqrt(v*corr)+eps)
// and the bf16 shadow of w refreshed in the same pass.
__global__ void __launch_bounds__(256)
rmsprop_kernel(float *__restrict__ w, const float *__restrict__ g, float *__restrict__ v,
               bf16 *__restrict__ shadow, size_t n4, float lr, float beta2, float eps,
               float clip, float corr, const float *__restrict__ hyper)
{
    pdl_trigger();
    pdl_wait();
    if (hyper) { // {lr, corr} from device memory: a captured launch must not freeze them
        lr = hyper[0];
        corr = hyper[1];
    }
    // grid-stride: correct for any grid; the library launches one thread per group of four
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += stride) {
    float4 ww = reinterpret_cast<float4 *>(w)[i];
    float4 gg = reinterpret_cast<const float4 *>(g)[i];
    float4 vv = reinterpret_cast<float4 *>(v)[i];
    float *pw = &ww.x, *pg = &gg.x, *pv = &vv.x;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        float x = pg[k];
        if (clip != 0.0f)
            x = fminf(fmaxf(x, -clip), clip);
        pv[k] = beta2 * pv[k] + (1.0f - beta2) * x * x;
        if (x != 0.0f)
            pw[k] -= lr * x / (sqrtf(pv[k] * corr) + eps);
    }
    reinterpret_cast<float4 *>(w)[i] = ww;
    reinterpret_cast<float4 *>(v)[i] = vv;
    if (shadow) {
        __nv_bfloat162 lo = __floats2bfloat162_rn(ww.x, ww.y);
        __nv_bfloat162 hi = __floats2bfloat162_rn(ww.z, ww.w);
        uint2 pk;
        pk.x = *reinterpret_cast<uint32_t *>(&lo);
        pk.y = *reinterpret_cast<uint32_t *>(&hi);
        reinterpret_cast<uint2 *>(shadow)[i] = pk;
    }
    }
}

__global__ void f32_to_bf16_kernel(const float *__restrict__ src, bf16 *__restrict__ dst, size_t n)
{
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n)
        dst[i] = __float2bfloat16_rn(src[i]);
}

// ------------------------------------------------------------------
// dense embedding gradient (adjoint of nc_get_col): g[v][:] = mult * sum over rows r with
// id[r]==v, in ascending r, of dx[r][:].  g must be zero on entry.
// first_rows_kernel leaves in first[v] the smallest row that carries symbol v (first[] holds a
// value >= rows on entry; integer atomicMin, so the result does not depend on the order of
// arrival).  embed_grad_kernel runs one block per row: the block of a symbol's first row lists the
// rows behind it that carry the symbol (ordered compaction by warp ballots), and every thread adds
// them, in ascending order, into the four columns it owns; the other blocks leave after two loads.
__global__ void first_rows_kernel(const int32_t *__restrict__ ids, int rows, int V, int *__restrict__ first)
{
    pdl_trigger();
    pdl_wait();
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= rows)
        return;
    int id = ids[r];
    id = id < 0 ? 0 : (id >= V ? V - 1 : id);
    atomicMin(first + id, r);
}

// blockIdx.y selects 256 columns, two of them a thread's.  A frequent symbol's sum is a chain of rows, bound
// by how many of their loads are in flight and by the list; four columns a thread, one range of 512 columns
// after the other, took 52 us for 2048 rows of 1024.
template <typename T>
__global__ void __launch_bounds__(128)
embed_grad_kernel(const int32_t *__restrict__ ids, const T *__restrict__ dx, float *__restrict__ g,
                  const int *__restrict__ first, int rows, int D, float mult, int V)
{
    pdl_trigger();
    pdl_wait();
    constexpr int SPAN = 2048, FLIGHT = 16; // rows listed per pass, rows loaded together
    __shared__ int list[SPAN];
    __shared__ int wcnt[2][4]; // per-warp hit counts of a chunk, double-buffered by chunk parity
    const int r0 = blockIdx.x, c0 = blockIdx.y * 256 + threadIdx.x;
    int v = ids[r0];
    v = v < 0 ? 0 : (v >= V ? V - 1 : v);
    if (first[v] != r0)
        return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool in0 = c0 < D, in1 = c0 + 128 < D;
    float acc[2] = {0.0f, 0.0f};
    for (int span0 = r0; span0 < rows; span0 += SPAN) {
        // ordered list of the rows of this span that carry the symbol (compaction by warp ballots).
        // Every thread keeps the running total in a register: the counts of a chunk are read by all
        // threads after one barrier, and the buffer they sit in is not written again before the
        // barrier of the next chunk has been passed by everyone.
        __syncthreads(); // the list of the span before has been read
        const int span1 = min(rows, span0 + SPAN);
        int idr[SPAN / 128]; // all of the span's ids are requested before the first is looked at
#pragma unroll
        for (int j = 0; j < SPAN / 128; j++) {
            const int r = span0 + 128 * j + threadIdx.x;
            idr[j] = r < span1 ? ids[r] : -1;
        }
        int n = 0;
#pragma unroll
        for (int j = 0; j < SPAN / 128; j++) {
            const int base = span0 + 128 * j;
            if (base >= span1)
                break;
            const int r = base + threadIdx.x;
            int id = idr[j];
            if (r < span1)
                id = id < 0 ? 0 : (id >= V ? V - 1 : id);
            const bool hit = id == v;
            const unsigned bal = __ballot_sync(0xffffffffu, hit);
            if (lane == 0)
                wcnt[j & 1][warp] = __popc(bal);
            __syncthreads();
            const int w0 = wcnt[j & 1][0], w1 = wcnt[j & 1][1], w2 = wcnt[j & 1][2], w3 = wcnt[j & 1][3];
            const int pos = n + (warp > 0 ? w0 : 0) + (warp > 1 ? w1 : 0) + (warp > 2 ? w2 : 0);
            if (hit)
                list[pos + __popc(bal & ((1u << lane) - 1u))] = r;
            n += w0 + w1 + w2 + w3;
        }
        __syncthreads(); // the list is complete
        // the rows' loads go out before the first is added: the sum of a frequent symbol is a
        // chain of additions in row order, but its loads need not wait for one another
        for (int k0 = 0; k0 < n; k0 += FLIGHT) {
            float x[FLIGHT][2];
#pragma unroll
            for (int u = 0; u < FLIGHT; u++) {
                const T *src = dx + (size_t)list[min(k0 + u, n - 1)] * D + c0;
                x[u][0] = in0 ? to_f(src[0]) : 0.0f;
                x[u][1] = in1 ? to_f(src[128]) : 0.0f;
            }
#pragma unroll
            for (int u = 0; u < FLIGHT; u++)
                if (k0 + u < n) {
                    acc[0] += x[u][0];
                    acc[1] += x[u][1];
                }
        }
    }
    if (in0)
        g[(size_t)v * D + c0] = acc[0] * mult;
    if (in1)
        g[(size_t)v * D + c0 + 128] = acc[1] * mult;
}

// ------------------------------------------------------------------
// dst[c][r] = src[r][c]  (bf16 32x32 tiles through shared memory)
__global__ void __launch_bounds__(256)
transpose_bf16_kernel(const bf16 *__restrict__ src, long lds, bf16 *__restrict__ dst, long ldd,
                      int R, int Ccols)
{
    __shared__ bf16 tile[32][33];
    int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
    int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    for (int j = ty; j < 32; j += 8) {
        int r = r0 + j, c = c0 + tx;
        if (r < R && c < Ccols)
            tile[j][tx] = src[(long)r * lds + c];
    }
    __syncthreads();
    for (int j = ty; j < 32; j += 8) {
        int c = c0 + j, r = r0 + tx;
        if (r < R && c < Ccols)
            dst[(long)c * ldd + r] = tile[tx][j];
    }
}

// ------------------------------------------------------------------
// order-independent 64-bit digest of a float buffer: sum of mix(index, bits) mod 2^64
__device__ __forceinline__ unsigned long long mix64(unsigned long long x)
{
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}
__global__ void hash_kernel(const float *__restrict__ w, size_t n, unsigned long long *out)
{
    unsigned long long s = 0;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x)
        s += mix64((i << 32) ^ (unsigned long long)__float_as_uint(w[i]));
    atomicAdd(out, s); // integer addition: the order of arrival does not change the sum
}
