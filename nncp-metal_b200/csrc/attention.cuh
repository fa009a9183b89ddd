// attention.cuh -- relative-position causal attention over [memory | segment],
// forward and backward, one CTA per (stream, head).
//
// Follows the sub-graph of trf_eval at nncp.c:722-800:
//   score(i,j) = ( q_i.k_j + q_i.w_r[max(r-(L-P),0)] + br_scale*b_r[r] ) / sqrt(dk)
//   r = j + (T-1) - i          nc_rel_shift(-(T-1))            nncp.c:784
//   left pad by duplication    nc_pad(L-P, NC_PAD_DUP)         nncp.c:777
//   key j visible to query i   iff 0 <= (i+M)-j < attn_len     nncp.c:357-361
// and its adjoint (LibNC's autograd is not part of the reference tree).
//
// CUDA-core kernels: at the sizes NNCP uses (T <= 64, L <= 576, dk <= 128 per
// (stream, head)) the op is bound by HBM traffic and launch latency, not by the
// tensor pipe.  K, V and the w_r table of the CTA's (stream, head) are staged
// once in shared memory; all reductions run in a fixed order (lanes own keys,
// butterflies combine them), so query row i gives the same bits whether it is
// computed alone (one-symbol step) or with the whole segment.
#pragma once
#include "attention_deal.h"
#include "common.cuh"

struct AttnArgs {
    const void *q, *kv, *out, *dout;
    const float *w_r, *b_r;
    const void *w_r16; // optional bf16 copy of w_r (same layout), used by the tensor-core kernels
    void *o, *dq, *dkv;
    float *lse, *dwr_part, *dbr_part;
    int *err_flag; // raised when a bounded wait runs out, may be NULL
    int B, H, dk, T, M, L, P, attn_len, t0, t1, qchunk;
    int sum;        // adjoint: dwr_part holds sums over the streams that a CTA takes (fab::Share), not one table a stream
    int ahead;      // one query: keys and values of other steps, and the tables, may be read before the wait for the predecessor
    int smem_pitch; // row pitch of the staged K and table rows (CUDA-core kernels)
    int qp, kvp, dqp, dkvp; // row pitches (elements) of q, kv, dq, dkv; K then V inside a kv row
    float br_scale, inv_sqrt;
};

// Row pitch (elements) of the K and table rows in shared memory.  Head sizes that are a multiple of
// four go through four-element loads: a pitch of dk + 4 puts the rows of eight neighbouring keys on
// different bank groups; where that does not fit, dk alone; any other head size keeps dk + an odd
// word and single-element loads.
template <typename T> struct SmemRow {
    static __host__ __device__ int wide(int dk) { return dk % 4 == 0 ? dk + 4 : dk + (sizeof(T) == 4 ? 1 : 2); }
    static __host__ __device__ int tight(int dk) { return dk % 4 == 0 ? dk : wide(dk); }
};

__device__ __forceinline__ float4 load_f4(const float *p) { return *reinterpret_cast<const float4 *>(p); }
__device__ __forceinline__ float4 load_f4(const bf16 *p)
{
    const uint2 u = *reinterpret_cast<const uint2 *>(p);
    const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162 *>(&u.x), b = *reinterpret_cast<const __nv_bfloat162 *>(&u.y);
    return make_float4(__low2float(a), __high2float(a), __low2float(b), __high2float(b));
}
__device__ __forceinline__ void store_f4(float *p, float4 v) { *reinterpret_cast<float4 *>(p) = v; }
__device__ __forceinline__ void store_f4(bf16 *p, float4 v)
{
    const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
    *reinterpret_cast<uint2 *>(p) = make_uint2(*reinterpret_cast<const uint32_t *>(&a), *reinterpret_cast<const uint32_t *>(&b));
}

// rows x dk elements (row pitch ld) into shared memory (row pitch lds), converted from S to D
template <typename D, typename S>
__device__ __forceinline__ void stage_rows(D *dst, int lds, const S *src, size_t ld, int rows, int dk)
{
    if (dk % 4 == 0 && ld % 4 == 0 && lds % 4 == 0 && (reinterpret_cast<uintptr_t>(src) & (4 * sizeof(S) - 1)) == 0) {
        const int cpr = dk / 4;
#pragma unroll 4
        for (int idx = threadIdx.x; idx < rows * cpr; idx += blockDim.x) {
            const int r = idx / cpr, e = (idx - r * cpr) * 4;
            store_f4(dst + (size_t)r * lds + e, load_f4(src + (size_t)r * ld + e));
        }
    } else {
        for (int idx = threadIdx.x; idx < rows * dk; idx += blockDim.x) {
            const int r = idx / dk, e = idx - r * dk;
            dst[(size_t)r * lds + e] = from_f<D>(to_f(src[(size_t)r * ld + e]));
        }
    }
}

template <typename T>
__device__ __forceinline__ float dot_q(const float *__restrict__ qf, const T *__restrict__ row, int dk)
{
    float s = 0.0f;
    if (dk % 4 == 0) {
#pragma unroll 4
        for (int e = 0; e < dk; e += 4) {
            const float4 a = load_f4(qf + e), b = load_f4(row + e);
            s = fmaf(a.x, b.x, s);
            s = fmaf(a.y, b.y, s);
            s = fmaf(a.z, b.z, s);
            s = fmaf(a.w, b.w, s);
        }
    } else {
        for (int e = 0; e < dk; e++)
            s = fmaf(qf[e], to_f(row[e]), s);
    }
    return s;
}

// score of (query i, key j) for an unmasked pair; br: the head's row of b_r, Rs NULL without a table
template <typename T>
__device__ __forceinline__ float score_ij(int i, int j, int Tn, int L, int P, int dk, float inv_sqrt, float br_scale,
                                          const float *qf, const T *Ks, const T *Rs, int ks, const float *br)
{
    const float s = dot_q<T>(qf, Ks + (size_t)j * ks, dk);
    const int r = j + (Tn - 1) - i;
    float z = __fmul_rn(br_scale, br[r]);
    if (Rs) {
        int pi = r - (L - P);
        pi = pi < 0 ? 0 : pi;
        z = __fadd_rn(z, dot_q<T>(qf, Rs + (size_t)pi * ks, dk));
    }
    return __fmul_rn(__fadd_rn(s, z), inv_sqrt);
}
__device__ __forceinline__ void attn_key_range(int L, int M, int attn_len, int i, int &jlo, int &jhi)
{
    jhi = min(L - 1, i + M);                 // (i+M)-j >= 0
    jlo = max(0, i + M - attn_len + 1);      // (i+M)-j < attn_len
}

// One query row by one warp: keys [jlo, jhi] over the lanes, output column e to out(e, value), log-sum-exp
// in lse.  qf: the query as floats; ps: scratch for the scores, indexed by key.
template <typename T, typename F>
__device__ __forceinline__ void attn_row(int i, int jlo, int jhi, int Tn, int L, int P, int dk, float inv_sqrt, float br_scale,
                                         const float *qf, const T *Ks, const T *Rs, int ks, const T *Vs, const float *br, float *ps,
                                         int lane, float &lse, F out)
{
    float mx = -INFINITY;
    for (int j = jlo + lane; j <= jhi; j += 32) {
        float s = score_ij<T>(i, j, Tn, L, P, dk, inv_sqrt, br_scale, qf, Ks, Rs, ks, br);
        ps[j] = s;
        mx = fmaxf(mx, s);
    }
    mx = warp_max(mx);
    float sum = 0.0f;
    for (int j = jlo + lane; j <= jhi; j += 32) {
        float p = expf(__fsub_rn(ps[j], mx));
        ps[j] = p;
        sum = __fadd_rn(sum, p);
    }
    sum = warp_sum(sum);
    const float rs = __fdiv_rn(1.0f, sum);
    __syncwarp();
    for (int e = lane; e < dk; e += 32) {
        float acc = 0.0f;
#pragma unroll 8
        for (int j = jlo; j <= jhi; j++)
            acc = fmaf(__fmul_rn(ps[j], rs), to_f(Vs[(size_t)j * dk + e]), acc);
        out(e, acc);
    }
    lse = __fadd_rn(mx, logf(sum));
    __syncwarp();
}

__device__ __forceinline__ void key_range(const AttnArgs &a, int i, int &jlo, int &jhi)
{
    attn_key_range(a.L, a.M, a.attn_len, i, jlo, jhi);
}

// floats a warp of the forward kernel keeps: the query row and its scores
__host__ __device__ inline int warp_floats(int dk, int L) { return dk % 4 == 0 ? (dk + L + 3) & ~3 : dk + L; }

template <typename T>
size_t attn_fwd_smem(int L, int P, int dk, bool has_wr, int ks)
{
    size_t b = (size_t)L * ks * sizeof(T) + (size_t)L * dk * sizeof(T);
    if (has_wr)
        b += (size_t)P * ks * sizeof(T);
    b = (b + 15) & ~(size_t)15;
    b += 8 * (size_t)warp_floats(dk, L) * sizeof(float);
    return b;
}

template <typename T>
__global__ void __launch_bounds__(256) attn_fwd_kernel(AttnArgs a)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    const int ks = a.smem_pitch;
    T *Ks = reinterpret_cast<T *>(smraw);
    T *Vs = Ks + (size_t)a.L * ks;
    T *Rs = Vs + (size_t)a.L * a.dk;
    size_t off = ((size_t)a.L * ks + (size_t)a.L * a.dk + (a.w_r ? (size_t)a.P * ks : 0)) * sizeof(T);
    off = (off + 15) & ~(size_t)15;
    float *fs = reinterpret_cast<float *>(smraw + off);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float *qf = fs + (size_t)warp * warp_floats(a.dk, a.L);
    float *ps = qf + a.dk;
    pdl_trigger();
    pdl_wait();

    const int b = blockIdx.x / a.H, h = blockIdx.x % a.H;
    const int HD = a.H * a.dk;
    const int i_first = a.t0 + blockIdx.y * a.qchunk;
    const int i_last = min(a.t1, i_first + a.qchunk) - 1;
    if (i_first > i_last)
        return;
    int jlo_all, jhi_all, tmp;
    key_range(a, i_first, jlo_all, tmp);
    key_range(a, i_last, tmp, jhi_all);

    const T *kv = reinterpret_cast<const T *>(a.kv) + ((size_t)jlo_all * a.B + b) * a.kvp + h * a.dk;
    const int nj = jhi_all - jlo_all + 1;
    stage_rows(Ks + (size_t)jlo_all * ks, ks, kv, (size_t)a.B * a.kvp, nj, a.dk);
    stage_rows(Vs + (size_t)jlo_all * a.dk, a.dk, kv + HD, (size_t)a.B * a.kvp, nj, a.dk);
    if (a.w_r)
        stage_rows(Rs, ks, a.w_r + (size_t)h * a.P * a.dk, (size_t)a.dk, a.P, a.dk);
    __syncthreads();

    const T *q = reinterpret_cast<const T *>(a.q);
    T *o = reinterpret_cast<T *>(a.o);
    for (int i = i_first + warp; i <= i_last; i += 8) {
        const T *qi = q + ((size_t)i * a.B + b) * a.qp + h * a.dk;
        for (int e = lane; e < a.dk; e += 32)
            qf[e] = to_f(qi[e]);
        __syncwarp();
        int jlo, jhi;
        key_range(a, i, jlo, jhi);
        float lse;
        attn_row<T>(i, jlo, jhi, a.T, a.L, a.P, a.dk, a.inv_sqrt, a.br_scale, qf, Ks, a.w_r ? Rs : nullptr, ks, Vs,
                    a.b_r + (size_t)h * a.L, ps, lane, lse,
                    [&](int e, float v) { o[((size_t)i * a.B + b) * HD + h * a.dk + e] = from_f<T>(v); });
        if (lane == 0 && a.lse)
            a.lse[((size_t)b * a.H + h) * a.T + i] = lse;
    }
}

template <typename T>
size_t attn_bwd_smem(int T_, int L, int P, int dk, bool has_wr, int ks)
{
    const int vs = dk % 4 == 0 ? ks : dk; // row pitch of V
    size_t b = (size_t)L * ks * sizeof(T) + (size_t)L * vs * sizeof(T);
    if (has_wr)
        b += (size_t)P * ks * sizeof(T);
    b = (b + 15) & ~(size_t)15;
    b += ((size_t)2 * T_ * dk + (size_t)2 * T_ * (L + 1) + T_) * sizeof(float);
    return b;
}

// W consecutive elements of a shared-memory row as floats (W = 4: one vector load)
template <int W, typename T> __device__ __forceinline__ void load_w(const T *p, float (&v)[W])
{
    if constexpr (W == 4) {
        const float4 x = load_f4(p);
        v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
    } else {
        v[0] = to_f(p[0]);
    }
}
template <int W, typename T> __device__ __forceinline__ void store_w(T *p, const float (&v)[W], bool vec)
{
    if constexpr (W == 4) {
        if (vec) {
            store_f4(p, make_float4(v[0], v[1], v[2], v[3]));
            return;
        }
    }
#pragma unroll
    for (int w = 0; w < W; w++)
        p[w] = from_f<T>(v[w]);
}

// A cluster of 1 to 8 CTAs per (stream, head).  The whole problem sits in the shared memory of each: a CTA takes
// every C-th group of eight query rows, writes their P and dS into all of the cluster's copies, and after the
// cluster's barrier every C-th part of the results; association and bits do not depend on C.  What bounds a CTA
// is the rate of shared-memory reads, so every inner loop reads W = 4 elements per access (head sizes that are
// a multiple of four; W = 1 otherwise) and each gradient row is a register tile of W columns.  One CTA per
// (stream, head) left the chip to 16 CTAs (4 streams x 4 heads of 32, 32 queries over 64 keys: 26 us a launch, 16.3 with
// four; a step of two such layers 208 -> 192 us) or to 128 of eight warps (16 x 8 heads: 26.4 us, 24.6 with two).
// the address of `p` in the shared memory of CTA `rank` of the cluster
__device__ __forceinline__ uint32_t peer_addr(const void *p, uint32_t rank)
{
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    return r;
}
__device__ __forceinline__ void peer_store(uint32_t at, float v)
{
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(at), "f"(v) : "memory");
}
template <typename T, int W, bool CLUSTER> // CLUSTER: the grid's second dimension is a cluster, else it is one
__global__ void __launch_bounds__(256) attn_bwd_kernel(AttnArgs a)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    const int ks = a.smem_pitch;
    const int Tn = a.T, L = a.L, dk = a.dk, P = a.P, M = a.M;
    const int vs = dk % 4 == 0 ? ks : dk;
    T *Ks = reinterpret_cast<T *>(smraw);
    T *Vs = Ks + (size_t)L * ks;
    T *Rs = Vs + (size_t)L * vs;
    size_t off = ((size_t)L * ks + (size_t)L * vs + (a.w_r ? (size_t)P * ks : 0)) * sizeof(T);
    off = (off + 15) & ~(size_t)15;
    float *qs = reinterpret_cast<float *>(smraw + off); // [T][dk]
    float *dos = qs + (size_t)Tn * dk;                  // [T][dk]
    float *Pm = dos + (size_t)Tn * dk;                  // [T][L+1]
    float *dS = Pm + (size_t)Tn * (L + 1);              // [T][L+1]
    float *Dr = dS + (size_t)Tn * (L + 1);              // [T]: D_i, later the row's sum over the left pad
    const int ls = L + 1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int C = CLUSTER ? gridDim.y : 1, rank = CLUSTER ? blockIdx.y : 0; // the cluster lies along y and is the whole of it
    const int b = blockIdx.x / a.H, h = blockIdx.x % a.H;
    const int HD = a.H * dk;
    const int tid = rank * blockDim.x + threadIdx.x, nthr = C * blockDim.x; // of the cluster
    if constexpr (CLUSTER) // the others are there before anything is written to them
        asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");
    pdl_trigger();
    pdl_wait();

    const T *kv = reinterpret_cast<const T *>(a.kv) + (size_t)b * a.kvp + h * dk;
    const T *q = reinterpret_cast<const T *>(a.q) + (size_t)b * a.qp + h * dk;
    const T *outp = reinterpret_cast<const T *>(a.out) + (size_t)b * HD + h * dk;
    const T *dout = reinterpret_cast<const T *>(a.dout) + (size_t)b * HD + h * dk;
    stage_rows(Ks, ks, kv, (size_t)a.B * a.kvp, L, dk);
    stage_rows(Vs, vs, kv + HD, (size_t)a.B * a.kvp, L, dk);
    stage_rows(qs, dk, q, (size_t)a.B * a.qp, Tn, dk);
    stage_rows(dos, dk, dout, (size_t)a.B * HD, Tn, dk);
    if (a.w_r)
        stage_rows(Rs, ks, a.w_r + (size_t)h * P * dk, (size_t)dk, P, dk);
    __syncthreads();
    if constexpr (CLUSTER)
        asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    // P and dS, zero where the pair is masked
    for (int i = rank * 8 + warp; i < Tn; i += 8 * C) {
        // D_i = dO_i . O_i  (= sum_j P_ij dP_ij)
        float D = 0.0f;
        for (int e = lane; e < dk; e += 32)
            D += dos[(size_t)i * dk + e] * to_f(outp[(size_t)i * a.B * HD + e]);
        D = warp_sum(D);
        int jlo, jhi;
        key_range(a, i, jlo, jhi);
        const float lse = a.lse[((size_t)b * a.H + h) * Tn + i];
        const float *qf = qs + (size_t)i * dk, *dof = dos + (size_t)i * dk;
        const int jpad = L - P - (Tn - 1) + i; // keys up to here share table row 0 (the left pad)
        float pad = 0.0f;
        for (int j = lane; j < L; j += 32) {
            float p = 0.0f, d = 0.0f;
            if (j >= jlo && j <= jhi) {
                p = expf(score_ij<T>(i, j, Tn, L, P, dk, a.inv_sqrt, a.br_scale, qf, Ks, a.w_r ? Rs : nullptr, ks, a.b_r + (size_t)h * L) - lse);
                d = p * (dot_q<T>(dof, Vs + (size_t)j * vs, dk) - D) * a.inv_sqrt;
            }
            if constexpr (!CLUSTER) {
                Pm[(size_t)i * ls + j] = p;
                dS[(size_t)i * ls + j] = d;
            } else {
                for (int c = 0; c < C; c++) {
                    peer_store(peer_addr(Pm + (size_t)i * ls + j, c), p);
                    peer_store(peer_addr(dS + (size_t)i * ls + j, c), d);
                }
            }
            if (j <= jpad)
                pad += d;
        }
        pad = warp_sum(pad);
        if constexpr (!CLUSTER) {
            if (lane == 0)
                Dr[i] = pad;
        } else if (lane < C) {
            peer_store(peer_addr(Dr + i, lane), pad);
        }
    }
    if constexpr (CLUSTER)
        asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
    else
        __syncthreads();
    const int nw = dk / W; // column groups
    const bool vec = (reinterpret_cast<uintptr_t>(a.dkv) & (4 * sizeof(T) - 1)) == 0 && (reinterpret_cast<uintptr_t>(a.dq) & (4 * sizeof(T) - 1)) == 0 &&
                     a.dkvp % 4 == 0 && a.dqp % 4 == 0;
    // dV[j] = sum_i P_ij dO_i ; dK[j] = sum_i dS_ij q_i     (i ascending), two keys per thread
    T *dkv = reinterpret_cast<T *>(a.dkv) + (size_t)b * a.dkvp + h * dk;
    const int half = (L + 1) / 2;
    for (int idx = tid; idx < half * nw; idx += nthr) {
        const int j0 = idx / nw, e = (idx - j0 * nw) * W, j1 = j0 + half < L ? j0 + half : j0;
        float av[2][W] = {}, ak[2][W] = {};
#pragma unroll 4
        for (int i = max(0, j0 - M); i < Tn; i++) {
            float x[W], y[W];
            load_w<W>(dos + (size_t)i * dk + e, x);
            load_w<W>(qs + (size_t)i * dk + e, y);
            const float p0 = Pm[(size_t)i * ls + j0], p1 = Pm[(size_t)i * ls + j1];
            const float d0 = dS[(size_t)i * ls + j0], d1 = dS[(size_t)i * ls + j1];
#pragma unroll
            for (int w = 0; w < W; w++) {
                av[0][w] = fmaf(p0, x[w], av[0][w]);
                av[1][w] = fmaf(p1, x[w], av[1][w]);
                ak[0][w] = fmaf(d0, y[w], ak[0][w]);
                ak[1][w] = fmaf(d1, y[w], ak[1][w]);
            }
        }
        T *dst = dkv + (size_t)j0 * a.B * a.dkvp + e;
        store_w<W>(dst, ak[0], vec);
        store_w<W>(dst + HD, av[0], vec && HD % 4 == 0);
        if (j1 != j0) {
            dst = dkv + (size_t)j1 * a.B * a.dkvp + e;
            store_w<W>(dst, ak[1], vec);
            store_w<W>(dst + HD, av[1], vec && HD % 4 == 0);
        }
    }
    // dQ[i] = sum_j dS_ij (k_j + w_r[pi(i,j)])               (j ascending)
    T *dq = reinterpret_cast<T *>(a.dq) + (size_t)b * a.dqp + h * dk;
    for (int idx = tid; idx < Tn * nw; idx += nthr) {
        const int i = idx / nw, e = (idx - i * nw) * W;
        int jlo, jhi;
        key_range(a, i, jlo, jhi);
        float acc[W] = {};
#pragma unroll 4
        for (int j = jlo; j <= jhi; j++) {
            float x[W];
            load_w<W>(Ks + (size_t)j * ks + e, x);
            if (a.w_r) {
                int pi = j + (Tn - 1) - i - (L - P);
                pi = pi < 0 ? 0 : pi;
                float y[W];
                load_w<W>(Rs + (size_t)pi * ks + e, y);
#pragma unroll
                for (int w = 0; w < W; w++)
                    x[w] += y[w];
            }
            const float d = dS[(size_t)i * ls + j];
#pragma unroll
            for (int w = 0; w < W; w++)
                acc[w] = fmaf(d, x[w], acc[w]);
        }
        store_w<W>(dq + (size_t)i * a.B * a.dqp + e, acc, vec);
    }
    // table gradients of this (stream, head): table row p collects the pairs (i, j = p + L - P - (T-1) + i),
    // row 0 the whole left pad
    if (a.w_r && a.dwr_part) {
        float *dst = a.dwr_part + ((size_t)b * a.H + h) * P * dk;
        for (int idx = tid; idx < P * nw; idx += nthr) {
            const int p = idx / nw, e = (idx - p * nw) * W, j0 = p + L - P - (Tn - 1);
            float acc[W] = {};
#pragma unroll 4
            for (int i = 0; i < Tn; i++) {
                const int j = j0 + i;
                float y[W], d = 0.0f;
                if (p == 0)
                    d = Dr[i];
                else if (j >= 0 && j < L)
                    d = dS[(size_t)i * ls + j];
                load_w<W>(qs + (size_t)i * dk + e, y);
#pragma unroll
                for (int w = 0; w < W; w++)
                    acc[w] = fmaf(d, y[w], acc[w]);
            }
#pragma unroll
            for (int w = 0; w < W; w++)
                dst[(size_t)p * dk + e + w] = acc[w];
        }
    }
    if (a.dbr_part) {
        float *dst = a.dbr_part + ((size_t)b * a.H + h) * L;
        for (int r = tid; r < L; r += nthr) {
            float acc = 0.0f;
#pragma unroll 4
            for (int i = 0; i < Tn; i++) {
                const int j = r - (Tn - 1) + i;
                if (j >= 0 && j < L)
                    acc += dS[(size_t)i * ls + j];
            }
            dst[r] = acc * a.br_scale;
        }
    }
}

static int attn_check_shape(const nncu_attn_shape *s)
{
    if (!s || s->n_streams < 1 || s->n_head < 1 || s->d_key < 1 || s->seg_len < 1 ||
        s->mem_len < 0 || s->d_pos < 1 || s->d_pos > s->mem_len + s->seg_len || s->t0 < 0 ||
        s->t1 > s->seg_len || s->t0 >= s->t1 || s->attn_len < 0 ||
        s->attn_len > s->mem_len + s->seg_len)
        return nncu_fail(NNCU_ERR_INVALID, "attention: bad shape");
    if (s->dtype_bf16 && (s->d_key & 1))
        return nncu_fail(NNCU_ERR_INVALID, "attention: bf16 needs an even d_key");
    return NNCU_OK;
}

// row pitches when q / kv / dq / dkv are column ranges of wider buffers (0 = packed)
struct AttnPitch {
    int qp, kvp, dqp, dkvp;
};

static AttnArgs attn_args(const nncu_attn_shape *s, const AttnPitch *pt = nullptr)
{
    AttnArgs a;
    memset(&a, 0, sizeof(a));
    a.B = s->n_streams; a.H = s->n_head; a.dk = s->d_key; a.T = s->seg_len; a.M = s->mem_len;
    a.L = s->mem_len + s->seg_len; a.P = s->d_pos;
    a.attn_len = s->attn_len ? s->attn_len : a.L;
    a.t0 = s->t0; a.t1 = s->t1;
    a.br_scale = s->br_scale;
    a.inv_sqrt = 1.0f / sqrtf((float)s->d_key);
    a.qp = a.dqp = a.H * a.dk;
    a.kvp = a.dkvp = 2 * a.H * a.dk;
    if (pt) {
        if (pt->qp) a.qp = pt->qp;
        if (pt->kvp) a.kvp = pt->kvp;
        if (pt->dqp) a.dqp = pt->dqp;
        if (pt->dkvp) a.dkvp = pt->dkvp;
    }
    return a;
}

// the row pitch for a shape and the shared memory it takes
template <typename T> static int fwd_pitch(const AttnArgs &a, bool has_wr, size_t &smem)
{
    int ks = SmemRow<T>::wide(a.dk);
    if (attn_fwd_smem<T>(a.L, a.P, a.dk, has_wr, ks) > 227 * 1024)
        ks = SmemRow<T>::tight(a.dk);
    smem = attn_fwd_smem<T>(a.L, a.P, a.dk, has_wr, ks);
    return ks;
}
template <typename T> static int bwd_pitch(const AttnArgs &a, bool has_wr, size_t &smem)
{
    int ks = SmemRow<T>::wide(a.dk);
    if (attn_bwd_smem<T>(a.T, a.L, a.P, a.dk, has_wr, ks) > 227 * 1024)
        ks = SmemRow<T>::tight(a.dk);
    smem = attn_bwd_smem<T>(a.T, a.L, a.P, a.dk, has_wr, ks);
    return ks;
}

template <typename T>
static int attn_forward_t(const nncu_attn_shape *s, const void *q, const void *kv, const float *w_r,
                          const float *b_r, void *out, float *lse, cudaStream_t st,
                          const AttnPitch *pt = nullptr)
{
    AttnArgs a = attn_args(s, pt);
    a.q = q; a.kv = kv; a.w_r = w_r; a.b_r = b_r; a.o = out; a.lse = lse;
    const int nq = a.t1 - a.t0;
    size_t smem = 0;
    a.smem_pitch = fwd_pitch<T>(a, w_r != nullptr, smem);
    if (smem > 227 * 1024)
        return nncu_fail(NNCU_ERR_RANGE, "attention forward: %zu bytes of shared memory needed", smem);
    a.qchunk = attn::queries_of_cta((long)a.B * a.H, nq, (long)smem);
    const int chunks = ceil_div(nq, a.qchunk);
    static DeviceOnce once;
    NNCU_TRY(smem_limit(once, attn_fwd_kernel<T>, SMEM_MOST));
    launch_kind(EDGE_ATTN, attn_fwd_kernel<T>, dim3(a.B * a.H, chunks), dim3(256), smem, st, a);
    KERNEL_CHECK();
    return NNCU_OK;
}

template <typename T>
static int attn_backward_t(const nncu_attn_shape *s, const void *q, const void *kv,
                           const float *w_r, const float *b_r, const void *out, const float *lse,
                           const void *dout, void *dq, void *dkv, float *dwr_part,
                           float *dbr_part, cudaStream_t st, const AttnPitch *pt = nullptr)
{
    AttnArgs a = attn_args(s, pt);
    if (a.t0 != 0 || a.t1 != a.T)
        return nncu_fail(NNCU_ERR_INVALID, "attention backward runs over the whole segment");
    a.q = q; a.kv = kv; a.w_r = w_r; a.b_r = b_r; a.out = out; a.lse = const_cast<float *>(lse);
    a.dout = dout; a.dq = dq; a.dkv = dkv; a.dwr_part = dwr_part; a.dbr_part = dbr_part;
    size_t smem = 0;
    a.smem_pitch = bwd_pitch<T>(a, w_r != nullptr, smem);
    if (smem > 227 * 1024)
        return nncu_fail(NNCU_ERR_RANGE, "attention backward: %zu bytes of shared memory needed", smem);
    const int C = attn::ctas_of_pair((long)a.B * a.H, a.T, (long)smem);
    const bool vec = a.dk % 4 == 0;
    auto kernel = C > 1 ? (vec ? attn_bwd_kernel<T, 4, true> : attn_bwd_kernel<T, 1, true>)
                        : (vec ? attn_bwd_kernel<T, 4, false> : attn_bwd_kernel<T, 1, false>);
    static DeviceOnce once[4];
    NNCU_TRY(smem_limit(once[2 * (C > 1) + vec], kernel, SMEM_MOST));
    if (C == 1) {
        launch_kind(EDGE_ATTN, kernel, dim3(a.B * a.H), dim3(256), smem, st, a);
        KERNEL_CHECK();
        return NNCU_OK;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(a.B * a.H, C);
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = attr[0].val.clusterDim.z = 1;
    attr[0].val.clusterDim.y = C;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = (g_nncu_edges & EDGE_ATTN) ? 2 : 1;
    CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, a));
    KERNEL_CHECK();
    return NNCU_OK;
}
