// attention_fa.cuh -- bf16 relative-position attention for head sizes 16, 32, 64 and 128 on
// warp-level tensor-core instructions (mma.sync m16n8k16, fp32 accumulation).
//
// Same math as attention.cuh (nncp.c:722-800 and its adjoint).  Per (stream, head) the
// contractions are 64 queries x 64-key blocks x head size, a few hundred warp-level products; what
// bounds the op is the chain load -> scores -> softmax -> product, not the tensor rate (measured
// 555 TFLOP/s for mma.sync on this part, of which the op needs a quarter).  A warp's products need
// no hand-off through tensor memory and barriers, two CTAs share an SM, and the relative shift is a
// 3 KB round trip through shared memory private to the warp.  The tcgen05 kernels these replace
// spent 47 k cycles per 128-key block of a stream pair (64 streams x 16 heads, 320 keys: backward
// 330 us, forward 70 us a launch).
//
// Geometry.  Keys go in blocks of 64 counted from key 0, queries in groups of 64 rows, a warp owns
// 16 rows.  Query i0 + ii and key j0 + jj meet table row max(wlo + w, 0), w = jj + 63 - ii, with
// wlo = j0 - i0 + P - M - 64: the window of a block is 128 table rows (rows below the table are
// loaded as row 0, which is what the left pad duplicates), and the next block's window starts 64
// rows further on.
//
// Association, the same for every launch: key blocks in ascending order; a block's probabilities are
// taken relative to the running maximum, the running output is rescaled and the block's products
// continue its chain (16 keys a step), a row's sum is kept in four parts (columns 2t, 2t + 1 of every
// eight) that meet at the end.  A block in which a row sees nothing changes no bit.  So whole
// segments and single queries, which go through different kernels, give the same bits.
#pragma once
#include "attention.cuh"
#include "gemm_tc.cuh"

namespace fa {

constexpr int KB = 64;  // keys per block
constexpr int ESC = 52; // floats per row of a warp's skew scratch (48 used)

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], const bf16 *p)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(smem_addr(p)));
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], const bf16 *p)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(smem_addr(p)));
}
__device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
                 "{%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack2(float lo, float hi)
{
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&h);
}
__device__ __forceinline__ void cp16(void *dst, const void *src, bool valid)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// 4 x 4 transpose of 32-bit values over the four lanes of a quad: lane t ends with what lane u held in
// v[t] at v[u] (turns four 4-byte column pairs per lane into one 16-byte run per lane)
__device__ __forceinline__ void quad_transpose(uint32_t (&v)[4], int t)
{
    const bool o1 = t & 1, o2 = t & 2;
    uint32_t a = o1 ? v[0] : v[1], b = o1 ? v[2] : v[3];
    a = __shfl_xor_sync(0xffffffffu, a, 1);
    b = __shfl_xor_sync(0xffffffffu, b, 1);
    if (o1) { v[0] = a; v[2] = b; } else { v[1] = a; v[3] = b; }
    a = o2 ? v[0] : v[2];
    b = o2 ? v[1] : v[3];
    a = __shfl_xor_sync(0xffffffffu, a, 2);
    b = __shfl_xor_sync(0xffffffffu, b, 2);
    if (o2) { v[0] = a; v[1] = b; } else { v[2] = a; v[3] = b; }
}

inline __host__ __device__ bool aligned_to(const void *p, int bytes) { return (reinterpret_cast<uintptr_t>(p) & (bytes - 1)) == 0; }

// One row of a warp tile out as bf16: lane t of the quad holds columns nt * 8 + 2t, + 1 of the N / 8
// column groups in x[nt][c], x[nt][c + 1].  Rows of 32 columns and more leave in 16-byte pieces where the
// destination is aligned to them (WIDE).
template <bool WIDE, int NT> __device__ __forceinline__ void store_row(bf16 *dst, const float (&x)[NT][4], int c, int t, bool act)
{
    if constexpr (WIDE && NT % 4 == 0) {
#pragma unroll
        for (int n4 = 0; n4 < NT; n4 += 4) {
            uint32_t v[4];
#pragma unroll
            for (int u = 0; u < 4; u++)
                v[u] = pack2(x[n4 + u][c], x[n4 + u][c + 1]);
            quad_transpose(v, t);
            if (act)
                *reinterpret_cast<uint4 *>(dst + (n4 + t) * 8) = make_uint4(v[0], v[1], v[2], v[3]);
        }
    } else {
#pragma unroll
        for (int nt = 0; nt < NT; nt++)
            if (act)
                *reinterpret_cast<uint32_t *>(dst + nt * 8 + 2 * t) = pack2(x[nt][c], x[nt][c + 1]);
    }
}

// rows [0, rows) of a bf16 matrix (row pitch `pitch`) -> shared tile, zero where !valid(r)
template <int DK, typename F>
__device__ __forceinline__ void load_rows(bf16 *dst, const bf16 *src, size_t pitch, int rows, int tid, int nthr, F valid)
{
    constexpr int LD = DK + 8, CPR = DK / 8;
    for (int idx = tid; idx < rows * CPR; idx += nthr) {
        const int r = idx / CPR, c = (idx % CPR) * 8;
        const bool ok = valid(r);
        cp16(dst + r * LD + c, ok ? src + (size_t)r * pitch + c : src, ok);
    }
}
// sixteen zero bytes, by words where the destination is not aligned to them
template <bool WIDE> __device__ __forceinline__ void zero16(void *p)
{
    if constexpr (WIDE) {
        *reinterpret_cast<uint4 *>(p) = make_uint4(0u, 0u, 0u, 0u);
    } else {
#pragma unroll
        for (int w = 0; w < 4; w++)
            reinterpret_cast<uint32_t *>(p)[w] = 0u;
    }
}
// eight consecutive fp32 table entries as bf16; one at a time where they are not aligned to 16 bytes
// (WIDE: they are known to be)
template <bool WIDE> __device__ __forceinline__ void table_piece(bf16 *dst, const float *p)
{
    if (WIDE || aligned_to(p, 16)) {
        const float4 u = *reinterpret_cast<const float4 *>(p), v = *reinterpret_cast<const float4 *>(p + 4);
        *reinterpret_cast<uint4 *>(dst) = make_uint4(pack2(u.x, u.y), pack2(u.z, u.w), pack2(v.x, v.y), pack2(v.z, v.w));
    } else {
#pragma unroll 1
        for (int e = 0; e < 8; e++)
            dst[e] = __float2bfloat16_rn(p[e]);
    }
}
// rows x0 .. x0 + rows - 1 of one head's position table, clamped to [0, P)
template <int DK, bool WIDE>
__device__ __forceinline__ void load_table(bf16 *dst, const AttnArgs &a, int h, int x0, int rows, int tid, int nthr)
{
    constexpr int LD = DK + 8, CPR = DK / 8;
    const bf16 *w16 = reinterpret_cast<const bf16 *>(a.w_r16) + (size_t)h * a.P * DK;
    const float *w32 = a.w_r + (size_t)h * a.P * DK;
    for (int idx = tid; idx < rows * CPR; idx += nthr) {
        const int r = idx / CPR, c = (idx % CPR) * 8;
        const int x = min(max(x0 + r, 0), a.P - 1);
        if (a.w_r16) {
            cp16(dst + r * LD + c, w16 + (size_t)x * DK + c, true);
        } else {
            table_piece<WIDE>(dst + r * LD + c, w32 + (size_t)x * DK + c);
        }
    }
}

struct Blocks {
    int lo, hi; // first and last key block with a visible pair for query rows [t0, t1)
};
__host__ __device__ inline Blocks blocks_of(int M, int L, int attn_len, int t0, int t1)
{
    int jlo = t0 + M - attn_len + 1, jhi = t1 - 1 + M;
    jlo = jlo < 0 ? 0 : jlo;
    jhi = jhi > L - 1 ? L - 1 : jhi;
    return Blocks{jlo / KB, jhi / KB};
}

// b_r of one head, scaled, with room on both sides for the slots that masked pairs name
constexpr int BR_LO = 64, BR_PAD = BR_LO + 128;
__device__ __forceinline__ void load_br(float *brs, const AttnArgs &a, int h, int tid, int nthr)
{
    for (int r = tid; r < a.L + BR_PAD; r += nthr) {
        const int x = r - BR_LO;
        brs[r] = x >= 0 && x < a.L ? __fmul_rn(a.br_scale, a.b_r[(size_t)h * a.L + x]) : 0.0f;
    }
}
inline size_t br_bytes(int L) { return (size_t)((L + BR_PAD + 3) & ~3) * 4; }
// the score of a pair
__device__ __forceinline__ float score_of(float s, float e, float br, const AttnArgs &a)
{
    return __fmul_rn(__fadd_rn(s, __fadd_rn(br, e)), a.inv_sqrt);
}
// The scores of a warp's 16 x 32 pairs in place over s; first row i_w, first key j_w; rows from i_end on see
// nothing.  Whether a warp's pairs are all visible is the same for the whole warp, and for most tiles
// it is so: no masking there.
__device__ __forceinline__ void scores_16x32(float (&s)[4][4], const float (&e)[4][4], const float *brs, const AttnArgs &a, int i_w,
                                             int j_w, int i_end, int lane)
{
    const int g = lane >> 2, t = lane & 3, d0 = i_w + g + a.M - j_w - 2 * t; // query - key distance of element (0, 0)
    const float *br = brs + BR_LO + j_w + 2 * t + a.T - 1 - i_w - g;
#pragma unroll
    for (int n = 0; n < 4; n++)
#pragma unroll
        for (int c = 0; c < 4; c++)
            s[n][c] = score_of(s[n][c], e[n][c], br[n * 8 + (c & 1) - (c >> 1) * 8], a);
    if (j_w + 31 <= i_w + a.M && j_w > i_w + 15 + a.M - a.attn_len && i_w + 16 <= i_end)
        return;
#pragma unroll
    for (int n = 0; n < 4; n++)
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const int d = d0 - n * 8 - (c & 1) + (c >> 1) * 8; // visible iff 0 <= d < attn_len
            if ((unsigned)d >= (unsigned)a.attn_len || i_w + g + (c >> 1) * 8 >= i_end)
                s[n][c] = -INFINITY;
        }
}

// E of a warp's 16 rows (16 * qt ..) against 32 keys (32 * hf ..) of a block, skewed into the layout
// of the score fragments: e[nt][c] belongs to key 32 hf + 8 nt + 2 t + (c & 1), row g + 8 (c >> 1).
// window(p): the 16 rows of piece p of the block's window (row 16 p).
template <int DK, typename W>
__device__ __forceinline__ void skewed_positions(float (&e)[4][4], const bf16 *Qt, W window, int qt, int hf, float *es, int lane)
{
    constexpr int LD = DK + 8;
    const int g = lane >> 2, t = lane & 3;
    float x[6][4];
#pragma unroll
    for (int n = 0; n < 6; n++)
#pragma unroll
        for (int c = 0; c < 4; c++)
            x[n][c] = 0.0f;
#pragma unroll
    for (int ks = 0; ks < DK / 16; ks++) {
        uint32_t q[4];
        ldsm4(q, Qt + (lane & 15) * LD + ks * 16 + (lane >> 4) * 8);
#pragma unroll
        for (int p = 0; p < 3; p++) {
            uint32_t b[4];
            ldsm4(b, window(2 * hf + 3 - qt + p) + ((lane & 7) + (lane >> 4) * 8) * LD + ks * 16 + ((lane >> 3) & 1) * 8);
            mma(x[2 * p], q, b[0], b[1]);
            mma(x[2 * p + 1], q, b[2], b[3]);
        }
    }
    __syncwarp();
#pragma unroll
    for (int n = 0; n < 6; n++) {
        *reinterpret_cast<float2 *>(es + g * ESC + n * 8 + 2 * t) = make_float2(x[n][0], x[n][1]);
        *reinterpret_cast<float2 *>(es + (g + 8) * ESC + n * 8 + 2 * t) = make_float2(x[n][2], x[n][3]);
    }
    __syncwarp();
#pragma unroll
    for (int n = 0; n < 4; n++)
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const int row = g + (c >> 1) * 8;
            e[n][c] = es[row * ESC + n * 8 + 2 * t + (c & 1) + 15 - row];
        }
}

// s[nt][c] (same layout) = rows of At (16 rows) against 32 rows of Bt
template <int DK>
__device__ __forceinline__ void product_16x32(float (&s)[4][4], const bf16 *At, const bf16 *Bt, int lane)
{
    constexpr int LD = DK + 8;
#pragma unroll
    for (int n = 0; n < 4; n++)
#pragma unroll
        for (int c = 0; c < 4; c++)
            s[n][c] = 0.0f;
#pragma unroll
    for (int ks = 0; ks < DK / 16; ks++) {
        uint32_t q[4];
        ldsm4(q, At + (lane & 15) * LD + ks * 16 + (lane >> 4) * 8);
#pragma unroll
        for (int p = 0; p < 2; p++) {
            uint32_t b[4];
            ldsm4(b, Bt + (p * 16 + (lane & 7) + (lane >> 4) * 8) * LD + ks * 16 + ((lane >> 3) & 1) * 8);
            mma(s[2 * p], q, b[0], b[1]);
            mma(s[2 * p + 1], q, b[2], b[3]);
        }
    }
}

// ---------------- forward, a group of queries ----------------
//
// One CTA of eight warps per (stream, head, 64 queries).  Per key block, warp (q tile, half) takes the
// scores of 16 rows x 32 keys and then the value product of all 64 keys into half of the columns; the two
// warps of a tile exchange maxima and probabilities through shared memory under a barrier of
// their own.  The next block's tiles are fetched under the present block.  109 KB of shared memory at
// head size 64: two CTAs per SM.
template <int DK> struct FwdSmem {
    static constexpr int LD = DK + 8, TILE = 64 * LD * 2;
    static constexpr int Q = 0, K = TILE, V = K + 2 * TILE, R = V + 2 * TILE, ES = R + 3 * TILE, PF = ES + 8 * 16 * ESC * 4,
                         MX = PF + 4 * 4 * 512, BRS = MX + 4 * 6 * 32 * 4;
    static size_t bytes(int L) { return (size_t)BRS + br_bytes(L); }
};

template <int DK, bool WIDE> // WIDE: out takes 16-byte stores, an fp32 table 16-byte loads
__global__ void __launch_bounds__(256, 2) attn_fwd_kernel(const __grid_constant__ AttnArgs a)
{
    using SM = FwdSmem<DK>;
    constexpr int LD = SM::LD, NCH = DK >= 32 ? 2 : 1, NTC = DK / 8 / NCH; // column halves, 8-column groups in one
    extern __shared__ __align__(16) unsigned char sm[];
    bf16 *Qs = reinterpret_cast<bf16 *>(sm + SM::Q), *Ks = reinterpret_cast<bf16 *>(sm + SM::K),
         *Vs = reinterpret_cast<bf16 *>(sm + SM::V), *Rs = reinterpret_cast<bf16 *>(sm + SM::R);
    float *brs = reinterpret_cast<float *>(sm + SM::BRS);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int qt = warp & 3, hf = warp >> 2;
    const int b = blockIdx.x / a.H, h = blockIdx.x % a.H, HD = a.H * DK, T = a.T, M = a.M, L = a.L;
    const int i0 = (a.t0 & ~63) + blockIdx.y * 64;
    const Blocks blk = blocks_of(M, L, a.attn_len, max(i0, a.t0), min(i0 + 64, a.t1));
    float *es = reinterpret_cast<float *>(sm + SM::ES) + warp * 16 * ESC;
    // of this tile: [half][row A, row B][8] maxima, then [row A, row B][32] sums of half 0
    float *mx = reinterpret_cast<float *>(sm + SM::MX) + qt * 6 * 32, *sums = mx + 32;
    uint4 *pfs = reinterpret_cast<uint4 *>(sm + SM::PF) + qt * 4 * 32; // A fragments of the tile's probabilities, [16-key step][lane]
    pdl_wait(); // no early trigger: successors resident beside these CTAs cost more than their launch (33 % of the op alone)

    const bf16 *q = reinterpret_cast<const bf16 *>(a.q) + ((size_t)i0 * a.B + b) * a.qp + h * DK;
    const bf16 *kv = reinterpret_cast<const bf16 *>(a.kv) + (size_t)b * a.kvp + h * DK;
    auto fetch_r = [&](int gr) { // table group gr: window rows 0-63 of block gr, 64-127 of block gr - 1
        if (a.w_r)
            load_table<DK, WIDE>(Rs + (gr % 3) * 64 * LD, a, h, gr * KB - i0 + a.P - M - 64, 64, threadIdx.x, 256);
    };
    auto fetch = [&](int kb) {
        const int j0 = kb * KB;
        load_rows<DK>(Ks + (kb & 1) * 64 * LD, kv + (size_t)j0 * a.B * a.kvp, (size_t)a.B * a.kvp, 64, threadIdx.x, 256,
                      [&](int r) { return j0 + r < L; });
        load_rows<DK>(Vs + (kb & 1) * 64 * LD, kv + HD + (size_t)j0 * a.B * a.kvp, (size_t)a.B * a.kvp, 64, threadIdx.x, 256,
                      [&](int r) { return j0 + r < L; });
        fetch_r(kb + 1);
    };
    load_rows<DK>(Qs, q, (size_t)a.B * a.qp, 64, threadIdx.x, 256, [&](int r) { return i0 + r >= a.t0 && i0 + r < a.t1; });
    fetch_r(blk.lo);
    fetch(blk.lo);
    cp_commit();
    load_br(brs, a, h, threadIdx.x, 256);
    const int iA = i0 + qt * 16 + g, iB = iA + 8; // this thread's two rows
    const bool active = i0 + qt * 16 < a.t1 && i0 + qt * 16 + 16 > a.t0;

    float o[NTC][4], mA = -INFINITY, mB = -INFINITY, lA = 0.0f, lB = 0.0f;
#pragma unroll
    for (int n = 0; n < NTC; n++)
#pragma unroll
        for (int c = 0; c < 4; c++)
            o[n][c] = 0.0f;

    for (int kb = blk.lo; kb <= blk.hi; kb++) {
        const int j0 = kb * KB;
        cp_wait<0>();
        __syncthreads(); // this block's tiles have landed, the one before has been read
        if (kb < blk.hi)
            fetch(kb + 1);
        cp_commit();
        if (!active)
            continue;
        float s[4][4], mbA = -INFINITY, mbB = -INFINITY;
        {
            float e[4][4] = {};
            product_16x32<DK>(s, Qs + qt * 16 * LD, Ks + ((kb & 1) * 64 + hf * 32) * LD, lane);
            if (a.w_r)
                skewed_positions<DK>(e, Qs + qt * 16 * LD, [&](int p) { return Rs + (((kb + (p >> 2)) % 3) * 64 + (p & 3) * 16) * LD; },
                                     qt, hf, es, lane);
            scores_16x32(s, e, brs, a, i0 + qt * 16, j0 + hf * 32, 1 << 30, lane);
        }
#pragma unroll
        for (int n = 0; n < 4; n++) {
            mbA = fmaxf(mbA, fmaxf(s[n][0], s[n][1]));
            mbB = fmaxf(mbB, fmaxf(s[n][2], s[n][3]));
        }
        mbA = fmaxf(mbA, __shfl_xor_sync(0xffffffffu, mbA, 1));
        mbB = fmaxf(mbB, __shfl_xor_sync(0xffffffffu, mbB, 1));
        mbA = fmaxf(mbA, __shfl_xor_sync(0xffffffffu, mbA, 2));
        mbB = fmaxf(mbB, __shfl_xor_sync(0xffffffffu, mbB, 2));
        if (t == 0) {
            mx[hf * 16 + g] = mbA;
            mx[hf * 16 + 8 + g] = mbB;
        }
        asm volatile("bar.sync %0, 64;" ::"r"(1 + qt) : "memory");
        mbA = fmaxf(mbA, mx[(hf ^ 1) * 16 + g]);
        mbB = fmaxf(mbB, mx[(hf ^ 1) * 16 + 8 + g]);
        const float nA = fmaxf(mA, mbA), nB = fmaxf(mB, mbB);
        const float uA = nA == -INFINITY ? 0.0f : nA, uB = nB == -INFINITY ? 0.0f : nB;
        const float scA = __expf(__fsub_rn(mA, uA)), scB = __expf(__fsub_rn(mB, uB));
        mA = nA;
        mB = nB;
        float sA = 0.0f, sB = 0.0f, xA[4], xB[4];
#pragma unroll
        for (int n = 0; n < 4; n++) {
            s[n][0] = __expf(__fsub_rn(s[n][0], uA));
            s[n][1] = __expf(__fsub_rn(s[n][1], uA));
            s[n][2] = __expf(__fsub_rn(s[n][2], uB));
            s[n][3] = __expf(__fsub_rn(s[n][3], uB));
            xA[n] = __fadd_rn(s[n][0], s[n][1]);
            xB[n] = __fadd_rn(s[n][2], s[n][3]);
            sA = __fadd_rn(sA, xA[n]);
            sB = __fadd_rn(sB, xB[n]);
        }
#pragma unroll
        for (int ks = 0; ks < 2; ks++)
            pfs[(hf * 2 + ks) * 32 + lane] = make_uint4(pack2(s[2 * ks][0], s[2 * ks][1]), pack2(s[2 * ks][2], s[2 * ks][3]),
                                                        pack2(s[2 * ks + 1][0], s[2 * ks + 1][1]), pack2(s[2 * ks + 1][2], s[2 * ks + 1][3]));
        if (hf == 0) {
            sums[lane] = sA;
            sums[32 + lane] = sB;
        }
        asm volatile("bar.sync %0, 64;" ::"r"(1 + qt) : "memory");
        if (hf == 1) { // the row's sum runs over the keys in order: half 1 carries on from half 0
            sA = sums[lane];
            sB = sums[32 + lane];
#pragma unroll
            for (int n = 0; n < 4; n++) {
                sA = __fadd_rn(sA, xA[n]);
                sB = __fadd_rn(sB, xB[n]);
            }
            lA = __fmaf_rn(lA, scA, sA);
            lB = __fmaf_rn(lB, scB, sB);
        }
        if (hf < NCH) {
#pragma unroll
            for (int n = 0; n < NTC; n++) {
                o[n][0] = __fmul_rn(o[n][0], scA);
                o[n][1] = __fmul_rn(o[n][1], scA);
                o[n][2] = __fmul_rn(o[n][2], scB);
                o[n][3] = __fmul_rn(o[n][3], scB);
            }
            const bf16 *vb = Vs + ((kb & 1) * 64 + (lane & 7) + ((lane >> 3) & 1) * 8) * LD + hf * (DK / 2) * (NCH - 1) + (lane >> 4) * 8;
#pragma unroll
            for (int ks = 0; ks < 4; ks++) {
                const uint4 u = pfs[ks * 32 + lane];
                const uint32_t pf[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
                for (int p = 0; p < NTC / 2; p++) {
                    uint32_t bb[4];
                    ldsm4t(bb, vb + ks * 16 * LD + p * 16);
                    mma(o[2 * p], pf, bb[0], bb[1]);
                    mma(o[2 * p + 1], pf, bb[2], bb[3]);
                }
            }
        }
    }
    if (!active)
        return;
    if (hf == 1) {
        lA = __fadd_rn(lA, __shfl_xor_sync(0xffffffffu, lA, 1));
        lB = __fadd_rn(lB, __shfl_xor_sync(0xffffffffu, lB, 1));
        lA = __fadd_rn(lA, __shfl_xor_sync(0xffffffffu, lA, 2));
        lB = __fadd_rn(lB, __shfl_xor_sync(0xffffffffu, lB, 2));
        sums[lane] = lA;
        sums[32 + lane] = lB;
    }
    asm volatile("bar.sync %0, 64;" ::"r"(1 + qt) : "memory");
    lA = sums[lane];
    lB = sums[32 + lane];
    const bool okA = iA >= a.t0 && iA < a.t1, okB = iB >= a.t0 && iB < a.t1;
    if (hf < NCH) {
        const float rA = __fdiv_rn(1.0f, lA), rB = __fdiv_rn(1.0f, lB);
#pragma unroll
        for (int n = 0; n < NTC; n++) {
            o[n][0] = __fmul_rn(o[n][0], rA);
            o[n][1] = __fmul_rn(o[n][1], rA);
            o[n][2] = __fmul_rn(o[n][2], rB);
            o[n][3] = __fmul_rn(o[n][3], rB);
        }
        bf16 *out = reinterpret_cast<bf16 *>(a.o) + ((size_t)iA * a.B + b) * HD + h * DK + hf * (DK / 2) * (NCH - 1);
        store_row<WIDE>(out, o, 0, t, okA);
        store_row<WIDE>(out + (size_t)8 * a.B * HD, o, 2, t, okB);
    }
    if (hf == 0 && t == 0 && a.lse) {
        float *lse = a.lse + ((size_t)b * a.H + h) * T;
        if (okA)
            lse[iA] = mA + logf(lA);
        if (okB)
            lse[iB] = mB + logf(lB);
    }
}

// ---------------- forward, one query ----------------
//
// A decoding step: one query per stream, so the op is a stream of K and V through the chip (151 MB a
// layer at 128 streams x 8 heads x 576 keys) and what bounds it is HBM.  One CTA of four warps per
// (stream, head), four key blocks a round: a warp takes one block's scores from tiles of its own, then
// the four share the round's value products by 16-column slices.  The next round's K and table rows are
// fetched as soon as the scores are taken; 220 KB an SM are in flight.  The operand roles are
// exchanged: keys (and table rows, of which a single query needs exactly one per key) fill the 16 rows
// of a product, the query is the other operand, broadcast to its 8 columns; a product of 16 terms gives
// the same bits either way round.
template <int DK> struct OneSmem {
    static constexpr int LD = DK + 8, TILE = 64 * LD * 2;
    static constexpr int K = 0, R = 4 * TILE, V = 8 * TILE, S = 12 * TILE, MB = S + 4 * 64 * 4, TOTAL = MB + 16;
};

template <int DK>
__global__ void __launch_bounds__(128) attn_one_kernel(const __grid_constant__ AttnArgs a)
{
    using SM = OneSmem<DK>;
    constexpr int LD = SM::LD, MT = DK / 16, MW = (MT + 3) / 4; // 16-column slices, and those of one warp
    extern __shared__ __align__(16) unsigned char sm[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    bf16 *Ks = reinterpret_cast<bf16 *>(sm + SM::K) + warp * 64 * LD, *Rs = reinterpret_cast<bf16 *>(sm + SM::R) + warp * 64 * LD,
         *Vall = reinterpret_cast<bf16 *>(sm + SM::V);
    float *sc = reinterpret_cast<float *>(sm + SM::S), *mbs = reinterpret_cast<float *>(sm + SM::MB); // [4][64] scores, [4] maxima
    const int b = blockIdx.x / a.H, h = blockIdx.x % a.H, HD = a.H * DK, T = a.T, M = a.M, L = a.L, i = a.t0;
    const Blocks blk = blocks_of(M, L, a.attn_len, i, i + 1);
    pdl_trigger();
    const bf16 *kv = reinterpret_cast<const bf16 *>(a.kv) + (size_t)b * a.kvp + h * DK;
    auto fetch_kr = [&](int kb) { // this warp's block of a round
        const int j0 = kb * KB;
        if (kb > blk.hi)
            return;
        load_rows<DK>(Ks, kv + (size_t)j0 * a.B * a.kvp, (size_t)a.B * a.kvp, 64, lane, 32, [&](int r) { return j0 + r < L; });
        if (a.w_r)
            load_table<DK, false>(Rs, a, h, j0 - i + a.P - M - 1, 64, lane, 32);
    };
    auto fetch_v = [&](int kb) {
        const int j0 = kb * KB;
        if (kb <= blk.hi)
            load_rows<DK>(Vall + warp * 64 * LD, kv + HD + (size_t)j0 * a.B * a.kvp, (size_t)a.B * a.kvp, 64, lane, 32,
                          [&](int r) { return j0 + r < L; });
    };
    const bool early = a.ahead && blk.lo + warp < blk.hi; // the last block holds this step's own key, which the predecessor writes
    if (!early)
        pdl_wait();
    fetch_kr(blk.lo + warp);
    cp_commit();
    fetch_v(blk.lo + warp);
    cp_commit();
    if (early)
        pdl_wait();
    // the query as the second operand: k = 2t, 2t + 1 (+ 8) of every 16-wide slice, the same for all columns
    uint32_t qf[DK / 16][2];
    {
        const bf16 *q = reinterpret_cast<const bf16 *>(a.q) + ((size_t)i * a.B + b) * a.qp + h * DK;
#pragma unroll
        for (int ks = 0; ks < DK / 16; ks++) {
            qf[ks][0] = *reinterpret_cast<const uint32_t *>(q + ks * 16 + 2 * t);
            qf[ks][1] = *reinterpret_cast<const uint32_t *>(q + ks * 16 + 8 + 2 * t);
        }
    }
    float o[MW][4], m_run = -INFINITY, l = 0.0f; // l: the part of the sum that lane t of a quad keeps
#pragma unroll
    for (int w = 0; w < MW; w++)
#pragma unroll
        for (int c = 0; c < 4; c++)
            o[w][c] = 0.0f;
    for (int kb0 = blk.lo; kb0 <= blk.hi; kb0 += 4) {
        const int kb = kb0 + warp, j0 = kb * KB, nb = min(4, blk.hi - kb0 + 1);
        cp_wait<1>(); // K and the table rows
        __syncwarp();
        if (kb <= blk.hi) {
            float mb = -INFINITY;
#pragma unroll
            for (int m = 0; m < 4; m++) {
                float x[4] = {0.0f, 0.0f, 0.0f, 0.0f}, e[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
                for (int ks = 0; ks < DK / 16; ks++) {
                    uint32_t k4[4];
                    ldsm4(k4, Ks + (m * 16 + (lane & 15)) * LD + ks * 16 + (lane >> 4) * 8);
                    mma(x, k4, qf[ks][0], qf[ks][1]);
                    if (a.w_r) {
                        ldsm4(k4, Rs + (m * 16 + (lane & 15)) * LD + ks * 16 + (lane >> 4) * 8);
                        mma(e, k4, qf[ks][0], qf[ks][1]);
                    }
                }
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    const int j = j0 + m * 16 + g + c * 8, d = i + M - j, r = min(max(j + T - 1 - i, 0), L - 1);
                    const float br = __fmul_rn(a.br_scale, __ldg(a.b_r + (size_t)h * L + r));
                    const float v = (unsigned)d < (unsigned)a.attn_len ? score_of(x[2 * c], e[2 * c], br, a) : -INFINITY;
                    mb = fmaxf(mb, v);
                    if (t == 0)
                        sc[warp * 64 + m * 16 + g + c * 8] = v;
                }
            }
            mb = fmaxf(mb, __shfl_xor_sync(0xffffffffu, mb, 4));
            mb = fmaxf(mb, __shfl_xor_sync(0xffffffffu, mb, 8));
            mb = fmaxf(mb, __shfl_xor_sync(0xffffffffu, mb, 16));
            if (lane == 0)
                mbs[warp] = mb;
        }
        __syncwarp();
        if (kb0 + 4 <= blk.hi)
            fetch_kr(kb + 4);
        cp_commit();
        cp_wait<1>(); // V
        __syncthreads(); // scores, maxima and V of the round are there for everyone
        for (int s = 0; s < nb; s++) {
            const float n = fmaxf(m_run, mbs[s]), u = n == -INFINITY ? 0.0f : n, scale = __expf(__fsub_rn(m_run, u));
            m_run = n;
            float sum = 0.0f;
            uint32_t pf[4][2];
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const float2 v = *reinterpret_cast<const float2 *>(sc + s * 64 + k * 8 + 2 * t);
                const float p0 = __expf(__fsub_rn(v.x, u)), p1 = __expf(__fsub_rn(v.y, u));
                sum = __fadd_rn(sum, __fadd_rn(p0, p1));
                pf[k >> 1][k & 1] = pack2(p0, p1);
            }
            l = __fmaf_rn(l, scale, sum);
#pragma unroll
            for (int w = 0; w < MW; w++) {
                const int m = warp + 4 * w;
                if (MT % 4 != 0 && m >= MT)
                    break;
#pragma unroll
                for (int c = 0; c < 4; c++)
                    o[w][c] = __fmul_rn(o[w][c], scale);
#pragma unroll
                for (int ks = 0; ks < 4; ks++) {
                    uint32_t v4[4]; // V^T: rows are columns of V, so the 8 x 8 blocks come transposed
                    ldsm4t(v4, Vall + (s * 64 + ks * 16 + (lane & 7) + (lane >> 4) * 8) * LD + m * 16 + ((lane >> 3) & 1) * 8);
                    mma(o[w], v4, pf[ks][0], pf[ks][1]);
                }
            }
        }
        __syncthreads(); // the round has been read
        if (kb0 + 4 <= blk.hi)
            fetch_v(kb + 4);
        cp_commit();
    }
    l = __fadd_rn(l, __shfl_xor_sync(0xffffffffu, l, 1));
    l = __fadd_rn(l, __shfl_xor_sync(0xffffffffu, l, 2));
    const float inv = __fdiv_rn(1.0f, l);
    bf16 *out = reinterpret_cast<bf16 *>(a.o) + ((size_t)i * a.B + b) * HD + h * DK;
#pragma unroll
    for (int w = 0; w < MW; w++) {
        const int m = warp + 4 * w;
        if (t == 0 && (MT % 4 == 0 || m < MT)) {
            out[m * 16 + g] = __float2bfloat16_rn(__fmul_rn(o[w][0], inv));
            out[m * 16 + g + 8] = __float2bfloat16_rn(__fmul_rn(o[w][2], inv));
        }
    }
    if (threadIdx.x == 0 && a.lse)
        a.lse[((size_t)b * a.H + h) * T + i] = m_run + logf(l);
}

// The same for head sizes 64 and 128 with tiles that arrive by TMA: 64 rows x 64 columns a copy, 128-byte
// rows, chunk c of row r at c ^ (r % 8).  The loop above spends most of its instructions on addresses (some 600
// a block of a warp against 200 of products, on eight warps an SM), and at 128 streams x 8 heads x 576 keys
// it took 57 us of which HBM needs 23; this loop takes 39.
template <int DK> struct OneTmaSmem {
    static constexpr int NS = DK / 64, TILE = NS * 8192;
    static constexpr int K = 0, R = 4 * TILE, V = 8 * TILE, S = 12 * TILE, MB = S + 4 * 64 * 4, BRS = MB + 16;
    static size_t bytes(int L) { return (size_t)BRS + (size_t)L * 4 + 1024; }
};
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap *map, uint32_t bar, int x, int y, int z)
{
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(dst),
                 "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y), "r"(z)
                 : "memory");
}
__device__ __forceinline__ void ldsm4_at(uint32_t (&r)[4], uint32_t at)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at));
}
__device__ __forceinline__ void ldsm4t_at(uint32_t (&r)[4], uint32_t at)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(at));
}
// byte offset of 16-byte chunk c of row r in a tile
__device__ __forceinline__ uint32_t tile_at(int r, int c) { return (uint32_t)((c >> 3) * 8192 + r * 128 + (((c & 7) ^ (r & 7)) << 4)); }

template <int DK, bool WIDE> // WIDE: an fp32 table takes 16-byte loads
__global__ void __launch_bounds__(128) attn_one_tma_kernel(const __grid_constant__ AttnArgs a, const __grid_constant__ CUtensorMap map_kv,
                                                           const __grid_constant__ CUtensorMap map_r, int stage_br)
{
    using SM = OneTmaSmem<DK>;
    constexpr int NS = SM::NS, TILE = SM::TILE, MT = DK / 16, MW = MT / 4; // 16-column slices, and those of one warp
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ __align__(8) uint64_t bars[8]; // K and table, V of each warp
    __shared__ int abort_s, dummy;
    unsigned char *sm = smraw + ((1024u - (smem_addr(smraw) & 1023u)) & 1023u);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const uint32_t base = smem_addr(sm), Kt = base + SM::K + warp * TILE, Rt = base + SM::R + warp * TILE, Vt = base + SM::V;
    const uint32_t bar_k = smem_addr(bars + warp), bar_v = smem_addr(bars + 4 + warp);
    float *sc = reinterpret_cast<float *>(sm + SM::S), *mbs = reinterpret_cast<float *>(sm + SM::MB); // [4][64] scores, [4] maxima
    float *brs = reinterpret_cast<float *>(sm + SM::BRS);
    const int b = blockIdx.x / a.H, h = blockIdx.x % a.H, HD = a.H * DK, T = a.T, M = a.M, L = a.L, i = a.t0;
    const Blocks blk = blocks_of(M, L, a.attn_len, i, i + 1);
    pdl_trigger();
    if (threadIdx.x == 0) {
        abort_s = 0;
        for (int k = 0; k < 8; k++)
            tc::mbar_init(smem_addr(bars + k), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    int *ef = a.err_flag ? a.err_flag : &dummy;
    bool ok = true; // this lane's waits: after one that ran out it issues no copy and waits no more
    auto fetch_kr = [&](int kb) { // this warp's block of a round
        if (kb > blk.hi)
            return;
        const int j0 = kb * KB, x0 = j0 - i + a.P - M - 1;
        // rows below the table stand for row 0, and a table in fp32 has to be rounded: such tiles are loaded by hand
        const bool by_hand = a.w_r && (!a.w_r16 || x0 < 0);
        if (lane == 0 && ok) {
            const bool r = a.w_r && !by_hand;
            tc::mbar_expect_tx(bar_k, (uint32_t)(r ? 2 * TILE : TILE));
#pragma unroll
            for (int n = 0; n < NS; n++) {
                tma_load_3d(Kt + n * 8192, &map_kv, bar_k, h * DK + n * 64, b, j0);
                if (r)
                    tma_load_3d(Rt + n * 8192, &map_r, bar_k, n * 64, x0, h);
            }
        }
        if (by_hand) {
            const bf16 *w16 = reinterpret_cast<const bf16 *>(a.w_r16) + (size_t)h * a.P * DK;
            const float *w32 = a.w_r + (size_t)h * a.P * DK;
            for (int idx = lane; idx < 64 * (DK / 8); idx += 32) {
                const int r = idx / (DK / 8), c = idx % (DK / 8), x = min(max(x0 + r, 0), a.P - 1);
                if constexpr (WIDE) {
                    uint4 v;
                    if (a.w_r16) {
                        v = *reinterpret_cast<const uint4 *>(w16 + (size_t)x * DK + c * 8);
                    } else {
                        const float4 u = *reinterpret_cast<const float4 *>(w32 + (size_t)x * DK + c * 8);
                        const float4 w = *reinterpret_cast<const float4 *>(w32 + (size_t)x * DK + c * 8 + 4);
                        v = make_uint4(pack2(u.x, u.y), pack2(u.z, u.w), pack2(w.x, w.y), pack2(w.z, w.w));
                    }
                    *reinterpret_cast<uint4 *>(sm + SM::R + warp * TILE + tile_at(r, c)) = v;
                } else {
                    table_piece<false>(reinterpret_cast<bf16 *>(sm + SM::R + warp * TILE + tile_at(r, c)), w32 + (size_t)x * DK + c * 8);
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); // a later round's tile may come by TMA to the same place
        }
    };
    auto fetch_v = [&](int kb) {
        if (kb > blk.hi || lane != 0 || !ok)
            return;
        tc::mbar_expect_tx(bar_v, (uint32_t)TILE);
#pragma unroll
        for (int n = 0; n < NS; n++)
            tma_load_3d(Vt + warp * TILE + n * 8192, &map_kv, bar_v, HD + h * DK + n * 64, b, kb * KB);
    };
    // the last block holds this step's own key, which the predecessor writes
    const bool early = a.ahead && blk.lo + warp < blk.hi;
    if (!a.ahead)
        pdl_wait();
    if (early) {
        fetch_kr(blk.lo + warp);
        fetch_v(blk.lo + warp);
    }
    if (stage_br) // the head's b_r, scaled
        for (int r = threadIdx.x; r < L; r += 128)
            brs[r] = __fmul_rn(a.br_scale, a.b_r[(size_t)h * L + r]);
    if (a.ahead)
        pdl_wait();
    if (!early) {
        fetch_kr(blk.lo + warp);
        fetch_v(blk.lo + warp);
    }
    // the query as the second operand: k = 2t, 2t + 1 (+ 8) of every 16-wide slice, the same for all columns
    uint32_t qf[DK / 16][2];
    {
        const bf16 *q = reinterpret_cast<const bf16 *>(a.q) + ((size_t)i * a.B + b) * a.qp + h * DK;
#pragma unroll
        for (int ks = 0; ks < DK / 16; ks++) {
            qf[ks][0] = *reinterpret_cast<const uint32_t *>(q + ks * 16 + 2 * t);
            qf[ks][1] = *reinterpret_cast<const uint32_t *>(q + ks * 16 + 8 + 2 * t);
        }
    }
    __syncthreads();
    float o[MW][4], m_run = -INFINITY, l = 0.0f; // l: the part of the sum that lane t of a quad keeps
#pragma unroll
    for (int w = 0; w < MW; w++)
#pragma unroll
        for (int c = 0; c < 4; c++)
            o[w][c] = 0.0f;
    uint32_t phase = 0;
    for (int kb0 = blk.lo; kb0 <= blk.hi; kb0 += 4, phase ^= 1) {
        const int kb = kb0 + warp, j0 = kb * KB, nb = min(4, blk.hi - kb0 + 1);
        if (kb <= blk.hi) {
            ok = ok && tc::mbar_wait(bar_k, phase, &abort_s, ef, 44); // K and the table rows
            __syncwarp();
            float mb = -INFINITY;
#pragma unroll
            for (int m = 0; m < 4; m++) {
                float x[4] = {0.0f, 0.0f, 0.0f, 0.0f}, e[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                const int r = m * 16 + (lane & 15);
#pragma unroll
                for (int ks = 0; ks < DK / 16; ks++) {
                    uint32_t k4[4];
                    ldsm4_at(k4, Kt + tile_at(r, ks * 2 + (lane >> 4)));
                    mma(x, k4, qf[ks][0], qf[ks][1]);
                    if (a.w_r) {
                        ldsm4_at(k4, Rt + tile_at(r, ks * 2 + (lane >> 4)));
                        mma(e, k4, qf[ks][0], qf[ks][1]);
                    }
                }
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    const int j = j0 + m * 16 + g + c * 8, d = i + M - j, rr = min(max(j + T - 1 - i, 0), L - 1);
                    const float br = stage_br ? brs[rr] : __fmul_rn(a.br_scale, __ldg(a.b_r + (size_t)h * L + rr));
                    const float v = (unsigned)d < (unsigned)a.attn_len ? score_of(x[2 * c], e[2 * c], br, a) : -INFINITY;
                    mb = fmaxf(mb, v);
                    if (t == 0)
                        sc[warp * 64 + m * 16 + g + c * 8] = v;
                }
            }
            mb = fmaxf(mb, __shfl_xor_sync(0xffffffffu, mb, 4));
            mb = fmaxf(mb, __shfl_xor_sync(0xffffffffu, mb, 8));
            mb = fmaxf(mb, __shfl_xor_sync(0xffffffffu, mb, 16));
            if (lane == 0)
                mbs[warp] = mb;
            __syncwarp();
            fetch_kr(kb + 4);
            ok = ok && tc::mbar_wait(bar_v, phase, &abort_s, ef, 45);
        }
        __syncthreads(); // scores, maxima and V of the round are there for everyone
        for (int s = 0; s < nb; s++) {
            const float n = fmaxf(m_run, mbs[s]), u = n == -INFINITY ? 0.0f : n, scale = __expf(__fsub_rn(m_run, u));
            m_run = n;
            float sum = 0.0f;
            uint32_t pf[4][2];
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const float2 v = *reinterpret_cast<const float2 *>(sc + s * 64 + k * 8 + 2 * t);
                const float p0 = __expf(__fsub_rn(v.x, u)), p1 = __expf(__fsub_rn(v.y, u));
                sum = __fadd_rn(sum, __fadd_rn(p0, p1));
                pf[k >> 1][k & 1] = pack2(p0, p1);
            }
            l = __fmaf_rn(l, scale, sum);
#pragma unroll
            for (int w = 0; w < MW; w++) {
                const int m = warp + 4 * w;
#pragma unroll
                for (int c = 0; c < 4; c++)
                    o[w][c] = __fmul_rn(o[w][c], scale);
#pragma unroll
                for (int ks = 0; ks < 4; ks++) {
                    uint32_t v4[4]; // V^T: rows are columns of V, so the 8 x 8 blocks come transposed
                    ldsm4t_at(v4, Vt + s * TILE + tile_at(ks * 16 + (lane & 7) + (lane >> 4) * 8, m * 2 + ((lane >> 3) & 1)));
                    mma(o[w], v4, pf[ks][0], pf[ks][1]);
                }
            }
        }
        __syncthreads(); // the round has been read
        fetch_v(kb + 4);
    }
    if (lane == 0 && !ok) { // copies still in flight land in this CTA's shared memory: both phases get a bounded chance to finish
        for (uint32_t parity = 0; parity < 2; parity++) {
            tc::mbar_wait(bar_k, parity, &abort_s, ef, 44, tc::DRAIN_TRIES);
            tc::mbar_wait(bar_v, parity, &abort_s, ef, 45, tc::DRAIN_TRIES);
        }
    }
    __syncwarp();
    l = __fadd_rn(l, __shfl_xor_sync(0xffffffffu, l, 1));
    l = __fadd_rn(l, __shfl_xor_sync(0xffffffffu, l, 2));
    if (*static_cast<volatile int *>(&abort_s)) // a wait ran out: no result
        l = __int_as_float(0x7fffffff);
    const float inv = __fdiv_rn(1.0f, l);
    bf16 *out = reinterpret_cast<bf16 *>(a.o) + ((size_t)i * a.B + b) * HD + h * DK;
#pragma unroll
    for (int w = 0; w < MW; w++) {
        const int m = warp + 4 * w;
        if (t == 0) {
            out[m * 16 + g] = __float2bfloat16_rn(__fmul_rn(o[w][0], inv));
            out[m * 16 + g + 8] = __float2bfloat16_rn(__fmul_rn(o[w][2], inv));
        }
    }
    if (threadIdx.x == 0 && a.lse)
        a.lse[((size_t)b * a.H + h) * T + i] = m_run + logf(l);
}

// Many streams and heads: a warp of its own for every (stream, head), a CTA each, up to eight on an SM (four at head size 128).  The four warps
// of the kernel above meet twice a round and its CTAs take turns at loading and at computing; here nothing
// meets, K and the table rows of the next block are on their way as soon as the scores are taken and V as soon as
// its products are, and 128 streams x 8 heads are one wave.  128 x 8 pairs of 576
// keys: 26.4 us, the kernel above 40.6, HBM 23.  Same association.
template <int DK> struct OneWarpSmem {
    static constexpr int NS = DK / 64, TILE = NS * 8192, K = 0, R = TILE, V = 2 * TILE, S = 3 * TILE, TOTAL = S + 64 * 4 + 1024;
};
template <int DK>
__global__ void __launch_bounds__(32) attn_one_warp_kernel(const __grid_constant__ AttnArgs a, const __grid_constant__ CUtensorMap map_kv,
                                                           const __grid_constant__ CUtensorMap map_r)
{
    using SM = OneWarpSmem<DK>;
    constexpr int NS = SM::NS, TILE = SM::TILE, MT = DK / 16; // 16-column slices
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ __align__(8) uint64_t bars[2]; // K and table, V
    __shared__ int abort_s, dummy;
    unsigned char *sm = smraw + ((1024u - (smem_addr(smraw) & 1023u)) & 1023u);
    const int lane = threadIdx.x, g = lane >> 2, t = lane & 3;
    const uint32_t base = smem_addr(sm), Kt = base + SM::K, Rt = base + SM::R, Vt = base + SM::V;
    const uint32_t bar_k = smem_addr(bars), bar_v = smem_addr(bars + 1);
    float *sc = reinterpret_cast<float *>(sm + SM::S);
    const int b = blockIdx.x / a.H, h = blockIdx.x % a.H, HD = a.H * DK, T = a.T, M = a.M, L = a.L, i = a.t0;
    const Blocks blk = blocks_of(M, L, a.attn_len, i, i + 1);
    pdl_trigger();
    if (lane == 0) {
        abort_s = 0;
        tc::mbar_init(bar_k, 1);
        tc::mbar_init(bar_v, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    int *ef = a.err_flag ? a.err_flag : &dummy;
    bool ok = true; // this lane's waits: after one that ran out it issues no copy and waits no more
    float br[4][2]; // of the block that is being fetched
    auto fetch_kr = [&](int kb) {
        if (kb > blk.hi)
            return;
        const int j0 = kb * KB, x0 = j0 - i + a.P - M - 1;
        // rows below the table stand for row 0: such tiles are loaded by hand
        const bool by_hand = a.w_r && x0 < 0;
        if (lane == 0 && ok) {
            const bool r = a.w_r && !by_hand;
            tc::mbar_expect_tx(bar_k, (uint32_t)(r ? 2 * TILE : TILE));
#pragma unroll
            for (int n = 0; n < NS; n++) {
                tma_load_3d(Kt + n * 8192, &map_kv, bar_k, h * DK + n * 64, b, j0);
                if (r)
                    tma_load_3d(Rt + n * 8192, &map_r, bar_k, n * 64, x0, h);
            }
        }
        if (by_hand) {
            const bf16 *w16 = reinterpret_cast<const bf16 *>(a.w_r16) + (size_t)h * a.P * DK;
            for (int idx = lane; idx < 64 * (DK / 8); idx += 32) {
                const int r = idx / (DK / 8), c = idx % (DK / 8), x = min(max(x0 + r, 0), a.P - 1);
                *reinterpret_cast<uint4 *>(sm + SM::R + tile_at(r, c)) = *reinterpret_cast<const uint4 *>(w16 + (size_t)x * DK + c * 8);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); // a later block's tile may come by TMA to the same place
        }
#pragma unroll
        for (int m = 0; m < 4; m++)
#pragma unroll
            for (int c = 0; c < 2; c++)
                br[m][c] = __ldg(a.b_r + (size_t)h * L + min(max(j0 + m * 16 + g + c * 8 + T - 1 - i, 0), L - 1));
    };
    auto fetch_v = [&](int kb) {
        if (kb > blk.hi || lane != 0 || !ok)
            return;
        tc::mbar_expect_tx(bar_v, (uint32_t)TILE);
#pragma unroll
        for (int n = 0; n < NS; n++)
            tma_load_3d(Vt + n * 8192, &map_kv, bar_v, HD + h * DK + n * 64, b, kb * KB);
    };
    const bool early = a.ahead && blk.lo < blk.hi; // the last block holds this step's own key, which the predecessor writes
    if (!early)
        pdl_wait();
    fetch_kr(blk.lo);
    fetch_v(blk.lo);
    if (early)
        pdl_wait();
    // the query as the second operand: k = 2t, 2t + 1 (+ 8) of every 16-wide slice, the same for all columns
    uint32_t qf[DK / 16][2];
    {
        const bf16 *q = reinterpret_cast<const bf16 *>(a.q) + ((size_t)i * a.B + b) * a.qp + h * DK;
#pragma unroll
        for (int ks = 0; ks < DK / 16; ks++) {
            qf[ks][0] = *reinterpret_cast<const uint32_t *>(q + ks * 16 + 2 * t);
            qf[ks][1] = *reinterpret_cast<const uint32_t *>(q + ks * 16 + 8 + 2 * t);
        }
    }
    float o[MT][4], m_run = -INFINITY, l = 0.0f; // l: the part of the sum that lane t of a quad keeps
#pragma unroll
    for (int m = 0; m < MT; m++)
#pragma unroll
        for (int c = 0; c < 4; c++)
            o[m][c] = 0.0f;
    uint32_t phase = 0;
    for (int kb = blk.lo; kb <= blk.hi; kb++, phase ^= 1) {
        const int j0 = kb * KB;
        ok = ok && tc::mbar_wait(bar_k, phase, &abort_s, ef, 46); // K and the table rows
        __syncwarp();
        float mb = -INFINITY;
#pragma unroll
        for (int m = 0; m < 4; m++) {
            float x[4] = {0.0f, 0.0f, 0.0f, 0.0f}, e[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            const int r = m * 16 + (lane & 15);
#pragma unroll
            for (int ks = 0; ks < DK / 16; ks++) {
                uint32_t k4[4];
                ldsm4_at(k4, Kt + tile_at(r, ks * 2 + (lane >> 4)));
                mma(x, k4, qf[ks][0], qf[ks][1]);
                if (a.w_r) {
                    ldsm4_at(k4, Rt + tile_at(r, ks * 2 + (lane >> 4)));
                    mma(e, k4, qf[ks][0], qf[ks][1]);
                }
            }
#pragma unroll
            for (int c = 0; c < 2; c++) {
                const int j = j0 + m * 16 + g + c * 8, d = i + M - j;
                const float v = (unsigned)d < (unsigned)a.attn_len ? score_of(x[2 * c], e[2 * c], __fmul_rn(a.br_scale, br[m][c]), a) : -INFINITY;
                mb = fmaxf(mb, v);
                if (t == 0)
                    sc[m * 16 + g + c * 8] = v;
            }
        }
        mb = fmaxf(mb, __shfl_xor_sync(0xffffffffu, mb, 4));
        mb = fmaxf(mb, __shfl_xor_sync(0xffffffffu, mb, 8));
        mb = fmaxf(mb, __shfl_xor_sync(0xffffffffu, mb, 16));
        __syncwarp(); // the scores are there, K and the table rows have been read
        fetch_kr(kb + 1);
        const float n = fmaxf(m_run, mb), u = n == -INFINITY ? 0.0f : n, scale = __expf(__fsub_rn(m_run, u));
        m_run = n;
        float sum = 0.0f;
        uint32_t pf[4][2];
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const float2 v = *reinterpret_cast<const float2 *>(sc + k * 8 + 2 * t);
            const float p0 = __expf(__fsub_rn(v.x, u)), p1 = __expf(__fsub_rn(v.y, u));
            sum = __fadd_rn(sum, __fadd_rn(p0, p1));
            pf[k >> 1][k & 1] = pack2(p0, p1);
        }
        l = __fmaf_rn(l, scale, sum);
        ok = ok && tc::mbar_wait(bar_v, phase, &abort_s, ef, 47);
        __syncwarp();
#pragma unroll
        for (int m = 0; m < MT; m++) {
#pragma unroll
            for (int c = 0; c < 4; c++)
                o[m][c] = __fmul_rn(o[m][c], scale);
#pragma unroll
            for (int ks = 0; ks < 4; ks++) {
                uint32_t v4[4]; // V^T: rows are columns of V, so the 8 x 8 blocks come transposed
                ldsm4t_at(v4, Vt + tile_at(ks * 16 + (lane & 7) + (lane >> 4) * 8, m * 2 + ((lane >> 3) & 1)));
                mma(o[m], v4, pf[ks][0], pf[ks][1]);
            }
        }
        __syncwarp(); // V and the scores have been read
        fetch_v(kb + 1);
    }
    if (lane == 0 && !ok) { // copies still in flight land in this CTA's shared memory: both phases get a bounded chance to finish
        for (uint32_t parity = 0; parity < 2; parity++) {
            tc::mbar_wait(bar_k, parity, &abort_s, ef, 46, tc::DRAIN_TRIES);
            tc::mbar_wait(bar_v, parity, &abort_s, ef, 47, tc::DRAIN_TRIES);
        }
    }
    __syncwarp();
    l = __fadd_rn(l, __shfl_xor_sync(0xffffffffu, l, 1));
    l = __fadd_rn(l, __shfl_xor_sync(0xffffffffu, l, 2));
    if (*static_cast<volatile int *>(&abort_s)) // a wait ran out: no result
        l = __int_as_float(0x7fffffff);
    const float inv = __fdiv_rn(1.0f, l);
    bf16 *out = reinterpret_cast<bf16 *>(a.o) + ((size_t)i * a.B + b) * HD + h * DK;
#pragma unroll
    for (int m = 0; m < MT; m++)
        if (t == 0) {
            out[m * 16 + g] = __float2bfloat16_rn(__fmul_rn(o[m][0], inv));
            out[m * 16 + g + 8] = __float2bfloat16_rn(__fmul_rn(o[m][2], inv));
        }
    if (lane == 0 && a.lse)
        a.lse[((size_t)b * a.H + h) * T + i] = m_run + logf(l);
}

// ---------------- forward, a group of queries, by TMA ----------------
//
// The same for head sizes 64 and 128 with tiles that arrive by TMA, issued by one thread, in 128-byte rows, chunk c of row r
// at c ^ (r % 8) (tile_at): copies by every thread were a sixth of the instructions of the loop above.  Training
// steps: 12 layers, 128 streams, 576 keys 10617 -> 10477 us; 20 layers, 320 keys 16416 -> 16320; 8 heads of 128 9654 -> 9579.  Table groups
// that have to be rounded from fp32, or hold copies of row 0, are still written by all threads.
template <int DK> struct FwdTmaSmem {
    static constexpr int NS = DK / 64, TILE = NS * 8192;
    static constexpr int Q = 0, K = TILE, V = K + 2 * TILE, R = V + 2 * TILE, ES = R + 3 * TILE, PF = ES + 8 * 16 * ESC * 4, MX = PF + 4 * 4 * 512,
                         BRS = MX + 4 * 6 * 32 * 4;
    static size_t bytes(int L) { return (size_t)BRS + br_bytes(L) + 1024; }
};
// s[nt][c] = 16 rows at `at` against 32 rows at `bt`; oa, ob: this lane's swizzled chunk of 16-wide step k (mod 4) in either
template <int DK>
__device__ __forceinline__ void product_16x32_at(float (&s)[4][4], uint32_t at, uint32_t bt, const uint32_t (&oa)[4], const uint32_t (&ob)[4])
{
#pragma unroll
    for (int n = 0; n < 4; n++)
#pragma unroll
        for (int c = 0; c < 4; c++)
            s[n][c] = 0.0f;
#pragma unroll
    for (int ks = 0; ks < DK / 16; ks++) {
        uint32_t q[4];
        ldsm4_at(q, at + (ks >> 2) * 8192 + oa[ks & 3]);
#pragma unroll
        for (int p = 0; p < 2; p++) {
            uint32_t b[4];
            ldsm4_at(b, bt + (ks >> 2) * 8192 + p * 2048 + ob[ks & 3]);
            mma(s[2 * p], q, b[0], b[1]);
            mma(s[2 * p + 1], q, b[2], b[3]);
        }
    }
}
template <int DK, typename W>
__device__ __forceinline__ void skewed_positions_at(float (&e)[4][4], uint32_t Qt, W window, int qt, int hf, float *es, int lane, const uint32_t (&oa)[4],
                                                    const uint32_t (&ob)[4])
{
    const int g = lane >> 2, t = lane & 3;
    float x[6][4];
#pragma unroll
    for (int n = 0; n < 6; n++)
#pragma unroll
        for (int c = 0; c < 4; c++)
            x[n][c] = 0.0f;
#pragma unroll
    for (int ks = 0; ks < DK / 16; ks++) {
        uint32_t q[4];
        ldsm4_at(q, Qt + (ks >> 2) * 8192 + oa[ks & 3]);
#pragma unroll
        for (int p = 0; p < 3; p++) {
            uint32_t b[4];
            ldsm4_at(b, window(2 * hf + 3 - qt + p) + (ks >> 2) * 8192 + ob[ks & 3]);
            mma(x[2 * p], q, b[0], b[1]);
            mma(x[2 * p + 1], q, b[2], b[3]);
        }
    }
    __syncwarp();
#pragma unroll
    for (int n = 0; n < 6; n++) {
        *reinterpret_cast<float2 *>(es + g * ESC + n * 8 + 2 * t) = make_float2(x[n][0], x[n][1]);
        *reinterpret_cast<float2 *>(es + (g + 8) * ESC + n * 8 + 2 * t) = make_float2(x[n][2], x[n][3]);
    }
    __syncwarp();
#pragma unroll
    for (int n = 0; n < 4; n++)
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const int row = g + (c >> 1) * 8;
            e[n][c] = es[row * ESC + n * 8 + 2 * t + (c & 1) + 15 - row];
        }
}

template <int DK, bool WIDE> // WIDE: out takes 16-byte stores, an fp32 table 16-byte loads
__global__ void __launch_bounds__(256, DK <= 64 ? 2 : 1) attn_fwd_tma_kernel(const __grid_constant__ AttnArgs a, const __grid_constant__ CUtensorMap map_q,
                                                                                    const __grid_constant__ CUtensorMap map_kv,
                                                                                    const __grid_constant__ CUtensorMap map_r)
{
    using SM = FwdTmaSmem<DK>;
    constexpr int TILE = SM::TILE, NTC = DK / 16; // 8-column groups in one column half
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ __align__(8) uint64_t bars[2];
    __shared__ int abort_s, dummy;
    unsigned char *sm = smraw + ((1024u - (smem_addr(smraw) & 1023u)) & 1023u);
    const uint32_t base = smem_addr(sm), bar0 = smem_addr(bars);
    float *brs = reinterpret_cast<float *>(sm + SM::BRS);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int qt = warp & 3, hf = warp >> 2;
    const int b = blockIdx.x / a.H, h = blockIdx.x % a.H, HD = a.H * DK, T = a.T, M = a.M, L = a.L;
    const int i0 = (a.t0 & ~63) + blockIdx.y * 64;
    const Blocks blk = blocks_of(M, L, a.attn_len, max(i0, a.t0), min(i0 + 64, a.t1));
    float *es = reinterpret_cast<float *>(sm + SM::ES) + warp * 16 * ESC;
    // of this tile: [half][row A, row B][8] maxima, then [row A, row B][32] sums of half 0
    float *mx = reinterpret_cast<float *>(sm + SM::MX) + qt * 6 * 32, *sums = mx + 32;
    uint4 *pfs = reinterpret_cast<uint4 *>(sm + SM::PF) + qt * 4 * 32; // A fragments of the tile's probabilities, [16-key step][lane]
    if (threadIdx.x == 0) {
        abort_s = 0;
        tc::mbar_init(bar0, 1);
        tc::mbar_init(bar0 + 8, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    pdl_wait(); // no early trigger: successors resident beside these CTAs cost more than their launch (33 % of the op alone)
    int *ef = a.err_flag ? a.err_flag : &dummy;
    bool ok = true; // thread 0's waits: after one that ran out it issues no copy and waits no more

    const bool fold = a.P < L; // rows below the table stand for row 0; otherwise no visible pair names one
    auto group0 = [&](int gr) { return gr * KB - i0 + a.P - M - 64; }; // first table row of group gr: window rows 0-63 of block gr, 64-127 of block gr - 1
    auto by_hand = [&](int gr) { return a.w_r && (!a.w_r16 || (fold && group0(gr) < 0)); };
    auto group_by_hand = [&](int gr) {
        const bf16 *w16 = reinterpret_cast<const bf16 *>(a.w_r16) + (size_t)h * a.P * DK;
        const float *w32 = a.w_r + (size_t)h * a.P * DK;
        for (int idx = threadIdx.x; idx < 64 * (DK / 8); idx += 256) {
            const int r = idx / (DK / 8), c = idx % (DK / 8), x = min(max(group0(gr) + r, 0), a.P - 1);
            bf16 *to = reinterpret_cast<bf16 *>(sm + SM::R + (gr % 3) * TILE + tile_at(r, c));
            if (a.w_r16)
                *reinterpret_cast<uint4 *>(to) = *reinterpret_cast<const uint4 *>(w16 + (size_t)x * DK + c * 8);
            else
                table_piece<WIDE>(to, w32 + (size_t)x * DK + c * 8);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); // a later group may come by TMA to the same place
    };
    // block kb: its keys and values, the upper half of its window, and with the first block Q and the lower half
    auto fetch = [&](int kb) {
        const bool first = kb == blk.lo, lower = first && a.w_r && !by_hand(kb), upper = a.w_r && !by_hand(kb + 1);
        if (threadIdx.x == 0 && ok) {
            const uint32_t bar = bar0 + 8 * (kb & 1);
            tc::mbar_expect_tx(bar, (uint32_t)((2 + (first ? 1 : 0) + (lower ? 1 : 0) + (upper ? 1 : 0)) * TILE));
#pragma unroll
            for (int n = 0; n < SM::NS; n++) {
                if (first)
                    tma_load_3d(base + SM::Q + n * 8192, &map_q, bar, h * DK + n * 64, b, i0);
                tma_load_3d(base + SM::K + (kb & 1) * TILE + n * 8192, &map_kv, bar, h * DK + n * 64, b, kb * KB);
                if (lower)
                    tma_load_3d(base + SM::R + (kb % 3) * TILE + n * 8192, &map_r, bar, n * 64, group0(kb), h);
                if (upper)
                    tma_load_3d(base + SM::R + ((kb + 1) % 3) * TILE + n * 8192, &map_r, bar, n * 64, group0(kb + 1), h);
                tma_load_3d(base + SM::V + (kb & 1) * TILE + n * 8192, &map_kv, bar, HD + h * DK + n * 64, b, kb * KB);
            }
        }
        if (first && by_hand(kb))
            group_by_hand(kb);
        if (by_hand(kb + 1))
            group_by_hand(kb + 1);
    };
    fetch(blk.lo);
    load_br(brs, a, h, threadIdx.x, 256);
    uint32_t oa[4], ob[4]; // swizzled chunks of this lane's rows: of an operand of 16 rows, and of one of 8 x 2
#pragma unroll
    for (int n = 0; n < 4; n++) {
        oa[n] = (uint32_t)((lane & 15) * 128 + (((n * 2 + (lane >> 4)) ^ (lane & 7)) << 4));
        ob[n] = (uint32_t)(((lane & 7) + (lane >> 4) * 8) * 128 + (((n * 2 + ((lane >> 3) & 1)) ^ (lane & 7)) << 4));
    }
    const uint32_t Qt = base + SM::Q + qt * 2048;
    const int iA = i0 + qt * 16 + g, iB = iA + 8; // this thread's two rows
    const bool active = i0 + qt * 16 < a.t1 && i0 + qt * 16 + 16 > a.t0;

    float o[NTC][4], mA = -INFINITY, mB = -INFINITY, lA = 0.0f, lB = 0.0f;
#pragma unroll
    for (int n = 0; n < NTC; n++)
#pragma unroll
        for (int c = 0; c < 4; c++)
            o[n][c] = 0.0f;

    for (int kb = blk.lo; kb <= blk.hi; kb++) {
        const int j0 = kb * KB;
        if (threadIdx.x == 0)
            ok = ok && tc::mbar_wait(bar0 + 8 * (kb & 1), (uint32_t)(((kb - blk.lo) >> 1) & 1), &abort_s, ef, 48);
        __syncthreads(); // this block's tiles have landed, the one before has been read
        if (kb < blk.hi)
            fetch(kb + 1);
        if (!active)
            continue;
        float s[4][4], mbA = -INFINITY, mbB = -INFINITY;
        {
            float e[4][4] = {};
            product_16x32_at<DK>(s, Qt, base + SM::K + (kb & 1) * TILE + hf * 4096, oa, ob);
            if (a.w_r)
                skewed_positions_at<DK>(e, Qt, [&](int p) { return base + SM::R + ((kb + (p >> 2)) % 3) * TILE + (p & 3) * 2048; }, qt, hf, es, lane, oa, ob);
            scores_16x32(s, e, brs, a, i0 + qt * 16, j0 + hf * 32, 1 << 30, lane);
        }
#pragma unroll
        for (int n = 0; n < 4; n++) {
            mbA = fmaxf(mbA, fmaxf(s[n][0], s[n][1]));
            mbB = fmaxf(mbB, fmaxf(s[n][2], s[n][3]));
        }
        mbA = fmaxf(mbA, __shfl_xor_sync(0xffffffffu, mbA, 1));
        mbB = fmaxf(mbB, __shfl_xor_sync(0xffffffffu, mbB, 1));
        mbA = fmaxf(mbA, __shfl_xor_sync(0xffffffffu, mbA, 2));
        mbB = fmaxf(mbB, __shfl_xor_sync(0xffffffffu, mbB, 2));
        if (t == 0) {
            mx[hf * 16 + g] = mbA;
            mx[hf * 16 + 8 + g] = mbB;
        }
        asm volatile("bar.sync %0, 64;" ::"r"(1 + qt) : "memory");
        mbA = fmaxf(mbA, mx[(hf ^ 1) * 16 + g]);
        mbB = fmaxf(mbB, mx[(hf ^ 1) * 16 + 8 + g]);
        const float nA = fmaxf(mA, mbA), nB = fmaxf(mB, mbB);
        const float uA = nA == -INFINITY ? 0.0f : nA, uB = nB == -INFINITY ? 0.0f : nB;
        const float scA = __expf(__fsub_rn(mA, uA)), scB = __expf(__fsub_rn(mB, uB));
        mA = nA;
        mB = nB;
        float sA = 0.0f, sB = 0.0f, xA[4], xB[4];
#pragma unroll
        for (int n = 0; n < 4; n++) {
            s[n][0] = __expf(__fsub_rn(s[n][0], uA));
            s[n][1] = __expf(__fsub_rn(s[n][1], uA));
            s[n][2] = __expf(__fsub_rn(s[n][2], uB));
            s[n][3] = __expf(__fsub_rn(s[n][3], uB));
            xA[n] = __fadd_rn(s[n][0], s[n][1]);
            xB[n] = __fadd_rn(s[n][2], s[n][3]);
            sA = __fadd_rn(sA, xA[n]);
            sB = __fadd_rn(sB, xB[n]);
        }
#pragma unroll
        for (int ks = 0; ks < 2; ks++)
            pfs[(hf * 2 + ks) * 32 + lane] = make_uint4(pack2(s[2 * ks][0], s[2 * ks][1]), pack2(s[2 * ks][2], s[2 * ks][3]),
                                                        pack2(s[2 * ks + 1][0], s[2 * ks + 1][1]), pack2(s[2 * ks + 1][2], s[2 * ks + 1][3]));
        if (hf == 0) {
            sums[lane] = sA;
            sums[32 + lane] = sB;
        }
        asm volatile("bar.sync %0, 64;" ::"r"(1 + qt) : "memory");
        if (hf == 1) { // the row's sum runs over the keys in order: half 1 carries on from half 0
            sA = sums[lane];
            sB = sums[32 + lane];
#pragma unroll
            for (int n = 0; n < 4; n++) {
                sA = __fadd_rn(sA, xA[n]);
                sB = __fadd_rn(sB, xB[n]);
            }
            lA = __fmaf_rn(lA, scA, sA);
            lB = __fmaf_rn(lB, scB, sB);
        }
        {
#pragma unroll
            for (int n = 0; n < NTC; n++) {
                o[n][0] = __fmul_rn(o[n][0], scA);
                o[n][1] = __fmul_rn(o[n][1], scA);
                o[n][2] = __fmul_rn(o[n][2], scB);
                o[n][3] = __fmul_rn(o[n][3], scB);
            }
            const uint32_t vb = base + SM::V + (kb & 1) * TILE + ((lane & 7) + ((lane >> 3) & 1) * 8) * 128 + (DK == 128 ? hf * 8192 : 0);
            const int vc = (DK == 64 ? hf * 4 : 0) + (lane >> 4);
#pragma unroll
            for (int ks = 0; ks < 4; ks++) {
                const uint4 u = pfs[ks * 32 + lane];
                const uint32_t pf[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
                for (int p = 0; p < NTC / 2; p++) {
                    uint32_t bb[4];
                    ldsm4t_at(bb, vb + ks * 2048 + (((vc + p * 2) ^ (lane & 7)) << 4));
                    mma(o[2 * p], pf, bb[0], bb[1]);
                    mma(o[2 * p + 1], pf, bb[2], bb[3]);
                }
            }
        }
    }
    if (threadIdx.x == 0 && !ok) // copies still in flight land in this CTA's shared memory: both get a bounded chance to finish
        for (uint32_t n = 0; n < 4; n++)
            tc::mbar_wait(bar0 + 8 * (n & 1), n >> 1, &abort_s, ef, 48, tc::DRAIN_TRIES);
    if (!active)
        return;
    if (hf == 1) {
        lA = __fadd_rn(lA, __shfl_xor_sync(0xffffffffu, lA, 1));
        lB = __fadd_rn(lB, __shfl_xor_sync(0xffffffffu, lB, 1));
        lA = __fadd_rn(lA, __shfl_xor_sync(0xffffffffu, lA, 2));
        lB = __fadd_rn(lB, __shfl_xor_sync(0xffffffffu, lB, 2));
        sums[lane] = lA;
        sums[32 + lane] = lB;
    }
    asm volatile("bar.sync %0, 64;" ::"r"(1 + qt) : "memory");
    lA = sums[lane];
    lB = sums[32 + lane];
    const bool okA = iA >= a.t0 && iA < a.t1, okB = iB >= a.t0 && iB < a.t1;
    if (*static_cast<volatile int *>(&abort_s)) // a wait ran out: no result
        lA = lB = __int_as_float(0x7fffffff);
    {
        const float rA = __fdiv_rn(1.0f, lA), rB = __fdiv_rn(1.0f, lB);
#pragma unroll
        for (int n = 0; n < NTC; n++) {
            o[n][0] = __fmul_rn(o[n][0], rA);
            o[n][1] = __fmul_rn(o[n][1], rA);
            o[n][2] = __fmul_rn(o[n][2], rB);
            o[n][3] = __fmul_rn(o[n][3], rB);
        }
        bf16 *out = reinterpret_cast<bf16 *>(a.o) + ((size_t)iA * a.B + b) * HD + h * DK + hf * (DK / 2);
        store_row<WIDE>(out, o, 0, t, okA);
        store_row<WIDE>(out + (size_t)8 * a.B * HD, o, 2, t, okB);
    }
    if (hf == 0 && t == 0 && a.lse) {
        float *lse = a.lse + ((size_t)b * a.H + h) * T;
        if (okA)
            lse[iA] = mA + logf(lA);
        if (okB)
            lse[iB] = mB + logf(lB);
    }
}

// ---------------- backward ----------------
//
// One CTA of eight warps per (stream, head), key blocks in ascending order; per block
//
//   A   warp (q tile, key half): scores and table products again, P = exp(a - lse), dP = dO V^T,
//       dS = P (dP - D) / sqrt(dk); P, dS and the inverse-skewed dE (row ii, window column jj + 63 - ii)
//       go to shared memory as bf16
//   B1  dQ += dS K + dE Rwin                 (registers over all blocks; 16 rows x half the columns)
//   B2  dV = P^T dO, dK = dS^T Q             (complete for the block: stored)
//       dR += dE^T Q and the column sums of dE, per 64-row group of the table
//
// A table group is touched by two consecutive blocks only (upper half of one window, lower half of
// the next), so warps 0-3 keep the even groups' sums in registers and warps 4-7 the odd ones', and
// every table row is stored once; nothing is read back.  Rows that stand for table row 0 (the
// left pad) are folded into it at the end.  K, the table window and V of the next block are fetched
// as soon as phases B1 and A have read the present ones.  109 KB of shared memory at head size 64:
// two CTAs per SM.
template <int DK> struct BwdSmem {
    static constexpr int LD = DK + 8, TILE = 64 * LD * 2;
    static constexpr int LPS = 152, LDE = 136; // row pitches: [P 64 | pad 8 | dS 64 | pad 16], dE window
    static constexpr int Q = 0, DO = Q + TILE, K = DO + TILE, V = K + TILE, R = V + TILE, PS = R + 2 * TILE,
                         DE = PS + 64 * LPS * 2, ES = DE + 64 * LDE * 2, ROW = ES + 4 * 16 * ESC * 4, PAD = ROW + 2 * 64 * 4, BRS = PAD + 8 * DK * 4;
    static size_t bytes(int L) { return (size_t)BRS + br_bytes(L); }
};

template <int DK, bool WIDE> // WIDE: dq, dkv and the table's partials take 16-byte stores, an fp32 table 16-byte loads
__global__ void __launch_bounds__(256, DK <= 64 ? 2 : 1) attn_bwd_kernel(const __grid_constant__ AttnArgs a)
{
    using SM = BwdSmem<DK>;
    constexpr int LD = SM::LD, LPS = SM::LPS, LDE = SM::LDE;
    constexpr int NCH = DK >= 32 ? 2 : 1, NTC = DK / 8 / NCH; // column halves of dQ, dV, dK; 8-column groups in one
    constexpr int NT = DK / 8;
    extern __shared__ __align__(16) unsigned char sm[];
    bf16 *Qs = reinterpret_cast<bf16 *>(sm + SM::Q), *Os = reinterpret_cast<bf16 *>(sm + SM::DO),
         *Ks = reinterpret_cast<bf16 *>(sm + SM::K), *Vs = reinterpret_cast<bf16 *>(sm + SM::V),
         *Rs = reinterpret_cast<bf16 *>(sm + SM::R), *PS = reinterpret_cast<bf16 *>(sm + SM::PS),
         *DE = reinterpret_cast<bf16 *>(sm + SM::DE);
    float *lses = reinterpret_cast<float *>(sm + SM::ROW), *Dr = lses + 64, *brs = reinterpret_cast<float *>(sm + SM::BRS);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int qt = warp & 3, hf = warp >> 2; // phase A: q tile, key half; B: row tile, column half or table set
    const int b = blockIdx.x / a.H, h = blockIdx.x % a.H, HD = a.H * DK, T = a.T, M = a.M, L = a.L, P = a.P;
    const Blocks blk = blocks_of(M, L, a.attn_len, 0, T);
    const int nqt = (T + 15) >> 4; // q tiles in use
    // skew scratch: the warps of key half 0 use their tile's rows of PS (written after both warps of the tile
    // have read their scratch), the others an area of their own
    float *es = hf == 0 ? reinterpret_cast<float *>(PS + qt * 16 * LPS) : reinterpret_cast<float *>(sm + SM::ES) + qt * 16 * ESC;
    pdl_wait(); // no early trigger: successors resident beside these CTAs cost more than their launch (33 % of the op alone)

    const bf16 *kv = reinterpret_cast<const bf16 *>(a.kv) + (size_t)b * a.kvp + h * DK;
    const bf16 *dout = reinterpret_cast<const bf16 *>(a.dout) + (size_t)b * HD + h * DK;
    const bf16 *outp = reinterpret_cast<const bf16 *>(a.out) + (size_t)b * HD + h * DK;
    bf16 *dkv = reinterpret_cast<bf16 *>(a.dkv) + (size_t)b * a.dkvp + h * DK;
    float *dwr = (a.w_r && a.dwr_part) ? a.dwr_part + ((size_t)b * a.H + h) * P * DK : nullptr;
    float *dbr = a.dbr_part ? a.dbr_part + ((size_t)b * a.H + h) * L : nullptr;
    auto window0 = [&](int kb) { return kb * KB + P - M - 64; }; // table row of window row 0
    auto fetch_k = [&](int kb) {
        const int j0 = kb * KB;
        load_rows<DK>(Ks, kv + (size_t)j0 * a.B * a.kvp, (size_t)a.B * a.kvp, 64, threadIdx.x, 256, [&](int r) { return j0 + r < L; });
    };
    auto fetch_v = [&](int kb) {
        const int j0 = kb * KB;
        load_rows<DK>(Vs, kv + HD + (size_t)j0 * a.B * a.kvp, (size_t)a.B * a.kvp, 64, threadIdx.x, 256, [&](int r) { return j0 + r < L; });
    };
    // table group gr (window rows 0-63 of block gr, 64-127 of block gr - 1) into its slot of the two
    auto fetch_r = [&](int gr) {
        if (a.w_r)
            load_table<DK, WIDE>(Rs + (gr & 1) * 64 * LD, a, h, window0(gr), 64, threadIdx.x, 256);
    };
    load_rows<DK>(Qs, reinterpret_cast<const bf16 *>(a.q) + (size_t)b * a.qp + h * DK, (size_t)a.B * a.qp, 64, threadIdx.x, 256,
                  [&](int r) { return r < T; });
    load_rows<DK>(Os, dout, (size_t)a.B * HD, 64, threadIdx.x, 256, [&](int r) { return r < T; });
    fetch_k(blk.lo);
    fetch_v(blk.lo);
    fetch_r(blk.lo);
    fetch_r(blk.lo + 1);
    cp_commit();
    load_br(brs, a, h, threadIdx.x, 256);
    // D_i = dO_i . O_i and the log-sum-exp, a warp for eight rows
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const int r = warp * 8 + k;
        float D = 0.0f;
        if (r < T) {
            const bf16 *x = dout + (size_t)r * a.B * HD, *y = outp + (size_t)r * a.B * HD;
#pragma unroll
            for (int e = lane; e < DK; e += 32)
                D = __fmaf_rn(to_f(x[e]), to_f(y[e]), D);
        }
        D = warp_sum(D);
        if (lane == 0) {
            Dr[r] = D;
            lses[r] = r < T ? a.lse[((size_t)b * a.H + h) * T + r] : 0.0f;
        }
    }
    // outside the rows' bands the dE window is zero for every block; unused q tiles of P, dS and dE stay zero
    for (int idx = threadIdx.x; idx < (64 * LPS + 64 * LDE) / 8; idx += 256)
        reinterpret_cast<uint4 *>(PS)[idx] = make_uint4(0u, 0u, 0u, 0u);
    // what no block reaches: keys' gradients, table rows, b_r slots
    for (int kb = 0; kb * KB < L; kb++) {
        if (kb >= blk.lo && kb <= blk.hi)
            continue;
        for (int idx = threadIdx.x; idx < 64 * (DK / 8); idx += 256) {
            const int j = kb * KB + idx / (DK / 8), c = (idx % (DK / 8)) * 8;
            if (j < L) {
                zero16<WIDE>(dkv + (size_t)j * a.B * a.dkvp + c);
                zero16<WIDE>(dkv + (size_t)j * a.B * a.dkvp + HD + c);
            }
        }
    }
    const int x_lo = window0(blk.lo), x_hi = window0(blk.hi) + 127, r_off = T - P + M; // b_r slot = table row + r_off
    if (dwr)
        for (int idx = threadIdx.x; idx < P * DK / 4; idx += 256) {
            const int x = idx / (DK / 4);
            if (x < x_lo || x > x_hi)
                zero16<WIDE>(reinterpret_cast<float4 *>(dwr) + idx);
        }
    if (dbr)
        for (int r = threadIdx.x; r < L; r += 256)
            if (r < x_lo + r_off || r > x_hi + r_off)
                dbr[r] = 0.0f;

    float dq[NTC][4], dqr[NTC][4], dr[NT][4], cs[4] = {0.0f, 0.0f, 0.0f, 0.0f}; // dq: through the keys, dqr: through the table
#pragma unroll
    for (int n = 0; n < NTC; n++)
#pragma unroll
        for (int c = 0; c < 4; c++)
            dq[n][c] = dqr[n][c] = 0.0f;
#pragma unroll
    for (int n = 0; n < NT; n++)
#pragma unroll
        for (int c = 0; c < 4; c++)
            dr[n][c] = 0.0f;
    // this warp's share of table row 0: its window rows at or below it
    float *pad = reinterpret_cast<float *>(sm + SM::PAD) + warp * DK;
    for (int d = lane; d < DK; d += 32)
        pad[d] = 0.0f;
    // the finished sums of table group gr (this warp: its rows 16 qt ..) out, and the registers cleared
    auto store_group = [&](int gr) {
        const int xA = window0(gr) + qt * 16 + g, xB = xA + 8;
        if (dwr) {
#pragma unroll
            for (int n = 0; n < NT; n++) {
                if (xA > 0 && xA < P)
                    *reinterpret_cast<float2 *>(dwr + (size_t)xA * DK + n * 8 + 2 * t) = make_float2(dr[n][0], dr[n][1]);
                if (xB > 0 && xB < P)
                    *reinterpret_cast<float2 *>(dwr + (size_t)xB * DK + n * 8 + 2 * t) = make_float2(dr[n][2], dr[n][3]);
            }
            if (window0(gr) + qt * 16 <= 0) { // the same for the whole warp
#pragma unroll
                for (int n = 0; n < NT; n++)
#pragma unroll
                    for (int c = 0; c < 2; c++) {
                        float v = (xA <= 0 ? dr[n][c] : 0.0f) + (xB <= 0 ? dr[n][c + 2] : 0.0f);
                        v += __shfl_xor_sync(0xffffffffu, v, 4);
                        v += __shfl_xor_sync(0xffffffffu, v, 8);
                        v += __shfl_xor_sync(0xffffffffu, v, 16);
                        if (g == 0)
                            pad[n * 8 + 2 * t + c] += v;
                    }
            }
        }
        if (dbr && t == 0) {
            const int rA = xA + r_off, rB = xB + r_off;
            if (rA >= 0 && rA < L)
                dbr[rA] = a.br_scale * cs[0];
            if (rB >= 0 && rB < L)
                dbr[rB] = a.br_scale * cs[2];
        }
#pragma unroll
        for (int n = 0; n < NT; n++)
#pragma unroll
            for (int c = 0; c < 4; c++)
                dr[n][c] = 0.0f;
        cs[0] = cs[1] = cs[2] = cs[3] = 0.0f;
    };
    const int iA = qt * 16 + g, iB = iA + 8;
    cp_wait<0>();
    __syncthreads();

    for (int kb = blk.lo; kb <= blk.hi; kb++) {
        const int j0 = kb * KB;
        auto window = [&](int p) { return Rs + (((kb + (p >> 2)) & 1) * 64 + (p & 3) * 16) * LD; }; // piece p of the window
        // ---- A
        if (qt < nqt) {
            float s[4][4], e[4][4] = {};
            product_16x32<DK>(s, Qs + qt * 16 * LD, Ks + hf * 32 * LD, lane);
            if (a.w_r)
                skewed_positions<DK>(e, Qs + qt * 16 * LD, window, qt, hf, es, lane);
            const float lA = lses[iA], lB = lses[iB], DA = Dr[iA], DB = Dr[iB];
            scores_16x32(s, e, brs, a, qt * 16, j0 + hf * 32, T, lane);
#pragma unroll
            for (int n = 0; n < 4; n++)
#pragma unroll
                for (int c = 0; c < 4; c++)
                    s[n][c] = __expf(__fsub_rn(s[n][c], c < 2 ? lA : lB));
            product_16x32<DK>(e, Os + qt * 16 * LD, Vs + hf * 32 * LD, lane); // dP
            asm volatile("bar.sync %0, 64;" ::"r"(1 + qt) : "memory"); // both warps of the tile are done with their scratch
            bf16 *pA = PS + (qt * 16 + g) * LPS + hf * 32 + 2 * t, *pB = pA + 8 * LPS;
#pragma unroll
            for (int n = 0; n < 4; n++) {
                *reinterpret_cast<uint32_t *>(pA + n * 8) = pack2(s[n][0], s[n][1]);
                *reinterpret_cast<uint32_t *>(pB + n * 8) = pack2(s[n][2], s[n][3]);
                const __nv_bfloat162 dA = __floats2bfloat162_rn(s[n][0] * (e[n][0] - DA) * a.inv_sqrt, s[n][1] * (e[n][1] - DA) * a.inv_sqrt);
                const __nv_bfloat162 dB = __floats2bfloat162_rn(s[n][2] * (e[n][2] - DB) * a.inv_sqrt, s[n][3] * (e[n][3] - DB) * a.inv_sqrt);
                *reinterpret_cast<__nv_bfloat162 *>(pA + 72 + n * 8) = dA;
                *reinterpret_cast<__nv_bfloat162 *>(pB + 72 + n * 8) = dB;
                // window column of key jj is jj + 63 - ii: odd rows' pairs are aligned, even rows' are not
                const int w = hf * 32 + n * 8 + 2 * t + 63 - iA;
                bf16 *eA = DE + iA * LDE + w, *eB = DE + iB * LDE + w - 8;
                if (iA & 1) {
                    *reinterpret_cast<__nv_bfloat162 *>(eA) = dA;
                    *reinterpret_cast<__nv_bfloat162 *>(eB) = dB;
                } else {
                    eA[0] = dA.x; eA[1] = dA.y;
                    eB[0] = dB.x; eB[1] = dB.y;
                }
            }
        }
        __syncthreads(); // P, dS, dE complete; V has been read
        if (kb < blk.hi)
            fetch_v(kb + 1);
        // ---- B1: dQ of rows 16 qt .., columns of half hf
        if (qt < nqt && hf < NCH) {
            const bf16 *arow = PS + (qt * 16 + (lane & 15)) * LPS + 72 + (lane >> 4) * 8;
            const int vrow = (lane & 7) + ((lane >> 3) & 1) * 8, vcol = hf * (DK / 2) * (NCH - 1) + (lane >> 4) * 8;
#pragma unroll
            for (int ks = 0; ks < 4; ks++) {
                uint32_t x[4];
                ldsm4(x, arow + ks * 16);
#pragma unroll
                for (int p = 0; p < NTC / 2; p++) {
                    uint32_t bb[4];
                    ldsm4t(bb, Ks + (ks * 16 + vrow) * LD + vcol + p * 16);
                    mma(dq[2 * p], x, bb[0], bb[1]);
                    mma(dq[2 * p + 1], x, bb[2], bb[3]);
                }
            }
            if (a.w_r) {
                const bf16 *erow = DE + (qt * 16 + (lane & 15)) * LDE + (lane >> 4) * 8;
#pragma unroll
                for (int pc = 0; pc < 5; pc++) { // the five pieces of the window that the tile's band touches
                    const int pp = 3 - qt + pc;
                    uint32_t x[4];
                    ldsm4(x, erow + pp * 16);
                    const bf16 *rw = window(pp) + vrow * LD + vcol;
#pragma unroll
                    for (int p = 0; p < NTC / 2; p++) {
                        uint32_t bb[4];
                        ldsm4t(bb, rw + p * 16);
                        mma(dqr[2 * p], x, bb[0], bb[1]);
                        mma(dqr[2 * p + 1], x, bb[2], bb[3]);
                    }
                }
            }
        }
        __syncthreads(); // K and the table window have been read
        if (kb < blk.hi) {
            fetch_k(kb + 1);
            fetch_r(kb + 2); // the slot of group kb
        }
        cp_commit();
        // ---- B2: dV and dK of keys j0 + 16 qt .., columns of half hf
        if (hf < NCH) {
            const bf16 *pcol = PS + ((lane & 7) + (lane >> 4) * 8) * LPS + qt * 16 + ((lane >> 3) & 1) * 8;
            const int vrow = (lane & 7) + ((lane >> 3) & 1) * 8, vcol = hf * (DK / 2) * (NCH - 1) + (lane >> 4) * 8;
#pragma unroll
            for (int which = 0; which < 2; which++) { // 0: dV = P^T dO, 1: dK = dS^T Q
                const bf16 *ac = pcol + which * 72, *bm = (which ? Qs : Os) + vrow * LD + vcol;
                float acc[NTC][4];
#pragma unroll
                for (int n = 0; n < NTC; n++)
#pragma unroll
                    for (int c = 0; c < 4; c++)
                        acc[n][c] = 0.0f;
                for (int ks = 0; ks < nqt; ks++) {
                    uint32_t x[4];
                    ldsm4t(x, ac + ks * 16 * LPS);
#pragma unroll
                    for (int p = 0; p < NTC / 2; p++) {
                        uint32_t bb[4];
                        ldsm4t(bb, bm + ks * 16 * LD + p * 16);
                        mma(acc[2 * p], x, bb[0], bb[1]);
                        mma(acc[2 * p + 1], x, bb[2], bb[3]);
                    }
                }
                const int jA = j0 + qt * 16 + g, jB = jA + 8;
                bf16 *dst = dkv + (which ? 0 : HD) + hf * (DK / 2) * (NCH - 1) + (size_t)(jA < L ? jA : 0) * a.B * a.dkvp;
                store_row<WIDE>(dst, acc, 0, t, jA < L);
                dst += (size_t)(jB < L ? 8 : 0) * a.B * a.dkvp;
                store_row<WIDE>(dst, acc, 2, t, jB < L);
            }
        }
        // dR and the column sums of one table group: the lower one (window columns 0-63) belongs to the warps of
        // set kb & 1, the upper one to the others
        {
            const bool upper = hf != (kb & 1);
            const int piece = (upper ? 4 : 0) + qt, k0 = upper ? 0 : 3 - qt, k1 = min(nqt, upper ? 4 - qt : 4); // q tiles whose band meets the piece
            const bf16 *ecol = DE + ((lane & 7) + (lane >> 4) * 8) * LDE + piece * 16 + ((lane >> 3) & 1) * 8;
            const bf16 *qrow = Qs + ((lane & 7) + ((lane >> 3) & 1) * 8) * LD + (lane >> 4) * 8;
            for (int ks = k0; ks < k1; ks++) {
                uint32_t x[4];
                ldsm4t(x, ecol + ks * 16 * LDE);
                mma(cs, x, 0x3F803F80u, 0x3F803F80u);
                if (dwr) {
#pragma unroll
                    for (int p = 0; p < NT / 2; p++) {
                        uint32_t bb[4];
                        ldsm4t(bb, qrow + ks * 16 * LD + p * 16);
                        mma(dr[2 * p], x, bb[0], bb[1]);
                        mma(dr[2 * p + 1], x, bb[2], bb[3]);
                    }
                }
            }
            if (!upper)
                store_group(kb);
            else if (kb == blk.hi)
                store_group(kb + 1);
        }
        cp_wait<0>();
        __syncthreads(); // the next block's tiles have landed; P, dS and dE may be written again
    }
    if (qt < nqt && hf < NCH) {
#pragma unroll
        for (int n = 0; n < NTC; n++)
#pragma unroll
            for (int c = 0; c < 4; c++)
                dq[n][c] = __fadd_rn(dq[n][c], dqr[n][c]);
        bf16 *dst = reinterpret_cast<bf16 *>(a.dq) + ((size_t)(iA < T ? iA : 0) * a.B + b) * a.dqp + h * DK + hf * (DK / 2) * (NCH - 1);
        store_row<WIDE>(dst, dq, 0, t, iA < T);
        dst += (size_t)(iB < T ? 8 : 0) * a.B * a.dqp;
        store_row<WIDE>(dst, dq, 2, t, iB < T);
    }
    if (dwr && x_lo <= 0) // table row 0: the warps' shares, in warp order (the loop's last barrier is behind them)
        for (int d = threadIdx.x; d < DK; d += 256) {
            const float *all = reinterpret_cast<const float *>(sm + SM::PAD);
            float v = 0.0f;
#pragma unroll
            for (int w = 0; w < 8; w++)
                v += all[w * DK + d];
            dwr[d] = v;
        }
}

// ---------------- host side ----------------

// head sizes and operand placements the kernels take: 16-byte copies of the bf16 operands, stores of two
// elements at least; the fp32 table and `out` as an input may lie anywhere
inline bool head_size(int dk) { return dk == 16 || dk == 32 || dk == 64 || dk == 128; }
inline bool supported(const AttnArgs &a)
{
    return head_size(a.dk) && a.qp % 8 == 0 && a.kvp % 8 == 0 && aligned_to(a.q, 16) && aligned_to(a.kv, 16) && aligned_to(a.o, 4) &&
           aligned_to(a.w_r16, 16);
}
inline bool supported_bwd(const AttnArgs &a)
{
    return supported(a) && a.T <= 64 && a.t0 == 0 && a.t1 == a.T && a.dqp % 8 == 0 && a.dkvp % 8 == 0 && aligned_to(a.dq, 4) &&
           aligned_to(a.dkv, 4) && aligned_to(a.dout, 16) && aligned_to(a.dwr_part, 8) && a.lse;
}
// Shared memory both kernels of a shape need.  At head sizes 64 and 128 the forward kernel by TMA needs a little less than
// FwdSmem, which stays the line between what is taken and what goes to the CUDA-core kernels.
inline bool fits(int dk, int L)
{
    const size_t most = 227 * 1024;
    switch (dk) {
    case 16: return FwdSmem<16>::bytes(L) <= most && BwdSmem<16>::bytes(L) <= most;
    case 32: return FwdSmem<32>::bytes(L) <= most && BwdSmem<32>::bytes(L) <= most;
    case 64: return FwdSmem<64>::bytes(L) <= most && BwdSmem<64>::bytes(L) <= most;
    default: return FwdSmem<128>::bytes(L) <= most && BwdSmem<128>::bytes(L) <= most;
    }
}

// tiles of 64 columns x `rows` of a three-dimensional bf16 tensor whose rows are `mid` or `outer` apart
inline int tile_map(const void *p, const cuuint64_t (&dims)[3], const cuuint64_t (&strides)[2], bool rows_outer, CUtensorMap *out,
                    cuuint32_t rows = 64)
{
    tc::EncodeTiledFn fn = tc::encode_fn();
    if (!fn)
        return nncu_fail(NNCU_ERR_CUDA, "cuTensorMapEncodeTiled is not available");
    cuuint32_t box[3] = {64, rows_outer ? 1u : rows, rows_outer ? rows : 1u}, estr[3] = {1, 1, 1};
    CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void *>(p), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? NNCU_OK : nncu_fail(NNCU_ERR_CUDA, "cuTensorMapEncodeTiled failed: %d", (int)r);
}
// (stream, head) pairs from which a warp each is better than four: the warps have to fill the chip.  Steps of four
// layers over 528 keys, with four warps and with one: head size 64, 256 pairs 177 / 203 us, 384 225 / 221, 768 294 / 270;
// head size 128, 128 pairs 184 / 210 us, 256 252 / 244, 512 377 / 300.
template <int DK> constexpr int one_warp_pairs() { return DK == 64 ? 384 : 256; }
template <int DK> static int forward_one(const AttnArgs &a, cudaStream_t st)
{
    static DeviceOnce once[2];
    if constexpr (DK < 64) {
        NNCU_TRY(smem_limit(once[0], attn_one_kernel<DK>, OneSmem<DK>::TOTAL));
        launch_kind(EDGE_ATTN, attn_one_kernel<DK>, dim3(a.B * a.H), dim3(128), OneSmem<DK>::TOTAL, st, a);
    } else {
        CUtensorMap kv, r;
        const cuuint64_t B = a.B, L = a.L, kvp = a.kvp, H = a.H, P = a.P;
        NNCU_TRY(tile_map(a.kv, {2 * H * DK, B, L}, {kvp * 2, B * kvp * 2}, true, &kv));
        r = kv;
        if (a.w_r16)
            NNCU_TRY(tile_map(a.w_r16, {DK, P, H}, {DK * 2, P * DK * 2}, false, &r));
        if (a.B * a.H >= one_warp_pairs<DK>() && (!a.w_r || a.w_r16)) {
            static DeviceOnce once_warp;
            NNCU_TRY(smem_limit(once_warp, attn_one_warp_kernel<DK>, OneWarpSmem<DK>::TOTAL));
            launch_kind(EDGE_ATTN, attn_one_warp_kernel<DK>, dim3(a.B * a.H), dim3(32), OneWarpSmem<DK>::TOTAL, st, a, kv, r);
            KERNEL_CHECK();
            return NNCU_OK;
        }
        const bool wide = a.w_r16 || aligned_to(a.w_r, 16);
        auto kernel = wide ? attn_one_tma_kernel<DK, true> : attn_one_tma_kernel<DK, false>;
        NNCU_TRY(smem_limit(once[wide], kernel, 226 * 1024)); // its barriers are static
        const size_t most = 226 * 1024, all = OneTmaSmem<DK>::bytes(a.L);
        launch_kind(EDGE_ATTN, kernel, dim3(a.B * a.H), dim3(128), all <= most ? all : OneTmaSmem<DK>::bytes(0), st, a, kv, r,
                 all <= most ? 1 : 0);
    }
    KERNEL_CHECK();
    return NNCU_OK;
}
template <int DK> static int forward_dk(const AttnArgs &a, cudaStream_t st)
{
    if (a.t1 - a.t0 == 1)
        return forward_one<DK>(a, st);
    static DeviceOnce once[2];
    const bool wide = aligned_to(a.o, 16) && aligned_to(a.w_r, 16);
    const dim3 grid(a.B * a.H, (a.t1 - (a.t0 & ~63) + 63) / 64);
    if constexpr (DK >= 64) {
        CUtensorMap q, kv, r;
        const cuuint64_t B = a.B, T = a.T, L = a.L, qp = a.qp, kvp = a.kvp, H = a.H, P = a.P;
        NNCU_TRY(tile_map(a.q, {H * DK, B, T}, {qp * 2, B * qp * 2}, true, &q));
        NNCU_TRY(tile_map(a.kv, {2 * H * DK, B, L}, {kvp * 2, B * kvp * 2}, true, &kv));
        r = kv;
        if (a.w_r16)
            NNCU_TRY(tile_map(a.w_r16, {DK, P, H}, {DK * 2, P * DK * 2}, false, &r));
        auto kernel = wide ? attn_fwd_tma_kernel<DK, true> : attn_fwd_tma_kernel<DK, false>;
        NNCU_TRY(smem_limit(once[wide], kernel, SMEM_MOST - 1024)); // its barriers are static
        launch_kind(EDGE_ATTN, kernel, grid, dim3(256), FwdTmaSmem<DK>::bytes(a.L), st, a, q, kv, r);
    } else {
        auto kernel = wide ? attn_fwd_kernel<DK, true> : attn_fwd_kernel<DK, false>;
        NNCU_TRY(smem_limit(once[wide], kernel, SMEM_MOST));
        launch_kind(EDGE_ATTN, kernel, grid, dim3(256), FwdSmem<DK>::bytes(a.L), st, a);
    }
    KERNEL_CHECK();
    return NNCU_OK;
}
template <int DK> static int backward_dk(const AttnArgs &a, cudaStream_t st)
{
    static DeviceOnce once[2];
    const bool wide = aligned_to(a.dq, 16) && aligned_to(a.dkv, 16) && aligned_to(a.dwr_part, 16) && aligned_to(a.w_r, 16);
    auto kernel = wide ? attn_bwd_kernel<DK, true> : attn_bwd_kernel<DK, false>;
    NNCU_TRY(smem_limit(once[wide], kernel, SMEM_MOST));
    launch_kind(EDGE_ATTN, kernel, dim3(a.B * a.H), dim3(256), BwdSmem<DK>::bytes(a.L), st, a);
    KERNEL_CHECK();
    return NNCU_OK;
}
static int forward(const AttnArgs &a, cudaStream_t st)
{
    switch (a.dk) {
    case 16: return forward_dk<16>(a, st);
    case 32: return forward_dk<32>(a, st);
    case 64: return forward_dk<64>(a, st);
    default: return forward_dk<128>(a, st);
    }
}
static int backward(const AttnArgs &a, cudaStream_t st)
{
    switch (a.dk) {
    case 16: return backward_dk<16>(a, st);
    case 32: return backward_dk<32>(a, st);
    case 64: return backward_dk<64>(a, st);
    default: return backward_dk<128>(a, st);
    }
}

} // namespace fa

namespace fab { // attention_bwd.cuh
static bool takes(const AttnArgs &a);
static bool sums(const AttnArgs &a);
static int backward(const AttnArgs &a, cudaStream_t st);
} // namespace fab

// ---- dispatch: bf16 goes to the tensor-core kernels when the shape allows, everything else to the
// CUDA-core kernels of attention.cuh.  The choice depends on the shape only, never on the query
// range, so one-symbol steps and whole segments take the same arithmetic.
template <typename T>
static int attn_forward_any(const nncu_attn_shape *s, const void *q, const void *kv, const float *w_r,
                            const float *b_r, void *out, float *lse, cudaStream_t st,
                            const AttnPitch *pt = nullptr, const void *w_r16 = nullptr, int *err_flag = nullptr, bool ahead = false)
{
    if (sizeof(T) == 2) {
        AttnArgs a = attn_args(s, pt);
        a.q = q; a.kv = kv; a.w_r = w_r; a.b_r = b_r; a.o = out; a.lse = lse; a.err_flag = err_flag; a.ahead = ahead ? 1 : 0;
        a.w_r16 = w_r ? w_r16 : nullptr;
        if (fa::supported(a) && fa::fits(a.dk, a.L))
            return fa::forward(a, st);
    }
    return attn_forward_t<T>(s, q, kv, w_r, b_r, out, lse, st, pt);
}

// With `sums` dwr_part may come back as sums over streams in fewer parts (fab::slots_of); *sums says whether.  It has room for
// `parts` of them (attn_table_parts).
template <typename T>
static int attn_backward_any(const nncu_attn_shape *s, const void *q, const void *kv, const float *w_r,
                             const float *b_r, const void *out, const float *lse, const void *dout,
                             void *dq, void *dkv, float *dwr_part, float *dbr_part, cudaStream_t st,
                             const AttnPitch *pt = nullptr, const void *w_r16 = nullptr, int *err_flag = nullptr, bool *sums = nullptr, int parts = 0)
{
    const auto room = [&]() {
        return sums && w_r && parts < s->n_streams ? nncu_fail(NNCU_ERR_INVALID, "attention backward: no room for a table a stream") : NNCU_OK;
    };
    if (sizeof(T) == 2) {
        AttnArgs a = attn_args(s, pt);
        a.w_r16 = w_r ? w_r16 : nullptr;
        a.err_flag = err_flag;
        a.q = q; a.kv = kv; a.w_r = w_r; a.b_r = b_r; a.out = out; a.lse = const_cast<float *>(lse);
        a.dout = dout; a.dq = dq; a.dkv = dkv; a.dwr_part = dwr_part; a.dbr_part = dbr_part;
        if (fa::supported_bwd(a) && fa::fits(a.dk, a.L)) {
            if (!fab::takes(a)) {
                NNCU_TRY(room());
                return fa::backward(a, st);
            }
            if (sums)
                *sums = a.sum = fab::sums(a);
            if (!a.sum)
                NNCU_TRY(room());
            return fab::backward(a, st);
        }
    }
    NNCU_TRY(room());
    return attn_backward_t<T>(s, q, kv, w_r, b_r, out, lse, dout, dq, dkv, dwr_part, dbr_part, st, pt);
}

// Whether some kernel pair can run the forward and the backward pass of this shape (asked once,
// when a model is created, so that an unsupported shape is refused there and not in the middle
// of a file).  Mirrors the dispatch of attn_forward_any / attn_backward_any.
template <typename T>
static int attn_shape_supported(const nncu_attn_shape *s, bool has_wr)
{
    AttnArgs a = attn_args(s, nullptr);
    const bool tensor = sizeof(T) == 2 && fa::head_size(a.dk) && fa::fits(a.dk, a.L);
    if (!tensor) {
        size_t smem = 0;
        fwd_pitch<T>(a, has_wr, smem);
        if (smem > 227 * 1024)
            return nncu_fail(NNCU_ERR_RANGE,
                             "attention forward of this shape (%d keys, d_pos %d, d_key %d) needs %zu bytes of "
                             "shared memory; the limit is %d",
                             a.L, a.P, a.dk, smem, 227 * 1024);
    }
    if (!(tensor && a.T <= 64)) {
        size_t smem = 0;
        bwd_pitch<T>(a, has_wr, smem);
        if (smem > 227 * 1024)
            return nncu_fail(NNCU_ERR_RANGE,
                             "attention backward of this shape (seg_len %d, %d keys, d_pos %d, d_key %d) needs %zu "
                             "bytes of shared memory; the limit is %d",
                             a.T, a.L, a.P, a.dk, smem, 227 * 1024);
    }
    return NNCU_OK;
}
