// gemm_tc2.cuh -- the bf16 GEMM of gemm_tc.cuh for outputs of many tiles: CTA pairs, persistent,
// epilogue under the next tile's mainloop.
//
// Two CTAs of a cluster share a 256 x BN tile (tcgen05.mma cta_group::2, M = 256): each loads its own
// 128 rows of A and half of the B rows by TMA, so an SM reads 32 KB of shared
// memory per 64-wide k-block for the products of a single-CTA 128 x BN tile, which reads 48 KB; below
// that width the single-CTA kernel is bound by shared-memory reads (128 x 128: 64 cycles of reads for 32
// of products).  One pair per two SMs walks the tiles in order.
//
// Same bits as gemm_tc.cuh: an output is (chain of the even 64-wide k-blocks) + (chain of the odd
// ones).  Here a tile runs its even blocks first, into TMEM columns [0, BN), then its odd ones into
// [BN, 2 BN).  The epilogue warps take the even sums into registers as soon as they are complete,
// which frees those columns for the next tile while the odd chain is still running, and add the odd
// sums when they come: both accumulators are double-buffered by each other.
//
//   warp 0      TMA producer (one lane), in each CTA for its own halves
//   warp 1      MMA issue (one lane of the leader CTA)
//   warp 2      TMEM allocation and release
//   warps 4-11  epilogue: warp w has TMEM lanes 32 * (w % 4) .. +31 and half of the columns
//
// Barriers: full (leader's: bytes of both CTAs), empty (each CTA's: commits of the leader), acc_full
// (each CTA's: commits of the leader), acc_empty (leader's: the sixteen epilogue warps of the pair).
// Every wait is bounded as in gemm_tc.cuh.  The loads carry no multicast.
#pragma once
#include "gemm_tc.cuh"

namespace tc2 {

using tc::BK;
using tc::fence_after_sync;
using tc::fence_before_sync;
using tc::mbar_expect_tx;
using tc::mbar_init;
using tc::mbar_wait;
using tc::smem_u32;
using tc::tmem_ld32;
using tc::tmem_ld_wait;

constexpr int BN = 256; // columns of a tile
constexpr uint32_t LEADER = 0xFEFFFFFFu; // clears the CTA bit of a shared::cluster address: the leader's copy

__device__ __forceinline__ uint32_t cta_rank()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}
__device__ __forceinline__ void tma_load_pair(uint32_t dst, const CUtensorMap *map, uint32_t bar, int x, int y)
{
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
                 " [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
                 "l"(reinterpret_cast<uint64_t>(map)), "r"(bar & LEADER), "r"(x), "r"(y)
                 : "memory");
}
// arrives on the barrier at this offset in both CTAs when the MMAs issued so far have retired
__device__ __forceinline__ void commit_pair(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
                 "h"((uint16_t)3)
                 : "memory");
}
// One arrival on the leader's barrier at this offset.  Relaxed: what it hands over is tensor memory,
// ordered by the tcgen05 fences on both sides; a release would first wait for the warp's shared-memory
// traffic (1700 cycles measured) and hold up the next chain.
__device__ __forceinline__ void arrive_leader(uint32_t bar)
{
    asm volatile("{\n\t.reg .b32 r;\n\tmapa.shared::cluster.u32 r, %0, 0;\n\t"
                 "mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [r];\n\t}" ::"r"(bar)
                 : "memory");
}
// the four 16-wide steps of one k-block (tc::umma_bf16_x4 for a CTA pair)
template <uint32_t ASTEP, uint32_t BSTEP>
__device__ __forceinline__ void umma_pair_x4(uint32_t tmem_d, uint32_t alo, uint32_t blo, uint32_t idesc, uint32_t accumulate)
{
    asm volatile("{\n\t.reg .pred p, t;\n\t.reg .b64 da, db;\n\t.reg .b32 la, lb;\n\t"
                 "setp.ne.b32 p, %4, 0;\n\t"
                 "setp.eq.b32 t, %4, %4;\n\t"
                 "mov.b64 da, {%1, %5};\n\t"
                 "mov.b64 db, {%2, %5};\n\t"
                 "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %3, p;\n\t"
                 "add.u32 la, %1, %6;\n\t"
                 "add.u32 lb, %2, %7;\n\t"
                 "mov.b64 da, {la, %5};\n\t"
                 "mov.b64 db, {lb, %5};\n\t"
                 "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %3, t;\n\t"
                 "add.u32 la, %1, %8;\n\t"
                 "add.u32 lb, %2, %9;\n\t"
                 "mov.b64 da, {la, %5};\n\t"
                 "mov.b64 db, {lb, %5};\n\t"
                 "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %3, t;\n\t"
                 "add.u32 la, %1, %10;\n\t"
                 "add.u32 lb, %2, %11;\n\t"
                 "mov.b64 da, {la, %5};\n\t"
                 "mov.b64 db, {lb, %5};\n\t"
                 "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %3, t;\n\t}" ::"r"(tmem_d),
                 "r"(alo), "r"(blo), "r"(idesc), "r"(accumulate), "r"(tc::DESC_HI), "n"(ASTEP), "n"(BSTEP),
                 "n"(2 * ASTEP), "n"(2 * BSTEP), "n"(3 * ASTEP), "n"(3 * BSTEP)
                 : "memory");
}

// What a launch computes, and what of it is left out: rows [0, hole_m) x columns [0, hole_n) of the
// output are not needed (whole tiles are skipped); output rows below skip_m have nothing in the first
// skip_k terms of the contraction.
struct Shape {
    int M, N, K;
    int hole_m, hole_n;
    int skip_m, skip_k;
    int ksplit; // pairs per tile, each a run of k-blocks; part z goes to rows z * M .. of the output (a workspace)
    int bias_n;
    int act; // activation whose value goes to a second output (-1: none)
};

struct Smem {
    static constexpr int A_BYTES = 128 * BK * 2, B_BYTES = BN / 2 * BK * 2, STAGE = A_BYTES + B_BYTES;
    static constexpr int STAGES = 5;
    static constexpr int C = STAGES * STAGE;       // two 32-row x 128-byte blocks for each epilogue warp
    static constexpr int BIAS = C + 8 * 8192;      // BN floats
    static constexpr int BAR = BIAS + BN * 4;      // full, empty [STAGES]; acc_full, acc_empty [2]; TMEM slot; abort flag
    static constexpr int TOTAL = BAR + (2 * STAGES + 4) * 8 + 16 + 1024; // + alignment slack
};

// One pair's piece of work: a tile and the k-blocks [kb0, kb1) of it
struct Unit {
    int tm, tn, z, kb0, kb1;
};
__device__ __forceinline__ void tile_at(int idx, int nt, int hm, int hn, int &tm, int &tn);
__device__ __forceinline__ Unit unit_at(int idx, const Shape &sh, int nt, int hm, int hn)
{
    Unit u;
    u.z = idx % sh.ksplit;
    tile_at(idx / sh.ksplit, nt, hm, hn, u.tm, u.tn);
    const int all = (sh.K + BK - 1) / BK, first = u.tm * 256 + 256 <= sh.skip_m ? sh.skip_k / BK : 0;
    const int per = (all - first + sh.ksplit - 1) / sh.ksplit;
    u.kb0 = min(all, first + u.z * per);
    u.kb1 = min(all, u.kb0 + per);
    return u;
}
// the tile with linear index `idx` (hole left out), N fastest
__device__ __forceinline__ void tile_at(int idx, int nt, int hm, int hn, int &tm, int &tn)
{
    const int first = hm * (nt - hn);
    if (idx < first) {
        tm = idx / (nt - hn);
        tn = hn + idx % (nt - hn);
    } else {
        tm = hm + (idx - first) / nt;
        tn = (idx - first) % nt;
    }
}

template <typename TC, bool AMN, bool BMN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(384, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                 const __grid_constant__ CUtensorMap map_c, const __grid_constant__ CUtensorMap map_c2,
                 const __grid_constant__ Shape sh, const float *__restrict__ bias, const TC *addsrc, long ldc, int *err_flag)
{
    using SL = Smem;
    constexpr int ST = SL::STAGES;
    extern __shared__ unsigned char smraw_[];
    unsigned char *sm = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smraw_) + 1023) & ~(uintptr_t)1023);
    uint64_t *bars = reinterpret_cast<uint64_t *>(sm + SL::BAR);
    const uint32_t full0 = smem_u32(bars), empty0 = full0 + 8 * ST, accf0 = empty0 + 8 * ST, acce0 = accf0 + 16;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * ST + 4);
    volatile int *abort_s = reinterpret_cast<volatile int *>(tmem_slot + 1);
    float *bias_s = reinterpret_cast<float *>(sm + SL::BIAS);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cta_rank();
    const int mt = (sh.M + 255) / 256, nt = (sh.N + BN - 1) / BN, hm = sh.hole_m / 256, hn = sh.hole_n / BN;
    const int units = (hm * (nt - hn) + (mt - hm) * nt) * sh.ksplit, stride = gridDim.x / 2;
    pdl_trigger();

    if (threadIdx.x == 0) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_a)) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_b)) : "memory");
        for (int s = 0; s < ST; s++) {
            mbar_init(full0 + 8 * s, 1);
            mbar_init(empty0 + 8 * s, 1);
        }
        for (int b = 0; b < 2; b++) {
            mbar_init(accf0 + 8 * b, 1);
            mbar_init(acce0 + 8 * b, 16);
        }
        *abort_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(2 * BN) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    fence_before_sync();
    __syncthreads();
    cluster_sync(); // the peer's barriers are there
    fence_after_sync();
    pdl_wait();
    const uint32_t tmem = *tmem_slot, sm0 = smem_u32(sm);

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
        if (warp == 0 && lane == 0) {
            int it = 0;
            bool ok = true;
            for (int idx = blockIdx.x / 2; ok && idx < units; idx += stride) {
                const Unit u = unit_at(idx, sh, nt, hm, hn);
                const int ma = u.tm * 256 + (int)rank * 128, nb = u.tn * BN + (int)rank * (BN / 2);
                for (int par = 0; ok && par < 2; par++)
                    for (int kb = u.kb0 + ((u.kb0 ^ par) & 1); kb < u.kb1; kb += 2, it++) {
                        const int s = it % ST, kx = kb * BK;
                        const uint32_t dst = sm0 + s * SL::STAGE, fb = full0 + 8 * s;
                        if (it >= ST && !mbar_wait(empty0 + 8 * s, (uint32_t)((it / ST - 1) & 1), abort_s, err_flag, 51)) {
                            ok = false;
                            break;
                        }
                        if (rank == 0)
                            mbar_expect_tx(fb, 2 * SL::STAGE);
                        if (AMN) {
#pragma unroll
                            for (int i = 0; i < 2; i++)
                                tma_load_pair(dst + i * 8192, &map_a, fb, ma + i * 64, kx);
                        } else {
                            tma_load_pair(dst, &map_a, fb, kx, ma);
                        }
                        if (BMN) {
#pragma unroll
                            for (int i = 0; i < BN / 128; i++)
                                tma_load_pair(dst + SL::A_BYTES + i * 8192, &map_b, fb, nb + i * 64, kx);
                        } else {
                            tma_load_pair(dst + SL::A_BYTES, &map_b, fb, kx, nb);
                        }
                    }
            }
            // The last commits of the leader arrive on this CTA's empty barriers; it must still be here then.
            for (int k = max(0, it - ST); ok && k < it; k++)
                ok = mbar_wait(empty0 + 8 * (k % ST), (uint32_t)((k / ST) & 1), abort_s, err_flag, 52);
        } else if (warp == 1 && lane == 0 && rank == 0) {
            constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((AMN ? 1u : 0u) << 15) | ((BMN ? 1u : 0u) << 16) |
                                       ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
            const uint32_t alo0 = (uint32_t)(AMN ? tc::smem_desc_sw128_mn(sm0) : tc::smem_desc_sw128(sm0));
            const uint32_t blo0 = (uint32_t)(BMN ? tc::smem_desc_sw128_mn(sm0 + SL::A_BYTES) : tc::smem_desc_sw128(sm0 + SL::A_BYTES));
            constexpr uint32_t astep = AMN ? 128u : 2u, bstep = BMN ? 128u : 2u;
            int it = 0, ti = 0;
            bool ok = true;
            for (int idx = blockIdx.x / 2; ok && idx < units; idx += stride, ti++) {
                const Unit u = unit_at(idx, sh, nt, hm, hn);
                for (int par = 0; ok && par < 2; par++) {
                    // the accumulator of this parity has been read by both CTAs (of the tile before)
                    ok = mbar_wait(acce0 + 8 * par, (uint32_t)((ti & 1) ^ 1), abort_s, err_flag, 53);
                    if (!ok)
                        break;
                    fence_after_sync();
                    uint32_t acc = 0;
                    for (int kb = u.kb0 + ((u.kb0 ^ par) & 1); kb < u.kb1; kb += 2, it++, acc = 1) {
                        const int s = it % ST;
                        ok = mbar_wait(full0 + 8 * s, (uint32_t)((it / ST) & 1), abort_s, err_flag, 54);
                        if (!ok)
                            break;
                        fence_after_sync();
                        umma_pair_x4<astep, bstep>(tmem + (uint32_t)(par * BN), alo0 + s * (SL::STAGE >> 4), blo0 + s * (SL::STAGE >> 4),
                                                   idesc, acc);
                        commit_pair(empty0 + 8 * s);
                    }
                    if (ok)
                        commit_pair(accf0 + 8 * par);
                }
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
        const int quarter = warp & 3, half = (warp >> 2) - 1;
        constexpr int NCH = BN / 64;                               // 32-column chunks of this warp
        constexpr int CPB = sizeof(TC) == 2 ? 2 : 1;               // chunks per 128-byte block
        unsigned char *stg0 = sm + SL::C + (warp - 4) * 8192;
        const uint32_t trow = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(half * (BN / 2));
        int ti = 0, blk = 0; // blk: blocks staged, alternating between the two buffers
        bool ok = true;
        // the next buffer: the store before the last has been read out of it
        auto next_buffer = [&]() {
            if (lane == 0)
                asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
            __syncwarp();
            return stg0 + (blk++ & 1) * 4096;
        };
        unsigned char *stg = stg0;
        // a warp whose wait ran out goes on to the end without working: the barriers of its half count on it
        for (int idx = blockIdx.x / 2; idx < units; idx += stride, ti++) {
            const Unit u = unit_at(idx, sh, nt, hm, hn);
            const int row0 = u.tm * 256 + (int)rank * 128 + quarter * 32, row = row0 + lane, n0 = u.tn * BN + half * (BN / 2);
            if (bias) { // this half's columns, by the four warps that use them
                asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory");
                for (int i = (threadIdx.x & 127); i < BN / 2; i += 128)
                    bias_s[half * (BN / 2) + i] = n0 + i < min(sh.N, sh.bias_n) ? __ldg(bias + n0 + i) : 0.0f;
                asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory");
            }
            if (!ok)
                continue;
            // even sums into registers
            uint32_t e[NCH][32];
            const bool has_even = u.kb0 + (u.kb0 & 1) < u.kb1, has_odd = u.kb0 + ((u.kb0 ^ 1) & 1) < u.kb1;
            if (lane == 0)
                ok = mbar_wait(accf0, (uint32_t)(ti & 1), abort_s, err_flag, 55);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok)
                continue;
            fence_after_sync();
#pragma unroll
            for (int c = 0; c < NCH; c++) {
                if (has_even) {
                    tmem_ld32(trow + (uint32_t)(c * 32), e[c]);
                } else {
#pragma unroll
                    for (int j = 0; j < 32; j++)
                        e[c][j] = 0u;
                }
            }
            tmem_ld_wait();
            fence_before_sync();
            __syncwarp();
            if (lane == 0) {
                arrive_leader(acce0);
                ok = mbar_wait(accf0 + 8, (uint32_t)(ti & 1), abort_s, err_flag, 56);
            }
            ok = __all_sync(0xffffffffu, ok);
            if (!ok)
                continue;
            fence_after_sync();
#pragma unroll
            for (int c = 0; c < NCH; c++)
                if (has_odd) {
                    uint32_t q[32];
                    tmem_ld32(trow + (uint32_t)(BN + c * 32), q);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 32; j++)
                        e[c][j] = __float_as_uint(__uint_as_float(e[c][j]) + __uint_as_float(q[j]));
                }
            fence_before_sync(); // the odd accumulator is out of TMEM
            __syncwarp();
            if (lane == 0)
                arrive_leader(acce0 + 8);
#pragma unroll
            for (int c = 0; c < NCH; c++) {
                const int cc = c % CPB, col = n0 + c * 32, c0 = n0 + (c / CPB) * 32 * CPB;
                // a block that lies outside is not staged either: only stores count for next_buffer()
                if (c0 >= sh.N || row0 >= sh.M)
                    continue;
                float x[32];
#pragma unroll
                for (int j = 0; j < 32; j++)
                    x[j] = __uint_as_float(e[c][j]);
                if (cc == 0)
                    stg = next_buffer();
                if (bias) {
                    const float4 *bp = reinterpret_cast<const float4 *>(bias_s + half * (BN / 2) + c * 32);
#pragma unroll
                    for (int v = 0; v < 8; v++) {
                        const float4 t = bp[v];
                        x[v * 4] += t.x; x[v * 4 + 1] += t.y; x[v * 4 + 2] += t.z; x[v * 4 + 3] += t.w;
                    }
                }
                if (addsrc && row < sh.M && col < sh.N) {
                    const TC *add = addsrc + (long)row * ldc + col;
                    if (col + 32 <= sh.N) {
                        const uint4 *a4 = reinterpret_cast<const uint4 *>(add);
#pragma unroll
                        for (int v = 0; v < (int)(32 * sizeof(TC) / 16); v++) {
                            const uint4 t = a4[v];
                            const TC *p = reinterpret_cast<const TC *>(&t);
#pragma unroll
                            for (int w = 0; w < (int)(16 / sizeof(TC)); w++)
                                x[v * (int)(16 / sizeof(TC)) + w] += to_f(p[w]);
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < 32; j++)
                            if (col + j < sh.N)
                                x[j] += to_f(add[j]);
                    }
                }
                unsigned char *rowp = stg + lane * 128;
                if (sizeof(TC) == 2) {
#pragma unroll
                    for (int v = 0; v < 4; v++)
                        *reinterpret_cast<uint4 *>(rowp + (((cc * 4 + v) ^ (lane & 7)) << 4)) =
                            make_uint4(tc::pack_bf16(x[v * 8], x[v * 8 + 1]), tc::pack_bf16(x[v * 8 + 2], x[v * 8 + 3]),
                                       tc::pack_bf16(x[v * 8 + 4], x[v * 8 + 5]), tc::pack_bf16(x[v * 8 + 6], x[v * 8 + 7]));
                } else {
#pragma unroll
                    for (int v = 0; v < 8; v++)
                        *reinterpret_cast<float4 *>(rowp + ((v ^ (lane & 7)) << 4)) = make_float4(x[v * 4], x[v * 4 + 1], x[v * 4 + 2], x[v * 4 + 3]);
                }
                if (cc == CPB - 1) {
                    auto store = [&](const CUtensorMap *map) {
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                        __syncwarp();
                        if (lane == 0) {
                            asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(
                                             reinterpret_cast<uint64_t>(map)),
                                         "r"(smem_u32(stg)), "r"(c0), "r"(u.z * sh.M + row0)
                                         : "memory");
                            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                        }
                    };
                    store(&map_c);
                    if (sizeof(TC) == 2 && sh.act >= 0) {
                        // the activation of the values just stored (rounded as stored), to the second output
                        stg = next_buffer();
#pragma unroll
                        for (int v = 0; v < 8; v++) {
                            uint4 t = *reinterpret_cast<const uint4 *>(rowp + (v << 4));
                            uint32_t *w = &t.x;
#pragma unroll
                            for (int k = 0; k < 4; k++) {
                                const __nv_bfloat162 h = *reinterpret_cast<const __nv_bfloat162 *>(&w[k]);
                                float a0 = __low2float(h), a1 = __high2float(h);
                                a0 = sh.act == NNCU_FF_RELU ? (a0 > 0.0f ? a0 : 0.0f) : gelu_hw(a0);
                                a1 = sh.act == NNCU_FF_RELU ? (a1 > 0.0f ? a1 : 0.0f) : gelu_hw(a1);
                                w[k] = tc::pack_bf16(a0, a1);
                            }
                            *reinterpret_cast<uint4 *>(stg + lane * 128 + (v << 4)) = t;
                        }
                        store(&map_c2);
                    }
                }
            }
        }
        if (lane == 0)
            asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        __syncwarp();
    }
    // common exit: nobody touches TMEM, the peer's barriers or shared memory after this
    __syncwarp();
    fence_before_sync();
    __syncthreads();
    if (*abort_s) { // a wait gave up: let copies that are still in flight land before the CTA retires
        for (int i = 0; i < 2000; i++)
            __nanosleep(500);
    }
    cluster_sync();
    if (warp == 2) {
        fence_after_sync();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * BN) : "memory");
    }
}

// ---------------- host side ----------------

// Extras of a product: see Shape.  C2: second output of a bf16 product (activation), with C's layout.
struct Extra {
    int hole_m = 0, hole_n = 0, skip_m = 0, skip_k = 0, ksplit = 1, act = -1;
    void *C2 = nullptr;
    bool aside = false;   // runs beside the pass's own chain of launches (tc::gemm)
    bool weights = false; // B is one of the model's matrices (tc::gemm)
};
constexpr int PAIRS = 74; // CTA pairs the chip holds (148 SMs)
static int tile_count(int M, int N, const Extra &x)
{
    const int hm = x.hole_m / 256, hn = x.hole_n / BN, mt = ceil_div(M, 256), nt = ceil_div(N, BN);
    return hm * (nt - hn) + (mt - hm) * nt;
}

template <typename TC, bool AMN, bool BMN>
static int launch(cudaStream_t st, int M, int N, int K, const bf16 *A, long lda, const bf16 *B, long ldb, TC *C, long ldc,
                  const float *bias, const TC *addsrc, int *err_flag, int bias_n, const Extra &x)
{
    using SL = Smem;
    if (x.ksplit > 1 && (M % 256 || bias || addsrc || x.C2))
        return nncu_fail(NNCU_ERR_INVALID, "split-K needs whole row tiles and a bare product");
    CUtensorMap ma, mb, mc, mc2;
    if (AMN)
        NNCU_TRY(tc::make_tmap(A, K, M, lda, 64, &ma));
    else
        NNCU_TRY(tc::make_tmap(A, M, K, lda, 128, &ma));
    if (BMN)
        NNCU_TRY(tc::make_tmap(B, K, N, ldb, 64, &mb));
    else
        NNCU_TRY(tc::make_tmap(B, N, K, ldb, BN / 2, &mb));
    NNCU_TRY(tc::make_tmap(C, (long)M * x.ksplit, N, ldc, 32, &mc, 128 / (int)sizeof(TC), (int)sizeof(TC)));
    mc2 = mc;
    if (x.C2)
        NNCU_TRY(tc::make_tmap(x.C2, M, N, ldc, 32, &mc2, 128 / (int)sizeof(TC), (int)sizeof(TC)));
    static DeviceOnce once;
    NNCU_TRY(smem_limit(once, gemm_pair_kernel<TC, AMN, BMN>, SL::TOTAL));
    Shape sh;
    sh.M = M; sh.N = N; sh.K = K;
    sh.hole_m = x.hole_m; sh.hole_n = x.hole_n; sh.skip_m = x.skip_m; sh.skip_k = x.skip_k;
    sh.ksplit = x.ksplit; sh.bias_n = bias_n; sh.act = x.C2 ? x.act : -1;
    const int units = tile_count(M, N, x) * x.ksplit;
    GemmProfiler *pr = g_nncu_prof;
    const bool timed = pr && pr->n < GemmProfiler::MAX_EV;
    if (timed)
        cudaEventRecord(pr->ev[2 * pr->n], st);
    launch_kind(EDGE_GEMM, gemm_pair_kernel<TC, AMN, BMN>, dim3(2 * std::min(units, PAIRS)), dim3(384), SL::TOTAL, st, ma, mb, mc, mc2, sh, bias,
             addsrc, ldc, err_flag);
    if (timed) {
        cudaEventRecord(pr->ev[2 * pr->n + 1], st);
        // what is left out is no work: the hole's tiles, and the terms that whole row tiles skip
        const double hole = (double)(x.hole_m / 256 * 256) * (x.hole_n / BN * BN), skipped = (double)(x.skip_m / 256 * 256) * (x.skip_k / BK * BK);
        pr->flops[pr->n++] = 2.0 * (((double)M * N - hole) * K - skipped * N);
    }
    KERNEL_CHECK();
    return NNCU_OK;
}

// Whether the pair kernel (256-wide tiles) is the better one for an output.  Times of both kernels in us as
// fitted to launches of 256..73728 rows (ncu, cold): a pair launch costs 8 and each round of tiles over
// the 74 pairs 0.34 per 64-wide k-block plus 1 (the epilogue of the last is exposed, the others mostly
// run under the next mainloop); the single-CTA kernel 1 plus, per round of CTAs, 4.4 + 0.13 per k-block
// (64-wide tiles, one per SM) or 4.4 + 0.46 (128-wide, two per SM).  So the pair kernel takes outputs
// of more than one round and long contractions: 20480 x 3072 x 1024 141 -> 94 us, 73728 x 1536 x 512
// 187 -> 101, 4096 x 4096 x 1024 45 -> 34, while 4096 x 1024 x 1024 (64 tiles) stays at 12.9 (14.3).
template <typename TC> static bool pair_better(int M, int N, int K, const void *C, long ldc, const void *addsrc, const Extra &x)
{
    if ((reinterpret_cast<uintptr_t>(C) & 15) || (ldc * sizeof(TC)) % 16 || (reinterpret_cast<uintptr_t>(addsrc) & 15))
        return false;
    const double kb = ceil_div(K, BK), rounds = ceil_div(tile_count(M, N, x), PAIRS);
    const double pair = 8.0 + rounds * (0.34 * kb + 1.0);
    const long mt = ceil_div(M, 128), c64 = mt * ceil_div(N, 64), c128 = mt * ceil_div(N, 128);
    const bool wide = c128 >= 200 || N <= 64; // what tc::gemm takes, its 256-wide tiles (bf16 outputs of 200 and more) counted as 128-wide
    const double one = wide ? 1.0 + std::max(1.0, c128 / 296.0) * (4.4 + 0.46 * kb) : 1.0 + std::max(1.0, c64 / 148.0) * (4.4 + 0.13 * kb);
    return pair < one;
}

// tc::gemm or the pair kernel, by the size of the output.  x.C2 is written by the pair kernel only:
// *did_act says whether it was.
template <typename TC, bool AMN, bool BMN>
static int gemm(cudaStream_t st, int M, int N, int K, const bf16 *A, long lda, const bf16 *B, long ldb, TC *C, long ldc,
                const float *bias, const TC *addsrc, int *err_flag, int bias_n = 1 << 30, const Extra &x = Extra(), bool *did_act = nullptr)
{
    if (did_act)
        *did_act = false;
    if (M <= 0 || N <= 0)
        return NNCU_OK;
    if (!tc::usable(A, lda, B, ldb, K))
        return nncu_fail(NNCU_ERR_INVALID, "tcgen05 GEMM needs 16-byte aligned operands and strides");
    if (pair_better<TC>(M, N, K, C, ldc, addsrc, x)) {
        if (did_act)
            *did_act = x.C2 != nullptr;
        return launch<TC, AMN, BMN>(st, M, N, K, A, lda, B, ldb, C, ldc, bias, addsrc, err_flag, bias_n, x);
    }
    return tc::gemm<TC, AMN, BMN>(st, M, N, K, A, lda, B, ldb, C, ldc, bias, addsrc, err_flag, bias_n, x.weights, x.aside);
}

} // namespace tc2
