// attention_bwd.cuh -- adjoint of the bf16 relative-position attention on tcgen05, head sizes 64 and 128.
//
// Same math as fa::attn_bwd_kernel (nncp.c:722-800).  The products of a (stream, head) run on the tensor
// pipe with keys, or rows of the position table, in the 128 rows of a tile, so that a thread owns one key and a
// run of queries:
//
//   E^T  = Rwin Q^T   (two tiles: window rows 0-127 and 128-191)         S^T = K Q^T,  dP^T = V dO^T
//   dV   = P^T dO,  dK = dS^T Q,  dQ += dS K + dE Rwin,  dR += dE^T Q
//
// Query i0 = 0 and key j0 + jj meet window row jj + 63 - ii; the window of a 128-key block is 192 rows from table
// row j0 + P - M - 64, and the next block's starts 128 rows further on.  E^T is skewed on its way through
// shared memory ([query][key], fp32), dE = [query][window row] is dS skewed back (bf16; zero outside the band,
// which no block writes).
//
// What bounds it.  The warp-level kernel (fa::attn_bwd_kernel) runs 27500 instructions for 128 keys, most of them to
// feed and place operand fragments, and two CTAs took 17200 cycles of an SM for them (8 x 128 pairs of 576 keys: 287 us
// a launch; 16 x 64 of 320: 176).  Here a block of 128 keys is 52 products, issued by one thread, and a chain of phases
// that the sixteen warps go through together, 9300 cycles: scores out of tensor memory and skewed 2100, P and dS 1300,
// their stores 750, the products of the results 2600, the table's sums out 1300, dK and dV out 900.  Training steps:
// 12 layers, 128 streams, 576 keys 11508 -> 10741 us; 20 layers, 64 streams, 320 keys 17177 -> 16445; 20 layers, 8 heads of
// 128 10228 -> 9735; 6 layers, 128 keys 732 -> 678; the op alone, 16 x 8 pairs of 128 keys 27.2 -> 20.8.
// Errors against 64 bits as before (dq 2.41, dk and dv 2.36, tables 1.70 of 1000).
//
//   warps 0-15   compute: warp w has TMEM lanes 32 (w % 4) .. and queries (columns) 16 (w / 4) ..; drains results
//   warp 16      TMA producer (one lane)
//   warp 17      TMEM allocation, product issue (one lane)
//   warps 18, 19 D = dO . O and the log-sum-exp of the next item, b_r, column sums of dE (the b_r gradient)
//
// One CTA per SM walks the (stream, head) pairs; loads run ahead over their borders.  Every wait is bounded; a
// compute warp whose wait ran out goes on without waiting (the barriers count on it), and every result of the CTA's
// pairs becomes NaN.
#pragma once
#include <algorithm>

#include "attention_fa.cuh"

namespace fab {

using tc::fence_after_sync;
using tc::fence_before_sync;
using tc::mbar_expect_tx;
using tc::mbar_init;
using tc::smem_u32;

constexpr int KB = 128;                // keys per block
constexpr int CT = 512;                // compute threads
constexpr int THREADS = CT + 4 * 32;   // 20 warps: 96 registers a thread
constexpr float LOG2E = 1.4426950408889634f;
constexpr int SMEM_LIMIT = SMEM_MOST - 1024; // a kilobyte is static
constexpr int BR_LO = 64, BR_PAD = BR_LO + 192; // zero slots on both sides of b_r that masked pairs name

template <int DK> struct Smem {
    static constexpr int NA = DK / 64;           // 64-column atoms of a row
    static constexpr int NB = DK == 64 ? 2 : 1;  // buffers of everything that is loaded
    static constexpr int QT = NA * 8192, KT = NA * 16384, RT = NA * 24576;
    static constexpr int Q = 0, K = Q + NB * 2 * QT, V = K + NB * KT, R = V + NB * KT, DE = R + NB * RT, PS = DE + 32768,
                         ROW = PS + 32768, SUMS = ROW + 2 * 2 * 64 * 4, PAD = SUMS + 2 * 192 * 4, BAR = PAD + 4 * DK * 4, BRS = BAR + 320;
    static __host__ __device__ int br_floats(int L) { return (L + BR_PAD + 3) & ~3; }
    static size_t bytes(int L) { return (size_t)BRS + 2 * (size_t)br_floats(L) * 4 + 1024; }
};
// tensor memory columns: of head size 128 dV lies over E, dK over S and dP
template <int DK> struct Tmem {
    static constexpr int E = 0, S = 128, D = 192, V = DK == 64 ? 256 : 0, K = V + (DK == 64 ? 64 : 128), Q = DK == 64 ? 384 : 256,
                         R = Q + DK;
};

#ifndef NNCU_FAB_POLLS
#define NNCU_FAB_POLLS (1u << 24)
#endif
// tc::mbar_wait by polling: the waits of a block are short
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int *abort_s, int *err_flag, int code)
{
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p, q;\n\t.reg .u32 c;\n\t"
                 "mov.u32 c, 0;\n"
                 "NNCU_WAIT:\n\t"
                 "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "@p bra NNCU_DONE;\n\t"
                 "add.u32 c, c, 1;\n\t"
                 "setp.lt.u32 q, c, %3;\n\t"
                 "@q bra NNCU_WAIT;\n"
                 "NNCU_DONE:\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok)
                 : "r"(bar), "r"(parity), "r"(NNCU_FAB_POLLS)
                 : "memory");
    if (!ok) {
        *abort_s = 1;
        atomicExch(err_flag, code);
    }
    return ok != 0;
}
__device__ __forceinline__ void umma(uint32_t d, uint32_t alo, uint32_t blo, uint32_t idesc, uint32_t accumulate)
{
    asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
                 "setp.ne.b32 p, %4, 0;\n\t"
                 "mov.b64 da, {%1, %5};\n\t"
                 "mov.b64 db, {%2, %5};\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n\t}" ::"r"(d),
                 "r"(alo), "r"(blo), "r"(idesc), "r"(accumulate), "r"(tc::DESC_HI)
                 : "memory");
}
// low descriptor words: a K-major tile, and an MN-major tile whose 64-wide boxes are `lbo` bytes apart
__device__ __forceinline__ uint32_t kmaj(uint32_t addr) { return ((addr & 0x3FFFFu) >> 4) | (1u << 16); }
__device__ __forceinline__ uint32_t mnmaj(uint32_t addr, uint32_t lbo) { return ((addr & 0x3FFFFu) >> 4) | ((lbo >> 4) << 16); }
__host__ __device__ constexpr uint32_t idesc_of(int m, int n, bool amn, bool bmn)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((amn ? 1u : 0u) << 15) | ((bmn ? 1u : 0u) << 16) | ((uint32_t)(n >> 3) << 17) |
           ((uint32_t)(m >> 4) << 24);
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t *r)
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                   "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ float exp2_hw(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ void arrive(uint32_t bar)
{
    asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tma_store_3d(const CUtensorMap *map, uint32_t src, int x, int y, int z)
{
    asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(reinterpret_cast<uint64_t>(map)),
                 "r"(src), "r"(x), "r"(y), "r"(z)
                 : "memory");
}
// 32 lanes x 16 fp32 columns as fragments of 16 x 8: r[8 c + 4 u + 2 v + e] is row 16 u + 8 v + lane / 4, column 8 c + 2 (lane % 4) + e
__device__ __forceinline__ void tmem_ld_frag16(uint32_t taddr, uint32_t *r)
{
#pragma unroll
    for (int c = 0; c < 2; c++)
#pragma unroll
        for (int u = 0; u < 2; u++)
            asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(r[8 * c + 4 * u]), "=r"(r[8 * c + 4 * u + 1]), "=r"(r[8 * c + 4 * u + 2]), "=r"(r[8 * c + 4 * u + 3])
                         : "r"(taddr + ((uint32_t)(16 * u) << 16) + (uint32_t)(8 * c))
                         : "memory");
}
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void bar_compute() { asm volatile("bar.sync 1, 512;" ::: "memory"); }

// The pairs, all streams of a head after another, in as even runs as there are CTAs: where CTA c starts, and the CTA that
// has a place of the sequence.
struct Share {
    int q, r; // r CTAs with q + 1 pairs, the others with q
    __host__ __device__ Share(int pairs, int ctas) : q(pairs / ctas), r(pairs % ctas) {}
    __host__ __device__ int start(int c) const { return c * q + (c < r ? c : r); }
    __host__ __device__ int cta_of(int at) const { return at < r * (q + 1) ? at / (q + 1) : r + (at - r * (q + 1)) / q; }
};
inline __host__ __device__ int ctas_of(int pairs) { return pairs < 148 ? pairs : 148; }
// how many CTAs have pairs of head h: with AttnArgs::sum its table's partial sums are in that many slots
inline __host__ __device__ int slots_of(int B, int H, int h)
{
    const Share s(B * H, ctas_of(B * H));
    return s.cta_of(h * B + B - 1) - s.cta_of(h * B) + 1;
}

// the CTA's items (stream, head) and their key blocks as one sequence; each role steps through it on its own
template <bool SUM> struct Walk {
    int lo, nkb, B, H, start, step, item, n, kb, b, h; // n: items before this one
    __device__ void at(int k)
    {
        const int i = start + k * step;
        if (SUM) {
            h = i / B;
            b = i - h * B;
        } else {
            b = i / H;
            h = i - b * H;
        }
        item = b * H + h;
        n = k;
    }
    __device__ bool first() const { return kb == lo; }
    __device__ bool last() const { return kb == lo + nkb - 1; }
    __device__ void next()
    {
        if (!last()) {
            kb++;
            return;
        }
        kb = lo;
        at(n + 1);
    }
};

template <int DK, bool WIDE, bool SUM> // SUM: AttnArgs::sum; WIDE: out, w_r, dq, dkv and the table's partials take 16-byte accesses
__global__ void __launch_bounds__(THREADS, 1)
attn_bwd_tc_kernel(const __grid_constant__ AttnArgs a, const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_o,
                   const __grid_constant__ CUtensorMap map_kv, const __grid_constant__ CUtensorMap map_r,
                   const __grid_constant__ CUtensorMap map_dkv)
{
    using SM = Smem<DK>;
    using TM = Tmem<DK>;
    constexpr int NB = SM::NB, NA = SM::NA, NC = DK / 4; // columns of a result that one thread drains
    extern __shared__ __align__(16) unsigned char smraw_[];
    __shared__ int dummy;
    unsigned char *sm = smraw_ + ((1024u - (smem_u32(smraw_) & 1023u)) & 1023u);
    const uint32_t sm0 = smem_u32(sm);
    uint64_t *bars = reinterpret_cast<uint64_t *>(sm + SM::BAR);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 32);
    volatile int *abort_s = reinterpret_cast<volatile int *>(tmem_slot + 1);
    // full and free buffers; what the issuer has finished (P1: E, S and dP; P2: the lower table group, dV,
    // dK and dQ through the keys); READY: P, dS and dE are written; TR_FREE, DRAINED: results read; DE_FREE: dE read by the issuer's
    // products (the upper table group is the last of them) and the column sums
    enum { FULL_QO = 0, FREE_QO = 2, FULL_KV = 4, FULL_R = 6, FREE_KV = 8, FREE_R = 10, ROWS_FULL = 12, ROWS_FREE = 14, P1_DONE = 16, READY, P2_DONE, TR_FREE, DE_FREE, DRAINED, N_BARS };
    static_assert(N_BARS <= 32, "barrier slots");
    const uint32_t bar0 = smem_u32(bars);
    auto bar = [&](int i) { return bar0 + 8 * (uint32_t)i; };
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int B = a.B, HD = a.H * DK, T = a.T, M = a.M, L = a.L, P = a.P;
    // 64-key blocks with a visible pair.  The half of a first or last block that is none of them, and the table rows that only it
    // meets, count as zeros, and their gradients are: what lies there need not be finite
    const fa::Blocks all = fa::blocks_of(M, L, a.attn_len, 0, T);
    auto seen = [&](int b64) { return b64 >= all.lo && b64 <= all.hi; };
    auto met = [&](int g64) { return g64 >= all.lo && g64 <= all.hi + 1; }; // 64 rows of the window, 0-63 of block g64
    Walk<SUM> wk;
    {
        wk.lo = wk.kb = all.lo / 2;
        wk.nkb = all.hi / 2 - wk.lo + 1;
        wk.B = B;
        wk.H = a.H;
    }
    int n_items;
    if (SUM) {
        const Share share(B * a.H, gridDim.x);
        wk.start = share.start(blockIdx.x);
        wk.step = 1;
        n_items = share.start(blockIdx.x + 1) - wk.start;
    } else {
        wk.start = blockIdx.x;
        wk.step = gridDim.x;
        n_items = (B * a.H - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
    }
    wk.at(0);
    const int lo = wk.lo, G = n_items * wk.nkb;
    // where an item's table gradient goes; with a.sum all items of a head that this CTA has share a slot, and add to it but for the first
    auto table_at = [&](int item, int h) {
        return a.dwr_part + (SUM ? (size_t)((int)blockIdx.x - Share(B * a.H, gridDim.x).cta_of(h * B)) * a.H + h : (size_t)item) * P * DK;
    };
    auto adds = [&](int n, int b) { return SUM && n > 0 && b > 0; };
    constexpr int LB = NB - 1; // log2 NB
    constexpr bool STAGED = NB == 2 && WIDE; // dK and dV leave from the places of K and V by TMA
    auto window0 = [&](int kb) { return kb * KB + P - M - 64; }; // table row of window row 0
    const bool fold = P < L; // rows below the table stand for row 0; otherwise no visible pair names one
    auto by_hand = [&](int kb) { return a.w_r && (!a.w_r16 || (fold && window0(kb) < 0)); };
    float *dwr0 = a.w_r ? a.dwr_part : nullptr;

    if (threadIdx.x == 0) {
        for (int i = 0; i < N_BARS; i++)
            mbar_init(bar(i), i == READY || i == TR_FREE || i == DRAINED || (i & ~1) == ROWS_FREE || (STAGED && (i & ~1) == FREE_KV) ? 16
                              : i == DE_FREE ? 3 : (i & ~1) == ROWS_FULL ? 2 : 1);
        *abort_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 17)
        tc::tmem_alloc(smem_u32(tmem_slot), 512);
    for (int i = threadIdx.x; i < 32768 / 16; i += THREADS)
        reinterpret_cast<uint4 *>(sm + SM::DE)[i] = make_uint4(0u, 0u, 0u, 0u);
    fence_async();
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    pdl_wait(); // no early trigger: successors resident beside these CTAs cost more than their launch
    const uint32_t tmem = *tmem_slot;
    int *ef = a.err_flag ? a.err_flag : &dummy;

    if (warp == 16) {
        if (lane == 0) {
            bool ok = true;
            // the results of block g out of the places of its K and V; `w` stands at it
            auto store = [&](const Walk<SUM> &w, int g) {
                const int s = g & (NB - 1);
                if (!(ok = mbar_wait(bar(FREE_KV + s), (uint32_t)((g >> LB) & 1), abort_s, ef, 62)))
                    return;
                tma_store_3d(&map_dkv, sm0 + SM::K + s * SM::KT, w.h * DK, w.b, w.kb * KB);
                tma_store_3d(&map_dkv, sm0 + SM::V + s * SM::KT, HD + w.h * DK, w.b, w.kb * KB);
                asm volatile("cp.async.bulk.commit_group;\n\tcp.async.bulk.wait_group.read 0;" ::: "memory");
            };
            auto ws = wk; // where the stores are
            for (int g = 0; ok && g < G; g++, wk.next()) {
                const int s = g & (NB - 1), b = wk.b, h = wk.h, kb = wk.kb, j0 = kb * KB;
                if (wk.first()) {
                    const int n = wk.n, qs = n & (NB - 1);
                    if (n >= NB && !(ok = mbar_wait(bar(FREE_QO + qs), (uint32_t)(((n >> LB) - 1) & 1), abort_s, ef, 59)))
                        break;
                    mbar_expect_tx(bar(FULL_QO + qs), 2 * SM::QT);
                    const uint32_t dst = sm0 + SM::Q + qs * 2 * SM::QT;
#pragma unroll
                    for (int c = 0; c < NA; c++) {
                        fa::tma_load_3d(dst + c * 8192, &map_q, bar(FULL_QO + qs), h * DK + c * 64, b, 0);
                        fa::tma_load_3d(dst + SM::QT + c * 8192, &map_o, bar(FULL_QO + qs), h * DK + c * 64, b, 0);
                    }
                }
                if (g >= NB) {
                    if constexpr (STAGED) {
                        store(ws, g - NB);
                        ws.next();
                    } else {
                        ok = mbar_wait(bar(FREE_KV + s), (uint32_t)(((g >> LB) - 1) & 1), abort_s, ef, 62);
                    }
                    if (!ok)
                        break;
                }
                mbar_expect_tx(bar(FULL_KV + s), 2 * SM::KT);
#pragma unroll
                for (int c = 0; c < NA; c++)
#pragma unroll
                    for (int p = 0; p < 2; p++) {
                        const int j = seen(2 * kb + p) ? j0 + p * 64 : L; // rows from L on are zeros
                        fa::tma_load_3d(sm0 + SM::K + s * SM::KT + c * 16384 + p * 8192, &map_kv, bar(FULL_KV + s), h * DK + c * 64, b, j);
                        fa::tma_load_3d(sm0 + SM::V + s * SM::KT + c * 16384 + p * 8192, &map_kv, bar(FULL_KV + s), HD + h * DK + c * 64, b, j);
                    }
                if (a.w_r && !by_hand(kb)) {
                    if (g >= NB && !(ok = mbar_wait(bar(FREE_R + s), (uint32_t)(((g >> LB) - 1) & 1), abort_s, ef, 60)))
                        break;
                    mbar_expect_tx(bar(FULL_R + s), SM::RT);
#pragma unroll
                    for (int c = 0; c < NA; c++)
#pragma unroll
                        for (int p = 0; p < 3; p++)
                            fa::tma_load_3d(sm0 + SM::R + s * SM::RT + c * 24576 + p * 8192, &map_r, bar(FULL_R + s), c * 64,
                                            met(2 * kb + p) ? window0(kb) + p * 64 : P, h);
                }
            }
            if constexpr (STAGED)
                for (int g = max(0, G - NB); ok && g < G; g++, ws.next())
                    store(ws, g);
        }
    } else if (warp == 17) {
        if (lane == 0) {
            bool ok = true;
            auto wait = [&](int i, int phase, int code) {
                ok = ok && mbar_wait(bar(i), (uint32_t)(phase & 1), abort_s, ef, code);
                return ok;
            };
            // scores, positions and dP of block g
            auto w1 = wk; // where phase1 is
            auto phase1 = [&](int g) {
                const int s = g & (NB - 1), n = w1.n, qs = n & (NB - 1);
                const bool first = w1.first();
                w1.next();
                if (first && !wait(FULL_QO + qs, n >> LB, 63))
                    return;
                if (!wait(FULL_KV + s, g >> LB, 64) || (a.w_r && !wait(FULL_R + s, g >> LB, 65)))
                    return;
                if (DK == 128 && g > 0 && !wait(DRAINED, g - 1, 66))
                    return;
                fence_after_sync();
                constexpr uint32_t id = idesc_of(128, 64, false, false);
                const uint32_t q = kmaj(sm0 + SM::Q + qs * 2 * SM::QT), o = kmaj(sm0 + SM::Q + qs * 2 * SM::QT + SM::QT),
                               k = kmaj(sm0 + SM::K + s * SM::KT), v = kmaj(sm0 + SM::V + s * SM::KT), r = kmaj(sm0 + SM::R + s * SM::RT);
#pragma unroll
                for (int ks = 0; ks < DK / 16; ks++) {
                    const uint32_t at64 = (ks >> 2) * (8192 >> 4) + (ks & 3) * 2, at128 = (ks >> 2) * (16384 >> 4) + (ks & 3) * 2,
                                   at192 = (ks >> 2) * (24576 >> 4) + (ks & 3) * 2;
                    if (a.w_r) {
                        umma(tmem + TM::E, r + at192, q + at64, id, ks > 0);
                        umma(tmem + TM::E + 64, r + at192 + (16384 >> 4), q + at64, id, ks > 0);
                    }
                    umma(tmem + TM::S, k + at128, q + at64, id, ks > 0);
                    umma(tmem + TM::D, v + at128, o + at64, id, ks > 0);
                }
                tc::umma_commit(bar(P1_DONE));
            };
            phase1(0);
            for (int g = 0; ok && g < G; g++, wk.next()) {
                const int s = g & (NB - 1), qs = wk.n & (NB - 1);
                const bool first = wk.first(), last = wk.last();
                const uint32_t qa = sm0 + SM::Q + qs * 2 * SM::QT;
                const uint32_t q = mnmaj(qa, 8192), o = mnmaj(qa + SM::QT, 8192), k = mnmaj(sm0 + SM::K + s * SM::KT, 16384),
                               r = mnmaj(sm0 + SM::R + s * SM::RT, 24576), ps = sm0 + SM::PS, de = sm0 + SM::DE;
                if (!wait(READY, g, 67))
                    break;
                fence_after_sync();
                // dQ has 64 rows; rows 64-127 of its products are whatever lies behind dS (P) and behind a box of dE (the next), so that
                // all accumulators have one layout
#pragma unroll
                for (int ks = 0; ks < 8; ks++) {
                    umma(tmem + TM::Q, mnmaj(ps, 16384) + ks * 128, k + ks * 128, idesc_of(128, DK, true, true), ks > 0 || !first);
                    if (ks < 4) {
                        umma(tmem + TM::V, kmaj(ps + 16384) + ks * 2, o + ks * 128, idesc_of(128, DK, false, true), ks > 0);
                        umma(tmem + TM::K, kmaj(ps) + ks * 2, q + ks * 128, idesc_of(128, DK, false, true), ks > 0);
                        if (dwr0)
                            umma(tmem + TM::R, mnmaj(de, 8192) + ks * 128, q + ks * 128, idesc_of(128, DK, true, true), ks > 0 || !first);
                    }
                }
                tc::umma_commit(bar(P2_DONE));
                if (!STAGED)
                    tc::umma_commit(bar(FREE_KV + s));
                if (NB == 2 && g + 1 < G)
                    phase1(g + 1); // runs while the results are drained
                if (a.w_r) {
#pragma unroll
                    for (int ks = 0; ks < 12; ks++)
                        umma(tmem + TM::Q, kmaj(de) + (ks >> 2) * (8192 >> 4) + (ks & 3) * 2, r + ks * 128, idesc_of(128, DK, false, true), 1u);
                }
                tc::umma_commit(bar(FREE_R + s));
                if (!wait(TR_FREE, g, 68))
                    break;
                fence_after_sync();
                if (dwr0) {
#pragma unroll
                    for (int ks = 0; ks < 4; ks++)
                        umma(tmem + TM::R, mnmaj(de + 16384, 8192) + ks * 128, q + ks * 128, idesc_of(128, DK, true, true), ks > 0);
                }
                tc::umma_commit(bar(DE_FREE));
                if (last)
                    tc::umma_commit(bar(FREE_QO + qs));
                if (NB == 1 && g + 1 < G)
                    phase1(g + 1);
            }
        }
    } else if (warp >= 18) {
        const int aw = warp - 18, tid = threadIdx.x - 18 * 32;
        bool ok = true;
        float *sums = reinterpret_cast<float *>(sm + SM::SUMS), carry = 0.0f;
        const int x_lo = window0(lo), x_hi = window0(lo + wk.nkb - 1) + 191, r_off = T - P + M; // b_r slot = table row + r_off
        // what the compute warps need of item n, and the parts of its results that no block reaches
        auto rows_of = [&](int n) {
            if (n >= 2) {
                if (lane == 0 && ok)
                    ok = mbar_wait(bar(ROWS_FREE + (n & 1)), (uint32_t)((n / 2 - 1) & 1), abort_s, ef, 69);
                __syncwarp();
            }
            auto of = wk;
            of.at(n);
            const int b = of.b, h = of.h, item = of.item;
            float *lses = reinterpret_cast<float *>(sm + SM::ROW) + (n & 1) * 128, *Dr = lses + 64;
            float *brs = reinterpret_cast<float *>(sm + SM::BRS) + (n & 1) * SM::br_floats(L);
            constexpr int LPR = DK / 8, RPW = 32 / LPR, IT = 32 / RPW; // lanes per row, rows at a time, times for a warp's 32 rows
            const bf16 *dout = reinterpret_cast<const bf16 *>(a.dout) + (size_t)b * HD + h * DK + (lane % LPR) * 8;
            const bf16 *outp = reinterpret_cast<const bf16 *>(a.out) + (size_t)b * HD + h * DK + (lane % LPR) * 8;
            lses[tid] = tid < T ? __ldg(a.lse + (size_t)item * T + tid) * LOG2E : 0.0f;
#pragma unroll 1
            for (int i0 = 0; i0 < IT; i0 += 4) { // four rows' loads in flight
                uint4 x[4], y[4];
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int r = aw * 32 + (i0 + i) * RPW + lane / LPR;
                    x[i] = y[i] = make_uint4(0u, 0u, 0u, 0u);
                    if (r < T) {
                        x[i] = __ldg(reinterpret_cast<const uint4 *>(dout + (size_t)r * B * HD));
                        if constexpr (WIDE) {
                            y[i] = __ldg(reinterpret_cast<const uint4 *>(outp + (size_t)r * B * HD));
                        } else {
#pragma unroll
                            for (int e = 0; e < 8; e++)
                                reinterpret_cast<bf16 *>(&y[i])[e] = outp[(size_t)r * B * HD + e];
                        }
                    }
                }
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const bf16 *xp = reinterpret_cast<const bf16 *>(&x[i]), *yp = reinterpret_cast<const bf16 *>(&y[i]);
                    float D = 0.0f;
#pragma unroll
                    for (int e = 0; e < 8; e++)
                        D = __fmaf_rn(to_f(xp[e]), to_f(yp[e]), D);
#pragma unroll
                    for (int o = LPR / 2; o > 0; o >>= 1)
                        D += __shfl_xor_sync(0xffffffffu, D, o);
                    if (lane % LPR == 0)
                        Dr[aw * 32 + (i0 + i) * RPW + lane / LPR] = D * a.inv_sqrt;
                }
            }
            for (int r0 = tid; r0 < L + BR_PAD; r0 += 8 * 64) { // eight loads in flight
                float v[8];
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    const int x = r0 + k * 64 - BR_LO;
                    v[k] = x >= 0 && x < L ? __ldg(a.b_r + (size_t)h * L + x) : 0.0f;
                }
#pragma unroll
                for (int k = 0; k < 8; k++)
                    if (r0 + k * 64 < L + BR_PAD)
                        brs[r0 + k * 64] = __fmul_rn(a.br_scale, v[k]);
            }
            bf16 *dkv = reinterpret_cast<bf16 *>(a.dkv) + (size_t)b * a.dkvp + h * DK;
            const int j_lo = STAGED ? lo * KB : all.lo * 64, j_hi = STAGED ? (lo + wk.nkb) * KB : (all.hi + 1) * 64, outside = j_lo + max(0, L - j_hi);
            for (int idx = tid; idx < outside * (DK / 8); idx += 64) {
                const int k = idx / (DK / 8), j = k < j_lo ? k : j_hi + k - j_lo, c = (idx % (DK / 8)) * 8;
                fa::zero16<WIDE>(dkv + (size_t)j * B * a.dkvp + c);
                fa::zero16<WIDE>(dkv + (size_t)j * B * a.dkvp + HD + c);
            }
            const int below = min(P, max(0, x_lo)), above = max(0, P - 1 - x_hi);
            if (dwr0 && !adds(n, b)) {
                float *dwr = table_at(item, h);
                for (int idx = tid; idx < (below + above) * (DK / 4); idx += 64) {
                    const int k = idx / (DK / 4), x = k < below ? k : x_hi + 1 + k - below;
                    fa::zero16<WIDE>(dwr + (size_t)x * DK + (idx % (DK / 4)) * 4);
                }
            }
            if (a.dbr_part) {
                float *dbr = a.dbr_part + (size_t)item * L;
                for (int r = tid; r < L; r += 64)
                    if (r < x_lo + r_off || r > x_hi + r_off)
                        dbr[r] = 0.0f;
            }
            __syncwarp();
            if (lane == 0)
                arrive(bar(ROWS_FULL + (n & 1)));
        };
        rows_of(0);
        for (int g = 0; g < G; g++, wk.next()) {
            const int n = wk.n, item = wk.item, kb = wk.kb;
            const bool first = wk.first(), last = wk.last();
            if (lane == 0 && ok)
                ok = mbar_wait(bar(READY), (uint32_t)(g & 1), abort_s, ef, 70);
            __syncwarp();
            if (a.dbr_part) {
                // column sums of the window: each warp half of the queries, a lane columns 2 lane, + 1 of the three boxes
                float s[3][2] = {};
                const unsigned char *at = sm + SM::DE + aw * 4096 + (lane & 3) * 4;
#pragma unroll 8
                for (int q = 0; q < 32; q++)
#pragma unroll
                    for (int p = 0; p < 3; p++) {
                        const uint32_t w = *reinterpret_cast<const uint32_t *>(at + p * 8192 + q * 128 + (((lane >> 2) ^ (q & 7)) << 4));
                        const __nv_bfloat162 v = *reinterpret_cast<const __nv_bfloat162 *>(&w);
                        s[p][0] += __low2float(v);
                        s[p][1] += __high2float(v);
                    }
                __syncwarp();
                if (lane == 0)
                    arrive(bar(DE_FREE));
#pragma unroll
                for (int p = 0; p < 3; p++)
                    *reinterpret_cast<float2 *>(sums + aw * 192 + p * 64 + 2 * lane) = make_float2(s[p][0], s[p][1]);
                asm volatile("bar.sync 2, 64;" ::: "memory");
                // columns 0-63 of a block are columns 128-191 of the one before: the same thread has both
                float *dbr = a.dbr_part + (size_t)item * L;
#pragma unroll
                for (int p = 0; p < 3; p++) {
                    float v = sums[p * 64 + tid] + sums[192 + p * 64 + tid];
                    if (p == 0 && !first)
                        v += carry;
                    if (p == 2)
                        carry = v;
                    const int r = window0(kb) + r_off + p * 64 + tid;
                    if ((p < 2 || last) && r >= 0 && r < L)
                        dbr[r] = a.br_scale * v;
                }
                asm volatile("bar.sync 2, 64;" ::: "memory");
            } else if (lane == 0) {
                arrive(bar(DE_FREE));
            }
            if (first && n + 1 < n_items)
                rows_of(n + 1);
        }
    } else {
        const int qd = warp & 3, cg = warp >> 2, jj = qd * 32 + lane, t4 = lane & 3, lane4 = lane & ~3;
        const uint32_t trow = tmem + ((uint32_t)(qd * 32) << 16);
        bool ok = true;
        auto wait = [&](int i, int phase, int code) {
            if (lane == 0 && ok)
                ok = mbar_wait(bar(i), (uint32_t)(phase & 1), abort_s, ef, code);
            __syncwarp();
            fence_after_sync();
        };
        // all compute warps, once the barrier has completed: warp 0 watches it, because every poll is a shared-memory access that
        // the products' operands and the other warps' work queue behind
        auto meet = [&](int i, int phase, int code) {
            if (threadIdx.x == 0 && ok)
                ok = mbar_wait(bar(i), (uint32_t)(phase & 1), abort_s, ef, code);
            bar_compute();
            fence_after_sync();
        };
        auto signal = [&](int i) { // what this warp has read from tensor memory, or written to shared memory, is behind it
            fence_before_sync();
            __syncwarp();
            if (lane == 0)
                arrive(bar(i));
        };
        // the table window of block g, which `w` stands at, by ordinary stores (rounded from fp32, or with copies of row 0)
        auto window_by_hand = [&](const Walk<SUM> &w, int g) {
            const int h = w.h, x0 = window0(w.kb);
            unsigned char *dst = sm + SM::R + (g & (NB - 1)) * SM::RT;
            const bf16 *w16 = reinterpret_cast<const bf16 *>(a.w_r16) + (size_t)h * P * DK;
            const float *w32 = a.w_r + (size_t)h * P * DK;
#pragma unroll 3
            for (int idx = threadIdx.x; idx < 192 * (DK / 8); idx += CT) {
                const int r = idx / (DK / 8), c = idx % (DK / 8), x = min(max(x0 + r, 0), P - 1);
                bf16 *at = reinterpret_cast<bf16 *>(dst + (c >> 3) * 24576 + r * 128 + (((c & 7) ^ (r & 7)) << 4));
                if (!met(2 * w.kb + (r >> 6)))
                    *reinterpret_cast<uint4 *>(at) = make_uint4(0u, 0u, 0u, 0u);
                else if (a.w_r16)
                    *reinterpret_cast<uint4 *>(at) = *reinterpret_cast<const uint4 *>(w16 + (size_t)x * DK + c * 8);
                else
                    fa::table_piece<WIDE>(at, w32 + (size_t)x * DK + c * 8);
            }
            fence_async();
            bar_compute();
            if (threadIdx.x == 0)
                arrive(bar(FULL_R + (g & (NB - 1))));
        };
        // rows of bf16 results out: this thread's row `x` (NC columns), four neighbouring lanes exchange pieces so that
        // each row leaves in runs of NC columns; row(u) is the destination of row lane4 + u or NULL
        auto store_bf16 = [&](const uint32_t *x, auto row) {
            constexpr int W = NC / 8; // words per piece: 2 or 4
            uint32_t v[W][4];
#pragma unroll
            for (int w = 0; w < W; w++) {
#pragma unroll
                for (int p = 0; p < 4; p++)
                    v[w][p] = fa::pack2(__uint_as_float(x[(p * W + w) * 2]), __uint_as_float(x[(p * W + w) * 2 + 1]));
                fa::quad_transpose(v[w], t4);
            }
#pragma unroll
            for (int u = 0; u < 4; u++) {
                bf16 *dst = row(u);
                if (dst) {
                    if constexpr (!WIDE) {
#pragma unroll
                        for (int w = 0; w < W; w++)
                            *reinterpret_cast<uint32_t *>(dst + (t4 * W + w) * 2) = v[w][u];
                    } else if constexpr (W == 2)
                        *reinterpret_cast<uint2 *>(dst + t4 * 4) = make_uint2(v[0][u], v[1][u]);
                    else
                        *reinterpret_cast<uint4 *>(dst + t4 * 8) = make_uint4(v[0][u], v[1][u], v[2][u], v[3][u]);
                }
            }
        };
        auto load_nc = [&](int col, uint32_t *x) {
#pragma unroll
            for (int c = 0; c < NC; c += 16)
                tmem_ld16(trow + (uint32_t)(col + cg * NC + c), x + c);
            tc::tmem_ld_wait();
        };
        float *pad = reinterpret_cast<float *>(sm + SM::PAD);
        // sums of table rows xb + 0 .. 127 out, as load_table has them
        auto store_table = [&](float *dwr, int xb, const uint32_t *x, bool add) {
            if (fold && xb + qd * 32 <= 0) { // the same for the whole warp: rows at or below 0 go to this warp's share of row 0
#pragma unroll
                for (int c = 0; c < NC / 8; c++)
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        float v = 0.0f;
#pragma unroll
                        for (int k = 0; k < 4; k++)
                            if (xb + qd * 32 + 8 * k + (lane >> 2) <= 0)
                                v += __uint_as_float(x[8 * c + 2 * k + e]);
                        v += __shfl_xor_sync(0xffffffffu, v, 4);
                        v += __shfl_xor_sync(0xffffffffu, v, 8);
                        v += __shfl_xor_sync(0xffffffffu, v, 16);
                        if (lane < 4)
                            pad[qd * DK + cg * NC + 8 * c + 2 * lane + e] += v;
                    }
            }
            const int r0 = xb + qd * 32 + (lane >> 2), least = fold ? 1 : 0;
            float *dst = dwr + (ptrdiff_t)r0 * DK + cg * NC + 2 * t4;
            auto rows = [&](auto f) {
#pragma unroll
                for (int k = 0; k < 4; k++)
                    if (r0 + 8 * k >= least && r0 + 8 * k < P)
#pragma unroll
                        for (int c = 0; c < NC / 8; c++)
                            f(dst + 8 * k * DK + 8 * c, x[8 * c + 2 * k], x[8 * c + 2 * k + 1]);
            };
            if (add) // no other thread has these places, so the sums are taken in the order of the items
                rows([](float *p, uint32_t v0, uint32_t v1) {
                    asm volatile("red.relaxed.gpu.global.add.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(__uint_as_float(v0)), "f"(__uint_as_float(v1)) : "memory");
                });
            else
                rows([](float *p, uint32_t v0, uint32_t v1) { *reinterpret_cast<uint2 *>(p) = make_uint2(v0, v1); });
        };
        auto load_table = [&](uint32_t *x) {
#pragma unroll
            for (int c = 0; c < NC; c += 16)
                tmem_ld_frag16(trow + (uint32_t)(TM::R + cg * NC + c), x + c);
            tc::tmem_ld_wait();
        };
        if (by_hand(lo))
            window_by_hand(wk, 0);
        // byte offset of window column jj + 63 - 16 cg in a row of dE, the 128-byte boxes spread 8 KB apart: bits 7 to 12 stay free
        const uint32_t de0 = (uint32_t)(((jj + 63 - cg * 16) * 2) & 127) | ((uint32_t)((jj + 63 - cg * 16) >> 6) << 13);
        const float sc2 = a.inv_sqrt * LOG2E;
        for (int g = 0; g < G; g++) {
            const int n = wk.n, b = wk.b, h = wk.h, kb = wk.kb, j0 = kb * KB, s = g & (NB - 1);
            const bool first = wk.first(), last = wk.last();
            const float *lses = reinterpret_cast<const float *>(sm + SM::ROW) + (n & 1) * 128 + cg * 16;
            const float *br = reinterpret_cast<const float *>(sm + SM::BRS) + (n & 1) * SM::br_floats(L) + BR_LO + j0 + jj + T - 1 - cg * 16;
            float *dwr = dwr0 ? table_at(wk.item, h) : nullptr;
            const bool add = adds(n, b);
            if (first) {
                if (fold && dwr) { // own shares
                    for (int c = lane; c < NC; c += 32)
                        pad[qd * DK + cg * NC + c] = 0.0f;
                    __syncwarp();
                }
                wait(ROWS_FULL + (n & 1), n >> 1, 71); // once an item
            }
            meet(P1_DONE, g, 72);
            float e[16];
            if (a.w_r) {
                float *es = reinterpret_cast<float *>(sm + SM::PS) + cg * 16 * 128;
                uint32_t x[16];
#pragma unroll
                for (int t = 0; t < 2; t++) {
                    if (t == 1 && qd >= 2)
                        break;
                    // window row t * 128 + jj and query 16 cg + c: key k0 + c.  Where no lane's key is in the block, or all are,
                    // the whole warp knows
                    const int k0 = t * 128 + jj - 63 + cg * 16, kw = k0 - lane;
                    if (kw + 46 < 0 || kw >= 128)
                        continue;
                    tmem_ld16(trow + (uint32_t)(TM::E + t * 64 + cg * 16), x);
                    tc::tmem_ld_wait();
                    float *to = es + k0;
                    if (kw >= 0 && kw + 46 < 128) {
#pragma unroll
                        for (int c = 0; c < 16; c++)
                            to[c * 129] = __uint_as_float(x[c]);
                    } else {
#pragma unroll
                        for (int c = 0; c < 16; c++)
                            if ((unsigned)(k0 + c) < 128u)
                                to[c * 129] = __uint_as_float(x[c]);
                    }
                }
                bar_compute();
#pragma unroll
                for (int c = 0; c < 16; c++)
                    e[c] = es[c * 128 + jj];
                // P and dS take the place; the dE of the block before has been read
                if (g > 0)
                    meet(DE_FREE, g - 1, 74);
                else
                    bar_compute();
            } else {
                if (g > 0)
                    meet(DE_FREE, g - 1, 74);
#pragma unroll
                for (int c = 0; c < 16; c++)
                    e[c] = 0.0f;
            }
            uint32_t pk[8], dk[8];
            const int ib = cg * 16, jw = j0 + qd * 32; // first query and key of the warp
            if (jw > ib + 15 + M || jw + 31 <= ib + M - a.attn_len || ib >= T) { // nothing visible
#pragma unroll
                for (int c = 0; c < 8; c++)
                    pk[c] = dk[c] = 0u;
            } else {
                uint32_t z[16], d[16];
                tmem_ld16(trow + (uint32_t)(TM::S + cg * 16), z);
                tmem_ld16(trow + (uint32_t)(TM::D + cg * 16), d);
                tc::tmem_ld_wait();
                const bool all = jw + 31 <= ib + M && jw > ib + 15 + M - a.attn_len && ib + 16 <= T;
                float p[16], ds[16];
#pragma unroll
                for (int c4 = 0; c4 < 16; c4 += 4) { // lses holds log2 e times the log-sum-exp, behind it D / sqrt(dk)
                    const float4 l4 = *reinterpret_cast<const float4 *>(lses + c4), D4 = *reinterpret_cast<const float4 *>(lses + 64 + c4);
                    const float lv[4] = {l4.x, l4.y, l4.z, l4.w}, Dv[4] = {D4.x, D4.y, D4.z, D4.w};
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const int c = c4 + k;
                        p[c] = exp2_hw(fmaf(__uint_as_float(z[c]) + (br[-c] + e[c]), sc2, -lv[k]));
                        ds[c] = p[c] * fmaf(__uint_as_float(d[c]), a.inv_sqrt, -Dv[k]);
                    }
                }
                if (!all) {
                    const int d0 = ib + M - (j0 + jj); // query - key distance; visible iff 0 <= d < attn_len
#pragma unroll
                    for (int c = 0; c < 16; c++)
                        if ((unsigned)(d0 + c) >= (unsigned)a.attn_len || ib + c >= T)
                            p[c] = ds[c] = 0.0f;
                }
#pragma unroll
                for (int c = 0; c < 8; c++) {
                    pk[c] = fa::pack2(p[2 * c], p[2 * c + 1]);
                    dk[c] = fa::pack2(ds[2 * c], ds[2 * c + 1]);
                }
            }
            {
                unsigned char *pr = sm + SM::PS + jj * 128;
                *reinterpret_cast<uint4 *>(pr + (((2 * cg) ^ (jj & 7)) << 4)) = make_uint4(dk[0], dk[1], dk[2], dk[3]);
                *reinterpret_cast<uint4 *>(pr + (((2 * cg + 1) ^ (jj & 7)) << 4)) = make_uint4(dk[4], dk[5], dk[6], dk[7]);
                pr += 16384;
                *reinterpret_cast<uint4 *>(pr + (((2 * cg) ^ (jj & 7)) << 4)) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
                *reinterpret_cast<uint4 *>(pr + (((2 * cg + 1) ^ (jj & 7)) << 4)) = make_uint4(pk[4], pk[5], pk[6], pk[7]);
                unsigned char *er = sm + SM::DE + cg * 16 * 128;
#pragma unroll
                for (int c = 0; c < 16; c++) // column 16 cg + c back: a borrow passes through the free bits; row c & 7 of the swizzle
                    *reinterpret_cast<uint16_t *>(er + (((de0 - 2 * c) & ~0x1f80u) ^ ((c & 7) << 4)) + c * 128) =
                        (uint16_t)(dk[c >> 1] >> ((c & 1) * 16));
            }
            fence_async();
            signal(READY);
            if (last)
                if (lane == 0)
                    arrive(bar(ROWS_FREE + (n & 1)));
            auto following = wk;
            following.next();
            const bool hand = g + 1 < G && by_hand(following.kb);
            if (NB == 2 && hand)
                window_by_hand(following, g + 1);
            uint32_t x[NC];
            meet(P2_DONE, g, 75);
            auto drop_unless = [&](bool there) { // the same for the whole warp
                if (!there) {
#pragma unroll
                    for (int c = 0; c < NC; c++)
                        x[c] = 0u;
                }
            };
            if (dwr) {
                load_table(x);
                drop_unless(met(2 * kb + (qd >> 1)));
            }
            signal(TR_FREE);
            if (dwr)
                store_table(dwr, window0(kb), x, add);
            if constexpr (STAGED) { // into the places of V and K, which the producer sends out
                auto park = [&](unsigned char *tile) {
                    unsigned char *row = tile + jj * 128;
#pragma unroll
                    for (int k = 0; k < 2; k++) {
                        uint32_t v[4];
#pragma unroll
                        for (int w = 0; w < 4; w++)
                            v[w] = fa::pack2(__uint_as_float(x[8 * k + 2 * w]), __uint_as_float(x[8 * k + 2 * w + 1]));
                        *reinterpret_cast<uint4 *>(row + (((2 * cg + k) ^ (jj & 7)) << 4)) = make_uint4(v[0], v[1], v[2], v[3]);
                    }
                };
                load_nc(TM::V, x);
                drop_unless(seen(2 * kb + (qd >> 1)));
                park(sm + SM::V + s * SM::KT);
                load_nc(TM::K, x);
                drop_unless(seen(2 * kb + (qd >> 1)));
                park(sm + SM::K + s * SM::KT);
                fence_async();
                signal(FREE_KV + s);
            } else {
                bf16 *dkv = reinterpret_cast<bf16 *>(a.dkv) + (size_t)b * a.dkvp + h * DK + cg * NC;
                auto key_row = [&](int u, int off) {
                    const int j = j0 + qd * 32 + lane4 + u;
                    return j < L ? dkv + (size_t)j * B * a.dkvp + off : nullptr;
                };
                const bool there = seen(2 * kb + (qd >> 1));
                if (there) {
                    load_nc(TM::V, x);
                    store_bf16(x, [&](int u) { return key_row(u, HD); });
                    load_nc(TM::K, x);
                }
                if (DK == 128 && !last)
                    signal(DRAINED);
                if (there)
                    store_bf16(x, [&](int u) { return key_row(u, 0); });
            }
            if (last || (NB == 1 && hand))
                meet(DE_FREE, g, 78); // and everything else
            if (NB == 1 && hand)
                window_by_hand(following, g + 1);
            if (last) {
                load_nc(TM::Q, x); // rows 0-63; the others are the products of what lies behind dS and dE
                if (DK == 128)
                    signal(DRAINED);
                bf16 *dq = reinterpret_cast<bf16 *>(a.dq) + (size_t)b * a.dqp + h * DK + cg * NC;
                store_bf16(x, [&](int u) {
                    const int i = qd * 32 + lane4 + u;
                    return qd < 2 && i < T ? dq + (size_t)i * B * a.dqp : nullptr;
                });
                if (dwr) {
                    if (qd < 2) { // the upper 64 rows of the last window
                        load_table(x);
                        drop_unless(met(2 * kb + 2));
                        store_table(dwr, window0(kb) + 128, x, add);
                    }
                    if (fold) {
                        bar_compute();
                        if (window0(lo) <= 0)
                            for (int c = threadIdx.x; c < DK; c += CT)
                                dwr[c] = (add ? dwr[c] : 0.0f) + ((pad[c] + pad[DK + c]) + (pad[2 * DK + c] + pad[3 * DK + c]));
                        bar_compute();
                    }
                }
            }
            wk = following;
        }
        fence_before_sync();
    }
    // common exit: nobody touches tensor memory or the barriers after this
    __syncwarp();
    __syncthreads();
    if (*abort_s) { // a wait gave up: copies and products that are still in flight finish before the CTA retires, then there is no result
        for (int i = 0; i < 2000; i++)
            __nanosleep(500);
        if (threadIdx.x == 16 * 32)
            asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
        __syncthreads();
        auto fill = [&](void *p, int words) {
            for (int i = threadIdx.x; i < words; i += THREADS)
                reinterpret_cast<uint32_t *>(p)[i] = 0x7fff7fffu; // NaN as fp32 and as two bf16
        };
        auto of = wk;
        for (int n = 0; n < n_items; n++) {
            of.at(n);
            const int col = of.h * DK;
            for (int i = 0; i < T; i++)
                fill(reinterpret_cast<bf16 *>(a.dq) + ((size_t)i * B + of.b) * a.dqp + col, DK / 2);
            for (int j = 0; j < L; j++) {
                fill(reinterpret_cast<bf16 *>(a.dkv) + ((size_t)j * B + of.b) * a.dkvp + col, DK / 2);
                fill(reinterpret_cast<bf16 *>(a.dkv) + ((size_t)j * B + of.b) * a.dkvp + HD + col, DK / 2);
            }
            if (dwr0)
                fill(table_at(of.item, of.h), P * DK);
            if (a.dbr_part)
                fill(a.dbr_part + (size_t)of.item * L, L);
        }
    }
    if (warp == 17) {
        fence_after_sync();
        tc::tmem_dealloc(tmem, 512);
    }
}

// ---------------- host side ----------------

// Head sizes 64 and 128 whose two copies of b_r find room, where it is the faster kernel; other shapes stay with the warp-level one.
static bool takes(const AttnArgs &a)
{
    const bool room = a.dk == 64 ? Smem<64>::bytes(a.L) <= (size_t)SMEM_LIMIT : a.dk == 128 && Smem<128>::bytes(a.L) <= (size_t)SMEM_LIMIT;
    const fa::Blocks blk = fa::blocks_of(a.M, a.L, a.attn_len, 0, a.T);
    return room && attn::adjoint_by_128(a.dk, (long)a.B * a.H, a.T, blk.lo, blk.hi);
}
// Table gradients added up by the CTA, in its own slot, instead of a table for each stream that the reduction reads again: where it
// has four pairs or more.  The tables of 1024 pairs are 84 (320 rows) or 151 MB (576) a layer each way; steps of 20 layers 16196 -> 15999 us,
// of 12 10469 -> 10359.  With 256 pairs, two to a CTA, it cost 0.5 % (2261 -> 2272 us): the tables stay in L2 and the added rows are slower.
static bool sums(const AttnArgs &a) { return a.B * a.H >= 4 * 148; }
template <int DK> static int launch(const AttnArgs &a, cudaStream_t st)
{
    CUtensorMap q, o, kv, r, dkv;
    const cuuint64_t B = a.B, T = a.T, L = a.L, H = a.H, P = a.P, qp = a.qp, kvp = a.kvp, HD = H * DK;
    NNCU_TRY(fa::tile_map(a.q, {HD, B, T}, {qp * 2, B * qp * 2}, true, &q));
    NNCU_TRY(fa::tile_map(a.dout, {HD, B, T}, {HD * 2, B * HD * 2}, true, &o));
    NNCU_TRY(fa::tile_map(a.kv, {2 * HD, B, L}, {kvp * 2, B * kvp * 2}, true, &kv));
    r = kv;
    if (a.w_r16)
        NNCU_TRY(fa::tile_map(a.w_r16, {DK, P, H}, {DK * 2, P * DK * 2}, false, &r));
    const bool wide = fa::aligned_to(a.out, 16) && fa::aligned_to(a.w_r, 16) && fa::aligned_to(a.dq, 16) && fa::aligned_to(a.dkv, 16) &&
                      fa::aligned_to(a.dwr_part, 16);
    dkv = kv;
    if (wide && Smem<DK>::NB == 2)
        NNCU_TRY(fa::tile_map(a.dkv, {2 * HD, B, L}, {(cuuint64_t)a.dkvp * 2, B * a.dkvp * 2}, true, &dkv, KB));
    auto kernel = a.sum ? (wide ? attn_bwd_tc_kernel<DK, true, true> : attn_bwd_tc_kernel<DK, false, true>)
                        : (wide ? attn_bwd_tc_kernel<DK, true, false> : attn_bwd_tc_kernel<DK, false, false>);
    static DeviceOnce once[4];
    NNCU_TRY(smem_limit(once[2 * a.sum + wide], kernel, SMEM_LIMIT));
    launch_kind(EDGE_ATTN, kernel, dim3(ctas_of(a.B * a.H)), dim3(THREADS), Smem<DK>::bytes(a.L), st, a, q, o, kv, r, dkv);
    KERNEL_CHECK();
    return NNCU_OK;
}
static int backward(const AttnArgs &a, cudaStream_t st) { return a.dk == 64 ? launch<64>(a, st) : launch<128>(a, st); }

} // namespace fab

// How many tables attn_backward_any leaves in dwr_part for this shape when it may leave sums: the slots of the head with the
// most CTAs, or one a stream.  Operands as a model places them, 16-byte aligned.
static int attn_table_parts(const nncu_attn_shape *s, const AttnPitch *pt)
{
    AttnArgs a = attn_args(s, pt);
    float lse; // supported_bwd asks that there be one
    a.lse = &lse;
    if (!s->dtype_bf16 || !fa::supported_bwd(a) || !fa::fits(a.dk, a.L) || !fab::takes(a) || !fab::sums(a))
        return s->n_streams;
    int most = 0;
    for (int h = 0; h < a.H; h++)
        most = std::max(most, fab::slots_of(a.B, a.H, h));
    return most;
}
