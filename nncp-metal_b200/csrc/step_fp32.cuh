// step_fp32.cuh -- the forward pass of one time step of a small fp32 model in one launch.
//
// A decoder runs the model one symbol per stream at a time: for the fp32 models of the lower levels
// (fp32, post-LN, d_model up to 512 and like d_inner a multiple of 16, up to 56 streams) that was 37 launches of 3-5 us for 2 MFLOP a stream,
// 128 us a step (16 streams, 4 layers of 256; 62 us now, the serial decoder's 10 us included).  Streams do not meet in the forward pass, so a cluster of eight CTAs takes SP of them
// through the whole network by itself.  What bounds a step then is a chain: five exchanges of
// activations a layer (projection, attention, output projection, feed-forward up and down) with short
// dot products between them.
//   - Every product's output columns are dealt over the cluster in groups of eight, one warp a group.
//     Each warp has its own ring of weight pieces (8 rows x 256 columns, one TMA copy; a copy per row
//     cost the warp 1300 cycles a piece) and refills a slot once its results are on their way, so the
//     weights (8.4 MB a step at level 6, 1/8 per CTA) stream in beside the chain instead of in it.
//   - Results go to the other CTAs' shared memory by st.async, four columns a message, counted by a
//     barrier in the receiver; a cluster-wide barrier (1650 cycles with its release) stands only at
//     both ends of the launch.
//   - Norms are computed by every CTA for itself: cheaper than another exchange.
// Buffers need no second copy: whoever writes a buffer again has, through the exchanges between,
// heard from every CTA of the cluster since it last read it.  That takes a share for every CTA in two
// of the products (step_deal.h); models too narrow for it pay a cluster-wide barrier behind each norm.
//
// Same bits as the launches it replaces: a dot product is the four chains of gemm_simt.cuh, one thread
// each; attention, norm, softmax and tree rows are the device functions of those kernels.  Every value
// the backward pass reads is written where those launches write it.
#pragma once
#include "attention.cuh"
#include "coder.cuh"
#include "common.cuh"
#include "decoder.cuh"
#include "gemm_simt.cuh"
#include "gemm_tc.cuh"
#include "kernels.cuh"
#include "step_deal.h"

namespace stepf {

struct Layer {
    const float *b_q, *fb1, *fb2, *w_r, *b_r, *g1, *b1, *g2, *b2;
    float *x, *qkv, *o, *s1, *y, *hpre, *hact, *s2, *lse, *st1, *st2; // x: the layer's input rows (segment part of hcat)
    int attn_len;
};
struct Args {
    const Layer *layers;
    const CUtensorMap *maps; // the matrices in order: w_qkv, w_o, ff1, ff2 of each layer, then the output head
    const float *embed, *out_bias;
    const int32_t *ids;
    float *xlast, *probs, *dz;
    int *dz_fixed, *err_flag;
    uint16_t *trees; // [B][tree], NULL: not wanted
    int nl, D, H, dk, F, T, M, B, V, P, norm_mode, act, depth, slots; // norm_mode as residual_norm_kernel
    float emul, br_scale, inv_sqrt, scale;
};

constexpr int MAXD = 512;                    // row length that the norms' registers hold
constexpr int MAX_CLUSTERS = 14;             // clusters that are on the chip together (fifteen were, of 16)
constexpr int KC = 256, SLOT = 8 * KC;       // columns of a weight piece, floats of a ring slot
constexpr int MAX_SLOTS = 4;                 // ring slots per warp
constexpr int MAX_SMEM = 220 * 1024;         // of the plan

// weight pieces of a warp for N output columns, at most
__host__ __device__ inline int pieces_of(int N, int K) { return (per_cta(N) / 8 + 7) / 8 * ((K + KC - 1) / KC); }

// shared memory, in floats
struct Plan {
    int ring, layers, prods, list, cap, x, qkv, ob, tmp, y, ha, lg, S, kv, pair, ks, total;
};
__host__ __device__ inline Plan plan_of(int SP, int nl, int D, int H, int dk, int F, int L, int P, int V, int tree, int slots)
{
    Plan p;
    int at = 0;
    auto take = [&](int n) { int o = at; at += (n + 3) & ~3; return o; };
    const int HD = H * dk;
    p.ks = dk + 4;
    p.ring = take(8 * slots * SLOT); // first: its slots are 1024-byte aligned
    p.prods = take((4 * nl + 1) * 4);
    p.cap = nl * (pieces_of(3 * HD, D) + pieces_of(D, HD) + pieces_of(F, D) + pieces_of(D, F)) + pieces_of(V, D);
    p.list = take(8 * p.cap);
    p.layers = take(nl * (int)(sizeof(Layer) / 4));
    p.x = take(SP * D);
    p.qkv = take(SP * 3 * HD);
    p.ob = take(SP * HD);
    p.tmp = take(SP * D);
    p.y = take(SP * D);
    p.ha = take(SP * F);
    p.lg = take(V);
    p.S = take(2 * tree + 16);
    p.pair = L * p.ks + L * dk + P * p.ks + 3 * ((L + 3) & ~3) + dk; // K, V, table, b_r, both halves of the scores, the output
    p.kv = take((SP * H + CLUSTER - 1) / CLUSTER * p.pair);
    p.total = at + 256; // and the way to the first 1024-byte boundary
    return p;
}

__device__ __forceinline__ uint32_t mapa(uint32_t at, int rank)
{
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(at), "r"(rank));
    return r;
}
// four floats into a peer's shared memory, counted by its barrier
__device__ __forceinline__ void send4(uint32_t dst, uint32_t bar, int rank, float4 v)
{
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(mapa(dst, rank)),
                 "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"(mapa(bar, rank))
                 : "memory");
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }

// bounded; after the first wait that runs out every other one gives up at once
__device__ __forceinline__ void await(uint32_t bar, uint32_t parity, volatile int *abort_s, int *err_flag)
{
    const uint32_t tries = *abort_s ? 1u : (1u << 21);
    uint32_t ok = 0;
    for (uint32_t c = 0; c < tries && !ok; c++)
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok)
                     : "r"(bar), "r"(parity), "r"(1000u)
                     : "memory");
    if (!ok) {
        *abort_s = 1;
        atomicExch(err_flag, 61);
    }
}

// a matrix of the pass and the columns [n0, n0 + 8 groups) of its product that this CTA computes; turn: groups before it, mod 8
struct Product {
    int K, n0, groups, turn;
};
template <int SP>
__global__ void __launch_bounds__(256, 1) step_kernel(const __grid_constant__ Args a, int t)
{
    extern __shared__ __align__(1024) float smraw[];
    __shared__ float red[8];
    __shared__ __align__(8) uint64_t bars[6 + 8 * MAX_SLOTS]; // five exchanges of a layer, the logits, the rings
    __shared__ int abort_s;
    float *sm = smraw + (((1024u - (tc::smem_u32(smraw) & 1023u)) & 1023u) >> 2);
    uint32_t cr;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(cr));
    const int rank = (int)cr, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int D = a.D, H = a.H, dk = a.dk, HD = H * dk, F = a.F, B = a.B, M = a.M, V = a.V, P = a.P, L = a.M + a.T;
    const int b0 = (blockIdx.x / CLUSTER) * SP, nb = min(SP, B - b0), row0 = t * B + b0;
    const int treep = 1 << a.depth, slots = a.slots, np = 4 * a.nl + 1;
    const Plan pl = plan_of(SP, a.nl, D, H, dk, F, L, P, V, treep, slots);
    float *x = sm + pl.x, *qkv = sm + pl.qkv, *ob = sm + pl.ob, *tmp = sm + pl.tmp, *y = sm + pl.y, *ha = sm + pl.ha, *lg = sm + pl.lg,
          *S = sm + pl.S, *ring = sm + pl.ring + warp * slots * SLOT;
    const Layer *layers = reinterpret_cast<const Layer *>(sm + pl.layers);
    Product *prods = reinterpret_cast<Product *>(sm + pl.prods);
    enum { QKV, OB, T1, HA, T2, LG };
    const uint32_t bar0 = tc::smem_u32(bars), rbar = bar0 + 8 * (6 + warp * MAX_SLOTS), ring0 = tc::smem_u32(ring);
    const int npair = (nb * H + CLUSTER - 1 - rank) / CLUSTER; // (stream, head) pairs of this CTA: rank, rank + CLUSTER, ...
    const int V4 = (V + 3) & ~3;
    const bool ordered = exchanges_order_reuse(HD, F);
    auto expect = [&](int bar) { // bytes that an exchange brings to this CTA
        return (uint32_t)(bar == QKV ? npair * 3 * dk * 4 : bar == OB ? nb * HD * 4 : bar == HA ? nb * F * 4 : bar == LG ? (rank < nb ? V4 * 4 : 0) : nb * D * 4);
    };
    if (tid == 0) {
        abort_s = 0;
        for (int i = 0; i < 6 + 8 * MAX_SLOTS; i++)
            tc::mbar_init(bar0 + 8 * i, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        for (int i = 0; i < 6; i++)
            tc::mbar_expect_tx(bar0 + 8 * i, expect(i));
    }
    for (int i = tid; i < a.nl * (int)(sizeof(Layer) / 4); i += 256)
        reinterpret_cast<int *>(sm + pl.layers)[i] = reinterpret_cast<const int *>(a.layers)[i];
    if (tid == 32) {
        int turn = 0;
        for (int i = 0; i < np; i++) {
            const int j = i & 3, N = i == np - 1 ? V : (j == 0 ? 3 * HD : (j == 2 ? F : D));
            Product p;
            p.K = i == np - 1 ? D : (j == 1 ? HD : (j == 3 ? F : D));
            p.n0 = deal_from(N, rank);
            p.groups = (deal_from(N, rank + 1) - p.n0 + 7) >> 3;
            p.turn = turn;
            turn = (turn + p.groups) & 7;
            prods[i] = p;
        }
    }
    cluster_arrive(); // every CTA of the cluster has its barriers up before the first message
    __syncthreads();

    // This warp's stream of weight pieces: the groups of eight columns are dealt round robin over the warps
    // through all products, a group's pieces follow one another.  An entry of the list is (product, row / 8, piece).
    uint32_t *list = reinterpret_cast<uint32_t *>(sm + pl.list) + warp * pl.cap;
    int n_list = 0;
    for (int i = 0; i < np; i++) {
        const Product p = prods[i];
        const int pieces = (p.K + KC - 1) / KC;
        for (int g = (warp - p.turn) & 7; g < p.groups; g += 8)
            for (int k = 0; k < pieces; k++, n_list++)
                if (lane == 0)
                    list[n_list] = (uint32_t)(i | ((p.n0 >> 3) + g) << 8 | k << 22);
    }
    __syncwarp();
    int at_list = 0, aslot = 0, ahead = 0; // entries issued, slot of the next; pieces issued and not read yet
    uint32_t next = n_list ? list[0] : 0;
    auto issue = [&]() {
        if (at_list >= n_list)
            return;
        if (lane == 0) {
            tc::mbar_expect_tx(rbar + 8 * aslot, SLOT * 4);
            asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(
                             ring0 + aslot * SLOT * 4),
                         "l"(reinterpret_cast<uint64_t>(a.maps + (next & 255u))), "r"(rbar + 8 * aslot), "r"(0), "r"((next >> 8 & 0x3fffu) * 8),
                         "r"((next >> 22) * (KC / 32))
                         : "memory");
        }
        ahead++;
        aslot = aslot + 1 == slots ? 0 : aslot + 1;
        if (++at_list < n_list)
            next = list[at_list];
    };
    // The weights may be read ahead of the kernel before: a launch that overlaps it is only made behind a
    // decoder step of the same call, which writes none.
    for (int i = 0; i < slots; i++)
        issue();
    cluster_wait();
    pdl_wait();
    pdl_trigger();
    if (blockIdx.x == 0 && tid == 0)
        *a.dz_fixed = 0;
    int cslot = 0;
    uint32_t cphase = 0;
    // The groups of product i that this warp has.  Chain q of a column is a quarter of the warp's (lane / 8), the
    // column of eight is lane % 8; a row of a piece is cut into 128-byte lines, line k / 32 of all eight rows
    // together, swizzled (16-byte chunk c of row r sits at c ^ r): the eight lanes read eight bank groups.
    // f(first column of this lane's four, their biases, this lane's sums of the streams)
    constexpr int U = 2 * SP; // lanes as senders: unit lane % U is (stream ur, half uh of the group's columns),
    const int ur = (lane % U) >> 1, uh = (lane % U) & 1, peer0 = lane / U; // a unit has the peers lane / U, + 32 / U, ...
    const int q = lane >> 3, r8 = lane & 7;
    uint32_t off[4];
#pragma unroll
    for (int j = 0; j < 4; j++)
        off[j] = (uint32_t)((q >> 1) * 1024 + r8 * 128 + ((((q & 1) * 4 + j) ^ r8) << 4));
    auto product = [&](int i, const float *xs, const float *bias, int bias_n, auto f) {
        const Product p = prods[i];
        for (int g = (warp - p.turn) & 7; g < p.groups; g += 8) {
            const int n = p.n0 + g * 8 + uh * 4;
            float4 bv = make_float4(0.f, 0.f, 0.f, 0.f);
            if (bias && n < bias_n)
                bv = __ldg(reinterpret_cast<const float4 *>(bias + n));
            float acc[SP];
#pragma unroll
            for (int r = 0; r < SP; r++)
                acc[r] = 0.0f;
            int left = (p.K + KC - 1) / KC; // pieces of this group to come
            for (int k0 = 0; k0 < p.K; k0 += KC) {
                await(rbar + 8 * cslot, cphase, &abort_s, a.err_flag);
                const uint32_t w0 = ring0 + cslot * SLOT * 4;
                const int ns = min(KC, p.K - k0) >> 4;
                const float *xk = xs + k0 + q * 16;
                auto slice = [&](int m) { // slice q + 4 m of the piece
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        float4 w;
                        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                                     : "=f"(w.x), "=f"(w.y), "=f"(w.z), "=f"(w.w)
                                     : "r"(w0 + m * 2048 + off[j]));
#pragma unroll
                        for (int r = 0; r < SP; r++) {
                            const float4 v = *reinterpret_cast<const float4 *>(xk + r * p.K + m * 64 + j * 4);
                            acc[r] = fmaf(v.x, w.x, acc[r]);
                            acc[r] = fmaf(v.y, w.y, acc[r]);
                            acc[r] = fmaf(v.z, w.z, acc[r]);
                            acc[r] = fmaf(v.w, w.w, acc[r]);
                        }
                    }
                };
                if (ns == KC / 16) {
#pragma unroll
                    for (int m = 0; m < KC / 64; m++)
                        slice(m);
                } else {
                    for (int m = 0; q + 4 * m < ns; m++)
                        slice(m);
                    __syncwarp();
                }
                ahead--;
                left--;
                if (++cslot == slots) {
                    cslot = 0;
                    cphase ^= 1;
                }
                if (left > ahead) { // the group's next piece is not on its way yet
                    __syncwarp();
                    issue();
                }
            }
#pragma unroll
            for (int r = 0; r < SP; r++) {
                acc[r] = __fadd_rn(acc[r], __shfl_xor_sync(0xffffffffu, acc[r], 8));
                acc[r] = __fadd_rn(acc[r], __shfl_xor_sync(0xffffffffu, acc[r], 16));
            }
            f(n, bv, acc);
            while (ahead < slots && at_list < n_list)
                issue();
        }
    };
    auto gather = [&](const float (&acc)[SP]) {
        float4 v;
        float *e = &v.x;
#pragma unroll
        for (int r = 0; r < SP; r++)
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float s = __shfl_sync(0xffffffffu, acc[r], uh * 4 + j);
                if (r == 0 || r == ur)
                    e[j] = s;
            }
        return v;
    };
    auto add4 = [](float4 v, float4 b) { return make_float4(v.x + b.x, v.y + b.y, v.z + b.z, v.w + b.w); };
    auto to_all = [&](float *dst, int pitch, int bar, int n, float4 v, int N) {
        if (ur < nb && n < N)
#pragma unroll
            for (int c = peer0; c < CLUSTER; c += 32 / U)
                send4(tc::smem_u32(dst + ur * pitch + n), bar0 + 8 * bar, c, v);
    };
    auto landed = [&](int bar, int l) {
        await(bar0 + 8 * bar, (uint32_t)(l & 1), &abort_s, a.err_flag);
        if (tid == 0 && l + 1 < a.nl)
            tc::mbar_expect_tx(bar0 + 8 * bar, expect(bar));
    };
    // keys, values of the past and the position table of this CTA's pairs; a warp takes 32 / cpr rows at a time
    const int cpr = dk / 4, rpw = 32 / cpr, sub = lane / cpr, ce = (lane - sub * cpr) * 4;
    auto stage = [&](int l) {
        const Layer &ly = layers[l];
        int jlo, jhi;
        attn_key_range(L, M, ly.attn_len, t, jlo, jhi);
        for (int p = 0; p < npair; p++) {
            const int pair = rank + p * CLUSTER, r = pair / H, h = pair - r * H, b = b0 + r;
            float *Ks = sm + pl.kv + p * pl.pair, *Vs = Ks + L * pl.ks, *Rs = Vs + L * dk, *br = Rs + P * pl.ks;
            if (sub < rpw) {
                for (int j = jlo + warp * rpw + sub; j < jhi; j += 8 * rpw) { // all but the key of this step
                    const float *src = ly.qkv + ((size_t)j * B + b) * 3 * HD + HD + h * dk + ce;
                    simt::cp16(Ks + j * pl.ks + ce, src, 4);
                    simt::cp16(Vs + j * dk + ce, src + HD, 4);
                }
                if (ly.w_r)
                    for (int j = warp * rpw + sub; j < P; j += 8 * rpw)
                        simt::cp16(Rs + j * pl.ks + ce, ly.w_r + ((size_t)h * P + j) * dk + ce, 4);
            }
            for (int j = tid; j < L; j += 256)
                simt::cp4(br + j, ly.b_r + (size_t)h * L + j, 1);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    stage(0);
    // attention: 2^alog warps a pair; this warp's first pair
    const int alog = npair <= 1 ? 3 : (npair == 2 ? 2 : (npair <= 4 ? 1 : 0)), aw = 1 << alog, w = warp & (aw - 1);
    const int ar0 = (rank + (warp >> alog) * CLUSTER) / H, ah0 = rank + (warp >> alog) * CLUSTER - ar0 * H;

    // embedding rows (rows past the last stream stay zero)
    for (int i = tid; i < SP * D; i += 256) {
        const int r = i / D, c = i - r * D;
        float v = 0.0f;
        if (r < nb) {
            int id = a.ids[row0 + r];
            id = id < 0 ? 0 : (id >= V ? V - 1 : id);
            v = __fmul_rn(a.embed[(size_t)id * D + c], a.emul);
            if (rank == 0)
                layers[0].x[(size_t)(row0 + r) * D + c] = v;
        }
        x[i] = v;
    }
    __syncthreads();

    for (int l = 0; l < a.nl; l++) {
        const Layer &ly = layers[l];
        product(4 * l, x, ly.b_q, HD, [&](int n, float4 bv, const float(&acc)[SP]) {
            const int h = (n % HD) / dk;
            float4 v = gather(acc);
            if (ly.b_q && n < HD)
                v = add4(v, bv);
            if (ur < nb && n < 3 * HD) {
                if (peer0 == 0)
                    send4(tc::smem_u32(qkv + ur * 3 * HD + n), bar0 + 8 * QKV, (ur * H + h) % CLUSTER, v); // the CTA that has the pair
                else if (peer0 == 1)
                    *reinterpret_cast<float4 *>(ly.qkv + ((size_t)(M + t) * B + b0 + ur) * 3 * HD + n) = v;
            }
        });
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        if (npair)
            landed(QKV, l);
        __syncthreads();
        // Attention, aw warps a pair (attn_row's operations): the two dot products of 32 keys are two tasks, the
        // first warp takes the softmax, 32 output columns are a warp's.
        for (int p0 = 0; p0 < npair; p0 += 8 >> alog) {
            const int p = p0 + (warp >> alog), pair = rank + p * CLUSTER, r = p0 ? pair / H : ar0, h = p0 ? pair - r * H : ah0, b = b0 + r;
            const bool on = p < npair;
            float *Ks = sm + pl.kv + p * pl.pair, *Vs = Ks + L * pl.ks, *Rs = Vs + L * dk, *br = Rs + P * pl.ks, *ps = br + ((L + 3) & ~3),
                  *pz = ps + ((L + 3) & ~3), *os = pz + ((L + 3) & ~3);
            const float *qf = qkv + r * 3 * HD + h * dk, *kf = qf + HD, *vf = kf + HD;
            int jlo, jhi;
            attn_key_range(L, M, ly.attn_len, t, jlo, jhi);
            if (on)
                for (int i = w; i < 2 * ((jhi - jlo + 32) / 32); i += aw) {
                    const int j = jlo + (i >> 1) * 32 + lane;
                    if (j > jhi)
                        continue;
                    if (i & 1) {
                        const int rr = j + (a.T - 1) - t, pi = max(rr - (L - P), 0);
                        float z = __fmul_rn(a.br_scale, br[rr]);
                        if (ly.w_r)
                            z = __fadd_rn(z, dot_q<float>(qf, Rs + pi * pl.ks, dk));
                        pz[j] = z;
                    } else {
                        ps[j] = dot_q<float>(qf, j == jhi ? kf : Ks + j * pl.ks, dk);
                    }
                }
            __syncthreads();
            float lse = 0.0f;
            if (on && w == 0) {
                float mx = -INFINITY;
                for (int j = jlo + lane; j <= jhi; j += 32) {
                    const float s = __fmul_rn(__fadd_rn(ps[j], pz[j]), a.inv_sqrt);
                    ps[j] = s;
                    mx = fmaxf(mx, s);
                }
                mx = warp_max(mx);
                float sum = 0.0f;
                for (int j = jlo + lane; j <= jhi; j += 32) {
                    const float e = expf(__fsub_rn(ps[j], mx));
                    ps[j] = e;
                    sum = __fadd_rn(sum, e);
                }
                sum = warp_sum(sum);
                const float rs = __fdiv_rn(1.0f, sum);
                for (int j = jlo + lane; j <= jhi; j += 32)
                    ps[j] = __fmul_rn(ps[j], rs);
                lse = __fadd_rn(mx, logf(sum));
            }
            __syncthreads();
            if (on)
                for (int e0 = w * 32; e0 < dk; e0 += aw * 32) {
                    const int e = e0 + lane, n4 = min(8, (dk - e0) / 4);
                    if (e < dk) {
                        float acc = 0.0f;
#pragma unroll 16
                        for (int j = jlo; j < jhi; j++)
                            acc = fmaf(ps[j], Vs[j * dk + e], acc);
                        os[e] = fmaf(ps[jhi], vf[e], acc);
                    }
                    __syncwarp();
                    for (int i = lane; i < n4 * CLUSTER; i += 32) {
                        const int c = n4 == 8 ? i >> 3 : i / n4, at = e0 + (i - c * n4) * 4;
                        const float4 v = *reinterpret_cast<const float4 *>(os + at);
                        send4(tc::smem_u32(ob + r * HD + h * dk + at), bar0 + 8 * OB, c, v);
                        if (c == 0)
                            *reinterpret_cast<float4 *>(ly.o + (size_t)(row0 + r) * HD + h * dk + at) = v;
                    }
                }
            if (on && w == 0 && lane == 0)
                ly.lse[((size_t)b * H + h) * a.T + t] = lse;
        }
        // s = tmp + in, out = norm(s): every CTA for itself, CTA 0 keeps what the backward pass reads
        auto norm = [&](int bar, const float *in, float *out, const float *g, const float *b, float *s_out, float *y_out, float *stats) {
            float gv[4][4], bv[4][4]; // on their way before the wait
            if (warp < nb) {
                vec_load_f32<4, 4>(g, lane, D, gv);
                vec_load_f32<4, 4>(b, lane, D, bv);
            }
            landed(bar, l);
            for (int r = warp; r < nb; r += 8) {
                float v[4][4];
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    const int i = c * 128 + lane * 4;
                    float4 p = make_float4(0.f, 0.f, 0.f, 0.f), q = p;
                    if (i < D) {
                        p = *reinterpret_cast<const float4 *>(tmp + r * D + i);
                        q = *reinterpret_cast<const float4 *>(in + r * D + i);
                    }
                    v[c][0] = __fadd_rn(p.x, q.x); v[c][1] = __fadd_rn(p.y, q.y);
                    v[c][2] = __fadd_rn(p.z, q.z); v[c][3] = __fadd_rn(p.w, q.w);
                }
                const size_t at = (size_t)(row0 + r) * D;
                if (rank == 0)
                    row_store<float, 4, 4>(s_out + at, lane, D, v);
                norm_row<4, 4>(v, gv, bv, lane, D, a.norm_mode, rank == 0 ? stats + 2 * (row0 + r) : nullptr);
                if (rank == 0)
                    row_store<float, 4, 4>(y_out + at, lane, D, v);
                row_store<float, 4, 4>(out + r * D, lane, D, v);
            }
            __syncthreads();
            if (!ordered) {
                cluster_arrive();
                cluster_wait();
            }
        };
        landed(OB, l);
        product(4 * l + 1, ob, nullptr, 0, [&](int n, float4, const float(&acc)[SP]) { to_all(tmp, D, T1, n, gather(acc), D); });
        if (l + 1 < a.nl)
            stage(l + 1); // every CTA has finished this layer's attention
        norm(T1, x, y, ly.g1, ly.b1, ly.s1, ly.y, ly.st1);
        product(4 * l + 2, y, ly.fb1, F, [&](int n, float4 bv, const float(&acc)[SP]) {
            float4 hp = gather(acc), v;
            if (ly.fb1)
                hp = add4(hp, bv);
            const float *pp = &hp.x;
            float *vp = &v.x;
#pragma unroll
            for (int e = 0; e < 4; e++)
                vp[e] = a.act == NNCU_FF_RELU ? (pp[e] > 0.0f ? pp[e] : 0.0f) : gelu_f(pp[e]);
            to_all(ha, F, HA, n, v, F);
            if (ur < nb && n < F && peer0 < 2)
                *reinterpret_cast<float4 *>((peer0 ? ly.hact : ly.hpre) + (size_t)(row0 + ur) * F + n) = peer0 ? v : hp;
        });
        landed(HA, l);
        product(4 * l + 3, ha, ly.fb2, D, [&](int n, float4 bv, const float(&acc)[SP]) {
            float4 v = gather(acc);
            if (ly.fb2)
                v = add4(v, bv);
            to_all(tmp, D, T2, n, v, D);
        });
        norm(T2, y, x, ly.g2, ly.b2, ly.s2, l + 1 < a.nl ? layers[l + 1].x : a.xlast, ly.st2);
    }
    // output head: row r's logits to the CTA that finishes the row
    static_assert(SP <= CLUSTER, "a cluster has a CTA for every row");
    product(np - 1, x, a.out_bias, V4, [&](int n, float4 bv, const float(&acc)[SP]) { // the biases' slot is padded beyond the last symbol
        float4 v = gather(acc);
        if (a.out_bias)
            v = add4(v, bv);
        if (ur < nb && n < V4 && peer0 == 0)
            send4(tc::smem_u32(lg + n), bar0 + 8 * LG, ur, v);
    });
    cluster_arrive();
    if (rank < nb) {
        await(bar0 + 8 * LG, 0, &abort_s, a.err_flag);
        const size_t pr = (size_t)(row0 + rank) * V;
        if (softmax_by_fours(V)) {
            softmax_row_by_fours(lg, V, a.dz + pr, a.scale, red);
            __syncthreads(); // the copy below reads it column by column
        } else {
            softmax_row(lg, V, a.dz + pr, a.scale, red);
        }
        for (int i = tid; i < V; i += 256)
            a.probs[pr + i] = lg[i];
        __syncthreads();
        if (a.trees) {
            uint16_t *out = a.trees + (size_t)(b0 + rank) * treep;
            if (treep == V)
                coder_tree_row(S, lg, out, V);
            else
                coder_tree_row_any(S, lg, out, V, treep);
        }
    }
    cluster_wait(); // nobody leaves while a peer may still send to it
    for (; ahead > 0; ahead--) { // only after a wait that ran out: copies in flight land in this CTA's shared memory
        await(rbar + 8 * cslot, cphase, &abort_s, a.err_flag);
        if (++cslot == slots) {
            cslot = 0;
            cphase ^= 1;
        }
    }
}

// the tensor map of an N x K matrix for pieces of 8 rows x 256 columns, in lines of 32 columns
inline int piece_map(const float *W, int N, int K, CUtensorMap *out)
{
    tc::EncodeTiledFn fn = tc::encode_fn();
    if (!fn)
        return nncu_fail(NNCU_ERR_CUDA, "cuTensorMapEncodeTiled is not available");
    cuuint64_t dims[3] = {32, (cuuint64_t)N, (cuuint64_t)((K + 31) / 32)};
    cuuint64_t strides[2] = {(cuuint64_t)K * 4, 128};
    cuuint32_t box[3] = {32, 8, KC / 32}, estr[3] = {1, 1, 1};
    CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float *>(W), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS)
        return nncu_fail(NNCU_ERR_CUDA, "cuTensorMapEncodeTiled failed: %d (%d x %d in lines of 32)", (int)r, N, K);
    return NNCU_OK;
}

// ring slots per warp that fit beside the rest (0: the model does not fit)
inline int ring_slots(int sp, int nl, int D, int H, int dk, int F, int L, int P, int V, int tree)
{
    for (int s = MAX_SLOTS; s >= 2; s--)
        if (plan_of(sp, nl, D, H, dk, F, L, P, V, tree, s).total * 4 <= MAX_SMEM)
            return s;
    return 0;
}

template <int SP> static int launch_sp(cudaStream_t st, const Args &a, int t, bool chained)
{
    const Plan pl = plan_of(SP, a.nl, a.D, a.H, a.dk, a.F, a.M + a.T, a.P, a.V, 1 << a.depth, a.slots);
    static DeviceOnce once;
    NNCU_TRY(smem_limit(once, step_kernel<SP>, MAX_SMEM));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(CLUSTER * ceil_div(a.B, SP)));
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = (size_t)pl.total * 4;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CLUSTER;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = chained ? 2 : 1;
    CUDA_TRY(cudaLaunchKernelEx(&cfg, step_kernel<SP>, a, t));
    KERNEL_CHECK();
    return NNCU_OK;
}
// chained: the launch may begin while the kernel before it, a decoder step of the same model, is running
static int launch(cudaStream_t st, const Args &a, int t, int sp, bool chained)
{
    return sp == 1 ? launch_sp<1>(st, a, t, chained) : (sp == 2 ? launch_sp<2>(st, a, t, chained) : launch_sp<4>(st, a, t, chained));
}

} // namespace stepf
