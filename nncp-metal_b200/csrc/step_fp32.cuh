// step_fp32.cuh -- the forward pass of one time step of a small fp32 model in one launch.
//
// A decoder runs the model one symbol per stream at a time: for the fp32 models of the lower levels
// (2-4 layers, d_model 64-512, up to 64 streams) that was 37 launches of 3-5 us for 2 MFLOP a stream,
// 128 us a step.  Streams do not meet in the forward pass, so a cluster of eight CTAs takes SP of them
// through the whole network by itself.  What bounds a step then is a chain: five exchanges of
// activations a layer (projection, attention, output projection, feed-forward up and down) with short
// dot products between them.
//   - Every product's output columns are dealt over the cluster in groups of eight, one warp a group.
//     Each warp has its own ring of weight pieces (8 rows x 256 columns, bulk copies) and refills a
//     slot as soon as it has read it, so the weights (8.4 MB a step at level 6, 1/8 per CTA) stream in
//     beside the chain instead of in it.
//   - Results go to the other CTAs' shared memory by st.async, four columns a message, counted by a
//     barrier in the receiver; a cluster-wide barrier (1650 cycles with its release) stands only at
//     both ends of the launch.
//   - Norms are computed by every CTA for itself: cheaper than another exchange.
// Buffers need no second copy: whoever writes a buffer again has, through the exchanges between,
// heard from every CTA of the cluster since it last read it.
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

namespace stepf {

struct Layer {
    const float *w_qkv, *w_o, *ff1, *ff2, *b_q, *fb1, *fb2, *w_r, *b_r, *g1, *b1, *g2, *b2;
    float *x, *qkv, *o, *s1, *y, *hpre, *hact, *s2, *lse, *st1, *st2; // x: the layer's input rows (segment part of hcat)
    int attn_len;
};
struct Args {
    const Layer *layers;
    const float *embed, *w_out, *out_bias;
    const int32_t *ids;
    float *xlast, *probs, *dz;
    int *dz_fixed, *err_flag;
    uint16_t *trees; // [B][tree], NULL: not wanted
    int nl, D, H, dk, F, T, M, B, V, P, norm_mode, act, depth, slots; // norm_mode as residual_norm_kernel
    float emul, br_scale, inv_sqrt, scale;
};

constexpr int CLUSTER = 8;                   // CTAs that share a group of streams
constexpr int MAXD = 512;                    // row length that the norms' registers hold
constexpr int MAX_CLUSTERS = 14;             // clusters that are on the chip together (fifteen were, of 16)
constexpr int KC = 256, PITCH = KC + 4;      // columns of a weight piece and its row pitch: the eight rows that a
                                             // quarter of a warp reads together fall on different bank groups
constexpr int SLOT = 8 * PITCH;              // floats of a ring slot
constexpr int MAX_SLOTS = 4;                 // ring slots per warp

// shared memory, in floats
struct Plan {
    int layers, x, qkv, ob, tmp, y, ha, lg, S, kv, ring, pair, ks, total;
};
__host__ __device__ inline Plan plan_of(int SP, int nl, int D, int H, int dk, int F, int L, int P, int V, int tree, int slots)
{
    Plan p;
    int at = 0;
    auto take = [&](int n) { int o = at; at += (n + 3) & ~3; return o; };
    const int HD = H * dk;
    p.ks = dk + 4;
    p.layers = take(nl * (int)(sizeof(Layer) / 4));
    p.x = take(SP * D);
    p.qkv = take(SP * 3 * HD);
    p.ob = take(SP * HD);
    p.tmp = take(SP * D);
    p.y = take(SP * D);
    p.ha = take(SP * F);
    p.lg = take(V);
    p.S = take(2 * tree + 16);
    p.pair = L * p.ks + L * dk + P * p.ks + ((L + 3) & ~3) + ((dk + L + 3) & ~3);
    p.kv = take((SP * H + CLUSTER - 1) / CLUSTER * p.pair);
    p.ring = take(8 * slots * SLOT);
    p.total = at;
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
        atomicExch(err_flag, 51);
    }
}

// the products of a pass in order: 0-3 of each layer, then the output head
struct Product {
    const float *W;
    int K, n0, n1; // output columns [n0, n1) of this CTA, n0 a multiple of eight
};
// columns of an N-wide output per CTA, whole groups of eight
__device__ __forceinline__ int per_cta(int N) { return ((N + CLUSTER - 1) / CLUSTER + 7) & ~7; }

// a warp's place in its stream of weight pieces
struct Cursor {
    int l, j, g, k, turn; // layer, product, group of eight columns, first column of the piece, groups before this product mod 8
};

template <int SP>
__global__ void __launch_bounds__(256, 1) step_kernel(const __grid_constant__ Args a, int t)
{
    extern __shared__ __align__(128) float sm[];
    __shared__ float red[8];
    __shared__ __align__(8) uint64_t bars[6 + 8 * MAX_SLOTS]; // five exchanges of a layer, the logits, the rings
    __shared__ int abort_s;
    uint32_t cr;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(cr));
    const int rank = (int)cr, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int D = a.D, H = a.H, dk = a.dk, HD = H * dk, F = a.F, B = a.B, M = a.M, V = a.V, P = a.P, L = a.M + a.T;
    const int b0 = (blockIdx.x / CLUSTER) * SP, nb = min(SP, B - b0), row0 = t * B + b0;
    const int treep = 1 << a.depth, slots = a.slots;
    const Plan pl = plan_of(SP, a.nl, D, H, dk, F, L, P, V, treep, slots);
    float *x = sm + pl.x, *qkv = sm + pl.qkv, *ob = sm + pl.ob, *tmp = sm + pl.tmp, *y = sm + pl.y, *ha = sm + pl.ha, *lg = sm + pl.lg,
          *S = sm + pl.S, *ring = sm + pl.ring + warp * slots * SLOT;
    const Layer *layers = reinterpret_cast<const Layer *>(sm + pl.layers);
    enum { QKV, OB, T1, HA, T2, LG };
    const uint32_t bar0 = tc::smem_u32(bars), rbar = bar0 + 8 * (6 + warp * MAX_SLOTS);
    const int npair = (nb * H + CLUSTER - 1 - rank) / CLUSTER; // (stream, head) pairs of this CTA: rank, rank + CLUSTER, ...
    const int V4 = (V + 3) & ~3;
    uint32_t expect[6] = {(uint32_t)(npair * 3 * dk * 4), (uint32_t)(nb * HD * 4), (uint32_t)(nb * D * 4), (uint32_t)(nb * F * 4),
                          (uint32_t)(nb * D * 4), rank < nb ? (uint32_t)(V4 * 4) : 0u};
    if (tid == 0) {
        abort_s = 0;
        for (int i = 0; i < 6 + 8 * MAX_SLOTS; i++)
            tc::mbar_init(bar0 + 8 * i, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
#pragma unroll
        for (int i = 0; i < 6; i++)
            tc::mbar_expect_tx(bar0 + 8 * i, expect[i]);
    }
    for (int i = tid; i < a.nl * (int)(sizeof(Layer) / 4); i += 256)
        reinterpret_cast<int *>(sm + pl.layers)[i] = reinterpret_cast<const int *>(a.layers)[i];
    __syncthreads();

    auto product_of = [&](int l, int j) {
        Product p;
        int N = D;
        p.K = D;
        if (l == a.nl) {
            p.W = a.w_out;
            N = V;
        } else if (j == 0) {
            p.W = layers[l].w_qkv;
            N = 3 * HD;
        } else if (j == 1) {
            p.W = layers[l].w_o;
            p.K = HD;
        } else if (j == 2) {
            p.W = layers[l].ff1;
            N = F;
        } else {
            p.W = layers[l].ff2;
            p.K = F;
        }
        const int per = per_cta(N);
        p.n0 = min(N, rank * per);
        p.n1 = min(N, p.n0 + per);
        return p;
    };
    auto groups = [](const Product &p) { return (p.n1 - p.n0 + 7) >> 3; };
    // the first product at or behind the cursor's in which this warp has a group (groups are dealt round robin
    // over the warps through all products)
    auto settle = [&](Cursor &c) {
        while (c.l <= a.nl) {
            const Product p = product_of(c.l, c.j);
            if (c.g < groups(p))
                return;
            c.turn = (c.turn + groups(p)) & 7;
            c.g = (warp - c.turn) & 7;
            c.k = 0;
            if (c.l == a.nl || ++c.j == 4) {
                c.j = 0;
                c.l++;
            }
        }
    };
    Cursor ahead = {0, 0, warp, 0, 0};
    settle(ahead);
    int issued = 0, used = 0; // pieces
    auto issue = [&]() { // the next piece of this warp's stream into its slot
        if (ahead.l > a.nl)
            return;
        const Product p = product_of(ahead.l, ahead.j);
        const int n = p.n0 + ahead.g * 8, rows = min(8, p.n1 - n), kn = min(KC, p.K - ahead.k), slot = issued % slots;
        const uint32_t bar = rbar + 8 * slot;
        if (lane == 0)
            tc::mbar_expect_tx(bar, (uint32_t)(rows * kn * 4));
        __syncwarp();
        if (lane < rows)
            dec::bulk_load(tc::smem_u32(ring + slot * SLOT + lane * PITCH), p.W + (size_t)(n + lane) * p.K + ahead.k, (uint32_t)(kn * 4), bar);
        issued++;
        ahead.k += KC;
        if (ahead.k >= p.K) {
            ahead.k = 0;
            ahead.g += 8;
            settle(ahead);
        }
    };
    // The weights may be read ahead of the kernel before: a launch that overlaps it is only made behind a
    // decoder step of the same call, which writes none.
    for (int i = 0; i < slots; i++)
        issue();
    pdl_wait();
    pdl_trigger_late();
    if (blockIdx.x == 0 && tid == 0)
        *a.dz_fixed = 0;
    int turn = 0;
    // the groups of product p that this warp has: four chains over the lanes' quarters, a column per lane of
    // eight; f(first column, this lane's sums of the streams)
    auto product = [&](const Product &p, const float *xs, auto f) {
        for (int g = (warp - turn) & 7; g < groups(p); g += 8) {
            float acc[SP];
#pragma unroll
            for (int r = 0; r < SP; r++)
                acc[r] = 0.0f;
            for (int k0 = 0; k0 < p.K; k0 += KC) {
                const int slot = used % slots, ns = min(KC, p.K - k0) >> 4;
                await(rbar + 8 * slot, (uint32_t)((used / slots) & 1), &abort_s, a.err_flag);
                const float *wr = ring + slot * SLOT + (lane & 7) * PITCH;
#pragma unroll 4
                for (int s = lane >> 3; s < ns; s += 4) {
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const float4 w = *reinterpret_cast<const float4 *>(wr + s * 16 + j * 4);
#pragma unroll
                        for (int r = 0; r < SP; r++) {
                            const float4 v = *reinterpret_cast<const float4 *>(xs + r * p.K + k0 + s * 16 + j * 4);
                            acc[r] = fmaf(v.x, w.x, acc[r]);
                            acc[r] = fmaf(v.y, w.y, acc[r]);
                            acc[r] = fmaf(v.z, w.z, acc[r]);
                            acc[r] = fmaf(v.w, w.w, acc[r]);
                        }
                    }
                }
                used++;
                __syncwarp();
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                issue();
            }
#pragma unroll
            for (int r = 0; r < SP; r++) {
                acc[r] = __fadd_rn(acc[r], __shfl_xor_sync(0xffffffffu, acc[r], 8));
                acc[r] = __fadd_rn(acc[r], __shfl_xor_sync(0xffffffffu, acc[r], 16));
            }
            f(p.n0 + g * 8, acc);
        }
        turn = (turn + groups(p)) & 7;
    };
    // Lanes as senders: unit u = lane % (2 SP) is (stream r, half h of the group's columns); a unit has the peers
    // lane / (2 SP), + 16 / SP, ...
    constexpr int U = 2 * SP;
    const int ur = (lane % U) >> 1, uh = (lane % U) & 1, peer0 = lane / U;
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
    auto load4g = [](const float *p, int n) { return p ? __ldg(reinterpret_cast<const float4 *>(p + n)) : make_float4(0.f, 0.f, 0.f, 0.f); };
    auto add4 = [](float4 v, float4 b) { return make_float4(v.x + b.x, v.y + b.y, v.z + b.z, v.w + b.w); };
    auto to_all = [&](float *dst, int pitch, int bar, int n, float4 v, int N) {
        if (ur < nb && n < N)
            for (int c = peer0; c < CLUSTER; c += 32 / U)
                send4(tc::smem_u32(dst + ur * pitch + n), bar0 + 8 * bar, c, v);
    };
    auto landed = [&](int bar, int l) {
        await(bar0 + 8 * bar, (uint32_t)(l & 1), &abort_s, a.err_flag);
        if (tid == 0 && l + 1 < a.nl)
            tc::mbar_expect_tx(bar0 + 8 * bar, expect[bar]);
    };

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
    cluster_arrive(); // every CTA of the cluster has its barriers up before the first message
    cluster_wait();
    __syncthreads();

    for (int l = 0; l < a.nl; l++) {
        const Layer &ly = layers[l];
        // keys, values of the past and the position table of this CTA's pairs, on their way under the projection
        for (int p = 0; p < npair; p++) {
            const int pair = rank + p * CLUSTER, r = pair / H, h = pair % H, b = b0 + r;
            float *Ks = sm + pl.kv + p * pl.pair, *Vs = Ks + L * pl.ks, *Rs = Vs + L * dk, *br = Rs + P * pl.ks;
            int jlo, jhi;
            attn_key_range(L, M, ly.attn_len, t, jlo, jhi);
            const int cpr = dk / 4;
            for (int idx = tid; idx < (jhi - jlo) * cpr; idx += 256) { // all but the key of this step
                const int j = jlo + idx / cpr, e = (idx % cpr) * 4;
                const float *src = ly.qkv + ((size_t)j * B + b) * 3 * HD + HD + h * dk + e;
                simt::cp16(Ks + j * pl.ks + e, src, 4);
                simt::cp16(Vs + j * dk + e, src + HD, 4);
            }
            if (ly.w_r)
                for (int idx = tid; idx < P * cpr; idx += 256)
                    simt::cp16(Rs + (idx / cpr) * pl.ks + (idx % cpr) * 4, ly.w_r + ((size_t)h * P + idx / cpr) * dk + (idx % cpr) * 4, 4);
            for (int j = tid; j < L; j += 256)
                simt::cp4(br + j, ly.b_r + (size_t)h * L + j, 1);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        product(product_of(l, 0), x, [&](int n8, const float(&acc)[SP]) {
            const int n = n8 + uh * 4, h = (n % HD) / dk;
            float4 v = gather(acc);
            if (ly.b_q && n < HD)
                v = add4(v, load4g(ly.b_q, n));
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
        // attention, one warp a pair
        for (int p = warp; p < npair; p += 8) {
            const int pair = rank + p * CLUSTER, r = pair / H, h = pair % H, b = b0 + r;
            float *Ks = sm + pl.kv + p * pl.pair, *Vs = Ks + L * pl.ks, *Rs = Vs + L * dk, *br = Rs + P * pl.ks, *qf = br + ((L + 3) & ~3),
                  *ps = qf + dk;
            int jlo, jhi;
            attn_key_range(L, M, ly.attn_len, t, jlo, jhi);
            for (int e = lane; e < dk; e += 32) {
                qf[e] = qkv[r * 3 * HD + h * dk + e];
                Ks[jhi * pl.ks + e] = qkv[r * 3 * HD + HD + h * dk + e];
                Vs[jhi * dk + e] = qkv[r * 3 * HD + 2 * HD + h * dk + e];
            }
            __syncwarp();
            float lse;
            attn_row<float>(t, jlo, jhi, a.T, L, P, dk, a.inv_sqrt, a.br_scale, qf, Ks, ly.w_r ? Rs : nullptr, pl.ks, Vs, br, ps, lane, lse,
                            [&](int e, float v) { qf[e] = v; }); // the scores have been taken: the query's place is free
            if (lane == 0)
                ly.lse[((size_t)b * H + h) * a.T + t] = lse;
            const int n4 = dk / 4;
            for (int i = lane; i < n4 * CLUSTER; i += 32) {
                const float4 v = *reinterpret_cast<const float4 *>(qf + (i % n4) * 4);
                const int at = h * dk + (i % n4) * 4;
                send4(tc::smem_u32(ob + r * HD + at), bar0 + 8 * OB, i / n4, v);
                if (i < n4)
                    *reinterpret_cast<float4 *>(ly.o + (size_t)(row0 + r) * HD + at) = v;
            }
        }
        // s = tmp + in, out = norm(s): every CTA for itself, CTA 0 keeps what the backward pass reads
        auto norm = [&](int bar, const float *in, float *out, const float *g, const float *b, float *s_out, float *y_out, float *stats) {
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
                norm_row<4, 4>(v, g, b, lane, D, a.norm_mode, rank == 0 ? stats + 2 * (row0 + r) : nullptr);
                if (rank == 0)
                    row_store<float, 4, 4>(y_out + at, lane, D, v);
                row_store<float, 4, 4>(out + r * D, lane, D, v);
            }
            __syncthreads();
        };
        landed(OB, l);
        product(product_of(l, 1), ob, [&](int n8, const float(&acc)[SP]) { to_all(tmp, D, T1, n8 + uh * 4, gather(acc), D); });
        norm(T1, x, y, ly.g1, ly.b1, ly.s1, ly.y, ly.st1);
        product(product_of(l, 2), y, [&](int n8, const float(&acc)[SP]) {
            const int n = n8 + uh * 4;
            float4 hp = gather(acc), v;
            if (ly.fb1)
                hp = add4(hp, load4g(ly.fb1, n));
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
        product(product_of(l, 3), ha, [&](int n8, const float(&acc)[SP]) {
            const int n = n8 + uh * 4;
            float4 v = gather(acc);
            if (ly.fb2)
                v = add4(v, load4g(ly.fb2, n));
            to_all(tmp, D, T2, n, v, D);
        });
        norm(T2, y, x, ly.g2, ly.b2, ly.s2, l + 1 < a.nl ? layers[l + 1].x : a.xlast, ly.st2);
    }
    // output head: row r's logits to the CTA that finishes the row
    static_assert(SP <= CLUSTER, "a cluster has a CTA for every row");
    product(product_of(a.nl, 0), x, [&](int n8, const float(&acc)[SP]) {
        const int n = n8 + uh * 4;
        float4 v = gather(acc);
        if (a.out_bias)
            v = add4(v, load4g(a.out_bias, n)); // its slot is padded beyond the last symbol
        if (ur < nb && n < V4 && peer0 == 0)
            send4(tc::smem_u32(lg + n), bar0 + 8 * LG, ur, v);
    });
    cluster_arrive();
    if (rank < nb) {
        await(bar0 + 8 * LG, 0, &abort_s, a.err_flag);
        const size_t pr = (size_t)(row0 + rank) * V;
        softmax_row(lg, V, a.dz + pr, a.scale, red);
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
    while (used < issued) { // only after a wait that ran out: copies in flight land in this CTA's shared memory
        await(rbar + 8 * (used % slots), (uint32_t)((used / slots) & 1), &abort_s, a.err_flag);
        used++;
    }
}

// ring slots per warp that fit beside the rest (0: the model does not fit)
inline int ring_slots(int sp, int nl, int D, int H, int dk, int F, int L, int P, int V, int tree)
{
    for (int s = MAX_SLOTS; s >= 2; s--)
        if ((size_t)plan_of(sp, nl, D, H, dk, F, L, P, V, tree, s).total * 4 <= 220 * 1024)
            return s;
    return 0;
}

template <int SP> static int launch_sp(cudaStream_t st, const Args &a, int t, bool chained)
{
    const Plan pl = plan_of(SP, a.nl, a.D, a.H, a.dk, a.F, a.M + a.T, a.P, a.V, 1 << a.depth, a.slots);
    CUDA_TRY(cudaFuncSetAttribute(step_kernel<SP>, cudaFuncAttributeMaxDynamicSharedMemorySize, pl.total * 4));
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
