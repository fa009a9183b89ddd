// decoder.cuh -- the range decoder on the device: one step's symbols are decoded from the trees
// that coder_trees_kernel left in device memory, so a decode step needs no host round trip.
//
// The arithmetic is get_bit / read_sym of the reference coder (arith.c:241-310,
// cp_utils.c:326-349) bit for bit: split = (range * prob0) >> 15, bit = low >= split,
// renormalisation one byte at a time while range < 0xFF01, zero bytes past the end of the input.
// The streams of one step share ONE bit stream, so their symbols decode strictly one after the
// other: a single thread walks the trees, and its chain of operations per bit bounds the step.  What
// can run ahead is the data movement: a second warp fills a ring of shared-memory slots with the next
// streams' trees by bulk copies (2 V bytes each, completion on an mbarrier) while the current one is
// walked, and the payload bytes the step can consume at most (two per bit) are staged in shared memory
// up front.  128 streams of 14 bits: 156 us with one load of prob0 behind every decision, 95 now.
//
// An alphabet that is not a power of two has the uneven tree of write_sym (a node of n symbols
// sends n >> 1 left): the walk then carries the node's range beside its heap index and ends when
// one symbol is left (template argument ANY); a tree row has P = 2^ceil(log2 V) entries.
#pragma once
#include <type_traits>

#include "common.cuh"
#include "gemm_tc.cuh"

namespace dec {

struct State {
    unsigned long long pos, len; // next payload byte, payload size
    uint32_t low, range;
    int err, pad;
};

constexpr uint32_t R_LOW = (0xffu << 8) + 1u, R_TOP = 0xffu << 16;
constexpr int MAX_RING = 8, MAX_SMEM = 200 * 1024 + 16; // 16: the window's bytes to look ahead

__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(bar)
                 : "memory");
}

// window bytes a step of `B` streams with `nb` bits per symbol can consume, twelve to look ahead, as a multiple of 16
__host__ __device__ inline int window_bytes(int B, int nb) { return (2 * B * nb + 12 + 15) & ~15; }
// shared memory left for the ring
__host__ __device__ inline int ring_bytes(int B, int nb) { return MAX_SMEM - window_bytes(B, nb) - 128; }
// trees of P entries that share a ring slot: small ones come 16 KB at a time, fewer where a step of very many
// streams leaves no room for two such slots
__host__ __device__ inline int slot_trees(int B, int P, int nb)
{
    int n = P >= 8192 ? 1 : (8192 / P < B ? 8192 / P : B);
    while (n > 1 && 2 * n * P * 2 > ring_bytes(B, nb))
        n >>= 1;
    return n;
}

// slots of the ring for trees of P entries (0: the trees do not fit)
inline int ring_slots(int B, int P, int nb)
{
    const int n = ring_bytes(B, nb) / (slot_trees(B, P, nb) * P * 2);
    if (P < 8 || n < 2)
        return 0;
    return std::min(n, MAX_RING);
}
inline size_t smem_bytes(int B, int P, int nb, int ring) { return (size_t)ring * slot_trees(B, P, nb) * P * 2 + window_bytes(B, nb) + 128; }

// trees: [B][P] prob0 in heap order (entry 0 unused), P = 2^nb >= V.  sym_out[b] and ids_next[b]
// (when not null) receive the decoded symbol, 0 for the streams past the end of the block: those at
// step `t` are b >= limit_b when t == limit_t, and all of them when t > limit_t.
template <bool ANY, int NB>
__global__ void __launch_bounds__(64)
decode_step_kernel(const uint16_t *__restrict__ trees, const uint8_t *__restrict__ payload, State *state,
                   int32_t *__restrict__ sym_out, int32_t *__restrict__ ids_next, int t, int limit_t, int limit_b,
                   int B, int V, int P, int nb, int ring, int *err_flag)
{
    extern __shared__ __align__(128) uint8_t dsm[];
    uint64_t *bars = reinterpret_cast<uint64_t *>(dsm);           // [2][MAX_RING] of 8 bytes: 128
    const int G = slot_trees(B, P, nb);
    uint16_t *slots = reinterpret_cast<uint16_t *>(dsm + 128);    // [ring][G][P]
    uint8_t *win = dsm + 128 + (size_t)ring * G * P * 2;          // payload window
    __shared__ int abort_s;
    __shared__ int issued_s;
    const int tid = threadIdx.x;
    const int n_act = t < limit_t ? B : (t == limit_t ? min(limit_b, B) : 0);
    const uint32_t tree_bytes = (uint32_t)P * 2u;
    const int n_grp = (n_act + G - 1) / G;
    const unsigned long long pos0 = state->pos, len = state->len;
    uint64_t *done = bars + MAX_RING; // the walker has left a slot

    if (tid == 0) {
        abort_s = 0;
        for (int i = 0; i < ring; i++) {
            tc::mbar_init(tc::smem_u32(bars + i), 1);
            tc::mbar_init(tc::smem_u32(done + i), 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const int wbytes = window_bytes(B, nb);
    for (int i0 = tid; i0 < wbytes; i0 += 16 * 64) { // sixteen loads in flight
        uint8_t v[16];
#pragma unroll
        for (int k = 0; k < 16; k++) {
            const int i = i0 + k * 64;
            v[k] = i < wbytes && pos0 + i < len ? payload[pos0 + i] : (uint8_t)0;
        }
#pragma unroll
        for (int k = 0; k < 16; k++)
            if (i0 + k * 64 < wbytes)
                win[i0 + k * 64] = v[k];
    }
    // Up to here nothing depends on the kernels of this step: the state is what the step before left, and the step's first
    // kernel (embedding, or the whole step in one launch) lets its successors start only when that is complete.
    pdl_wait();
    pdl_trigger(); // a successor that was launched to overlap this kernel may start on what does not depend on it
    __syncthreads();

    if (tid == 32) { // the copies, on a warp of their own: the walk does not stop to issue them
        int g = 0;
        for (; g < n_grp; g++) {
            const int s = g % ring;
            if (g >= ring && !tc::mbar_wait(tc::smem_u32(done + s), (uint32_t)((g / ring - 1) & 1), &abort_s, err_flag, 43))
                break;
            const uint32_t bytes = (uint32_t)min(G, n_act - g * G) * tree_bytes;
            tc::mbar_expect_tx(tc::smem_u32(bars + s), bytes);
            bulk_load(tc::smem_u32(slots + (size_t)s * G * P), trees + (size_t)g * G * P, bytes, tc::smem_u32(bars + s));
        }
        issued_s = g;
    }
    int walked = 0; // groups whose copy has been waited for
    bool ok = true;
    if (tid == 0) {
        // What a bit costs is a chain of dependent instructions on one thread, so nothing in it branches: a node's
        // prob0 is in hand, and its children's (one 32-bit word) are on their way, before the branch at it is
        // known; (range * prob0) >> 15 is the high word of (range << 8) * (prob0 << 9), range staying below
        // 2^24; renormalisation shifts by 0, 8 or 16 (two bytes always suffice: range is at least 1) and draws
        // on the next eight payload bytes in two registers.  A branch costs some 15 cycles of this chain (53 a bit
        // without any, 76 with two every second bit), so up to eight bits go between two looks at the
        // payload: enough unless they draw more than the 32 bits that are certain to be there, and then they are
        // walked again one at a time.
        uint32_t low = state->low, range = state->range, used = 0, hi, lo, drawn; // drawn: bits taken from hi : lo
        const uint32_t *words = reinterpret_cast<const uint32_t *>(win);
        auto top_up = [&]() { // the eight window bytes from `used` on (zero past the payload's end)
            const uint32_t *w = words + (used >> 2);
            const uint32_t w0 = __byte_perm(w[0], 0, 0x0123), w1 = __byte_perm(w[1], 0, 0x0123), w2 = __byte_perm(w[2], 0, 0x0123);
            const uint32_t sh = (used & 3) * 8;
            hi = __funnelshift_l(w1, w0, sh);
            lo = __funnelshift_l(w2, w1, sh);
            drawn = 0;
        };
        const uint32_t last = (uint32_t)P / 2u - 1; // word of the last pair: below the tree's leaves there is nothing to load
        top_up();
        auto check = [&]() {
            if (drawn > 32) {
                used += drawn >> 3;
                top_up();
            }
        };
        int slot = ring - 1, in_slot = G; // the slot in use and the trees of it that have been walked
        uint32_t phase = 1;
        bool ready = false; // the next slot's copy was seen complete before the present slot's last tree
        int32_t *const next_in = ids_next ? ids_next : sym_out;
        int b = 0;
        for (; b < n_act; b++) {
            if (in_slot == G) {
                if (b > 0)
                    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::smem_u32(done + slot)) : "memory");
                in_slot = 0;
                slot = slot + 1 == ring ? 0 : slot + 1;
                phase ^= slot == 0 ? 1u : 0u;
                if (!ready && !tc::mbar_wait(tc::smem_u32(bars + slot), phase, &abort_s, err_flag, 41)) {
                    ok = false;
                    break;
                }
                walked++;
            }
            const uint32_t *pairs = reinterpret_cast<const uint32_t *>(slots + ((size_t)slot * G + in_slot) * P);
            if (++in_slot == G) { // asked here, needed behind the walk
                const bool wrap = slot + 1 == ring;
                uint32_t done_next;
                asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                             : "=r"(done_next)
                             : "r"(tc::smem_u32(bars + (wrap ? 0 : slot + 1))), "r"(phase ^ (wrap ? 1u : 0u))
                             : "memory");
                ready = done_next != 0;
            }
            uint32_t k = 1, p9 = (pairs[0] >> 16) << 9, kids = pairs[1];
            auto next_bit = [&]() { // get_bit at node k: the branch taken, the decoder's state advanced
                const uint32_t split = __umulhi(range << 8, p9);
                const bool bit = low >= split;
                k = 2 * k + (bit ? 1u : 0u);
                const uint32_t p1 = (kids >> 16) << 9, p0 = (kids & 0xffffu) << 9;
                p9 = bit ? p1 : p0;
                kids = pairs[min(k, last)];
                low = bit ? low - split : low;
                range = bit ? range - split : split;
                const uint32_t s = range < R_LOW ? (range < 0x100u ? 16u : 8u) : 0u;
                range <<= s;
                low = __funnelshift_l(hi, low, s);
                hi = __funnelshift_l(lo, hi, s);
                lo <<= s;
                drawn += s;
                return bit;
            };
            auto run = [&](auto count, auto step) { // `count` bits, step(bit, index); an index 0 starts over
                constexpr int N = decltype(count)::value;
                const uint32_t low0 = low, range0 = range, hi0 = hi, lo0 = lo, drawn0 = drawn, k0 = k, p0 = p9, kids0 = kids;
#pragma unroll
                for (int i = 0; i < N; i++)
                    step(next_bit(), i);
                if (drawn > 32) {
                    if (drawn > 64) { // a run of improbable branches
                        low = low0; range = range0; hi = hi0; lo = lo0; drawn = drawn0; k = k0; p9 = p0; kids = kids0;
#pragma unroll 1
                        for (int i = 0; i < N; i++) {
                            step(next_bit(), i);
                            check();
                        }
                    }
                    check();
                }
            };
            int c;
            if constexpr (ANY) { // every node above the last level is split, one of the last if it has two symbols
                int first = 0, n = V, first0 = 0, n0 = V;
                auto down = [&](bool bit) {
                    const int h = n >> 1;
                    first = bit ? first + h : first;
                    n = bit ? n - h : h;
                };
                int lvl = 1;
                for (; lvl + 3 < nb; lvl += 4) {
                    first0 = first;
                    n0 = n;
                    run(std::integral_constant<int, 4>(), [&](bool bit, int i) {
                        if (i == 0) {
                            first = first0;
                            n = n0;
                        }
                        down(bit);
                    });
                }
                for (; lvl < nb; lvl++) {
                    down(next_bit());
                    check();
                }
                if (n > 1) {
                    down(next_bit());
                    check();
                }
                c = first;
            } else {
                auto nothing = [](bool, int) {};
                constexpr int HALF = (NB + 1) / 2; // up to eight bits at once, else two halves
                if constexpr (NB <= 8) {
                    run(std::integral_constant<int, NB>(), nothing);
                } else {
                    run(std::integral_constant<int, HALF>(), nothing);
                    run(std::integral_constant<int, NB - HALF>(), nothing);
                }
                c = (int)k - V;
            }
            next_in[b] = c;
            sym_out[b] = c;
        }
        for (; b < B; b++) { // past the end of the block
            next_in[b] = 0;
            sym_out[b] = 0;
        }
        used += drawn >> 3;
        state->pos = min(pos0 + used, len);
        state->low = low;
        state->range = range;
        if (!ok)
            state->err = 1;
    }
    __syncthreads();
    if (tid == 0 && !ok) // copies still in flight land in this CTA's shared memory: each gets a bounded chance to finish
        for (int g = walked; g < issued_s; g++)
            tc::mbar_wait(tc::smem_u32(bars + g % ring), (uint32_t)((g / ring) & 1), &abort_s, err_flag, 42);
}

typedef void (*StepKernel)(const uint16_t *, const uint8_t *, State *, int32_t *, int32_t *, int, int, int, int, int, int, int, int, int *);
// the kernel for trees of depth nb
inline StepKernel step_kernel_of(bool pow2, int nb)
{
    if (!pow2)
        return decode_step_kernel<true, 0>;
    switch (nb) {
    case 3: return decode_step_kernel<false, 3>;
    case 4: return decode_step_kernel<false, 4>;
    case 5: return decode_step_kernel<false, 5>;
    case 6: return decode_step_kernel<false, 6>;
    case 7: return decode_step_kernel<false, 7>;
    case 8: return decode_step_kernel<false, 8>;
    case 9: return decode_step_kernel<false, 9>;
    case 10: return decode_step_kernel<false, 10>;
    case 11: return decode_step_kernel<false, 11>;
    case 12: return decode_step_kernel<false, 12>;
    case 13: return decode_step_kernel<false, 13>;
    default: return decode_step_kernel<false, 14>; // the tree kernels' shared memory ends here
    }
}

} // namespace dec
