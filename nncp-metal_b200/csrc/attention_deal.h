// attention_deal.h -- which kernel, how many CTAs and how many queries a CTA an attention launch takes, from its
// sizes alone.  Plain C++, so that the rules can be checked without a GPU.
#pragma once

namespace attn {

constexpr int SMS = 148;

// Whether the bf16 adjoint takes the kernel of 128-key blocks, one CTA to an SM (attention_bwd.cuh), rather than the
// warp-level one of 64-key blocks, two CTAs to an SM.  pairs: (stream, head) pairs; lo, hi: first and last 64-key
// block with a visible pair.
// A CTA of the former goes through 64 query rows and 128 keys whatever is in them.  At head size 64 it is the slower one where
//   * its blocks hold one 64-key block each and the pairs are more than one to an SM: 32 queries, 64 keys, 256 pairs 18.3
//     against 14.0 us, 1024 pairs 57.7 against 48.2 (a step of 4 layers, 128 streams, 8 heads 1138 against 1075); 148 pairs
//     10.5 against 11.6;
//   * one tile of queries meets three 64-key blocks and two CTAs to an SM take all pairs at once: 16 queries, 129 to 192
//     keys, 152 to 296 pairs 1.01 to 0.92 times as fast.
// Elsewhere it is the faster one: 64 queries, 128 keys 1.2 times, 193 keys 1.4 to 1.7 times; head size 128 from 1.02 times
// (one 64-key block) to 1.9.
inline bool adjoint_by_128(int dk, long pairs, int n_queries, int lo, int hi)
{
    if (dk != 64 || pairs <= SMS)
        return true;
    const int n64 = hi - lo + 1, n128 = hi / 2 - lo / 2 + 1;
    return n64 != n128 && !(n_queries <= 16 && n64 == 3 && pairs <= 2 * SMS);
}

// CTAs with `smem` bytes of shared memory that an SM holds, `most` at most
inline int resident(long smem, int most)
{
    const long n = 228 * 1024 / (smem + 1024);
    return n < most ? (int)n : most;
}

// fp32 forward: queries a CTA takes, its eight warps one each in a round; smem: its shared memory, most of it keys, values and
// table, which every CTA fills.  Eight while the CTAs that then are needed run at once, else whole rounds of eight for
// two CTAs an SM: 148 pairs of 32 queries, 232 keys (102 KB) 40.1 us in chunks of 8, 31.6 of 16; 64 keys (29 KB) 10.6 and 11.3.
inline int queries_of_cta(long pairs, int n_queries, long smem)
{
    const int rounds = (n_queries + 7) / 8;
    if (pairs * rounds <= resident(smem, 4) * SMS)
        return 8;
    const long chunks = (2 * SMS + pairs - 1) / pairs; // at least 1
    return (int)((n_queries + chunks - 1) / chunks + 7) & ~7;
}

// fp32 adjoint: CTAs that share a (stream, head) as a cluster; smem: the shared memory of each, which holds all operands and
// whose read rate bounds it.  Clusters pay while all run at once and leave no SM with a CTA more than the others for long:
//   * eight and four to a pair while they find room (clusters of four leave an eighth of the SMs over): 32 queries, 64 keys (51 KB), 37 / 74 pairs
//     in a training step's order 26.1 -> 21.0 / 26.2 -> 26.4 us, in a chain of the three calls of the op 59.1 -> 40.8 / 62.7 -> 45.5; 232 keys (164 KB,
//     one to an SM) 32 / 40 pairs 96.6 -> 55.2 / 99.9 -> 85.1, by two 73.1;
//   * two to a pair up to one to an SM, and exactly two to an SM where both have as many rounds of eight rows: 32 queries, 64 keys 148 pairs
//     26.4 -> 24.7, 16 queries 16.5 -> 15.7, but 24 queries 29.2 -> 32.2 in the op's chain; 232 keys 80.7 -> 104.8.
inline int ctas_of_pair(long pairs, int n_queries, long smem)
{
    const int rounds = (n_queries + 7) / 8;
    if (pairs <= 8 && rounds >= 8)
        return 8;
    if (rounds >= 4 && pairs <= SMS / 2 && 4 * pairs <= resident(smem, 4) * SMS * 7 / 8)
        return 4;
    return rounds >= 2 && (pairs <= SMS / 2 || (pairs <= SMS && rounds % 2 == 0 && resident(smem, 2) == 2)) ? 2 : 1;
}

} // namespace attn
