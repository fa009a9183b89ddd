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

} // namespace attn
