// step_deal.h -- how the one-launch time step (step_fp32.cuh) deals a product's output columns over the
// CTAs of a cluster, and for which models the exchanges alone order the reuse of its receive buffers.
// Plain C++, so that the order can be checked without a GPU.
#pragma once

#ifdef __CUDACC__
#define STEP_HD __host__ __device__
#else
#define STEP_HD
#endif

namespace stepf {

constexpr int CLUSTER = 8; // CTAs that share a group of streams

// Groups of eight columns as evenly as they go: CTA `rank` has the columns [deal_from(N, rank),
// deal_from(N, rank + 1)), at least one group when there are eight.
STEP_HD inline int deal_from(int N, int rank)
{
    const int at = (N + 7) / 8 * rank / CLUSTER * 8;
    return at < N ? at : N;
}
// columns of a CTA at most, whole groups
STEP_HD inline int per_cta(int N) { return ((N + CLUSTER - 1) / CLUSTER + 7) & ~7; }

// A CTA writes into its peers' buffers as soon as an exchange it needs is complete; that its peers have
// finished with the buffers follows where every CTA has had a share in an exchange between: columns of the
// feed-forward up product (between the two results that go through `tmp`, and between two layers'
// attention outputs) and columns of the projection (between the last result of a layer and the
// first of the next).  Where one of the two products leaves a CTA without columns, a cluster-wide
// barrier behind each norm takes their place.
STEP_HD inline bool exchanges_order_reuse(int HD, int F) { return F >= 8 * CLUSTER && 3 * HD >= 8 * CLUSTER; }

} // namespace stepf
