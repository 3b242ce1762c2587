// Rank of a block-matching candidate among the kept ones, by (cost,
// enumeration index). A cost that is NaN (float samples that are NaN or
// infinite) comes after every other one, so the ranks of the kept candidates
// are always 0, 1, 2, ... without a gap or a tie, and the best-4 list that they
// fill holds a candidate's position in every place that is read. Compiled for
// the device (k_bm_group) and for the host's sweep of cost patterns.
#pragma once

#ifdef __CUDACC__
#define LGCR_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define LGCR_HOST_DEVICE inline
#endif

namespace lgcr_b200 {

constexpr int kBmCandidates = 25;

LGCR_HOST_DEVICE int keptRank(const float *costs, unsigned kept, int me) {
    const float mine = costs[me];
    const bool last = mine != mine;
    int rank = 0;
    for (int d = 0; d < kBmCandidates; ++d) {
        if (d == me || !((kept >> d) & 1u))
            continue;
        const float c = costs[d];
        if (last ? (c == c || d < me) : (c < mine || (c == mine && d < me)))
            ++rank;
    }
    return rank;
}

} // namespace lgcr_b200
