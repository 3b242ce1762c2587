// Rank of a block-matching candidate among the kept ones, by (cost,
// enumeration index). A cost that is NaN (float samples that are NaN or
// infinite) comes after every other one, so the ranks of the kept candidates
// are always 0, 1, 2, ... without a gap or a tie, and the best-4 list that they
// fill holds a candidate's position in every place that is read. Compiled for
// the device (k_bm_group) and for the host's sweep of cost patterns.
#pragma once

#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define LGCR_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define LGCR_HOST_DEVICE inline
#endif

namespace lgcr_b200 {

constexpr int kBmCandidates = 25;

// A cost is a mean of squares, so it is not below zero and its bits order as
// its value; those of a NaN lie above infinity's.
LGCR_HOST_DEVICE uint32_t costBits(float c) {
    uint32_t b;
    memcpy(&b, &c, sizeof(b));
    return b & 0x7fffffffu;
}

LGCR_HOST_DEVICE int keptRank(const float *costs, unsigned kept, int me) {
    const uint32_t mine = costBits(costs[me]);
    int rank = 0;
    for (int d = 0; d < kBmCandidates; ++d)              // an earlier one of equal cost goes first
        rank += int((kept >> d) & 1u & unsigned(costBits(costs[d]) < mine + (d < me ? 1u : 0u)));
    return rank;
}

} // namespace lgcr_b200
