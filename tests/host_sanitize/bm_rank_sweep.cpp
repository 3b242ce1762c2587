// Ranks of block-matching candidates over cost patterns with equal, infinite
// and NaN costs: the kept candidates' ranks are a permutation of 0 .. count-1,
// and the ranked costs rise, NaN last. Exits non-zero on a difference.
#include "bm_rank.h"

#include <cmath>
#include <cstdio>
#include <limits>
#include <random>

using namespace lgcr_b200;

int main() {
    std::mt19937 rng(7);
    const float inf = std::numeric_limits<float>::infinity(), nan = std::numeric_limits<float>::quiet_NaN();
    const float values[] = {0.0f, 1e-6f, 1e-6f, 3e-5f, 4e-5f, 1.0f, inf, nan, nan, nan};
    int bad = 0;
    for (int round = 0; round < 20000; ++round) {
        float costs[kBmCandidates];
        const int span = 1 + int(rng() % 10);
        for (float &c : costs)
            c = values[9 - rng() % span];            // the first rounds' patterns are all NaN
        unsigned kept = rng() & ((1u << kBmCandidates) - 1u);
        if (!kept)
            kept = 1u;
        int at[kBmCandidates], count = 0;
        for (int &i : at)
            i = -1;
        for (int i = 0; i < kBmCandidates; ++i) {
            if (!((kept >> i) & 1u))
                continue;
            ++count;
            const int rank = keptRank(costs, kept, i);
            if (rank < 0 || rank >= kBmCandidates || at[rank] >= 0)
                ++bad;
            else
                at[rank] = i;
        }
        for (int r = 0; r < count; ++r) {
            if (at[r] < 0) {
                ++bad;
                continue;
            }
            if (r == 0 || at[r - 1] < 0)
                continue;
            const float a = costs[at[r - 1]], b = costs[at[r]];
            if (!(std::isnan(b) || a < b || a == b) || ((a == b || (std::isnan(a) && std::isnan(b))) && at[r - 1] > at[r]))
                ++bad;
        }
    }
    std::printf("%d differences\n", bad);
    return bad != 0;
}
