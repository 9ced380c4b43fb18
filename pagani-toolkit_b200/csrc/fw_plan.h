// fw_plan.h -- how a Floyd-Warshall batch is shared out (host only).
#pragma once
#include <algorithm>
#include <vector>

// Graphs in processing order (blocks of 64 per side, descending) are cut into
// bundles of consecutive graphs, bundle q being [bundle0[q], bundle0[q + 1]).
// Each team of CTAs takes one bundle after another and sweeps its graphs in
// step.
struct FwPlan {
    int teams = 1;
    std::vector<int> bundle0;
};

// One team and one bundle: all graphs in step over the whole GPU, so that the
// blocks of a round fill it.  Only where the batch has so many graphs that
// they fill it many times over do teams of four SMs do better, each with
// bundles of about 1 MB of matrices (an SM's share of a round is several
// blocks, what is being swept stays in L2, a barrier has four arrivals): the
// busiest team's work must be within a quarter of an even share.  Measured,
// teams against one: 512 graphs of 90 to 1024 nodes 10.6 / 10.9 ms, 512 of 90
// to 520 3.9 / 4.0; where this rule has one team, 64 graphs of 90 to 1024 3.6
// / 1.6 ms, 16 of 90 to 520 0.69 / 0.38, one of 1500 with 60 of 120 10.0 / 1.1.
inline FwPlan fw_batch_plan(const int* nb, int ng, int sm_count, int max_teams)
{
    constexpr double BUNDLE_BYTES = 1 << 20, UNEVEN = 1.25;
    FwPlan p;
    std::vector<double> work;   // per bundle
    double bytes = 0.0, all = 0.0;
    for (int q = 0; q < ng; q++) {
        const double side = 64.0 * nb[q], b = 4.0 * side * side, w = (double)nb[q] * nb[q] * nb[q];
        if (q == 0 || bytes + b > BUNDLE_BYTES) {
            p.bundle0.push_back(q);
            work.push_back(0.0);
            bytes = 0.0;
        }
        bytes += b;
        work.back() += w;
        all += w;
    }
    p.teams = std::max(1, std::min(max_teams, sm_count / 4));
    // the queue: each bundle goes to the team that is free first
    std::vector<double> busy((size_t)p.teams, 0.0);
    for (double w : work) *std::min_element(busy.begin(), busy.end()) += w;
    if (*std::max_element(busy.begin(), busy.end()) > UNEVEN * all / p.teams) {
        p.teams = 1;
        p.bundle0.assign(1, 0);
    }
    p.bundle0.push_back(ng);
    return p;
}
