// rb_launch.cuh -- the team size (CTAs per cluster) of a launch of one team per problem.
//
//   LAUNCH_FIXED   the caller's size;
//   LAUNCH_SERVE   the caller's size, doubled (up to 4×) until the local pass fits;
//   LAUNCH_BATCH   from 4 CTAs up, the smallest size that still gives no more teams than
//                  problems (a large batch runs many small teams, a small one a few large
//                  teams), among the sizes at which every 1D problem fits the local pass with its
//                  Gram-Schmidt slice in shared memory (else, fits it at all). Below 4 CTAs a team
//                  is slower per pass than the extra teams gain, measured on B200. A batch of 1D
//                  problems none of which can take the local pass keeps the caller's size: their
//                  team-wide pass gains nothing from more CTAs (150 cells, third-order DG in x and E,
//                  S16: one problem 2.82 s on 4 CTAs, 2.86 on 16; 24 problems 3.08 s on 4, 5.77 on 8,
//                  11.6 on 16). 2D and 3D problems gain (64×64, S8: one problem 10.4 ms on 4 CTAs,
//                  3.70 on 16; 24 problems 21.4 on 4, 20.2 on 8).
// Problems that do not fit the local pass take the team-wide pass.
#pragma once
#include <algorithm>
#include <vector>

#include "rb_local1d.cuh"

enum { LAUNCH_FIXED = 0, LAUNCH_SERVE = 1, LAUNCH_BATCH = 2 };

// `region`: bytes of shared memory beyond the per-CTA state; `hs`: host copies of the problems' records
static inline int choose_cluster(const std::vector<const DevProblem *> &hs, int cluster, int mode, int nsm, long long region) {
    bool any = false;  // some problem can use more CTAs
    for (const DevProblem *h : hs) any = any || h->ndims > 1 || rb::local1d_ok(*h, RB_MAXCLUSTER, 1LL << 40);
    if (!any) return cluster;
    auto fits = [&](int C, bool w) {  // every local-shaped 1D problem fits the local pass at cluster C
        for (const DevProblem *h : hs)
            if (rb::local1d_ok(*h, C, 1LL << 40) && !(w ? rb::local1d_w(*h, C, region) : rb::local1d_ok(*h, C, region)))
                return false;
        return true;
    };
    if (mode == LAUNCH_SERVE) {
        for (int c = cluster; c <= std::min(RB_MAXCLUSTER, 4 * cluster); c *= 2)
            if (fits(c, false)) return c;
    } else if (mode == LAUNCH_BATCH) {
        const int n = (int)hs.size();
        for (int w = 1; w >= 0; w--) {
            int best = -1, largest = -1;
            for (int c = 4; c <= RB_MAXCLUSTER; c *= 2) {
                if (!fits(c, w != 0)) continue;
                largest = c;
                if (best < 0 && nsm / c <= n + n / 20) best = c;
            }
            if (best < 0) best = largest;
            if (best > 0) return best;
        }
    }
    return cluster;
}
