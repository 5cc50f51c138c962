// Band groups of the density pass (calc_rhoe).
#pragma once

#include <algorithm>

namespace pwk {

// Each of the N3 G CTAs takes one z-plane of ceil(cnt / G) bands, per_sm of them
// resident on each of the 148 SMs, so the time goes with waves x bands per group,
// plus about 0.3 of a band for a CTA's set-up and plane and 0.1 a group for the
// reduction.  (75-point grid, 41 FP64 bands: 7 groups run 4 x 6 bands deep, 4 groups,
// "enough CTAs to fill the GPU twice", 3 x 11, their third wave nearly empty: 128
// bands 882 -> 812 us.)  per_sm is the launched kernel's: one or two a SM for every
// grid made 40 FP64 bands of 18 and 27 points 74 -> 96 and 53 -> 68 us, two FP32
// bands of 150 points 564 -> 712 us.
inline int rho_groups(int N3, int cnt, int per_sm) {
    const int slots = 148 * std::max(1, per_sm);
    int best = 1;
    double tbest = 1e300;
    for (int G = 1; G <= std::min(cnt, 16); ++G) {
        const int waves = (N3 * G + slots - 1) / slots, Bg = (cnt + G - 1) / G;
        const double t = waves * (Bg + 0.3) + 0.1 * G;
        if (t < tbest) {
            tbest = t;
            best = G;
        }
    }
    return best;
}

}  // namespace pwk
