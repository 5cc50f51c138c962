// Twiddle factors of the FFT tables (host).
#pragma once

#include <cmath>

namespace pwk {

// exp(-2 pi i m / n), 0 <= m < n, rounded once: the fraction of a turn is reduced to
// [0, 1/8] in integers first (cos and sin of the unreduced angle in double carry its
// rounding, up to 9e-16 near a whole turn).
inline void twiddle(int m, int n, double &re, double &im) {
    long p = m, q = n;
    bool neg_s = false, neg_c = false, swap = false;
    if (2 * p > q) {   // past half a turn
        p = q - p;
        neg_s = true;
    }
    if (4 * p > q) {   // past a quarter: half a turn less
        p = q - 2 * p;
        q *= 2;
        neg_c = true;
    }
    if (8 * p > q) {   // past an eighth: a quarter less
        p = q - 4 * p;
        q *= 4;
        swap = true;
    }
    const long double a = 2.0L * 3.14159265358979323846264338327950288L * p / q;
    const double c = (double)std::cos(a), s = (double)std::sin(a);
    re = neg_c ? -(swap ? s : c) : (swap ? s : c);
    im = neg_s ? (swap ? c : s) : -(swap ? c : s);
}

}  // namespace pwk
