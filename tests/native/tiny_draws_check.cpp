// Draws of tiny standard deviations (pair_math.h): a rounding that the motion kernel
// accepts for z stddev + mean is the double's, also where the products' low parts leave
// float's normal range.
#include "pair_math.h"

#include <stdio.h>
#include <stdlib.h>

#include <random>

using namespace tsdfl;

int main(int argc, char** argv)
{
    const long n = argc > 1 ? atol(argv[1]) : 2000000;
    std::mt19937_64 g(1);
    long draws = 0, left = 0, wrong = 0, ordinary = 0, ordinary_left = 0;
    for (long i = 0; i < n; ++i) {
        // radii and angles of every size, the smallest among them
        const uint64_t m = (1ull << 53) - 1 - (g() >> (12 + g() % 52));
        const uint64_t wa = (m - 1) << 11, wb = ((g() % 4) << 62) + (((g() >> 2) >> (g() % 52)) & ~2047ull);
        Pair z[2];
        if (!normal_pairs(wa, wb, z[0], z[1])) continue;
        const long double u2 = ldexpl((long double)(wb >> 11), -53);
        const long double r = sqrtl(-2 * logl(ldexpl((long double)m, -53)));
        const int q = (int)floorl(4 * u2 + 0.5L);
        const long double w = (4 * u2 - q) * 1.570796326794896619231321691639751442L;
        const long double s = sinl(w), c = cosl(w);
        const long double cs[4] = {c, -s, -c, s}, sn[4] = {s, c, -s, -c};
        const double exact[2] = {(double)(r * cs[q & 3]), (double)(r * sn[q & 3])};
        const int scale = -(int)(g() % 67);   // from 1 down to 1e-20
        const double stddev = ldexp(1.4 + 0.5 * ((double)(g() >> 11) * 0x1p-53), scale);
        const double mean = i % 3 ? 0.0 : ldexp(1.0, -(int)(g() % 66));
        for (int j = 0; j < 2; ++j) {
            float bound, f;
            const Pair v = normal_draw(z[j], from_double(stddev), from_double(mean), kDrawLow, bound);
            const double want = exact[j] * stddev + mean;
            const bool plain = fabs(exact[j] * stddev) > 0x1p-70;
            ++draws;
            ordinary += plain;
            if (!rounded(v, bound, f)) {
                ++left;
                ordinary_left += plain;
            } else if (f != (float)want) {
                if (++wrong < 5) printf("z %g stddev %g mean %g: %a, not %a\n", exact[j], stddev, mean, f, (float)want);
            }
        }
    }
    // a draw without noise stays exact
    float bound, f;
    const Pair v = normal_draw({0.75f, 0x1p-30f}, {0.0f, 0.0f}, {0.0f, 0.0f}, 0.0f, bound);
    if (bound != 0.0f || !rounded(v, bound, f) || f != 0.0f || signbit(f)) ++wrong;
    printf("draws %ld left %ld ordinary %ld left %ld wrong %ld\n", draws, left, ordinary, ordinary_left, wrong);
    return wrong != 0 || ordinary_left * 500 > ordinary;
}
