// fixed_shift and packs (tsdfl_internal.h): the scale of the likelihood sums is the
// largest, up to 2^40, at which n + 1 values sum below 2^62, and packs() says yes only
// where a lane's packed lookups leave the hits' bits alone.
#include <stdio.h>

#include "tsdfl_internal.h"

using namespace tsdfl;

int main()
{
    long wrong = 0, packed = 0, wide = 0;
    for (int e = -400; e <= 700; ++e) {
        const double top = std::exp2(e / 20.0);   // 1e-6 to 3e10
        for (double n : {1.0, 2.0, 72.0, 100.0, 1000.0, 4607.0, 4608.0, 65'535.0, 2e6, 2e9}) {
            const int shift = fixed_shift(top, n);
            const double sum = std::ldexp(top * (n + 1.0), shift);
            if (shift > 40 || !(sum <= 0x1p62)) ++wrong;
            if (shift < 40 && !(2.0 * sum > 0x1p62)) ++wrong;
            const double lane = std::ldexp(top * kPackedLookups, shift);
            if (packs(top, shift) != (lane <= 0x1p56)) ++wrong;
            ++(packs(top, shift) ? packed : wide);
        }
    }
    printf("packed %ld wide %ld wrong %ld\n", packed, wide, wrong);
    return wrong != 0 || !packed || !wide;
}
