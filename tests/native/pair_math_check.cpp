// pair_math.h against the double functions and against long double: how far the
// pairs are off, how often a rounding is left to the double function, and that no
// accepted rounding differs from "double function, rounded to float".
#include "pair_math.h"

#include <stdio.h>
#include <stdlib.h>

#include <algorithm>
#include <random>

using namespace tsdfl;

static long wrong = 0;
struct Stat {
    const char* name;
    long n = 0, left = 0;
    double worst = 0;   // relative error of the pair
};
static void report(const Stat& s)
{
    printf("%s %ld %ld %.3f\n", s.name, s.n, s.left, s.worst > 0 ? log2(s.worst) : -99.0);
}
static bool same(float a, float b) { return a == b && signbit(a) == signbit(b); }
static double rel(Pair p, long double v) { return v != 0 ? (double)fabsl(((long double)p.h + p.l - v) / v) : 0.0; }

static void angle(Stat& st, float x, double add)
{
    const Pair d = from_double(add);
    const double v = (double)x + add;
    if (fabs(add) > 0x1p-20 * fabs((double)x)) return;
    float s, c;
    ++st.n;
    if (!sincos_rounded(x, d.h, add == 0 ? 0.0f : (float)(fabs(v) * 0x1p-45), s, c)) ++st.left;
    else if (!same(s, (float)sin(v)) || !same(c, (float)cos(v))) ++wrong;
    Pair ps, pc;
    sincos_pair(x, d.h, ps, pc);
    const long double lv = (long double)x + (long double)d.h;
    st.worst = std::max({st.worst, rel(ps, sinl(lv)), rel(pc, cosl(lv))});
}

int main(int argc, char** argv)
{
    const long n = argc > 1 ? atol(argv[1]) : 2000000;
    std::mt19937_64 g(7);
    auto uni = [&](double a, double b) { return a + (b - a) * ((double)(g() >> 11) * 0x1p-53); };
    Stat tr{"angles"}, sm{"small"}, big{"large"}, near{"quarters"}, at{"atan2"}, as{"asin"}, lg{"log"}, nm{"normals"};
    for (long i = 0; i < n; ++i) {
        const double a = uni(-3.2, 3.2);
        angle(tr, (float)a, i & 1 ? 0.0 : a - (double)(float)a);
        const double b = ldexp(uni(-1, 1), -(int)(g() % 60));
        angle(sm, (float)b, i & 1 ? 0.0 : b - (double)(float)b);
        angle(big, (float)uni(-64, 64), 0.0);
        const float quarter = (float)((double)((long)(g() % 81) - 40) * 1.5707963267948966);
        float q = quarter;
        for (int k = (int)(g() % 5); k > 0; --k) q = nextafterf(q, 2e3f);
        angle(near, q, 0.0);

        const float y = (float)(i % 3 ? uni(-1, 1) : ldexp(uni(-1, 1), -(int)(g() % 45)));
        const float x = (float)(i % 5 ? uni(-1, 1) : ldexp(uni(-1, 1), -(int)(g() % 45)));
        // as the angles are formed: both divided by the pitch's cosine
        const double cp = cos((double)(float)uni(-1.5, 1.5));
        float o;
        ++at.n;
        if (!atan2_rounded(y, x, o)) ++at.left;
        else if (!same(o, (float)atan2((double)y / cp, (double)x / cp))) ++wrong;
        ++as.n;
        if (!asin_rounded(y, o)) ++as.left;
        else if (!same(o, (float)asin((double)y))) ++wrong;

        uint64_t m = (g() >> 11 >> (i % 4 ? 0 : g() % 52)) + 1;
        if (i % 7 == 0) m = (1ull << 53) - (g() >> 11 >> (g() % 53));
        if (m < (1ull << 53)) {
            ++lg.n;
            lg.worst = std::max(lg.worst, rel(minus_log(m), -logl(ldexpl((long double)m, -53))));
        }
        const uint64_t wa = (m - 1) << 11 | (g() & 2047);
        const uint64_t wb = i % 4 ? g() : (g() % 5 << 62) + (uint64_t)((int64_t)(g() >> 1) >> (1 + g() % 60));
        Pair z0, z1;
        ++nm.n;
        if (!normal_pairs(wa, wb, z0, z1)) ++nm.left;
        else {
            const long double u2 = ldexpl((long double)(wb >> 11), -53);
            const long double r = sqrtl(-2 * logl(ldexpl((long double)m, -53)));
            // reduced exactly, as 2 pi u2 near a quarter turn has no digits left otherwise
            const int qq = (int)floorl(4 * u2 + 0.5L);
            const long double w = (4 * u2 - qq) * 1.570796326794896619231321691639751442L;
            const long double s = sinl(w), c = cosl(w);
            const long double cs[4] = {c, -s, -c, s}, sn[4] = {s, c, -s, -c};
            nm.worst = std::max({nm.worst, rel(z0, r * cs[qq & 3]), rel(z1, r * sn[qq & 3])});
        }
    }
    for (float z : {0.0f, -0.0f}) {
        float s, c, o;
        if (!sincos_rounded(z, 0.0f, 0.0f, s, c) || !same(s, z) || c != 1.0f) ++wrong;
        if (!atan2_rounded(z, 0.5f, o) || !same(o, z)) ++wrong;
        if (!asin_rounded(z, o) || !same(o, z)) ++wrong;
    }
    for (float z : {INFINITY, -INFINITY, NAN, 2e3f, -1e30f}) {
        float s, c, o;
        if (sincos_rounded(z, 0.0f, 0.0f, s, c) || atan2_rounded(z, 0.5f, o) || atan2_rounded(0.5f, z, o) ||
            asin_rounded(z, o)) ++wrong;
    }
    for (const Stat* s : {&tr, &sm, &big, &near, &at, &as, &lg, &nm}) report(*s);
    printf("wrong %ld 0 0\n", wrong);
    return wrong != 0;
}
