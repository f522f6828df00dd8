// Float-pair arithmetic: values as the unevaluated sum of two floats (about 46
// bits), for trigonometry whose results are rounded to float.
//
// GB300 issues one FP64 instruction a warp every 16 cycles, an FP32 one every
// quarter cycle, so a double sine (some 30 FP64 instructions) costs what 2,000
// float instructions do; the pair form below takes about 100.  Results stay those
// of "double function, rounded to float" bit for bit: a pair is rounded only when
// every value within its error bound rounds to the same float (rounded()); for
// the rest, about one in 2^16, the caller evaluates the double function.  The
// double function's own error (about 2^-52) is far inside the bound.
//
// Pair sums and products: Dekker, "A floating-point technique for extending the
// available precision", 1971, with fused multiply-adds for the products' errors;
// the series are Taylor's (coefficients 1/n! and 1/n rounded to pairs).  Compiled
// without contraction on both sides (fmaf is explicit).
#pragma once
#include <math.h>
#include <stdint.h>

#ifdef __CUDACC__
#define PAIR_FN __host__ __device__ __forceinline__
#else
#define PAIR_FN inline
#endif

namespace tsdfl {

struct Pair {
    float h, l;
};

PAIR_FN Pair quick_sum(float a, float b)   // |a| >= |b|, or a == 0
{
    const float s = a + b;
    return {s, b - (s - a)};
}
PAIR_FN Pair two_sum(float a, float b)
{
    const float s = a + b, t = s - a;
    return {s, (a - (s - t)) + (b - t)};
}
PAIR_FN Pair two_prod(float a, float b)
{
    const float p = a * b;
    return {p, fmaf(a, b, -p)};
}
PAIR_FN Pair neg(Pair a) { return {-a.h, -a.l}; }
PAIR_FN Pair mul(Pair a, Pair b)
{
    const Pair p = two_prod(a.h, b.h);
    return quick_sum(p.h, p.l + fmaf(a.h, b.l, a.l * b.h));
}
PAIR_FN Pair mul(Pair a, float b)
{
    const Pair p = two_prod(a.h, b);
    return quick_sum(p.h, fmaf(a.l, b, p.l));
}
PAIR_FN Pair add(Pair a, Pair b)   // error about 2^-46 (|a| + |b|)
{
    const Pair s = two_sum(a.h, b.h);
    return quick_sum(s.h, s.l + (a.l + b.l));
}
PAIR_FN Pair quick_add(Pair a, Pair b)   // |a| >= |b|
{
    const Pair s = quick_sum(a.h, b.h);
    return quick_sum(s.h, s.l + (a.l + b.l));
}
PAIR_FN Pair div(Pair a, Pair b)
{
    const float r = 1.0f / b.h, q = a.h * r;
    const float rem = fmaf(-q, b.l, fmaf(-q, b.h, a.h) + a.l);
    return quick_sum(q, rem * r);
}
PAIR_FN Pair root(Pair a)   // a > 0
{
    const float q = sqrtf(a.h);
    return quick_sum(q, (fmaf(-q, q, a.h) + a.l) * (0.5f / q));
}
PAIR_FN Pair from_double(double v)   // |v| in float's normal range, or 0
{
    const float h = (float)v;
    return {h, (float)(v - (double)h)};
}

PAIR_FN float power_of_two(int e)   // -126 <= e <= 127
{
#ifdef __CUDA_ARCH__
    return __int_as_float((127 + e) << 23);
#else
    return ldexpf(1.0f, e);
#endif
}
PAIR_FN int leading_zeros(uint64_t v)   // v > 0
{
#ifdef __CUDA_ARCH__
    return __clzll((long long)v);
#else
    return __builtin_clzll(v);
#endif
}

// v 2^e of an integer |v| <= 2^53, to a relative 2^-48.
PAIR_FN Pair from_int(int64_t v, int e)
{
    const uint64_t a = (uint64_t)(v < 0 ? -v : v);
    if (a == 0) return {0.0f, 0.0f};
    const int sh = leading_zeros(a);
    const uint64_t b = a << sh;
    const float f = v < 0 ? -power_of_two(40 - sh + e) : power_of_two(40 - sh + e);
    return quick_sum((float)(uint32_t)(b >> 40) * f, (float)(uint32_t)(b >> 8) * (f * 0x1p-32f));
}

// The float that every value within `bound` of a rounds to; false when there is
// none such.
PAIR_FN bool rounded(Pair a, float bound, float& out)
{
    const float lo = a.h + (a.l - bound);
    out = a.h + (a.l + bound);
    return lo == out;
}

// Sine and cosine of |r| <= 0.8, each to a relative 2^-43.
PAIR_FN void sincos_reduced(Pair r, Pair& s, Pair& c)
{
    const Pair z = mul(r, r);
    float p = fmaf(z.h, fmaf(z.h, -0x1.ae7f3ep-41f, 0x1.612462p-33f), -0x1.ae6456p-26f);
    p = fmaf(z.h, p, 0x1.71de3ap-19f);
    Pair t = quick_add({-0x1.a01a02p-13f, 0x1.7f97fap-39f}, {z.h * p, 0.0f});
    t = quick_add({0x1.111112p-7f, -0x1.dddddep-32f}, mul(z, t));
    t = quick_add({-0x1.555556p-3f, 0x1.555556p-28f}, mul(z, t));
    s = quick_add(r, mul(r, mul(z, t)));
    p = fmaf(z.h, fmaf(z.h, 0x1.ae7f3ep-45f, -0x1.93974ap-37f), 0x1.1eed8ep-29f);
    p = fmaf(z.h, p, -0x1.27e4fcp-22f);
    t = quick_add({0x1.a01a02p-16f, -0x1.7f97fap-42f}, {z.h * p, 0.0f});
    t = quick_add({-0x1.6c16c2p-10f, 0x1.27d27ep-35f}, mul(z, t));
    t = quick_add({0x1.555556p-5f, -0x1.555556p-30f}, mul(z, t));
    t = quick_add({-0.5f, 0.0f}, mul(z, t));
    c = quick_add({1.0f, 0.0f}, mul(z, t));
}

// Sine and cosine from those of the angle less q quarter turns.
PAIR_FN void turn(int q, Pair& s, Pair& c)
{
    if (q & 1) {
        const Pair t = s;
        s = c;
        c = neg(t);
    }
    if (q & 2) {
        s = neg(s);
        c = neg(c);
    }
}

// Sine and cosine of x + d, |x| <= kPairAngle, |d| <= 2^-20 |x|; each to a relative
// 2^-42.5 (the worst near the zeros).
constexpr float kPairAngle = 64.0f;
PAIR_FN void sincos_pair(float x, float d, Pair& s, Pair& c)
{
    const float k = rintf(x * 0x1.45f306p-1f);
    // k pi/2 in three parts; the leading difference is exact
    const Pair a = two_prod(k, 0x1.921fb6p+0f), b = two_prod(k, -0x1.777a5cp-25f);
    Pair r = two_sum(x - a.h, -a.l);
    r = add(r, {-b.h, -b.l});
    r = add(r, {d, -(k * -0x1.ee59dap-50f)});
    sincos_reduced(r, s, c);
    turn((int)k, s, c);
}

// The floats nearest to the sine and cosine of the angle x + d, d known to within
// `bound`; false when one is not certain.
constexpr float kPairRel = 0x1p-41f;
PAIR_FN bool sincos_rounded(float x, float d, float bound, float& s, float& c)
{
    if (!(fabsf(x) <= kPairAngle)) return false;
    Pair ps, pc;
    sincos_pair(x, d, ps, pc);
    const bool a = rounded(ps, fmaf(fabsf(ps.h), kPairRel, bound), s);
    const bool b = rounded(pc, fmaf(fabsf(pc.h), kPairRel, bound), c);
    if (x == 0.0f && d == 0.0f) s = x;   // the sign of a zero
    return a && b;
}

// The float nearest to atan2(y, x); false when it is not certain.
PAIR_FN bool atan2_rounded(float y, float x, float& out)
{
    if (y == 0.0f && x > 0.0f) {
        out = y;
        return true;
    }
    const float ay = fabsf(y), ax = fabsf(x);
    if (!(ay >= 0x1p-40f && ax >= 0x1p-40f && ay <= 2.0f && ax <= 2.0f)) return false;
    const float t = atan2f(y, x);
    Pair s, c;
    sincos_pair(t, 0.0f, s, c);
    // the angle from (c, s) to (x, y), below 2^-20
    const Pair num = add(mul(c, y), neg(mul(s, x)));
    const float den = fmaf(x, c.h, y * s.h);
    return rounded({t, num.h / den}, fabsf(t) * kPairRel, out);
}

// The float nearest to asin(v); false when it is not certain.
PAIR_FN bool asin_rounded(float v, float& out)
{
    if (v == 0.0f) {
        out = v;
        return true;
    }
    const float a = fabsf(v);
    if (!(a >= 0x1p-40f && a <= 0.99f)) return false;
    const float t = asinf(v);
    Pair s, c;
    sincos_pair(t, 0.0f, s, c);
    const Pair num = add({v, 0.0f}, neg(s));
    const float d = num.h / c.h;
    // sin(t + d) = s + c d - s d^2 / 2
    return rounded({t, fmaf(0.5f * d * d, s.h / c.h, d)}, fabsf(t) * kPairRel, out);
}

// -ln(m 2^-53) of an integer 0 < m < 2^53, to a relative 2^-42.
PAIR_FN Pair minus_log(uint64_t m)
{
    const int up = leading_zeros(m) - 11;        // 0..52: m 2^up in [2^52, 2^53)
    const uint64_t f = m << up;
    const bool half = f > 6369051672525773ull;   // beyond sqrt(2): as f / 2 and one more
    const Pair t = half ? from_int((int64_t)f - (int64_t)(1ull << 53), -53)
                        : from_int((int64_t)f - (int64_t)(1ull << 52), -52);
    const float e = (float)(half ? -up : -up - 1);
    // ln(1 + t) = 2 atanh(t / (2 + t))
    const Pair s = div(t, quick_add({2.0f, 0.0f}, t));
    const Pair w = mul(s, s);
    float p = fmaf(w.h, 0x1.e1e1e2p-5f, 0x1.111112p-4f);
    p = fmaf(w.h, p, 0x1.3b13b2p-4f);
    p = fmaf(w.h, p, 0x1.745d18p-4f);
    p = fmaf(w.h, p, 0x1.c71c72p-4f);
    Pair q = quick_add({0x1.24924ap-3f, -0x1.b6db6ep-28f}, {w.h * p, 0.0f});
    q = quick_add({0x1.99999ap-3f, -0x1.99999ap-29f}, mul(w, q));
    q = quick_add({0x1.555556p-2f, -0x1.555556p-27f}, mul(w, q));
    q = mul(quick_add(s, mul(s, mul(w, q))), 2.0f);
    return neg(add(mul({0x1.62e43p-1f, -0x1.05c61p-29f}, e), q));
}

// Two standard normals from two 64-bit words (Box-Muller: u1 = ((a >> 11) + 1)
// 2^-53, u2 = (b >> 11) 2^-53, sqrt(-2 ln u1) (cos, sin)(2 pi u2)), each to a
// relative 2^-41; false for the few words where one is 0.
PAIR_FN bool normal_pairs(uint64_t a, uint64_t b, Pair& z0, Pair& z1)
{
    const uint64_t m = (a >> 11) + 1, n = b >> 11;
    const int q = (int)((n + (1ull << 50)) >> 51);   // quarter turns
    const int64_t t = (int64_t)(n - ((uint64_t)q << 51));
    if (m >= (1ull << 53) || t == 0) return false;
    const Pair r = root(mul(minus_log(m), 2.0f));
    Pair s, c;
    sincos_reduced(mul({0x1.921fb6p+0f, -0x1.777a5cp-25f}, from_int(t, -51)), s, c);
    turn(q, s, c);
    z0 = mul(r, c);
    z1 = mul(r, s);
    return true;
}

// The draw z stddev + mean of a normal z (normal_pairs), and the bound it is known to.
// `low` is kDrawLow for a stddev above 0, else 0: where z stddev is tiny the products'
// low parts leave the normal range, and the relative part of the bound with them.  The
// parts lost there are a few units of 2^-149; from 2^-75 up kDrawLow adds nothing.
constexpr float kDrawLow = 0x1p-120f;
PAIR_FN Pair normal_draw(Pair z, Pair stddev, Pair mean, float low, float& bound)
{
    const Pair n = mul(z, stddev);
    bound = fmaf(fabsf(n.h) + fabsf(mean.h), kPairRel, low);
    return add(n, mean);
}

}  // namespace tsdfl
