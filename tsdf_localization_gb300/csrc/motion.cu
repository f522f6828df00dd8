// Motion update on the device: ParticleCloud::apply_model
// (particle_cloud.cpp:499-617; the same loop body as motionUpdate(odom),
// :153-333).  Every particle draws six increments dx, dy, dz, roll, pitch,
// yaw, builds the odometry transform from them, rotates it by the particle's
// orientation and takes the translation and getAngleFromMat's angles
// (util.cpp:86-111) as its new pose; the weight is kept.
//
// Draws: the reference pulls them from one serial mt19937 through
// std::normal_distribution, a sequence no parallel generator reproduces.  Here
// each particle's six normals come from a counter-based generator instead:
// Philox4x64-10 (Salmon, Moraes, Dror, Shaw, "Parallel random numbers: as easy
// as 1, 2, 3", SC 2011) keyed by the seed, with the counter (particle index,
// block 0/1, step, 0), and Box-Muller pairs in FP64.  Callers that need the
// reference's own sequence draw it on the host and pass it in
// (tsdfl_motion_apply*): the pose composition is the reference's bit for bit.
//
// Arithmetic as the reference's x86-64 build does it: trig of the double draws
// in double rounded to float, trig of the float orientation through the
// double overloads, float products and sums with no contraction, float
// pitch re-used in double cos for roll and yaw.  The doubles are only ever rounded
// to float, so the kernel forms them as float pairs (pair_math.h) and evaluates
// the double functions where a pair leaves the rounding open.
#include <stdint.h>

#include <atomic>
#include <cmath>

#include "pair_math.h"
#include "philox.h"
#include "tsdfl_internal.h"

namespace tsdfl {

extern std::atomic<unsigned long long> g_launches;

namespace {

constexpr int kMotionBlock = 128;

struct MotionParams {
    float* particles;        // P x 7, updated in place
    uint32_t P;
    double mean[6], stddev[6];
    Pair mean2[6], stddev2[6];
    float low[6];            // normal_draw's
    int pairs;               // mean and stddev lie where pairs hold their digits
    unsigned long long key0, key1, step;
    const double* draws;     // P x 6 given draws, or null: generate
    double* draws_out;       // optional: the generated draws
};

// A standard normal pair from two 64-bit words: u1 in (0, 1], u2 in [0, 1),
// r = sqrt(-2 ln u1), (r cos 2 pi u2, r sin 2 pi u2).
__device__ __noinline__ double2 box_muller(unsigned long long a, unsigned long long b)
{
    const double u1 = ((double)(a >> 11) + 1.0) * 0x1.0p-53;
    const double u2 = (double)(b >> 11) * 0x1.0p-53;
    const double r = sqrt(-2.0 * log(u1));
    double s, c;
    sincospi(2.0 * u2, &s, &c);
    return make_double2(r * c, r * s);
}

// Draw of axis k in double: given, or generated again from its two words.
__device__ __noinline__ double axis_draw(const MotionParams& mp, uint32_t i, int k, unsigned long long a,
                                         unsigned long long b)
{
    if (mp.draws) return mp.draws[6 * (size_t)i + k];
    const double2 z = box_muller(a, b);
    return __dadd_rn(__dmul_rn(k & 1 ? z.y : z.x, mp.stddev[k]), mp.mean[k]);
}

__device__ __noinline__ float2 sincos_double(double v) { return make_float2((float)sin(v), (float)cos(v)); }

// util.cpp:86-111 with the double overloads of fabs, atan2, asin and cos.
__device__ __noinline__ float3 angles_double(float m8, float m9, float m10, float m4, float m0)
{
    float roll, pitch, yaw;
    if (fabs((double)m8) >= 1.0) {
        yaw = 0.0f;
        const double delta = atan2((double)m9, (double)m10);
        pitch = m8 < 0.0f ? (float)(3.14159265358979323846 / 2.0) : (float)(-3.14159265358979323846 / 2.0);
        roll = (float)delta;
    } else {
        pitch = (float)(-asin((double)m8));
        const double cp = cos((double)pitch);
        roll = (float)atan2(__ddiv_rn((double)m9, cp), __ddiv_rn((double)m10, cp));
        yaw = (float)atan2(__ddiv_rn((double)m4, cp), __ddiv_rn((double)m0, cp));
    }
    return make_float3(roll, pitch, yaw);
}

// The quotients by the pitch's cosine (positive) change atan2 by less than the
// pairs' bound, so the pairs do without them.
__device__ __forceinline__ void angles_from_mat(const float* m, float& roll, float& pitch, float& yaw)
{
    float as;
    if (asin_rounded(m[8], as) && atan2_rounded(m[9], m[10], roll) && atan2_rounded(m[4], m[0], yaw)) {
        pitch = -as;
        return;
    }
    const float3 a = angles_double(m[8], m[9], m[10], m[4], m[0]);
    roll = a.x;
    pitch = a.y;
    yaw = a.z;
}

__device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }

// sincos_rounded() as a call, (sine, cosine, certain): six copies of it in line ran
// the instruction cache out (26.5 against 24.7 us for 100,000 particles; the other
// pair functions as calls change nothing).
__device__ __noinline__ float3 sincos_call(float x, float d, float bound)
{
    float s = 0.0f, c = 0.0f;
    const bool ok = sincos_rounded(x, d, bound, s, c);
    return make_float3(s, c, ok ? 1.0f : 0.0f);
}

// A draw, known to within `bound`; axis_draw() is its exact form.
struct Draw {
    Pair v;
    float bound;
};

__device__ __forceinline__ float draw_float(const MotionParams& mp, uint32_t i, int k, const Draw& d,
                                            unsigned long long a, unsigned long long b)
{
    if (d.v.h == 0.0f && d.bound == 0.0f) return d.v.h;   // the sign of a zero
    float f;
    if (!rounded(d.v, d.bound, f)) f = (float)axis_draw(mp, i, k, a, b);
    return f;
}

__device__ __forceinline__ void draw_sincos(const MotionParams& mp, uint32_t i, int k, const Draw& d,
                                            unsigned long long a, unsigned long long b, float& s, float& c)
{
    const float3 r = sincos_call(d.v.h, d.v.l, d.bound);
    s = r.x;
    c = r.y;
    if (r.z == 0.0f) {
        const float2 f = sincos_double(axis_draw(mp, i, k, a, b));
        s = f.x;
        c = f.y;
    }
}

__device__ __forceinline__ void float_sincos(float v, float& s, float& c)
{
    const float3 r = sincos_call(v, 0.0f, 0.0f);
    s = r.x;
    c = r.y;
    if (r.z == 0.0f) {
        const float2 f = sincos_double((double)v);
        s = f.x;
        c = f.y;
    }
}

// particle_cloud.cpp:530-614 for one particle, its draws d[6] and the words w[6]
// they were generated from.
__device__ __forceinline__ void compose(const MotionParams& mp, uint32_t i, float* p, const Draw d[6],
                                        const unsigned long long w[6])
{
    float sr, cr, sp, cp, sy, cy;
    draw_sincos(mp, i, 3, d[3], w[2], w[3], sr, cr);
    draw_sincos(mp, i, 4, d[4], w[4], w[5], sp, cp);
    draw_sincos(mp, i, 5, d[5], w[4], w[5], sy, cy);
    float o[12];
    o[0] = mul(cp, cy);
    o[4] = mul(cp, sy);
    o[8] = -sp;
    o[3] = draw_float(mp, i, 0, d[0], w[0], w[1]);
    o[1] = sub(mul(mul(sr, sp), cy), mul(cr, sy));
    o[5] = add(mul(mul(sr, sp), sy), mul(cr, cy));
    o[9] = mul(sr, cp);
    o[7] = draw_float(mp, i, 1, d[1], w[0], w[1]);
    o[2] = add(mul(mul(cr, sp), cy), mul(sr, sy));
    o[6] = sub(mul(mul(cr, sp), sy), mul(sr, cy));
    o[10] = mul(cr, cp);
    o[11] = draw_float(mp, i, 2, d[2], w[2], w[3]);

    float sa, ca, sb, cb, sg, cg;
    float_sincos(p[3], sa, ca);
    float_sincos(p[4], sb, cb);
    float_sincos(p[5], sg, cg);
    float q[12];
    q[0] = mul(cb, cg);
    q[4] = mul(cb, sg);
    q[8] = -sb;
    q[3] = 0.0f;
    q[1] = sub(mul(mul(sa, sb), cg), mul(ca, sg));
    q[5] = add(mul(mul(sa, sb), sg), mul(ca, cg));
    q[9] = mul(sa, cb);
    q[7] = 0.0f;
    q[2] = add(mul(mul(ca, sb), cg), mul(sa, sg));
    q[6] = sub(mul(mul(ca, sb), sg), mul(sa, cg));
    q[10] = mul(ca, cb);
    q[11] = 0.0f;

    float t[12];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        const float a0 = q[4 * r], a1 = q[4 * r + 1], a2 = q[4 * r + 2];
        t[4 * r] = add(add(mul(a0, o[0]), mul(a1, o[4])), mul(a2, o[8]));
        t[4 * r + 1] = add(add(mul(a0, o[1]), mul(a1, o[5])), mul(a2, o[9]));
        t[4 * r + 2] = add(add(mul(a0, o[2]), mul(a1, o[6])), mul(a2, o[10]));
        t[4 * r + 3] = add(add(add(mul(a0, o[3]), mul(a1, o[7])), mul(a2, o[11])), q[4 * r + 3]);
    }
    float m[16];
#pragma unroll
    for (int k = 0; k < 12; ++k) m[k] = t[k];
    float roll, pitch, yaw;
    angles_from_mat(m, roll, pitch, yaw);
    p[0] = add(p[0], t[3]);
    p[1] = add(p[1], t[7]);
    p[2] = add(p[2], t[11]);
    p[3] = roll;
    p[4] = pitch;
    p[5] = yaw;
}

// A given draw as a pair; a value that a pair would not hold to 2^-46 leaves every
// rounding to the double functions (a bound that is not a number).
__device__ __forceinline__ Draw given_draw(double v)
{
    const double a = fabs(v);
    if (a == 0.0) return {{(float)v, 0.0f}, 0.0f};
    if (!(a >= 1e-20 && a <= 1e10)) return {{0.0f, 0.0f}, __int_as_float(0x7fffffff)};
    const Pair p = from_double(v);
    return {p, fabsf(p.h) * 0x1p-46f};
}

// One particle a thread.  In double it was bound by the FP64 pipe (some 800 FP64
// instructions a particle, 16 cycles a warp each: 137 us for 100,000 particles).  In
// pairs 4,300 instructions a warp, three quarters of them FP32: 24.7 us, issue two
// thirds busy.  Blocks of 64, 128 and 256 threads take the same time.
__global__ void __launch_bounds__(kMotionBlock) motion_kernel(const __grid_constant__ MotionParams mp)
{
    const uint32_t i = blockIdx.x * kMotionBlock + threadIdx.x;
    if (i >= mp.P) return;
    Draw d[6];
    unsigned long long w[6] = {0, 0, 0, 0, 0, 0};
    if (!mp.draws) {
        unsigned long long c0[4] = {i, 0, mp.step, 0};
        unsigned long long c1[4] = {i, 1, mp.step, 0};
        philox4x64_10(c0, mp.key0, mp.key1);
        philox4x64_10(c1, mp.key0, mp.key1);
#pragma unroll
        for (int k = 0; k < 4; ++k) w[k] = c0[k];
        w[4] = c1[0];
        w[5] = c1[1];
    }
    if (mp.pairs && !mp.draws && !mp.draws_out) {
#pragma unroll
        for (int k = 0; k < 6; k += 2) {
            Pair z[2];
            const bool ok = normal_pairs(w[k], w[k + 1], z[0], z[1]);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                float bound;
                d[k + j].v = normal_draw(z[j], mp.stddev2[k + j], mp.mean2[k + j], mp.low[k + j], bound);
                d[k + j].bound = ok ? bound : __int_as_float(0x7fffffff);
            }
        }
    } else {
#pragma unroll
        for (int k = 0; k < 6; k += 2) {
            double v[2];
            if (mp.draws) {
                v[0] = mp.draws[6 * (size_t)i + k];
                v[1] = mp.draws[6 * (size_t)i + k + 1];
            } else {
                const double2 z = box_muller(w[k], w[k + 1]);
                v[0] = __dadd_rn(__dmul_rn(z.x, mp.stddev[k]), mp.mean[k]);
                v[1] = __dadd_rn(__dmul_rn(z.y, mp.stddev[k + 1]), mp.mean[k + 1]);
            }
            if (mp.draws_out) {
                mp.draws_out[6 * (size_t)i + k] = v[0];
                mp.draws_out[6 * (size_t)i + k + 1] = v[1];
            }
            d[k] = given_draw(v[0]);
            d[k + 1] = given_draw(v[1]);
        }
    }
    float p[7];
    float* src = mp.particles + 7 * (size_t)i;
#pragma unroll
    for (int k = 0; k < 7; ++k) p[k] = src[k];
    compose(mp, i, p, d, w);
#pragma unroll
    for (int k = 0; k < 6; ++k) src[k] = p[k];
}

// mcl_3d.cpp:433-449: a particle as geometry_msgs::Pose (position, then the
// orientation quaternion x, y, z, w of tf2::Quaternion::setRPY(roll, pitch,
// yaw): half angles, ZYX composition, in double).
__global__ void pose_array_kernel(const float* __restrict__ particles, uint32_t P, double* __restrict__ poses)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P) return;
    const float* p = particles + 7 * (size_t)i;
    double sr, cr, sp, cp, sy, cy;
    sincos(__dmul_rn((double)p[3], 0.5), &sr, &cr);
    sincos(__dmul_rn((double)p[4], 0.5), &sp, &cp);
    sincos(__dmul_rn((double)p[5], 0.5), &sy, &cy);
    double* o = poses + 7 * (size_t)i;
    o[0] = p[0];
    o[1] = p[1];
    o[2] = p[2];
    o[3] = __dsub_rn(__dmul_rn(__dmul_rn(sr, cp), cy), __dmul_rn(__dmul_rn(cr, sp), sy));
    o[4] = __dadd_rn(__dmul_rn(__dmul_rn(cr, sp), cy), __dmul_rn(__dmul_rn(sr, cp), sy));
    o[5] = __dsub_rn(__dmul_rn(__dmul_rn(cr, cp), sy), __dmul_rn(__dmul_rn(sr, sp), cy));
    o[6] = __dadd_rn(__dmul_rn(__dmul_rn(cr, cp), cy), __dmul_rn(__dmul_rn(sr, sp), sy));
}

int check(cudaError_t e) { return e == cudaSuccess ? TSDFL_OK : TSDFL_ERR_DEVICE; }

}  // namespace

int launch_pose_array(const float* particles, size_t P, double* poses, cudaStream_t s)
{
    if (P == 0) return TSDFL_OK;
    pose_array_kernel<<<(unsigned)((P + 255) / 256), 256, 0, s>>>(particles, (uint32_t)P, poses);
    g_launches += 1;
    return check(cudaGetLastError());
}

int launch_motion(float* particles, size_t P, const double mean[6], const double stddev[6], uint64_t seed,
                  uint64_t step, const double* draws, double* draws_out, cudaStream_t s)
{
    if (P == 0) return TSDFL_OK;
    MotionParams mp{};
    mp.particles = particles;
    mp.P = (uint32_t)P;
    mp.pairs = 1;
    for (int k = 0; k < 6; ++k) {
        mp.mean[k] = mean ? mean[k] : 0.0;
        mp.stddev[k] = stddev ? stddev[k] : 0.0;
        for (const double v : {mp.mean[k], mp.stddev[k]})
            if (!(v == 0.0 ? !std::signbit(v) : std::fabs(v) >= 1e-20 && std::fabs(v) <= 1e10)) mp.pairs = 0;
        if (mp.pairs) {
            mp.mean2[k] = from_double(mp.mean[k]);
            mp.stddev2[k] = from_double(mp.stddev[k]);
            mp.low[k] = mp.stddev[k] != 0.0 ? kDrawLow : 0.0f;
        }
    }
    mp.key0 = seed;
    mp.key1 = kStreamMotion;
    mp.step = step;
    mp.draws = draws;
    mp.draws_out = draws_out;
    motion_kernel<<<(unsigned)((P + kMotionBlock - 1) / kMotionBlock), kMotionBlock, 0, s>>>(mp);
    g_launches += 1;
    return check(cudaGetLastError());
}

}  // namespace tsdfl
