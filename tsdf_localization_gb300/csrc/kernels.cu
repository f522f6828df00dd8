// Sensor-update kernels for sm_103a: pose build, scan staging, per-particle
// scoring, normalisation / mean pose, systematic resampling, map re-layout.
#include <cooperative_groups.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>
#include <utility>
#include <vector>

#include "chain.h"
#include "index_math.h"
#include "pair_math.h"
#include "subsample.h"
#include "tsdfl_internal.h"

namespace tsdfl {

namespace cg = cooperative_groups;

std::atomic<unsigned long long> g_launches{0};

namespace {

constexpr int kLutBytes = ((kNumCodes * 8 + 15) / 16) * 16;
constexpr int kLutFBytes = ((kNumCodes * 4 + 15) / 16) * 16;
static_assert(kLutBytes + 12 * kMaxPassPoints <= kMaxDynamicSmem, "eval_exact_kernel's longest pass");

__device__ __forceinline__ uint32_t smem_u32(const void* p)
{
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

// After a thread's last plain accesses to shared memory that a bulk copy will write
// next, before the barrier in front of that copy: bulk copies go another way into
// shared memory (the async proxy), and a barrier alone does not order the two.
__device__ __forceinline__ void before_bulk_reuse()
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// 1-D bulk copy global -> this CTA's shared memory, completing on bar
// (cp.async.bulk; src, dst 16-byte aligned, bytes a multiple of 16).
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar)
{
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t phase)
{
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(phase)
        : "memory");
    return ok != 0;
}

// Bounded wait: gives up after ~2^22 polls (try_wait itself suspends for a
// while each time), so a copy that never lands cannot hang the GPU.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t phase)
{
    for (uint32_t i = 0; i < (1u << 22); ++i)
        if (mbar_try_wait(bar, phase)) return true;
    return false;
}

// Stages n floats of three arrays into shared memory with bulk copies; every
// thread of the block must call it.  Returns false (and raises status) when
// the copies did not complete in time.
__device__ bool stage_xyz(float* xs, float* ys, float* zs, const float* gx, const float* gy, const float* gz,
                          int npad, uint64_t* bar, int32_t* status)
{
    if (threadIdx.x == 0) mbar_init(bar, 1);
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t bytes = (uint32_t)npad * 4u;
        mbar_expect_tx(bar, 3u * bytes);
        bulk_g2s(xs, gx, bytes, bar);
        bulk_g2s(ys, gy, bytes, bar);
        bulk_g2s(zs, gz, bytes, bar);
    }
    bool ok = mbar_wait_bounded(bar, 0);
    if (!ok) ok = mbar_wait_bounded(bar, 0);   // give copies in flight a second bound
    if (!ok && threadIdx.x == 0) atomicExch(status, TSDFL_ERR_TIMEOUT);
    return __syncthreads_and(ok ? 1 : 0) != 0;
}

__device__ __forceinline__ long long warp_sum_ll(long long v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ uint32_t warp_sum_u32(uint32_t v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Element-wise min (x, y) / max (z, w) over the warp; NaN entries are ignored.
__device__ __forceinline__ float4 warp_extent(float4 e)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        e.x = fminf(e.x, __shfl_xor_sync(0xffffffffu, e.x, o));
        e.y = fminf(e.y, __shfl_xor_sync(0xffffffffu, e.y, o));
        e.z = fmaxf(e.z, __shfl_xor_sync(0xffffffffu, e.z, o));
        e.w = fmaxf(e.w, __shfl_xor_sync(0xffffffffu, e.w, o));
    }
    return e;
}

__device__ __forceinline__ double warp_sum_d(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Code of the slot a point falls in (kCodeMiss when getIndex misses): the
// generic kernel's view of a map with the compact layout, read through the
// brick table.
__device__ __forceinline__ uint32_t dense_code(const MapView& m, float x, float y, float z)
{
    uint32_t idx = slot_index(m, x, y, z);
    return idx == kMissIndex ? (uint32_t)kCodeMiss : (uint32_t)__ldg(m.codes + idx);
}

struct PointParams {
    const float* points;  // N x 3
    int N, npad, npairs;
    const float* particles;  // P x 7 (the cloud's extent is taken from a sample)
    int P;
    float max_range_sq, c_in, c_out;
    const float* code_values;  // kNumCodes floats (device)
    int shift;                 // fixed-point scale 2^shift
    int order;                 // a spread cloud's particles will be put in spatial order
    int pose_warps;            // warps of a pose block that work
};

// Spatial order of the pair layout: the tiled kernels walk the scan in chunks
// of consecutive points with every particle at once, so the order decides how
// much of the map a chunk touches across the cloud; exact fixed-point sums make
// the result independent of it.  A compact cloud (tracking) gathers least with
// chunks that are compact in the sensor frame: azimuth sector, then range band
// (0.5 m).  A cloud spread over the map (global localisation, any yaw) gathers
// least with chunks of one height band (1 m), whose hits stay in one layer of
// the map whatever the particle's position and yaw: height, sector, then range
// band (2 m).  The cloud counts as spread when its x or y extent exceeds
// kWideCloud.
constexpr int kSortSectors = 16;
constexpr int kSortBins = 2048;
constexpr float kWideCloud = 10.0f;   // metres
constexpr int kPrepThreads = 1024;
constexpr int kPrepBlocks = 8;      // one cluster
constexpr int kBinCache = 16384;    // points whose bin the staging keeps in shared memory
static_assert(kSortBins == 2 * kPrepThreads, "two bins per thread in the scan");

// Sector of the diamond angle (|y| / (|x| + |y|) per quadrant, counter-clockwise
// from +x: monotone in the azimuth, no trigonometry), with the range band and,
// for a spread cloud, the height band.
__device__ __forceinline__ int spatial_bin(float x, float y, float z, bool wide)
{
    const float r1 = fabsf(x) + fabsf(y);
    if (!(r1 < 1e30f) || !(fabsf(z) < 1e30f)) return kSortBins - 1;   // NaN / huge: last
    const float t = r1 > 0.0f ? __fdividef(fabsf(y), r1) : 0.0f;
    const float a = x >= 0.0f ? (y >= 0.0f ? t : 4.0f - t) : (y >= 0.0f ? 2.0f - t : 2.0f + t);   // [0, 4]
    const int s = min((int)(a * (0.25f * kSortSectors)), kSortSectors - 1);
    const float r = sqrtf(x * x + y * y);
    if (!wide) return s * 128 + (int)fminf(r * 2.0f, 127.0f);   // 16 sectors x 128 bands of 0.5 m
    const int zb = (int)fminf(fmaxf(floorf(z) + 4.0f, 0.0f), 7.0f);   // [-4, 4) m in 1 m bands
    return (zb * 16 + (int)fminf(r * 0.5f, 15.0f)) * kSortSectors + s;   // x 16 bands of 2 m x 16 sectors
}

// Scan staging: AoS points -> SoA (padded with zeros to npad), the per-point
// score constant of tsdf_evaluator.cpp:56-65 and the number of points inside
// max_range; the pair layout of the tiled kernels in spatial order (a counting
// sort by spatial_bin; perm records each position's scan index); also the
// likelihood tables for this scan.  The first cluster of pose_prepare_kernel, beside
// the pose blocks: each of its kPrepBlocks blocks counts and places a slice of the
// scan, and reads the others' counts from their shared memory.  Bound by the
// scattered 4-byte stores of the pair layout, one tag a lane, so one block took
// 29 us for 16,384 points and 11 for 2,048 (a cloud update of 2,000 particles 230 us
// a pass, 219 with the cluster; an update and resampling of 1,000 x 2,048 55.9 and
// 54.1).  Which order suits the cloud (compact or spread) is decided on
// the x / y extent of a sample of at most kExtentSample particles, and the
// particle order's cells span that extent (clamped at its edges); both only
// decide how fast the scoring runs, never what it returns.
constexpr int kExtentSample = 4096;

__device__ __forceinline__ void prepare_points_block(const PointParams& p, const EvalBuffers& b, int rank)
{
    __shared__ int warp_counts[32];
    __shared__ int2 bins[kPrepThreads];      // this slice's points a bin, two bins a thread
    __shared__ int places[kSortBins];        // the next position of a bin's points of this slice
    __shared__ uint16_t sbin[kBinCache];
    __shared__ float4 s_ext[32];
    __shared__ int s_wide, s_in;
    cg::cluster_group cluster = cg::this_cluster();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int slice = ((p.npad + kPrepBlocks - 1) / kPrepBlocks + 31) & ~31;
    const int j0 = (int)min((long long)rank * slice, (long long)p.npad);
    const int jpad = min(p.npad - j0, slice) + j0, j1 = min(jpad, p.N);
    if (rank == 0 && threadIdx.x == 0) *b.status = 0;
    if (rank == 0 && p.order)
        for (int c = threadIdx.x; c < kCellBins; c += blockDim.x) b.phist[c] = 0;   // the particle order's histogram
    {   // the cloud's x / y extent from a sample of the particles
        const float inf = __int_as_float(0x7f800000);
        float4 e = make_float4(inf, inf, -inf, -inf);
        const int n_s = min(p.P, kExtentSample), stride = max(1, p.P / kExtentSample);
        for (int k = threadIdx.x; k < n_s; k += blockDim.x) {
            const float* q = p.particles + 7 * (size_t)k * (size_t)stride;
            const float x = q[0], y = q[1];
            e = make_float4(fminf(e.x, x), fminf(e.y, y), fmaxf(e.z, x), fmaxf(e.w, y));
        }
        e = warp_extent(e);
        if (lane == 0) s_ext[warp] = e;
        if (threadIdx.x == 0) s_in = 0;
        __syncthreads();
        if (warp == 0) e = warp_extent(s_ext[lane]);
        if (threadIdx.x == 0) {
            s_wide = fmaxf(e.z - e.x, e.w - e.y) > kWideCloud ? 1 : 0;   // no particles: -inf
            if (rank == 0) {
                b.counts[2] = p.order ? s_wide : 0;   // the particles are put in spatial order too
                for (int k = 0; k < kWorkWords; ++k) b.work[k] = 0u;
                b.cloud_ext[0] = e;
            }
        }
    }
    bins[threadIdx.x] = make_int2(0, 0);
    __syncthreads();
    const bool wide = s_wide != 0;
    int in = 0;
    for (int j = j0 + (int)threadIdx.x; j < jpad; j += blockDim.x) {
        float x = 0, y = 0, z = 0, c = 0;
        if (j < p.N) {
            x = __ldg(p.points + 3 * j);
            y = __ldg(p.points + 3 * j + 1);
            z = __ldg(p.points + 3 * j + 2);
            float sq = __fadd_rn(__fadd_rn(__fmul_rn(x, x), __fmul_rn(y, y)), __fmul_rn(z, z));
            bool inr = sq < p.max_range_sq;
            c = inr ? p.c_in : p.c_out;
            in += inr ? 1 : 0;
            const int bin = spatial_bin(x, y, z, wide);
            atomicAdd(&reinterpret_cast<int*>(bins)[bin], 1);
            if (j - j0 < kBinCache) sbin[j - j0] = (uint16_t)bin;
        }
        ((float*)b.xs)[j] = x;
        ((float*)b.ys)[j] = y;
        ((float*)b.zs)[j] = z;
        ((float*)b.cs)[j] = c;
    }
    in = (int)warp_sum_u32((uint32_t)in);
    if (lane == 0 && in) atomicAdd(&s_in, in);
    cluster.sync();   // every slice's counts are complete
    {   // exclusive scan of the bins' counts, and within a bin of the slices'
        int c0 = 0, c1 = 0, b0 = 0, b1 = 0, n_in = 0;
#pragma unroll
        for (int r = 0; r < kPrepBlocks; ++r) {
            const int2 c = *cluster.map_shared_rank(&bins[threadIdx.x], r);
            b0 += r < rank ? c.x : 0;
            b1 += r < rank ? c.y : 0;
            c0 += c.x;
            c1 += c.y;
        }
        if (rank == 0 && threadIdx.x < kPrepBlocks) n_in = *cluster.map_shared_rank(&s_in, threadIdx.x);
        if (rank == 0 && warp == 0) {
            n_in = (int)warp_sum_u32((uint32_t)n_in);
            if (lane == 0) b.counts[0] = n_in;
        }
        int v = c0 + c1;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += t;
        }
        if (lane == 31) warp_counts[warp] = v;
        __syncthreads();
        if (warp == 0) {
            int w = warp_counts[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, w, o);
                if (lane >= o) w += t;
            }
            warp_counts[lane] = w;   // inclusive over warps
        }
        __syncthreads();
        const int before = (warp ? warp_counts[warp - 1] : 0) + v - c0 - c1;
        places[2 * threadIdx.x] = before + b0;
        places[2 * threadIdx.x + 1] = before + c0 + b1;
    }
    __syncthreads();
    cg::cluster_group::arrival_token done = cluster.barrier_arrive();   // the other blocks' memory has been read
    // pair layout of the fast kernel: in every block of 64 positions, lane l of
    // a warp takes positions 64*blk + l and 64*blk + 32 + l
    for (int j = j0 + (int)threadIdx.x; j < j1; j += blockDim.x) {
        const float x = __ldg(p.points + 3 * j), y = __ldg(p.points + 3 * j + 1), z = __ldg(p.points + 3 * j + 2);
        const int q = atomicAdd(&places[j - j0 < kBinCache ? (int)sbin[j - j0] : spatial_bin(x, y, z, wide)], 1);
        const int pair = (q >> 6) * 32 + (q & 31), half = (q >> 5) & 1;
        float* xy = reinterpret_cast<float*>(b.pxy + pair);
        xy[half] = x;
        xy[2 + half] = y;
        reinterpret_cast<float*>(b.pz + pair)[half] = z;
        b.perm[q] = j;
    }
    const int at = rank * (int)blockDim.x + (int)threadIdx.x, step = kPrepBlocks * (int)blockDim.x;
    for (int q = p.N + at; q < 2 * p.npairs; q += step) {   // padding positions
        const int pair = (q >> 6) * 32 + (q & 31), half = (q >> 5) & 1;
        float* xy = reinterpret_cast<float*>(b.pxy + pair);
        xy[half] = 0.0f;
        xy[2 + half] = 0.0f;
        reinterpret_cast<float*>(b.pz + pair)[half] = 0.0f;
        b.perm[q] = 0;   // never read: padding lanes record no debug code
    }
    if (rank == kPrepBlocks - 1)
        for (int c = threadIdx.x; c < kNumCodes; c += blockDim.x) {
            float v = p.code_values[c];
            b.lut_f[c] = v;
            b.lut_fx[c] = __double2ll_rn(ldexp((double)v, p.shift));
        }
    cluster.barrier_wait(std::move(done));   // no block leaves while its counts may be read
}

// Spatial order of a spread cloud's particles (global localisation): 64 x 64
// cells over the particles' x / y extent, numbered along a Morton curve; a
// counting sort puts the particles in cell order.  The tiled kernel then walks
// regions of consecutive particles, so that at any time the grid scores
// particles from one part of the map and the gathers stay in the L2.  The
// order within a cell depends on the atomics, which changes nothing: every
// particle's sums are exact integers written to its own index.
constexpr int kCellScanThreads = 1024;
static_assert(kCellBins == 4 * kCellScanThreads, "four bins per thread in the scan");

__device__ __forceinline__ uint32_t morton2(uint32_t x, uint32_t y)
{
    uint32_t m = 0;
#pragma unroll
    for (int k = 0; k < kCellBits; ++k) m |= (((x >> k) & 1u) << (2 * k)) | (((y >> k) & 1u) << (2 * k + 1));
    return m;
}

__global__ void particle_cells_kernel(const float* particles, int P, EvalBuffers b)
{
    chain_enter();
    if (b.counts[2] == 0) return;   // a compact cloud keeps its order
    const float4 e = b.cloud_ext[0];
    const float n = (float)(1 << kCellBits);
    const float sx = n / fmaxf(e.z - e.x, 1e-3f), sy = n / fmaxf(e.w - e.y, 1e-3f);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < P; i += gridDim.x * blockDim.x) {
        const float x = particles[7 * (size_t)i], y = particles[7 * (size_t)i + 1];
        // fmaxf / fminf also send NaN positions to cell 0
        const uint32_t cx = (uint32_t)fminf(fmaxf((x - e.x) * sx, 0.0f), n - 1.0f);
        const uint32_t cy = (uint32_t)fminf(fmaxf((y - e.y) * sy, 0.0f), n - 1.0f);
        const uint32_t key = morton2(cx, cy);
        b.pkeys[i] = key;
        atomicAdd(&b.phist[key], 1);
    }
}

__global__ void __launch_bounds__(kCellScanThreads) particle_scan_kernel(EvalBuffers b)
{
    chain_enter();
    if (b.counts[2] == 0) return;
    __shared__ int warp_sums[kCellScanThreads / 32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    int c[4], v = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        c[k] = b.phist[4 * t + k];
        v += c[k];
    }
    int incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
    }
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        int w = warp_sums[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += u;
        }
        warp_sums[lane] = w;   // inclusive over warps
    }
    __syncthreads();
    int run = (warp ? warp_sums[warp - 1] : 0) + incl - v;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        b.phist[4 * t + k] = run;
        run += c[k];
    }
}

__global__ void particle_scatter_kernel(int P, EvalBuffers b)
{
    chain_enter();
    if (b.counts[2] == 0) return;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < P; i += gridDim.x * blockDim.x) {
        const int q = atomicAdd(&b.phist[b.pkeys[i]], 1);
        b.order[q] = (uint32_t)i;
    }
}

struct Tf16 {
    float v[16];
};

__device__ __noinline__ float2 sincos_double(float v)
{
    double s, c;
    sincos((double)v, &s, &c);
    return make_float2((float)s, (float)c);
}

// Laser pose of every particle (tsdf_evaluator.cpp:102-147): trig in double,
// rounded to float (formed in float pairs; the double functions only where a pair
// leaves the rounding open), products and sums in the
// reference's order without contraction.  Three lanes per particle, ten
// particles a warp (lanes 30 and 31 idle): lane 3p + k forms the sine and
// cosine of angle k (roll, pitch, yaw), the three exchange them by shuffles,
// and lane 3p + r forms row r of the 3 x 4 laser pose, so the latency of
// the three sincos is spread over three lanes.  Also zeros in the scoring
// sums, so no memset breaks the chain of kernels.  `blk` numbers the pose
// blocks of pose_prepare_kernel; of each, `warps` warps work (a small cloud is
// spread over the SMs, whose FP64 pipes are what it waits for).
__device__ __forceinline__ void pose_block(int blk, int warps, const float* particles, int P, const Tf16& tf,
                                           float* pose12, float* trig6, long long* sum_fx, uint32_t* hits)
{
    if ((int)(threadIdx.x >> 5) >= warps) return;
    const int lane = threadIdx.x & 31;
    const int slot = lane / 3, k = lane - 3 * slot;
    const int i = (blk * warps + (int)(threadIdx.x >> 5)) * kPoseSlots + slot;
    const bool active = slot < kPoseSlots && i < P;
    if (active && k == 0) {   // the tiled kernel's per-particle sums start at zero
        sum_fx[i] = 0;
        hits[i] = 0;
    }
    const float* p = particles + 7 * (size_t)(active ? i : 0);
    const float angle = p[3 + (k < 3 ? k : 0)];
    float sv, cv;
    if (!sincos_rounded(angle, 0.0f, 0.0f, sv, cv)) {
        const float2 v = sincos_double(angle);
        sv = v.x;
        cv = v.y;
    }
    const int base = 3 * slot;
    auto from = [&](float v, int j) { return __shfl_sync(0xffffffffu, v, min(base + j, 31)); };
    const float sin_alpha = from(sv, 0), cos_alpha = from(cv, 0);
    const float sin_beta = from(sv, 1), cos_beta = from(cv, 1);
    const float sin_gamma = from(sv, 2), cos_gamma = from(cv, 2);
    if (!active) return;
    float a[4];   // row k of the particle's transform
    if (k == 0) {
        a[0] = __fmul_rn(cos_beta, cos_gamma);
        a[1] = __fsub_rn(__fmul_rn(__fmul_rn(sin_alpha, sin_beta), cos_gamma), __fmul_rn(cos_alpha, sin_gamma));
        a[2] = __fadd_rn(__fmul_rn(__fmul_rn(cos_alpha, sin_beta), cos_gamma), __fmul_rn(sin_alpha, sin_gamma));
        a[3] = p[0];
    } else if (k == 1) {
        a[0] = __fmul_rn(cos_beta, sin_gamma);
        a[1] = __fadd_rn(__fmul_rn(__fmul_rn(sin_alpha, sin_beta), sin_gamma), __fmul_rn(cos_alpha, cos_gamma));
        a[2] = __fsub_rn(__fmul_rn(__fmul_rn(cos_alpha, sin_beta), sin_gamma), __fmul_rn(sin_alpha, cos_gamma));
        a[3] = p[1];
    } else {
        a[0] = -sin_beta;
        a[1] = __fmul_rn(sin_alpha, cos_beta);
        a[2] = __fmul_rn(cos_alpha, cos_beta);
        a[3] = p[2];
    }
    const float* f = tf.v;
    float o[4];
#pragma unroll
    for (int c = 0; c < 3; ++c)
        o[c] = __fadd_rn(__fadd_rn(__fmul_rn(a[0], f[c]), __fmul_rn(a[1], f[4 + c])), __fmul_rn(a[2], f[8 + c]));
    o[3] = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(a[0], f[3]), __fmul_rn(a[1], f[7])), __fmul_rn(a[2], f[11])), a[3]);
    reinterpret_cast<float4*>(pose12 + 12 * (size_t)i)[k] = make_float4(o[0], o[1], o[2], o[3]);
    float* tg = trig6 + 6 * (size_t)i;
    tg[2 * k] = sv;
    tg[2 * k + 1] = cv;
}

// First kernel of an update, in clusters of kPrepBlocks: the first cluster stages the
// scan (prepare_points_block), the others form the laser poses (pose_block); the two
// parts share no data, so they run side by side.
__global__ void __launch_bounds__(kPoseThreads) pose_prepare_kernel(Tf16 tf, PointParams p, EvalBuffers b)
{
    chain_enter();
    if (blockIdx.x < kPrepBlocks) prepare_points_block(p, b, (int)blockIdx.x);
    else pose_block((int)blockIdx.x - kPrepBlocks, p.pose_warps, p.particles, p.P, tf, b.pose12, b.trig6, b.sum_fx, b.hits);
}

struct EvalParams {
    MapView m;
    const float4* pxy;
    const float2* pz;
    const int32_t* perm;   // scan index of each pair-layout point (debug rows)
    const float* pose12;
    const float* xs;
    const float* ys;
    const float* zs;
    const float* cs;
    const long long* lut_fx;
    const float* lut_f;
    long long* sum_fx;   // exact mode, code storage
    double* sum_f64;     // exact mode, float storage
    float* raw;          // serial mode
    uint32_t* hits;
    uint32_t* dbg;       // optional: P x N_total slot index (brick) / code (dense)
    const uint32_t* order;   // spatial order of the particles (used when *sched != 0)
    const int32_t* sched;    // the staging kernel's spread-cloud flag (null: original order)
    int32_t* status;
    int P;
    int n0, n1;          // point range of this pass
    int n_total;
    int first_pass;
    float a_hit;
};

// Exact mode: one warp per particle, lanes stride over the scan (neighbouring
// lanes take neighbouring scan points, so their map gathers fall close
// together).  Likelihood values are summed in 64-bit fixed point, which is
// exact and independent of order; the weight is formed from the sum afterwards.
template <bool DENSE, int ST>
__global__ void __launch_bounds__(1024, 1) eval_exact_kernel(EvalParams p)
{
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ uint64_t bar;
    long long* lut = reinterpret_cast<long long*>(smem);
    const int n = p.n1 - p.n0;
    const int npad = (n + 3) & ~3;
    float* xs = reinterpret_cast<float*>(smem + kLutBytes);
    float* ys = xs + npad;
    float* zs = ys + npad;
    for (int c = threadIdx.x; c < kNumCodes; c += blockDim.x) lut[c] = p.lut_fx[c];
    if (!stage_xyz(xs, ys, zs, p.xs + p.n0, p.ys + p.n0, p.zs + p.n0, npad, &bar, p.status)) return;

    const int lane = threadIdx.x & 31;
    const int warps = (blockDim.x >> 5) * gridDim.x;
    const MapView& m = p.m;
    for (int pi = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); pi < p.P; pi += warps) {
        float t[12];
        const float4* src = reinterpret_cast<const float4*>(p.pose12 + 12 * (size_t)pi);
        float4 a = __ldg(src), b4 = __ldg(src + 1), c4 = __ldg(src + 2);
        t[0] = a.x; t[1] = a.y; t[2] = a.z; t[3] = a.w;
        t[4] = b4.x; t[5] = b4.y; t[6] = b4.z; t[7] = b4.w;
        t[8] = c4.x; t[9] = c4.y; t[10] = c4.z; t[11] = c4.w;
        long long acc = 0;
        double accd = 0.0;
        uint32_t h = 0;
        for (int j = lane; j < n; j += 32) {
            float tx, ty, tz;
            transform_point(t, xs[j], ys[j], zs[j], tx, ty, tz);
            if (DENSE) {
                uint32_t code = dense_code(m, tx, ty, tz);
                h += code != (uint32_t)kCodeMiss ? 1u : 0u;
                acc += lut[code];
                if (p.dbg) p.dbg[(size_t)pi * p.n_total + p.n0 + j] = code;
            } else {
                uint32_t idx = slot_index(m, tx, ty, tz);
                if (ST == 1) {
                    float v = idx != kMissIndex ? __ldg(m.data + idx) : m.init_value;
                    accd += (double)v;
                } else if (ST == 2) {
                    float v = idx != kMissIndex ? __half2float(__ushort_as_half(__ldg(m.h16 + idx))) : m.init_value;
                    accd += (double)v;
                } else {
                    uint32_t code = idx != kMissIndex ? (uint32_t)__ldg(m.codes + idx) : (uint32_t)kCodeInit;
                    acc += lut[code];
                }
                h += idx != kMissIndex ? 1u : 0u;
                if (p.dbg) p.dbg[(size_t)pi * p.n_total + p.n0 + j] = idx;
            }
        }
        h = warp_sum_u32(h);
        if (ST != 0) accd = warp_sum_d(accd);
        else acc = warp_sum_ll(acc);
        if (lane == 0) {
            if (ST != 0) p.sum_f64[pi] = p.first_pass ? accd : p.sum_f64[pi] + accd;
            else p.sum_fx[pi] = p.first_pass ? acc : p.sum_fx[pi] + acc;
            p.hits[pi] = p.first_pass ? h : p.hits[pi] + h;
        }
    }
}

// ---------------------------------------------------------------- tiled kernel

typedef unsigned long long f2_t;   // two floats in one 64-bit register pair

__device__ __forceinline__ f2_t pk(float a, float b)
{
    f2_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void upk(f2_t v, float& a, float& b)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
// Packed additions: ptxas fuses a packed multiply feeding a packed add into an
// FMA even with explicit .rn, so products that feed additions stay scalar
// (__fmul_rn is never contracted).  mul2 is used only where its product is the
// addend of an FMA, which no contraction can absorb.
__device__ __forceinline__ f2_t add2(f2_t a, f2_t b)
{
    f2_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2_t add2_rz(f2_t a, f2_t b)
{
    f2_t r;
    asm("add.rz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2_t sub2(f2_t a, f2_t b)
{
    f2_t r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2_t and2(f2_t a, f2_t b)
{
    f2_t r;
    asm("and.b64 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2_t mul2(f2_t a, f2_t b)
{
    f2_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2_t fma2_rn(f2_t a, f2_t b, f2_t c)
{
    f2_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f2_t fma2_rz(f2_t a, f2_t b, f2_t c)
{
    f2_t r;
    asm("fma.rz.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

__device__ __forceinline__ f2_t or2(f2_t a, f2_t b)
{
    f2_t r;
    asm("or.b64 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

constexpr uint32_t kMagic = 0x4B000000u;     // bits of 2^23

// Code of a point the fast path does not cover: finite offsets go through the
// signed second tier, NaN / infinite / huge ones through the 64-bit emulation.
__device__ __forceinline__ uint32_t slow_code(const MapView& m, float x, float y, float z)
{
    const float ox = __fsub_rn(x, m.min_x), oy = __fsub_rn(y, m.min_y), oz = __fsub_rn(z, m.min_z);
    uint32_t idx = slot_index_tier2(m, m.grid_occ, ox, oy, oz);
    if (idx == kIdxSlow) idx = slot_index_slow(m, x, y, z);
    return idx == kMissIndex ? (uint32_t)kCodeMiss : (uint32_t)__ldg(m.codes + idx);
}

// Likelihood table entry in shared memory: the fixed-point value of a code,
// plus 2^kHitShift when the code is a slot's (a hit), so that one 64-bit sum
// counts both.  The values' part is a signed number below 2^(kHitShift - 1) for
// up to kPackedLookups lookups, so unpack() takes the two apart exactly.  Entries 8
// bytes apart spread a warp's random reads over 16 bank pairs.
// Where the values leave no room for that (packs() in tsdfl_internal.h), the wide
// form of the kernels (PACKED false) has the values alone in the table and counts
// the hits by the codes, two instructions a lookup more (building, us, packed / wide:
// 20,000 x 2,048 162 / 164, 100,000 x 3,000 867 / 888, spread 200,000 x 1,024 1,263 /
// 1,274).
struct __align__(8) LutEntry {
    long long v;
};
constexpr int kLutTableBytes = ((kNumCodes * 8 + 15) / 16) * 16;
constexpr int kHitShift = 57;
constexpr int kPackedSteps = 16;   // steps of two lookups a lane between two unpackings
static_assert(4 * (kPackedSteps + 1) + 1 < kPackedLookups && kPackedLookups < 128,
              "a lane's own lookups (with a partial step) and its share of the deferred ones");

__device__ __forceinline__ void unpack(long long acc, long long& v, uint32_t& hits)
{
    v = (long long)((unsigned long long)acc << (64 - kHitShift)) >> (64 - kHitShift);
    hits = (uint32_t)((unsigned long long)(acc - v) >> kHitShift);
}

// A lookup's table entry into the lane's sum (packed: with its hit) and, wide, its
// hit into the lane's count.
template <bool PACKED>
__device__ __forceinline__ void take(const LutEntry* lut, uint32_t code, long long& acc, uint32_t& hits)
{
    acc += lut[code].v;
    if (!PACKED) hits += code <= (uint32_t)kCodeInit ? 1u : 0u;
}

// Moves a packed sum's parts to the lane's 64-bit sum and its hits.
template <bool PACKED>
__device__ __forceinline__ void flush(long long& acc, long long& sum, uint32_t& hits)
{
    if (PACKED) {
        long long v;
        uint32_t h;
        unpack(acc, v, h);
        sum += v;
        hits += h;
    } else {
        sum += acc;
    }
    acc = 0;
}

// Settles a lookup the fast path left open where that takes a few compares.
__device__ __forceinline__ void settle(const MapView& m, float x, float y, float z, bool& slow)
{
    if (slow && certain_miss(m, __fsub_rn(x, m.min_x), __fsub_rn(y, m.min_y), __fsub_rn(z, m.min_z))) slow = false;
}

// Branch-free fast path of one lookup, from the packed pipeline's outputs: the
// offsets' float bits (x, y) and value (z), upb = kMagic + brick index and
// slb = bits(1.5 * 2^23) + sub-voxel offset.  Returns the gathered code: the
// slot's, or kCodeMiss from the sentinel behind the slots.  `slow` is set when
// the offsets lie outside the fast domain ([0, mmax + 1) on x and y, (-1, mmax +
// 1) on z): the code is then kCodeMiss, which stands if settle() says so, and
// otherwise the exact slow tiers decide.
// Inside the fast domain the brick index needs no test where the rank's table
// covers every index it can take (the bitmap is zero-padded and the brick table
// -1-padded to that: brick_reach in map_host.h).
// LAY: where the brick's rank comes from -- kLayBitmap: the shared-memory
// bitmap `occ`; kLayHash: the sparse brick hash (allocated bricks only, for
// maps whose bitmap does not fit shared memory); kLayTable: the brick table
// grid_occ (the reference's own); kLayGrid: no rank, the grid layout's codes
// of every brick of the bounding box are addressed by the brick index.
constexpr int kLayTable = 0, kLayBitmap = 1, kLayHash = 2, kLayGrid = 3;

template <int LAY>
__device__ __forceinline__ uint32_t fast_code(const MapView& m, const unsigned char* occ, uint32_t ox_b,
                                              uint32_t oy_b, float oz, uint32_t upb, uint32_t slb, bool& slow)
{
    const bool fast = ox_b < m.lim_x && oy_b < m.lim_y && oz > m.zlo && oz < m.zhi;
    slow = !fast;
    uint32_t idx;
    bool ok;
    if (LAY == kLayHash) {
        // open addressing, linear probing: every key lies within hash_probes
        // slots of its home, and every run of keys ends at an empty slot within
        // that bound (measured when the table is built)
        const uint32_t up = upb - kMagic;
        uint32_t rank = 0;
        ok = false;
        if (fast) {
            const uint32_t h = (up * 0x9E3779B1u) >> m.hash_shift;
            for (uint32_t t = 0; t < m.hash_probes; ++t) {
                const uint2 e = __ldg(m.hash + ((h + t) & m.hash_mask));
                if (e.x == up) {
                    rank = e.y;
                    ok = true;
                    break;
                }
                if (e.x == kHashEmpty) break;
            }
        }
        idx = rank * m.sub_dim_3 + slb;
    } else if (LAY == kLayGrid) {
        // every brick of the bounding box is stored: a miss is a miss code there
        const uint32_t up = upb - kMagic;
        ok = fast && upb < m.upb_lim;
        idx = (up + min(up, m.grid_uxy1)) * m.sub_dim_3 + slb;
    } else if (LAY == kLayBitmap) {
        // the masked offset stays inside the staged table whatever upb is
        const uint2 wb = *reinterpret_cast<const uint2*>(occ + ((upb >> 2) & m.occ_mask));
        const uint32_t v = __funnelshift_r(wb.x, 0u, upb);   // word >> (brick & 31)
        ok = fast && (v & 1u) != 0u;
        idx = (wb.y - (uint32_t)__popc(v)) * m.sub_dim_3 + slb;
    } else {
        const int32_t base = __ldg(m.grid_occ + (fast ? upb - kMagic : 0u));
        ok = fast && base >= 0;
        idx = (uint32_t)base + slb;
    }
    if (LAY == kLayGrid)
        return __ldg(reinterpret_cast<const uint16_t*>(m.grid_b + 2ull * (ok ? idx : m.gsent_miss)));
    return __ldg(reinterpret_cast<const uint16_t*>(m.codes_b + 2ull * (ok ? idx : m.sent_miss)));
}

// Constants of the packed index pipeline, each a pair of equal floats.
struct PipeConsts {
    f2_t NMX, NMY, NMZ;       // the map's min corner
    f2_t MAG, MAG15;          // 2^23, 1.5 * 2^23
    f2_t INV, INVLO;          // sub-voxel multiplier terms
    f2_t UX, UXY, SD, SD2;    // up_dim_x, up_dim_x * up_dim_y, sub_dim, sub_dim^2
};

__device__ __forceinline__ PipeConsts pipe_consts(const MapView& m)
{
    PipeConsts c;
    c.NMX = pk(m.min_x, m.min_x);
    c.NMY = pk(m.min_y, m.min_y);
    c.NMZ = pk(m.min_z, m.min_z);
    c.MAG = pk(8388608.0f, 8388608.0f);
    c.MAG15 = pk(12582912.0f, 12582912.0f);
    c.INV = pk(m.sub_inv, m.sub_inv);
    c.INVLO = pk(m.sub_inv_lo, m.sub_inv_lo);
    c.UX = pk(m.up_dim_x_f, m.up_dim_x_f);
    c.UXY = pk(m.up_dim_2_f, m.up_dim_2_f);
    c.SD = pk(m.sub_dim_f, m.sub_dim_f);
    c.SD2 = pk(m.sub_dim_2_f, m.sub_dim_2_f);
    return c;
}

// A laser pose (3 x 4, row-major) as pairs: both halves of R[k] hold entry k
// for a pose shared by the pair's two lookups, or entry k of two poses.
struct PosePairs {
    f2_t R[12];
};

__device__ __forceinline__ PosePairs pose_pairs(const float* pose12)
{
    const float4* src = reinterpret_cast<const float4*>(pose12);
    const float4 a = __ldg(src), b = __ldg(src + 1), c = __ldg(src + 2);
    PosePairs r;
    r.R[0] = pk(a.x, a.x); r.R[1] = pk(a.y, a.y); r.R[2] = pk(a.z, a.z); r.R[3] = pk(a.w, a.w);
    r.R[4] = pk(b.x, b.x); r.R[5] = pk(b.y, b.y); r.R[6] = pk(b.z, b.z); r.R[7] = pk(b.w, b.w);
    r.R[8] = pk(c.x, c.x); r.R[9] = pk(c.y, c.y); r.R[10] = pk(c.z, c.z); r.R[11] = pk(c.w, c.w);
    return r;
}

// Transform of two sensor-frame points (X, Y, Z pairs) as tsdf_evaluator.cpp:44-46
// does it: ((r0 x + r1 y) + r2 z) + r3, every product and sum rounded (products
// as FMAs with a +0 addend: exactly the rounded product but for the sign of a
// zero, which moves no offset into another slot).
__device__ __forceinline__ void pair_transform(const PosePairs& P, f2_t X, f2_t Y, f2_t Z, f2_t& TX, f2_t& TY, f2_t& TZ)
{
    const f2_t ZERO = 0ull;
    TX = add2(add2(add2(fma2_rn(P.R[0], X, ZERO), fma2_rn(P.R[1], Y, ZERO)), fma2_rn(P.R[2], Z, ZERO)), P.R[3]);
    TY = add2(add2(add2(fma2_rn(P.R[4], X, ZERO), fma2_rn(P.R[5], Y, ZERO)), fma2_rn(P.R[6], Z, ZERO)), P.R[7]);
    TZ = add2(add2(add2(fma2_rn(P.R[8], X, ZERO), fma2_rn(P.R[9], Y, ZERO)), fma2_rn(P.R[10], Z, ZERO)), P.R[11]);
}

// Transform and fast-path lookup of two sensor-frame points: the gathered codes
// k0, k1 and whether they lie outside the fast domain (s0, s1).
template <int LAY, bool TWO, bool MIN0>
__device__ __forceinline__ void pair_lookup(const MapView& m, const unsigned char* occ, const PosePairs& P,
                                            const PipeConsts& K, f2_t X, f2_t Y, f2_t Z, uint32_t& k0, uint32_t& k1,
                                            bool& s0, bool& s1)
{
    const f2_t ABS = 0x7fffffff7fffffffull, SGN = 0x8000000080000000ull;
    f2_t TX, TY, TZ;
    pair_transform(P, X, Y, Z, TX, TY, TZ);
    // offsets from the map's min corner (cuda_sub_voxel_map.tcc:52-54)
    const f2_t OX = MIN0 ? TX : sub2(TX, K.NMX), OY = MIN0 ? TY : sub2(TY, K.NMY);
    const f2_t OZ = MIN0 ? TZ : sub2(TZ, K.NMZ);
    const f2_t AZ = and2(OZ, ABS);   // |oz|: below the map, brick 0 and a negative sub-voxel index
    // 2^23 + trunc(o), trunc(o) and s = o - trunc(o), all exact
    const f2_t MX = add2_rz(OX, K.MAG), MY = add2_rz(OY, K.MAG), MZ = add2_rz(AZ, K.MAG);
    const f2_t FY = sub2(MY, K.MAG), FZ = sub2(MZ, K.MAG);
    const f2_t SX = sub2(OX, sub2(MX, K.MAG)), SY = sub2(OY, FY), SZ = sub2(AZ, FZ);
    f2_t CX, CY, CZ;   // 1.5 2^23 + sub-voxel index q
    if (TWO) {         // trunc(fl(s * hi + fl(s * lo)))
        CX = add2_rz(fma2_rn(SX, K.INV, mul2(SX, K.INVLO)), K.MAG15);
        CY = add2_rz(fma2_rn(SY, K.INV, mul2(SY, K.INVLO)), K.MAG15);
        CZ = add2_rz(fma2_rn(SZ, K.INV, mul2(SZ, K.INVLO)), K.MAG15);
    } else {           // floor(s * inv), the product unrounded
        CX = fma2_rz(SX, K.INV, K.MAG15);
        CY = fma2_rz(SY, K.INV, K.MAG15);
        CZ = fma2_rz(SZ, K.INV, K.MAG15);
    }
    // qz takes the sign of oz; slot and brick offsets as exact float sums
    const f2_t QY = sub2(CY, K.MAG15), QZ = or2(sub2(CZ, K.MAG15), and2(OZ, SGN));
    const f2_t SLB = fma2_rn(QZ, K.SD2, fma2_rn(QY, K.SD, CX));   // 1.5 2^23 + qx + qy S + qz S^2
    const f2_t UPB = fma2_rn(FZ, K.UXY, fma2_rn(FY, K.UX, MX));   // 2^23 + mx + my Ux + mz Ux Uy
    float ox0, ox1, oy0, oy1, oz0, oz1, u0, u1, l0, l1;
    upk(OX, ox0, ox1); upk(OY, oy0, oy1); upk(OZ, oz0, oz1); upk(UPB, u0, u1); upk(SLB, l0, l1);
    k0 = fast_code<LAY>(m, occ, __float_as_uint(ox0), __float_as_uint(oy0), oz0, __float_as_uint(u0),
                        __float_as_uint(l0), s0);
    k1 = fast_code<LAY>(m, occ, __float_as_uint(ox1), __float_as_uint(oy1), oz1, __float_as_uint(u1),
                        __float_as_uint(l1), s1);
}

// One CTA an SM.  100,000 x 8,192 on the compact layout / 23,457 x 5,003 on the brick
// table (us): 768 threads 2,167 / 305, 736 2,127 / 305, 704 2,134 / 307, 640 2,115 / 312.
constexpr int kTiledThreads = 736;
constexpr int kTiledWarps = kTiledThreads / 32;
constexpr int kSpreadThreads = 640;   // the spread kernel: registers before warps
constexpr int kSpreadWarps = kSpreadThreads / 32;
// The subsampling kernel, which waits on more gathers per lookup, so 1,024 threads;
// with a bitmap in shared memory their rings leave the L1 too little for the codes
// of neighbouring particles (150,000 x 200 of 4,096 points, warehouse, us: brick table
// 338 with 1,024 threads, 394 with 768, compact layout 515 and 427; 150,000 x 200 of 2,048,
// building, compact: 374 to 464 from one process to the next, and 416).  The layout
// decides the form too, which is not always the faster: every map has the brick
// table, and through it (1,024 threads, the scan in shared memory) 300,000 x 256 of
// 2,048 points on the compact building take 732 us, through the bitmap 791.
__host__ __device__ constexpr int sub_threads(bool dense) { return dense ? 768 : 1024; }
constexpr int kRing = 64;   // deferred lookups per warp (transformed point + scan index)
constexpr uint32_t kDbgSlow = 0x10000u;   // debug code flag: decided by the exact slow tiers

// Appends the lanes with `slow` set to the warp's ring of deferred lookups.
__device__ __forceinline__ void defer(float4* ring, uint32_t head, uint32_t& tail, bool slow, float tx, float ty,
                                      float tz, int j, int lane)
{
    const unsigned mask = __ballot_sync(0xffffffffu, slow);
    if (mask == 0u) return;
    const uint32_t pos = tail + (uint32_t)__popc(mask & ((1u << lane) - 1u));
    if (slow) ring[pos & (kRing - 1)] = make_float4(tx, ty, tz, __int_as_float(j));
    tail += (uint32_t)__popc(mask);
    __syncwarp();
}

// Scores `count` (<= 32) deferred lookups from the ring, one per lane, through
// the exact second tier / 64-bit emulation: the lane's code, kCodeNone beyond
// them.  The map view is read from a shared-memory copy so that no kernel
// parameter's address escapes.
__device__ __forceinline__ uint32_t drained_code(const MapView* m, const float4* ring, uint32_t head, int count,
                                                 int lane, uint32_t* dbg_row, const int32_t* perm)
{
    uint32_t code = (uint32_t)kCodeNone;
    if (lane < count) {
        const float4 e = ring[(head + (uint32_t)lane) & (kRing - 1)];
        code = slow_code(*m, e.x, e.y, e.z);
        if (dbg_row) dbg_row[perm[__float_as_int(e.w)]] = code | kDbgSlow;
    }
    __syncwarp();
    return code;
}

__device__ __noinline__ long long drain_packed(const MapView* m, const LutEntry* lut, const float4* ring,
                                               uint32_t head, int count, int lane, uint32_t* dbg_row,
                                               const int32_t* perm)
{
    return lut[drained_code(m, ring, head, count, lane, dbg_row, perm)].v;
}

__device__ __noinline__ uint32_t drain_wide(const MapView* m, const float4* ring, uint32_t head, int count, int lane,
                                            uint32_t* dbg_row, const int32_t* perm)
{
    return drained_code(m, ring, head, count, lane, dbg_row, perm);
}

template <bool PACKED>
__device__ __forceinline__ void drain(const MapView* m, const LutEntry* lut, const float4* ring, uint32_t head,
                                      int count, int lane, uint32_t* dbg_row, const int32_t* perm, long long& acc,
                                      uint32_t& hits)
{
    if (PACKED) acc += drain_packed(m, lut, ring, head, count, lane, dbg_row, perm);
    else take<false>(lut, drain_wide(m, ring, head, count, lane, dbg_row, perm), acc, hits);
}

constexpr int kTiledChunk = 1024;     // scan points per work item
constexpr int kTiledGroup = 4;        // particles per work item
struct TiledParams {
    EvalParams e;
    uint32_t* work;     // [0] next item, [1] CTAs done, both 0 between launches
    int chunk;          // points per work item (multiple of 64)
    int group;          // particles per work item
    int groups;         // particle groups
    int items;          // chunks * groups
};

// Exact mode, tiled.  The pass's scan points are staged once per CTA (bulk
// copies into shared memory, pair layout); then every warp takes (point chunk,
// particle group) work items in chunk-major order from one counter (next_item),
// so all SMs score the same part of the scan at a time and its map footprint
// stays in L2, with no block-wide barrier after staging.  Each lane scores two points per step:
// every floating-point operation of the transform and of the index is one
// packed f32x2 instruction for both points (products as FMAs with a zero addend,
// which round exactly like the reference's products), and the brick and
// sub-voxel offsets are formed as exact float sums whose bits are the biased
// integers, so the integer work per lookup is the rank, the address and the
// bounds.  Likelihood codes are summed in 64-bit fixed point and added to the
// particle's total with an integer atomic: exact and independent of order, so
// results equal eval_exact_kernel's bit for bit.
// Bound by the L1: every lookup's code lies in a cache line of its own (23 a
// warp's request of 32), the tag stage takes one line a cycle, and the shared-
// memory reads share its data pipe: 77 % of either's cycles at 20,000 x 8,192
// (477 us; 538 us before certain_miss(), the packed table and next_item()).
// Issue is 67 % busy, DRAM 12 %.
// One work item of the tiled scoring: the points [c0, c0 + chunk_pts) of the
// staged pass (pair layout in sxy/spz) against the particles of group grp.
// Sums go to p.sum_fx / p.hits with one integer atomic per particle.
// TWO: the sub-voxel index needs the two-term multiplier (sub_fast 1);
// DBG: per-point codes are written to the debug buffer; MIN0: the map's min
// corner is the origin, so offsets are the transformed coordinates.
// LONG: chunk_pts may exceed 64 kPackedSteps (the batch kernel's, whose steps
// stay single: in pairs 24 filters take 1.71 ms an update, singly 1.73); otherwise
// two steps' gathers are in flight at a time.
// PACKED: values and hits in one word (LutEntry).
template <int LAY, bool TWO, bool DBG, bool MIN0, bool LONG, bool PACKED>
__device__ __forceinline__ void tiled_item(const EvalParams& p, const MapView& m, const MapView* s_map,
                                           const unsigned char* occ, const float4* sxy, const float2* spz,
                                           const LutEntry* lut, float4* ring, int n, int chunk_pts, int group,
                                           int chunk, int grp, int lane)
{
    const PipeConsts K = pipe_consts(m);
    uint32_t head = 0, tail = 0;
    const int c0 = chunk * chunk_pts;
    const int cn = min(chunk_pts, n - c0);
    const int b0 = c0 >> 6, nblk = (cn + 63) >> 6, nfull = cn >> 6;
    for (int k = 0; k < group; ++k) {
        const int pi = grp * group + k;
        if (pi >= p.P) break;
        const PosePairs R = pose_pairs(p.pose12 + 12 * (size_t)pi);
        long long acc = 0, sum = 0;
        uint32_t hits = 0;
        // debug rows are indexed by scan index: perm maps the pass's pair-layout
        // positions back to it
        uint32_t* dbg_row = DBG ? p.dbg + (size_t)pi * p.n_total : nullptr;
        const int32_t* perm = DBG ? p.perm + p.n0 : nullptr;
        // the two points of block blk held by this lane
        auto points = [&](int blk, f2_t& X, f2_t& Y, f2_t& Z) {
            const float4 xy = sxy[(b0 + blk) * 32 + lane];
            const float2 zz = spz[(b0 + blk) * 32 + lane];
            X = pk(xy.x, xy.y);
            Y = pk(xy.z, xy.w);
            Z = pk(zz.x, zz.y);
        };
        auto look = [&](int blk, uint32_t& k0, uint32_t& k1, bool& s0, bool& s1) {
            f2_t X, Y, Z;
            points(blk, X, Y, Z);
            pair_lookup<LAY, TWO, MIN0>(m, occ, R, K, X, Y, Z, k0, k1, s0, s1);
        };
        // Block blk's lookups outside the fast domain (some lane of the warp has
        // one; its points are transformed again, so the fast path keeps none of
        // it in registers).  Those settle() cannot decide either are deferred to
        // the warp's ring and scored 32 at a time (kCodeLater contributes nothing
        // here), so no warp diverges into the slow tiers; at most 31 entries wait
        // between calls, so each append of <= 32 fits the ring.
        auto slow = [&](int blk, uint32_t& k0, uint32_t& k1, bool s0, bool s1) {
            f2_t X, Y, Z, TX, TY, TZ;
            points(blk, X, Y, Z);
            pair_transform(R, X, Y, Z, TX, TY, TZ);
            float x0, y0, z0, x1, y1, z1;
            upk(TX, x0, x1); upk(TY, y0, y1); upk(TZ, z0, z1);
            settle(m, x0, y0, z0, s0);
            settle(m, x1, y1, z1, s1);
            if (!__any_sync(0xffffffffu, s0 || s1)) return;
            k0 = s0 ? (uint32_t)kCodeLater : k0;
            k1 = s1 ? (uint32_t)kCodeLater : k1;
            defer(ring, head, tail, s0, x0, y0, z0, c0 + 64 * blk + lane, lane);
            if (tail - head >= 32) {
                drain<PACKED>(s_map, lut, ring, head, 32, lane, dbg_row, perm, acc, hits);
                head += 32;
            }
            defer(ring, head, tail, s1, x1, y1, z1, c0 + 64 * blk + 32 + lane, lane);
            if (tail - head >= 32) {
                drain<PACKED>(s_map, lut, ring, head, 32, lane, dbg_row, perm, acc, hits);
                head += 32;
            }
        };
        auto add = [&](int blk, uint32_t k0, uint32_t k1) {
            if (DBG) {
                const int j = c0 + 64 * blk + lane;
                if (k0 < (uint32_t)kCodeNone) dbg_row[perm[j]] = k0;
                if (k1 < (uint32_t)kCodeNone) dbg_row[perm[j + 32]] = k1;
            }
            take<PACKED>(lut, k0, acc, hits);
            take<PACKED>(lut, k1, acc, hits);
        };
        // one block (the chunk's partial last one masks its padding points)
        auto step = [&](int blk, bool partial) {
            uint32_t k0, k1;
            bool s0, s1;
            look(blk, k0, k1, s0, s1);
            if (partial) {
                const bool v0 = 64 * blk + lane < cn, v1 = 64 * blk + 32 + lane < cn;
                k0 = v0 ? k0 : (uint32_t)kCodeNone;
                k1 = v1 ? k1 : (uint32_t)kCodeNone;
                s0 = s0 && v0;
                s1 = s1 && v1;
            }
            if (__any_sync(0xffffffffu, s0 || s1)) slow(blk, k0, k1, s0, s1);
            add(blk, k0, k1);
        };
        // two blocks, their gathers in flight together
        auto step2 = [&](int blk) {
            uint32_t k0, k1, k2, k3;
            bool s0, s1, s2, s3;
            look(blk, k0, k1, s0, s1);
            look(blk + 1, k2, k3, s2, s3);
            if (__any_sync(0xffffffffu, s0 || s1 || s2 || s3)) {
                slow(blk, k0, k1, s0, s1);
                slow(blk + 1, k2, k3, s2, s3);
            }
            add(blk, k0, k1);
            add(blk + 1, k2, k3);
        };
        if constexpr (LONG) {   // chunks of any length: unpacked every kPackedSteps steps
            for (int blk = 0; blk < nfull;) {
                const int end = min(blk + kPackedSteps, nfull);
                for (; blk < end; ++blk) step(blk, false);
                flush<PACKED>(acc, sum, hits);
            }
        } else {
            int blk = 0;
            for (; blk + 2 <= nfull; blk += 2) step2(blk);
            if (blk < nfull) step(blk, false);
        }
        if (nfull < nblk) step(nfull, true);
        if (tail != head) {
            drain<PACKED>(s_map, lut, ring, head, (int)(tail - head), lane, dbg_row, perm, acc, hits);
            head = tail;
        }
        flush<PACKED>(acc, sum, hits);
        sum = warp_sum_ll(sum);
        hits = warp_sum_u32(hits);
        if (lane == 0) {
            atomicAdd(reinterpret_cast<unsigned long long*>(p.sum_fx + pi), (unsigned long long)sum);
            atomicAdd(p.hits + pi, hits);
        }
    }
}

// Shared memory of the tiled kernels: the likelihood table, the brick bitmap
// (compact layout), then the staged pass and the deferral rings.
template <bool PACKED>
__device__ __forceinline__ void fill_lut(LutEntry* lut, const long long* lut_fx)
{
    for (int c = threadIdx.x; c < kNumCodes; c += blockDim.x) {
        LutEntry e;
        e.v = lut_fx[c] + (PACKED && c <= kCodeInit ? 1ll << kHitShift : 0ll);
        lut[c] = e;
    }
}

// The next work item of a launch, the same on every lane: warps take items from
// one counter, so that all SMs stay on the same part of the scan and finish
// together.  (Dealt out in advance, item k to warp k mod W, the SMs drifted apart
// by whole chunks: the L2 then held the footprints of several, and the last SM
// finished late -- 20,000 particles x 4,099 points 428 -> 318 us, 100,000 x 8,192
// 2,325 -> 2,116 us.)
__device__ __forceinline__ uint32_t next_item(uint32_t* work, int lane)
{
    uint32_t item = 0;
    if (lane == 0) item = atomicAdd(work, 1u);
    return __shfl_sync(0xffffffffu, item, 0);
}

// Called by every thread of a CTA whose warps are done: the last CTA of the grid
// clears the counter for the next launch.
__device__ __forceinline__ void items_done(uint32_t* work)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicInc(work + 1, gridDim.x - 1u) == gridDim.x - 1u) atomicExch(work, 0u);
    }
}

// DBG scores any cloud; otherwise a spread cloud is eval_spread_kernel's and this
// kernel returns at once.
template <int LAY, bool TWO, bool DBG, bool MIN0, bool PACKED>
__global__ void __launch_bounds__(kTiledThreads, 1) eval_tiled_kernel(TiledParams tp)
{
    chain_enter();
    if (!DBG && *tp.e.sched != 0) return;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ uint64_t bar;
    __shared__ MapView s_map;   // the map view the slow tiers read
    const EvalParams& p = tp.e;
    const MapView& m = p.m;
    LutEntry* lut = reinterpret_cast<LutEntry*>(smem);
    const int n = p.n1 - p.n0;
    const int npairs = ((n + 63) >> 6) * 32;
    if (threadIdx.x == 0) s_map = m;
    const uint32_t occ_bytes = LAY == kLayBitmap ? m.occ_bytes : 0u;
    unsigned char* occ = smem + kLutTableBytes;
    float4* sxy = reinterpret_cast<float4*>(occ + occ_bytes);
    float2* spz = reinterpret_cast<float2*>(sxy + npairs);
    fill_lut<PACKED>(lut, p.lut_fx);
    if (threadIdx.x == 0) mbar_init(&bar, 1);
    __syncthreads();
    if (threadIdx.x == 0) {
        mbar_expect_tx(&bar, (uint32_t)npairs * 24u + occ_bytes);
        bulk_g2s(sxy, p.pxy + p.n0 / 2, (uint32_t)npairs * 16u, &bar);
        bulk_g2s(spz, p.pz + p.n0 / 2, (uint32_t)npairs * 8u, &bar);
        if (occ_bytes) bulk_g2s(occ, m.occ, occ_bytes, &bar);
    }
    bool staged = mbar_wait_bounded(&bar, 0);
    if (!staged) staged = mbar_wait_bounded(&bar, 0);   // give copies in flight a second bound
    if (!staged && threadIdx.x == 0) atomicExch(p.status, TSDFL_ERR_TIMEOUT);
    if (__syncthreads_and(staged ? 1 : 0) == 0) return;

    const int lane = threadIdx.x & 31;
    float4* ring = reinterpret_cast<float4*>(spz + npairs) + (threadIdx.x >> 5) * kRing;
    for (;;) {
        const uint32_t item = next_item(tp.work, lane);
        if (item >= (uint32_t)tp.items) break;
        const int chunk = (int)(item / (uint32_t)tp.groups), grp = (int)(item - (uint32_t)chunk * (uint32_t)tp.groups);
        tiled_item<LAY, TWO, DBG, MIN0, false, PACKED>(p, m, &s_map, occ, sxy, spz, lut, ring, n, tp.chunk, tp.group,
                                                       chunk, grp, lane);
    }
    items_done(tp.work);
}

// ------------------------------------------------------- spread-cloud kernel

constexpr int kSpreadBlocks = 2;      // 64-point blocks of the scan a work item holds in registers
constexpr int kSpreadGroup = 16;      // particles a work item scores against them
// a lane's packed sum of 2 kSpreadBlocks lookups, kPackedLookups of which stay below 2^56
static_assert((2ull * kSpreadBlocks << 29) / kPackedLookups < 1ull << 25, "eval_spread_kernel's parts of a sum");
constexpr int kRegionGroups = 1024;   // groups of neighbouring particles a region (512: 9.4, 2,048: 9.3, 8,192: 9.6 ms)

struct SpreadParams {
    EvalParams e;
    uint32_t* work;              // [0, 1] next item (64 bits), [2] CTAs done, all 0 between launches
    unsigned long long items;
    int chunks, groups;
};

// Scores `count` (<= 32) deferred lookups, one per lane, and adds each to its
// own particle (the ring entry's w).
template <bool PACKED>
__device__ __noinline__ void drain_to_particles(const MapView* m, const LutEntry* lut, const float4* ring,
                                                uint32_t head, int count, int lane, long long* sum_fx, uint32_t* hits)
{
    if (lane < count) {
        const float4 e = ring[(head + (uint32_t)lane) & (kRing - 1)];
        long long acc = 0, v = 0;
        uint32_t h = 0;
        take<PACKED>(lut, slow_code(*m, e.x, e.y, e.z), acc, h);
        flush<PACKED>(acc, v, h);
        const int pi = __float_as_int(e.w);
        if (v) atomicAdd(reinterpret_cast<unsigned long long*>(sum_fx + pi), (unsigned long long)v);
        if (h) atomicAdd(hits + pi, h);
    }
    __syncwarp();
}

// Exact mode for a cloud spread over the map (global localisation).  Its gathers
// come from DRAM unless the particles scored at a time see little of the map, so
// the walk is fine-grained: the particles in spatial order in regions of
// kRegionGroups x kSpreadGroup, and within a region all of them against 128 points
// of one height and range band before the next 128.  So small a chunk pays
// because a warp keeps its points in registers and takes the poses, as packed
// pairs, from shared memory; a particle's 128 lookups end in three 32-bit warp
// reductions of the packed sum's parts.  The scan is read from global memory
// once an item: no pass is staged, one launch covers any scan.
// One million particles x 2,048 points in the building: 1,024-point chunks of
// points in shared memory, dealt out in advance, 12.7 ms and 63 GB of DRAM; the
// same taken from a counter 10.9 ms and 49 GB; this walk 9.2 ms and 29 GB (3.2
// TB/s).  It waits on its gathers now (issue 47 %, L1 tags 48 %): 640 threads of
// 96 registers 9.1 ms, 768 of 80 9.6; two particles' gathers in flight a warp
// 10.4, four blocks of points an item 10.6, one 10.2.
template <int LAY, bool TWO, bool MIN0, bool PACKED>
__global__ void __launch_bounds__(kSpreadThreads, 1) eval_spread_kernel(SpreadParams sp)
{
    chain_enter();
    const EvalParams& p = sp.e;
    if (*p.sched == 0) return;   // a compact cloud is eval_tiled_kernel's
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ uint64_t bar;
    __shared__ MapView s_map;   // the map view the slow tiers read
    const MapView& m = p.m;
    LutEntry* lut = reinterpret_cast<LutEntry*>(smem);
    const uint32_t occ_bytes = LAY == kLayBitmap ? m.occ_bytes : 0u;
    unsigned char* occ = smem + kLutTableBytes;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    ulonglong2* poses = reinterpret_cast<ulonglong2*>(occ + occ_bytes) + warp * (6 * kSpreadGroup);
    float4* ring = reinterpret_cast<float4*>(occ + occ_bytes + kSpreadWarps * (6 * kSpreadGroup) * sizeof(ulonglong2)) +
                   warp * kRing;
    if (threadIdx.x == 0) s_map = m;
    fill_lut<PACKED>(lut, p.lut_fx);
    if (threadIdx.x == 0) mbar_init(&bar, 1);
    __syncthreads();
    bool staged = true;
    if (occ_bytes) {
        if (threadIdx.x == 0) {
            mbar_expect_tx(&bar, occ_bytes);
            bulk_g2s(occ, m.occ, occ_bytes, &bar);
        }
        staged = mbar_wait_bounded(&bar, 0);
        if (!staged) staged = mbar_wait_bounded(&bar, 0);   // give the copy in flight a second bound
    }
    if (!staged && threadIdx.x == 0) atomicExch(p.status, TSDFL_ERR_TIMEOUT);
    if (__syncthreads_and(staged ? 1 : 0) == 0) return;

    const PipeConsts K = pipe_consts(m);
    const int n = p.n_total;
    const unsigned long long per_region = (unsigned long long)sp.chunks * kRegionGroups;
    uint32_t head = 0, tail = 0;
    unsigned long long* next = reinterpret_cast<unsigned long long*>(sp.work);
    unsigned long long mine = 0;   // lane 0: the item after this one, fetched ahead
    if (lane == 0) mine = atomicAdd(next, 1ull);
    f2_t X[kSpreadBlocks], Y[kSpreadBlocks], Z[kSpreadBlocks];   // this lane's points: two of each block
    int held = -1;                                               // their chunk
    for (;;) {
        const unsigned long long item = __shfl_sync(0xffffffffu, mine, 0);
        if (item >= sp.items) break;
        if (lane == 0) mine = atomicAdd(next, 1ull);
        const unsigned long long r = item / per_region, rem = item - r * per_region;
        const int g0 = (int)r * kRegionGroups, rg = min(kRegionGroups, sp.groups - g0);
        const int chunk = (int)(rem / (unsigned)rg), grp = g0 + (int)(rem - (unsigned long long)chunk * (unsigned)rg);
        const int q0 = grp * kSpreadGroup, kn = min(kSpreadGroup, p.P - q0);
        int pi = 0;
        if (lane < kn) {   // the group's poses as pairs of equal floats
            pi = (int)p.order[q0 + lane];
            const PosePairs R = pose_pairs(p.pose12 + 12 * (size_t)pi);
#pragma unroll
            for (int j = 0; j < 6; ++j) poses[6 * lane + j] = make_ulonglong2(R.R[2 * j], R.R[2 * j + 1]);
        }
        const int first = 64 * kSpreadBlocks * chunk;
        const bool full = first + 64 * kSpreadBlocks <= n;
        if (chunk != held) {
            held = chunk;
#pragma unroll
            for (int b = 0; b < kSpreadBlocks; ++b) {
                const bool have = first + 64 * b < n;   // the pair layout is padded to whole blocks
                const size_t at = (size_t)(first / 2 + 32 * b + lane);
                const float4 xy = have ? __ldg(p.pxy + at) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                const float2 zz = have ? __ldg(p.pz + at) : make_float2(0.0f, 0.0f);
                X[b] = pk(xy.x, xy.y);
                Y[b] = pk(xy.z, xy.w);
                Z[b] = pk(zz.x, zz.y);
            }
        }
        __syncwarp();
        long long sum = 0;    // of the particle of this lane's place in the group
        uint32_t hits = 0;
        for (int k = 0; k < kn; ++k) {
            PosePairs R;
#pragma unroll
            for (int j = 0; j < 6; ++j) {
                const ulonglong2 v = poses[6 * k + j];
                R.R[2 * j] = v.x;
                R.R[2 * j + 1] = v.y;
            }
            uint32_t c0[kSpreadBlocks], c1[kSpreadBlocks];
            bool s0[kSpreadBlocks], s1[kSpreadBlocks], any = false;
#pragma unroll
            for (int b = 0; b < kSpreadBlocks; ++b)
                pair_lookup<LAY, TWO, MIN0>(m, occ, R, K, X[b], Y[b], Z[b], c0[b], c1[b], s0[b], s1[b]);
            if (!full) {
#pragma unroll
                for (int b = 0; b < kSpreadBlocks; ++b) {
                    const bool v0 = first + 64 * b + lane < n, v1 = first + 64 * b + 32 + lane < n;
                    c0[b] = v0 ? c0[b] : (uint32_t)kCodeNone;
                    c1[b] = v1 ? c1[b] : (uint32_t)kCodeNone;
                    s0[b] = s0[b] && v0;
                    s1[b] = s1[b] && v1;
                }
            }
#pragma unroll
            for (int b = 0; b < kSpreadBlocks; ++b) any = any || s0[b] || s1[b];
            if (__any_sync(0xffffffffu, any)) {
                const int who = __shfl_sync(0xffffffffu, pi, k);
#pragma unroll
                for (int b = 0; b < kSpreadBlocks; ++b) {
                    f2_t TX, TY, TZ;
                    pair_transform(R, X[b], Y[b], Z[b], TX, TY, TZ);
                    float x0, y0, z0, x1, y1, z1;
                    upk(TX, x0, x1); upk(TY, y0, y1); upk(TZ, z0, z1);
                    settle(m, x0, y0, z0, s0[b]);
                    settle(m, x1, y1, z1, s1[b]);
                    if (!__any_sync(0xffffffffu, s0[b] || s1[b])) continue;
                    c0[b] = s0[b] ? (uint32_t)kCodeLater : c0[b];
                    c1[b] = s1[b] ? (uint32_t)kCodeLater : c1[b];
                    defer(ring, head, tail, s0[b], x0, y0, z0, who, lane);
                    if (tail - head >= 32) {
                        drain_to_particles<PACKED>(&s_map, lut, ring, head, 32, lane, p.sum_fx, p.hits);
                        head += 32;
                    }
                    defer(ring, head, tail, s1[b], x1, y1, z1, who, lane);
                    if (tail - head >= 32) {
                        drain_to_particles<PACKED>(&s_map, lut, ring, head, 32, lane, p.sum_fx, p.hits);
                        head += 32;
                    }
                }
            }
            long long acc = 0, v = 0;
            uint32_t h = 0;
#pragma unroll
            for (int b = 0; b < kSpreadBlocks; ++b) {
                take<PACKED>(lut, c0[b], acc, h);
                take<PACKED>(lut, c1[b], acc, h);
            }
            flush<PACKED>(acc, v, h);
            h = __reduce_add_sync(0xffffffffu, h);
            if (PACKED) {
                // the warp's sum in parts that cannot overflow: 27 low bits (32 of them
                // below 2^32) and the signed rest (below 2^25 a lane)
                const uint32_t l = __reduce_add_sync(0xffffffffu, (uint32_t)v & 0x7ffffffu);
                const int u = __reduce_add_sync(0xffffffffu, (int)(v >> 27));
                v = ((long long)u << 27) + (long long)l;
            } else {
                v = warp_sum_ll(v);
            }
            if (lane == k) {
                sum = v;
                hits = h;
            }
        }
        if (lane < kn) {
            atomicAdd(reinterpret_cast<unsigned long long*>(p.sum_fx + pi), (unsigned long long)sum);
            atomicAdd(p.hits + pi, hits);
        }
        __syncwarp();   // the poses are overwritten by the next item's
    }
    if (tail != head) drain_to_particles<PACKED>(&s_map, lut, ring, head, (int)(tail - head), lane, p.sum_fx, p.hits);
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicInc(sp.work + 2, gridDim.x - 1u) == gridDim.x - 1u)
            atomicExch(reinterpret_cast<unsigned long long*>(sp.work), 0ull);
    }
}

size_t spread_smem_bytes(uint32_t occ_bytes)
{
    return (size_t)kLutTableBytes + occ_bytes + sizeof(ulonglong2) * 6 * kSpreadGroup * kSpreadWarps +
           sizeof(float4) * kRing * kSpreadWarps;
}

// Seeded per-particle scan subsampling (subsample.h): one warp per particle
// scores the particle's K kept points, two per lane per step, through the same
// packed pipeline as the tiled kernel.  Per particle: the fixed-point likelihood
// sum, the hits and the number of kept points within max_range (its weight's
// range term), written directly (one warp owns the particle).
// Waits on the codes' gathers.  300,000 particles x 256 of 2,048 points in the
// 100 x 100 m building, compact layout, a pass: 1,018 us with two 64-bit divisions a
// point for its stratum and particles dealt to the warps in turn; 791 with the
// strata stepped and particles from a counter (704 with 1,024 threads
// and the scan beside the bitmap, which larger scans lose more by: sub_threads).  STAGED: the scan in shared memory,
// one 16-byte read a point instead of four from the SoA arrays.
struct SubParams {
    EvalParams e;
    int K;
    unsigned long long seed;
    uint32_t* nin;
    float c_in;
    uint32_t* work;      // the item counter and the CTAs done
    int group, items;    // particles an item, items
};

template <bool DENSE, bool TWO, bool MIN0, bool STAGED, bool PACKED>
__global__ void __launch_bounds__(sub_threads(DENSE), 1) eval_subsample_kernel(SubParams sp)
{
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ uint64_t bar;
    __shared__ MapView s_map;   // the map view the slow tiers read
    const EvalParams& p = sp.e;
    const MapView& m = p.m;
    LutEntry* lut = reinterpret_cast<LutEntry*>(smem);
    const uint32_t occ_bytes = DENSE ? m.occ_bytes : 0u;
    unsigned char* occ = smem + kLutTableBytes;
    float4* rings = reinterpret_cast<float4*>(occ + occ_bytes);
    float4* pts = rings + kRing * (sub_threads(DENSE) / 32);
    if (threadIdx.x == 0) s_map = m;
    fill_lut<PACKED>(lut, p.lut_fx);
    if (STAGED)
        for (int j = threadIdx.x; j < p.n_total; j += sub_threads(DENSE))
            pts[j] = make_float4(p.xs[j], p.ys[j], p.zs[j], p.cs[j]);
    if (threadIdx.x == 0) mbar_init(&bar, 1);
    __syncthreads();
    bool staged = true;
    if (occ_bytes) {
        if (threadIdx.x == 0) {
            mbar_expect_tx(&bar, occ_bytes);
            bulk_g2s(occ, m.occ, occ_bytes, &bar);
        }
        staged = mbar_wait_bounded(&bar, 0);
        if (!staged) staged = mbar_wait_bounded(&bar, 0);   // give the copy in flight a second bound
    }
    if (!staged && threadIdx.x == 0) atomicExch(p.status, TSDFL_ERR_TIMEOUT);
    if (__syncthreads_and(staged ? 1 : 0) == 0) return;

    const int lane = threadIdx.x & 31;
    float4* ring = rings + (threadIdx.x >> 5) * kRing;
    const PipeConsts K = pipe_consts(m);
    const uint32_t N = (uint32_t)p.n_total, Ks = (uint32_t)sp.K;
    const bool ordered = p.sched && *p.sched;
    // The strata's bounds floor(k N / K) of a lane's k = lane, lane + 64, ... (and
    // lane + 32, ...), stepped with their remainders: exact, and no division a point.
    const uint32_t qn = N / Ks, rn = N - qn * Ks;
    const uint32_t q64 = (uint32_t)((64ull * N) / Ks), r64 = (uint32_t)(64ull * N - (uint64_t)q64 * Ks);
    const uint32_t first_a = (uint32_t)(((uint64_t)lane * N) / Ks),
                   first_b = (uint32_t)(((uint64_t)(lane + 32) * N) / Ks);
    const uint32_t rem_a = (uint32_t)((uint64_t)lane * N - (uint64_t)first_a * Ks),
                   rem_b = (uint32_t)((uint64_t)(lane + 32) * N - (uint64_t)first_b * Ks);
    // the kept point of the stratum from b (k N = b K + rem)
    auto kept = [&](uint64_t st, uint32_t b, uint32_t rem) {
        const uint32_t n = qn + (rem + rn >= Ks ? 1u : 0u);
        return b + __umulhi((uint32_t)(sub_mix64(st) >> 32), n);
    };
    int q = 0, q1 = 0;   // the item's particles
    for (;; ++q) {
        if (q == q1) {
            const uint32_t item = next_item(sp.work, lane);
            if (item >= (uint32_t)sp.items) break;
            q = (int)item * sp.group;
            q1 = min(q + sp.group, p.P);
        }
        const int pi = ordered ? (int)p.order[q] : q;   // neighbouring warps take neighbouring particles
        const PosePairs R = pose_pairs(p.pose12 + 12 * (size_t)pi);
        uint64_t st_a = sub_particle_state(sp.seed, (uint64_t)pi) + (uint64_t)(lane + 1) * kGoldenGamma;
        uint32_t b_a = first_a, m_a = rem_a, b_b = first_b, m_b = rem_b;
        long long acc = 0, sum = 0;
        uint32_t hits = 0, nin = 0, head = 0, tail = 0;
        int packed = 0;
        for (uint32_t base = 0; base < Ks; base += 64) {   // the same trip count on every lane
            const uint32_t ka = base + (uint32_t)lane, kb = ka + 32u;
            const bool va = ka < Ks, vb = kb < Ks;
            const uint32_t ja = va ? kept(st_a, b_a, m_a) : 0u;
            const uint32_t jb = vb ? kept(st_a + 32u * kGoldenGamma, b_b, m_b) : 0u;
            st_a += 64u * kGoldenGamma;
            b_a += q64 + (m_a + r64 >= Ks ? 1u : 0u);
            m_a = m_a + r64 >= Ks ? m_a + r64 - Ks : m_a + r64;
            b_b += q64 + (m_b + r64 >= Ks ? 1u : 0u);
            m_b = m_b + r64 >= Ks ? m_b + r64 - Ks : m_b + r64;
            float4 A, B;
            if (STAGED) {
                A = pts[ja];
                B = pts[jb];
            } else {
                A = make_float4(__ldg(p.xs + ja), __ldg(p.ys + ja), __ldg(p.zs + ja), __ldg(p.cs + ja));
                B = make_float4(__ldg(p.xs + jb), __ldg(p.ys + jb), __ldg(p.zs + jb), __ldg(p.cs + jb));
            }
            const float xa = A.x, ya = A.y, za = A.z, xb = B.x, yb = B.y, zb = B.z;
            nin += (va && A.w == sp.c_in ? 1u : 0u) + (vb && B.w == sp.c_in ? 1u : 0u);
            uint32_t k0, k1;
            bool s0, s1;
            pair_lookup<DENSE ? kLayBitmap : kLayTable, TWO, MIN0>(m, occ, R, K, pk(xa, xb), pk(ya, yb), pk(za, zb),
                                                                   k0, k1, s0, s1);
            k0 = va ? k0 : (uint32_t)kCodeNone;
            k1 = vb ? k1 : (uint32_t)kCodeNone;
            s0 = s0 && va;
            s1 = s1 && vb;
            if (__any_sync(0xffffffffu, s0 || s1)) {
                f2_t TX, TY, TZ;
                pair_transform(R, pk(xa, xb), pk(ya, yb), pk(za, zb), TX, TY, TZ);
                float tx, ty, tz, u;
                upk(TX, tx, u); upk(TY, ty, u); upk(TZ, tz, u);
                settle(m, tx, ty, tz, s0);
                k0 = s0 ? (uint32_t)kCodeLater : k0;
                defer(ring, head, tail, s0, tx, ty, tz, (int)ja, lane);
                if (tail - head >= 32) {
                    drain<PACKED>(&s_map, lut, ring, head, 32, lane, nullptr, nullptr, acc, hits);
                    head += 32;
                }
                upk(TX, u, tx); upk(TY, u, ty); upk(TZ, u, tz);
                settle(m, tx, ty, tz, s1);
                k1 = s1 ? (uint32_t)kCodeLater : k1;
                defer(ring, head, tail, s1, tx, ty, tz, (int)jb, lane);
                if (tail - head >= 32) {
                    drain<PACKED>(&s_map, lut, ring, head, 32, lane, nullptr, nullptr, acc, hits);
                    head += 32;
                }
            }
            take<PACKED>(lut, k0, acc, hits);
            take<PACKED>(lut, k1, acc, hits);
            if (++packed == kPackedSteps) {
                flush<PACKED>(acc, sum, hits);
                packed = 0;
            }
        }
        if (tail != head)
            drain<PACKED>(&s_map, lut, ring, head, (int)(tail - head), lane, nullptr, nullptr, acc, hits);
        flush<PACKED>(acc, sum, hits);
        sum = warp_sum_ll(sum);
        hits = warp_sum_u32(hits);
        nin = warp_sum_u32(nin);
        if (lane == 0) {
            p.sum_fx[pi] = sum;
            p.hits[pi] = hits;
            sp.nin[pi] = nin;
        }
    }
    items_done(sp.work);
}

// Work items per batch, the unit in which the persistent multi-filter launch's
// work is reported (tsdfl_batch_info).
constexpr int kBatchItems = kTiledWarps * 8;

struct BatchSeg {
    EvalParams e;
    int chunk, group, groups, items;
    uint32_t first_item;   // of the segments of its kind one after another
    uint32_t next;         // the next item to be taken; cleared before the launch
};

// Segment a CTA starts on: the one its share of the items begins in, so that the
// CTAs spread over the segments by their work.  One warp; the same in every lane.
__device__ __forceinline__ int batch_start(const BatchSeg* segs, int nseg, uint32_t total, int lane)
{
    const uint32_t at = (uint32_t)((unsigned long long)total * (2u * blockIdx.x + 1u) / (2u * gridDim.x));
    int best = 0;
    for (int k = lane; k < nseg; k += 32)
        if (segs[k].first_item <= at) best = k;   // ascending
    return __reduce_max_sync(0xffffffffu, best);
}

// Segment with the most items not taken yet, -1 when none has any.  One warp; the
// same in every lane.
__device__ __forceinline__ int batch_most_left(const BatchSeg* segs, int nseg, int lane)
{
    int left = 0, best = -1;
    for (int k = lane; k < nseg; k += 32) {
        const int v = segs[k].items - (int)min(*(const volatile uint32_t*)&segs[k].next, (uint32_t)segs[k].items);
        if (v > left) {
            left = v;
            best = k;
        }
    }
    const int most = __reduce_max_sync(0xffffffffu, left);
    if (most == 0) return -1;
    return __reduce_max_sync(0xffffffffu, left == most ? best : -1);
}

// Many filters in one persistent launch (one per map-layout kind present:
// compact or brick table, one- or two-term sub-voxel multiplier -- the same
// specialisations as eval_tiled_kernel).  The work is the filters' (filter, pass)
// segments, each of (point chunk, particle group) items that warps take from the
// segment's own counter.  A CTA stages a segment (the filter's code LUT, its map's
// occupancy bitmap, the pass's scan points), its warps score that segment's items
// with no barrier between them until none is left, and the CTA goes on to the
// segment with the most items left.  It begins where its share of all items
// begins: most CTAs stage one segment and help out in one or two others at the
// end.  (Batches of one queue, each taken by a CTA with barriers around it, put
// all CTAs through every segment and left warps idle before each: see the figures
// at the launch.)  Every item is taken once by the counter; a CTA leaves only
// when no segment has an item left, so none is missed.  Per-item scoring is
// eval_tiled_kernel's, so every filter's sums equal its single-filter sums bit for
// bit.
template <bool DENSE, bool TWO, bool MIN0, bool PACKED>
__global__ void __launch_bounds__(kTiledThreads, 1) eval_batch_kernel(BatchSeg* segs, int nseg, uint32_t total_items,
                                                                      int32_t* status)
{
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ uint64_t bar;
    __shared__ BatchSeg s_seg;
    __shared__ int s_segi;
    LutEntry* lut = reinterpret_cast<LutEntry*>(smem);
    unsigned char* occ = smem + kLutTableBytes;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) mbar_init(&bar, 1);
    if (warp == 0) {
        const int k = batch_start(segs, nseg, total_items, lane);
        if (lane == 0) s_segi = k;
    }
    __syncthreads();
    uint32_t phase = 0;
    for (;;) {
        const int segi = s_segi;
        if (segi < 0) break;
        for (unsigned k = threadIdx.x; k < sizeof(BatchSeg) / 4u; k += kTiledThreads)
            reinterpret_cast<uint32_t*>(&s_seg)[k] = reinterpret_cast<const uint32_t*>(segs + segi)[k];
        __syncthreads();
        const EvalParams& p = s_seg.e;
        const int n = p.n1 - p.n0;
        const int npairs = ((n + 63) >> 6) * 32;
        const uint32_t occ_bytes = DENSE ? p.m.occ_bytes : 0u;
        float4* sxy = reinterpret_cast<float4*>(occ + occ_bytes);
        float2* spz = reinterpret_cast<float2*>(sxy + npairs);
        float4* ring = reinterpret_cast<float4*>(spz + npairs) + warp * kRing;
        fill_lut<PACKED>(lut, p.lut_fx);
        if (threadIdx.x == 0) {
            mbar_expect_tx(&bar, (uint32_t)npairs * 24u + occ_bytes);
            bulk_g2s(sxy, p.pxy + p.n0 / 2, (uint32_t)npairs * 16u, &bar);
            bulk_g2s(spz, p.pz + p.n0 / 2, (uint32_t)npairs * 8u, &bar);
            if (occ_bytes) bulk_g2s(occ, p.m.occ, occ_bytes, &bar);
        }
        bool staged = mbar_wait_bounded(&bar, phase);
        if (!staged) staged = mbar_wait_bounded(&bar, phase);   // give copies in flight a second bound
        phase ^= 1u;
        if (!staged && threadIdx.x == 0) atomicExch(status, TSDFL_ERR_TIMEOUT);
        if (__syncthreads_and(staged ? 1 : 0) == 0) return;
        for (;;) {
            const uint32_t item = next_item(&segs[segi].next, lane);
            if (item >= (uint32_t)s_seg.items) break;
            const int chunk = (int)item / s_seg.groups, grp = (int)item - chunk * s_seg.groups;
            tiled_item<DENSE ? kLayBitmap : kLayTable, TWO, false, MIN0, true, PACKED>(
                p, p.m, &p.m, occ, sxy, spz, lut, ring, n, s_seg.chunk, s_seg.group, chunk, grp, lane);
        }
        before_bulk_reuse();   // the rings' place moves with the segment: the next one's copies may fall on them
        __syncthreads();       // every warp is done with the staged segment
        if (warp == 0) {
            const int k = batch_most_left(segs, nseg, lane);
            if (lane == 0) s_segi = k;
        }
        __syncthreads();
    }
}

// Serial mode: one thread per particle runs evaluatePose's loop
// (tsdf_evaluator.cpp:38-68) in scan order with float sums, reproducing the
// reference's un-normalised weight bit for bit.
template <bool F32>
__global__ void __launch_bounds__(256) eval_serial_kernel(EvalParams p)
{
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ uint64_t bar;
    float* lut = reinterpret_cast<float*>(smem);
    const int n = p.n1 - p.n0;
    const int npad = (n + 3) & ~3;
    float* xs = reinterpret_cast<float*>(smem + kLutFBytes);
    float* ys = xs + npad;
    float* zs = ys + npad;
    float* cs = zs + npad;
    for (int c = threadIdx.x; c < kNumCodes; c += blockDim.x) lut[c] = p.lut_f[c];
    for (int j = threadIdx.x; j < n; j += blockDim.x) cs[j] = p.cs[p.n0 + j];
    if (!stage_xyz(xs, ys, zs, p.xs + p.n0, p.ys + p.n0, p.zs + p.n0, npad, &bar, p.status)) return;
    int pi = blockIdx.x * blockDim.x + threadIdx.x;
    if (pi >= p.P) return;
    float t[12];
    for (int k = 0; k < 12; ++k) t[k] = p.pose12[12 * (size_t)pi + k];
    const MapView& m = p.m;
    float sum = p.first_pass ? 0.0f : p.raw[pi];
    uint32_t h = p.first_pass ? 0u : p.hits[pi];
    for (int j = 0; j < n; ++j) {
        float tx, ty, tz;
        transform_point(t, xs[j], ys[j], zs[j], tx, ty, tz);
        uint32_t idx = slot_index(m, tx, ty, tz);
        float v;
        if (F32) v = idx != kMissIndex ? m.data[idx] : m.init_value;
        else v = lut[idx != kMissIndex ? (uint32_t)m.codes[idx] : (uint32_t)kCodeInit];
        h += idx != kMissIndex ? 1u : 0u;
        if (p.dbg) p.dbg[(size_t)pi * p.n_total + p.n0 + j] = idx;
        v = __fadd_rn(__fmul_rn(p.a_hit, v), cs[j]);
        sum = __fadd_rn(sum, v);
    }
    p.raw[pi] = sum;
    p.hits[pi] = h;
}

constexpr int kNormBlocks = 256;
constexpr int kNormThreads = 256;
constexpr int kNormSums = 10;
constexpr int kNormalizeBlocks = 4 * 148;   // most blocks of normalize_kernel beside its first: about four an SM

struct NormParams {
    int P;
    int mode;            // 0 fixed point, 1 double sums, 2 serial raw
    int shift;
    double a_hit, c_in, c_out;
    int n_points;        // points every particle scored
    const uint32_t* nin; // per-particle points within max_range (subsampled scans), else null
};

// The block's sums of ten values per thread (blockDim.x == kNormThreads), in a
// fixed order: the values go to shared memory, 160 threads add sixteen each,
// ten threads add those sixteen partial sums.  Few FP64 instructions: a
// warp-shuffle tree would spend five FP64 additions a warp for every sum, and
// GB300's FP64 pipe is narrow.  Valid in threads 0..9 (out[k]).
constexpr int kNormSumsParts = 16;
static_assert(kNormSums * kNormSumsParts <= kNormThreads && kNormThreads % kNormSumsParts == 0,
              "the block's threads cover the partial sums");
__device__ __forceinline__ double block_sums10(const double (&acc)[kNormSums], double (*red)[kNormThreads],
                                               double (*red2)[kNormSumsParts])
{
    for (int k = 0; k < kNormSums; ++k) red[k][threadIdx.x] = acc[k];
    __syncthreads();
    if (threadIdx.x < kNormSums * kNormSumsParts) {
        const int k = threadIdx.x / kNormSumsParts, part = threadIdx.x % kNormSumsParts;
        double v = 0.0;
        for (int j = 0; j < kNormThreads / kNormSumsParts; ++j) v += red[k][part + kNormSumsParts * j];
        red2[k][part] = v;
    }
    __syncthreads();
    double v = 0.0;
    if (threadIdx.x < kNormSums)
        for (int j = 0; j < kNormSumsParts; ++j) v += red2[threadIdx.x][j];
    return v;
}

// Forms each particle's un-normalised weight from its likelihood sum and
// accumulates, in double and in a fixed order, the weight sum and the
// weighted pose sums of tsdf_evaluator.cpp:198-217.
__global__ void norm_partial_kernel(NormParams q, EvalBuffers b, const double* sum_f64)
{
    chain_enter();
    double acc[kNormSums];
    for (int k = 0; k < kNormSums; ++k) acc[k] = 0.0;
    const double n_in_all = (double)b.counts[0];
    const double scale = ldexp(1.0, -q.shift);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < q.P; i += gridDim.x * blockDim.x) {
        const double n_in = q.nin ? (double)q.nin[i] : n_in_all;
        const double n_out = (double)q.n_points - n_in;
        float raw;
        if (q.mode == 2) {
            raw = b.raw[i];
        } else {
            double sl = q.mode == 0 ? (double)b.sum_fx[i] * scale : sum_f64[i];
            raw = (float)(q.a_hit * sl + n_in * q.c_in + n_out * q.c_out);
            b.raw[i] = raw;
        }
        double w = (double)raw;
        const float* pp = b.particles + 7 * (size_t)i;
        const float* tg = b.trig6 + 6 * (size_t)i;
        acc[0] += w;
        acc[1] += (double)pp[0] * w;
        acc[2] += (double)pp[1] * w;
        acc[3] += (double)pp[2] * w;
        acc[4] += (double)tg[0] * w;
        acc[5] += (double)tg[1] * w;
        acc[6] += (double)tg[2] * w;
        acc[7] += (double)tg[3] * w;
        acc[8] += (double)tg[4] * w;
        acc[9] += (double)tg[5] * w;
    }
    __shared__ double red[kNormSums][kNormThreads];
    __shared__ double red2[kNormSums][kNormSumsParts];
    const double v = block_sums10(acc, red, red2);
    if (threadIdx.x < kNormSums) b.partials[blockIdx.x * kNormSums + threadIdx.x] = v;
}

// Final weight sum, the "No particle is valid!" check (tsdf_evaluator.cpp:159)
// and the mean pose with circular means of the angles (:219-221), by one block
// of kNormThreads threads: thread t takes block t's partial sums (nb blocks ran),
// then a fixed reduction tree (so the result does not depend on timing); the
// position and the three angles are formed by four threads side by side.
__device__ __forceinline__ void norm_final_block(const EvalBuffers& b, float* pose_out, int nb,
                                                 double (*red)[kNormThreads], double (*red2)[kNormSumsParts])
{
    static_assert(kNormBlocks == kNormThreads, "one partial per thread");
    __shared__ double s[kNormSums];
    const int t = threadIdx.x;
    double acc[kNormSums];
    for (int k = 0; k < kNormSums; ++k) acc[k] = t < nb ? b.partials[t * kNormSums + k] : 0.0;
    const double v = block_sums10(acc, red, red2);
    if (t < kNormSums) {
        s[t] = v;
        b.sums[t] = v;
    }
    __syncthreads();
    if (t >= 4) return;
    const bool degenerate = !((float)s[0] != 0.0f) || !isfinite(s[0]);
    if (t == 0) {
        b.weight_sum_f[0] = (float)s[0];
        if (degenerate) atomicExch(b.status, TSDFL_ERR_DEGENERATE);
    }
    if (degenerate || !pose_out) return;
    const double inv = 1.0 / s[0];
    if (t == 0) {
        pose_out[0] = (float)(s[1] * inv);
        pose_out[1] = (float)(s[2] * inv);
        pose_out[2] = (float)(s[3] * inv);
    } else {
        pose_out[2 + t] = (float)atan2(s[2 + 2 * t] * inv, s[3 + 2 * t] * inv);
    }
}

// Also the last step of an evaluation: one thread carries its device status into
// the sticky status word (when one is given and still clear).
__device__ __forceinline__ void fold_status(const int32_t* ev, int32_t* sticky)
{
    const int v = *ev;
    if (sticky && v && *sticky == 0) *sticky = v;
}

__global__ void fold_statuses_kernel(const int32_t* status, int n, int32_t* sticky)
{
    for (int i = 0; i < n && *sticky == 0; ++i) *sticky = status[i];
}

// particles[i].second = raw / weight_sum (tsdf_evaluator.cpp:203), skipped when
// the sum was degenerate so the caller's particles stay untouched.  Block 0
// forms the final sums and the mean pose meanwhile; the others add the weight
// sum's partials themselves, in its order, instead of waiting for a launch
// between.
__global__ void __launch_bounds__(kNormThreads) normalize_kernel(int P, EvalBuffers b, float* particles_out,
                                                                 float* pose_out, int nb, int32_t* sticky)
{
    chain_enter();
    __shared__ double red[kNormSums][kNormThreads];
    __shared__ double red2[kNormSums][kNormSumsParts];
    const int t = threadIdx.x;
    if (blockIdx.x == 0) {
        norm_final_block(b, pose_out, nb, red, red2);
        if (t == 0) fold_status(b.status, sticky);
        return;
    }
    red[0][t] = t < nb ? b.partials[t * kNormSums] : 0.0;
    __syncthreads();
    if (t < kNormSumsParts) {   // block_sums10's order
        double v = 0.0;
        for (int j = 0; j < kNormThreads / kNormSumsParts; ++j) v += red[0][t + kNormSumsParts * j];
        red2[0][t] = v;
    }
    __syncthreads();
    double sum = 0.0;
    for (int j = 0; j < kNormSumsParts; ++j) sum += red2[0][j];
    const float w = (float)sum;
    if (!(w != 0.0f) || !isfinite(sum)) return;
    const int step = (int)(gridDim.x - 1) * kNormThreads;
    for (int i = (int)(blockIdx.x - 1) * kNormThreads + t; i < P; i += step)
        particles_out[7 * (size_t)i + 6] = __fdiv_rn(b.raw[i], w);
}

__global__ void __launch_bounds__(kNormThreads) norm_final_kernel(EvalBuffers b, float* pose_out, int nb)
{
    chain_enter();
    __shared__ double red[kNormSums][kNormThreads];
    __shared__ double red2[kNormSums][kNormSumsParts];
    norm_final_block(b, pose_out, nb, red, red2);
}

// Log-domain normalisation (TSDFL_NORM_LOG), after norm_partial/final have
// formed the raw weights: the largest raw weight (positive floats order like
// their bits: one atomicMax), then sum_i exp(ln raw_i - ln max) in double
// (block partials in a fixed order), LSE, and w_i = exp(ln raw_i - LSE).
__global__ void log_max_kernel(int P, EvalBuffers b)
{
    uint32_t mx = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < P; i += gridDim.x * blockDim.x) {
        const float r = b.raw[i];
        if (r > 0.0f) mx = max(mx, __float_as_uint(r));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((threadIdx.x & 31) == 0 && mx) atomicMax(reinterpret_cast<unsigned int*>(b.counts + 1), mx);
}

__global__ void log_sum_kernel(int P, EvalBuffers b)
{
    const double lm = log((double)__uint_as_float((uint32_t)b.counts[1]));
    double acc = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < P; i += gridDim.x * blockDim.x) {
        const float r = b.raw[i];
        if (r > 0.0f) acc += exp(log((double)r) - lm);
    }
    __shared__ double red[kNormThreads / 32];
    acc = warp_sum_d(acc);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double v = 0.0;
        for (int w = 0; w < kNormThreads / 32; ++w) v += red[w];
        b.partials[blockIdx.x] = v;
    }
}

__global__ void __launch_bounds__(kNormBlocks) log_final_kernel(EvalBuffers b)
{
    __shared__ double red[kNormBlocks / 32];
    const double v = warp_sum_d(b.partials[threadIdx.x]);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int w = 0; w < kNormBlocks / 32; ++w) s += red[w];
        b.sums[10] = log((double)__uint_as_float((uint32_t)b.counts[1])) + log(s);   // LSE
    }
}

__global__ void normalize_log_kernel(int P, EvalBuffers b, float* particles_out, int32_t* sticky)
{
    if (blockIdx.x == 0 && threadIdx.x == 0) fold_status(b.status, sticky);
    if (*b.status == TSDFL_ERR_DEGENERATE) return;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P) return;
    const float r = b.raw[i];
    particles_out[7 * (size_t)i + 6] = r > 0.0f ? (float)exp(log((double)r) - b.sums[10]) : 0.0f;
}

// ---------------------------------------------------------------- resampling

constexpr int kScanThreads = 256;
constexpr int kScanItems = 4;
constexpr int kScanTile = kScanThreads * kScanItems;
constexpr int kMaxSegments = 1024;
constexpr int kSumsThreads = 1024;
constexpr int kSumsItems = 4;
constexpr int kSumsChunk = kSumsThreads * kSumsItems;   // a whole number of scan tiles
static_assert(kSumsChunk % kScanTile == 0, "chunks of the double sums are made of scan tiles");
static_assert(kSumsThreads == 1024, "the double sums scan one aggregate per warp in one warp");
constexpr int kNoBinade = 0x7fffffff;

// One chunk of kSumsChunk weights in the fallback's double sums (below).
struct SumsChunk {
    unsigned long long R0;   // the chunk's increment in units 2^(b-52), for a start of even parity
    unsigned long long P;    // the sum before the chunk in those units (par set)
    int b;                   // binade of every serial sum the chunk touches, or kNoBinade
    int delta;               // increment for an odd start minus R0 (+-1 at the first tie, else 0)
    int ok;                  // no weight reaches 2^(b+1): R0 and delta hold
    int par;                 // the chunk's sums follow from P and its increments
    double start;            // the sum before the chunk (par clear)
};

struct Segment {
    double u_start;   // exact float value
    double delta;     // exact float step
    long long j0;     // index of the first value
    long long n;      // number of values
};

struct ResampleWs {
    long long* cdf;         // M: inclusive fixed-point prefix within the tile
    long long* tile_sums;   // tiles
    long long* tile_off;    // tiles (exclusive)
    Segment* segs;          // kMaxSegments
    int* nseg;
    int* exact_ok;          // 1 when the parallel path reproduces the serial one
    long long* total;
    double* reach;          // the segments describe the draws below this
    int* serial;            // 1 when only the literal loop reproduces it
    double* sums;           // M serial double prefix sums (aliases cdf; used when !exact_ok)
    const float* u0p;       // the draw in device memory (replaces u0 when set)
    double* tile_dsum;      // tiles: double sum of each scan tile's weights (any order)
    int* tile_flag;         // tiles: kTileInexact, kTileWild
    int* err;               // the literal loop would never finish
    uint32_t* done;         // two block counters, 0 between calls (resample_finish_kernel)
    SumsChunk* chunks;      // ceil(M / kSumsChunk)
};

// Weight as an exact multiple of 2^-52 (its value in those units), or -1 when
// it is negative, not finite, not a multiple, or too large.
__device__ __forceinline__ long long weight_fx52(float w)
{
    uint32_t bits = __float_as_uint(w);
    if (bits == 0u || bits == 0x80000000u) return 0;
    if (bits >> 31) return -1;
    uint32_t e = (bits >> 23) & 0xffu;
    if (e == 0xffu) return -1;
    long long mant = e ? (long long)((bits & 0x7fffffu) | 0x800000u) : (long long)(bits & 0x7fffffu);
    int E = e ? (int)e - 150 : -149;
    int sh = E + 52;
    if (sh >= 0) {
        if (sh > 36) return -1;
        return mant << sh;
    }
    if (sh <= -63) return -1;
    if (mant & ((1ll << -sh) - 1)) return -1;
    return mant >> -sh;
}

// Whether the calling block is the grid's last to get here (the same on every
// thread): its writes before the call are visible to the last block, which may
// read the others' with __ldcg.  The counter returns to 0.
__device__ __forceinline__ bool last_block(uint32_t* counter)
{
    __shared__ int s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicInc(counter, gridDim.x - 1u) == gridDim.x - 1u;
    __syncthreads();
    if (s_last) __threadfence();
    return s_last != 0;
}

constexpr int kTileInexact = 1;   // a weight is not a multiple of 2^-52 (or too large)
constexpr int kTileWild = 2;      // a weight is negative or not finite

__device__ void offsets_warp(int tiles, const ResampleWs& ws);
__device__ double build_segments(int M, float u0, double s_total, const ResampleWs& ws);

// Tile-local inclusive scan of the fixed-point weights (exact integers).
// Also the tile's double sum of the weights for the fallback below, and its
// flags.  Block `tiles` describes the draws below 2 as segments meanwhile (the
// fixed-point sums stay below that); the last block to finish then forms the
// tiles' offsets.
__global__ void __launch_bounds__(kScanThreads) resample_scan_kernel(const float* w, int stride, int M, float u0,
                                                                     ResampleWs ws)
{
    chain_enter();
    if (blockIdx.x == gridDim.x - 1) {
        if (threadIdx.x == 0) *ws.reach = build_segments(M, ws.u0p ? *ws.u0p : u0, 2.0, ws);
        if (last_block(ws.done) && threadIdx.x < 32) offsets_warp((int)gridDim.x - 1, ws);
        return;
    }
    __shared__ long long warp_tot[kScanThreads / 32];
    __shared__ double warp_d[kScanThreads / 32];
    __shared__ int bad, wild;
    if (threadIdx.x == 0) bad = wild = 0;
    __syncthreads();
    const int base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    long long v[kScanItems];
    long long run = 0;
    double dsum = 0.0;
    for (int k = 0; k < kScanItems; ++k) {
        int i = base + k;
        long long f = 0;
        if (i < M) {
            const float x = w[(size_t)i * stride];
            f = weight_fx52(x);
            if (f < 0) { bad = 1; f = 0; }
            if (!(x >= 0.0f) || !(x < INFINITY)) wild = 1;
            else dsum += (double)x;
        }
        run += f;
        v[k] = run;
    }
    {
        const double d = warp_sum_d(dsum);
        if ((threadIdx.x & 31) == 0) warp_d[threadIdx.x >> 5] = d;
    }
    // inclusive scan of per-thread totals across the block
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    long long x = run;
    for (int o = 1; o < 32; o <<= 1) {
        long long y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_tot[warp] = x;
    __syncthreads();
    long long woff = 0;
    for (int k = 0; k < warp; ++k) woff += warp_tot[k];
    long long excl = woff + x - run;
    for (int k = 0; k < kScanItems; ++k) {
        int i = base + k;
        if (i < M) ws.cdf[i] = excl + v[k];
    }
    if (threadIdx.x == kScanThreads - 1) ws.tile_sums[blockIdx.x] = excl + run;
    if (threadIdx.x == 0) {
        double d = 0.0;
        for (int k = 0; k < kScanThreads / 32; ++k) d += warp_d[k];
        ws.tile_dsum[blockIdx.x] = d;
    }
    __syncthreads();
    if (threadIdx.x == 0) ws.tile_flag[blockIdx.x] = (bad ? kTileInexact : 0) | (wild ? kTileWild : 0);
    if (last_block(ws.done) && threadIdx.x < 32) offsets_warp((int)gridDim.x - 1, ws);
}

// 2^k for -1022 <= k <= 1023, exactly.
__device__ __forceinline__ double pow2(int k)
{
    return __longlong_as_double((long long)(k + 1023) << 52);
}

// V * 2^(b-52) for V in [2^52, 2^53): the double's bits directly.
__device__ __forceinline__ double binade_value(unsigned long long V, int b)
{
    return __longlong_as_double((long long)(((unsigned long long)(b + 1023) << 52) | (V - (1ull << 52))));
}

// Builds the piecewise-arithmetic description of the reference's float draw
// sequence U_{k+1} = (float)((double)U_k + 1.0/M) (novel_resampling.h:59-63)
// for all draws below s_total: inside one binade of float the step is constant
// except near its top, where single steps are taken literally.  Returns how far
// the description reaches: s_total (or the first draw past it), or less when it
// ends before (a step that would depend on the parity of U, a draw that stops
// advancing, more than kMaxSegments pieces).  Scalings by powers of two only.
__device__ double build_segments(int M, float u0, double s_total, const ResampleWs& ws)
{
    const double inv_m = 1.0 / (double)M;
    // 1/M = Mi 2^(Ei - 52): the binade arithmetic below is integer work on the
    // doubles' bits (one lane walks the binades; GB300's FP64 pipe is narrow)
    const unsigned long long ib = (unsigned long long)__double_as_longlong(inv_m);
    const unsigned long long Mi = (ib & ((1ull << 52) - 1ull)) | (1ull << 52);
    const int Ei = (int)((ib >> 52) & 0x7ff) - 1023;
    const unsigned long long kHalf29 = 1ull << 28, kMask29 = (1ull << 29) - 1ull, kTop = 1ull << 53;
    double U = (double)u0;
    long long j = 0;
    int ns = 0;
    if (!(s_total >= 0.0) || !(s_total < INFINITY)) {   // no sum of non-negative finite weights
        *ws.nseg = 0;
        return 0.0;
    }
    // the draws' and the sums' doubles are compared on their bits (a sum here
    // is >= +0, and a double >= +0 orders like its bits as a signed integer)
    const long long s_bits = __double_as_longlong(s_total);
    const long long kFltMinBits = 0x3810000000000000ll;   // 2^-126, the smallest normal float
    for (int iter = 0; __double_as_longlong(U) < s_bits; ++iter) {
        if (ns == kMaxSegments || iter > 4 * kMaxSegments) break;
        bool regular = false;
        long long cnt = 0;
        int e = 0;
        unsigned long long Ui = 0, D = 0;
        double delta = 0.0;
        if (__double_as_longlong(U) >= kFltMinBits) {   // normal float: binade [2^e, 2^(e+1))
            const unsigned long long ub = (unsigned long long)__double_as_longlong(U);
            e = (int)((ub >> 52) & 0x7ff) - 1023;
            Ui = (ub & ((1ull << 52) - 1ull)) | (1ull << 52);   // U in units g = 2^(e-52)
            // Y = rint(inv_m / g): (double)U + inv_m = U + Y g while inside the binade
            const int sh = Ei - e;
            unsigned long long Y = 0, low;   // low: Y's bits below the float ulp u = 2^29 g
            bool big = false;                // Y >= 2^53: the first step leaves the binade
            if (sh >= 0) {
                low = sh >= 29 ? 0ull : (Mi & ((1ull << (29 - sh)) - 1ull)) << sh;
                if (sh >= 11) {
                    big = true;
                } else {
                    Y = Mi << sh;
                    big = Y >= kTop;
                }
            } else {
                const int n = -sh;
                if (n < 64) {   // round half to even
                    const unsigned long long q = Mi >> n, rem = Mi & ((1ull << n) - 1ull), half = 1ull << (n - 1);
                    Y = q + ((rem > half || (rem == half && (q & 1ull))) ? 1ull : 0ull);
                }
                low = Y & kMask29;
            }
            if (low == kHalf29) break;   // step would depend on the parity of U
            if (!big) {
                // delta = rint(Y g / u) u = R 2^29 g
                const unsigned long long R = (Y >> 29) + (low > kHalf29 ? 1ull : 0ull);
                if (R == 0) break;        // U would stop advancing
                D = R << 29;
                {   // delta = R 2^(e-23), built from its bits (R < 2^25)
                    const int lz = __clzll((long long)R);
                    delta = __longlong_as_double(((long long)(63 - lz + e - 23 + 1023) << 52) |
                                                 (long long)((R << (lz - 11)) & ((1ull << 52) - 1ull)));
                }
                // values U + i delta below top = 2^(e+1) - Y g take the regular step
                const unsigned long long T = kTop - Y;
                if (Ui < T) {
                    const unsigned long long num = (T - Ui + D - 1ull) >> 29;   // below 2^24
                    cnt = (long long)((uint32_t)num / (uint32_t)R);
                    regular = cnt > 0;
                }
            }
        }
        if (regular) {
            ws.segs[ns].u_start = U;
            ws.segs[ns].delta = delta;
            ws.segs[ns].j0 = j;
            ws.segs[ns].n = cnt;
            ++ns;
            j += cnt;
            const unsigned long long V = Ui + (unsigned long long)cnt * D;   // at most 2^53 (a float value)
            U = V >= kTop ? pow2(e + 1) : binade_value(V, e);
        } else {
            ws.segs[ns].u_start = U;
            ws.segs[ns].delta = 0.0;
            ws.segs[ns].j0 = j;
            ws.segs[ns].n = 1;
            ++ns;
            j += 1;
            double next = (double)(float)(U + inv_m);
            if (!(next > U)) break;   // U stopped advancing
            U = next;
        }
    }
    *ws.nseg = ns;
    return U;
}

// The tiles' prefix offsets, and which of the forms below reproduces the
// reference (exact_ok, serial).
__device__ void offsets_warp(int tiles, const ResampleWs& ws)
{
    const int lane = threadIdx.x & 31;
    const int per = (tiles + 31) / 32, t0 = min(tiles, lane * per), t1 = min(tiles, t0 + per);
    long long loc = 0;
    int flags = 0;
    for (int t = t0; t < t1; ++t) {
        loc += __ldcg(ws.tile_sums + t);
        flags |= __ldcg(ws.tile_flag + t);
    }
    long long x = loc;   // inclusive scan over the lanes (exact integers)
    for (int o = 1; o < 32; o <<= 1) {
        const long long y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    long long off = x - loc;
    for (int t = t0; t < t1; ++t) {
        ws.tile_off[t] = off;
        off += __ldcg(ws.tile_sums + t);
    }
    const long long acc = __shfl_sync(0xffffffffu, x, 31);
    flags = __reduce_or_sync(0xffffffffu, (unsigned)flags);
    if (lane != 0) return;
    *ws.total = acc;
    *ws.err = 0;
    *ws.serial = flags & kTileWild ? 1 : 0;
    // partial sums >= 2 may round in the serial double sum
    *ws.exact_ok = !(flags & kTileInexact) && acc < (1ll << 53) && __ldcg(ws.reach) >= ldexp((double)acc, -52);
}

// Number of draws U_j below s (the count the serial loop has emitted once its
// running sum reaches s).
__device__ long long count_below(const Segment* seg, int ns, double s)
{
    int lo = 0, hi = ns;   // first segment with u_start >= s
    while (lo < hi) {
        int mid = (lo + hi) >> 1;
        if (seg[mid].u_start < s) lo = mid + 1;
        else hi = mid;
    }
    if (lo == 0) return 0;
    const Segment& g = seg[lo - 1];
    if (g.delta == 0.0) return g.j0 + 1;
    long long i = (long long)((s - g.u_start) / g.delta);
    if (i < 0) i = 0;
    while (i > 0 && g.u_start + (double)(i - 1) * g.delta >= s) --i;
    while (i < g.n && g.u_start + (double)i * g.delta < s) ++i;
    if (i > g.n) i = g.n;
    return g.j0 + i;
}

// count_below for s = c_fx 2^-52 (0 <= c_fx < 2^53), with integer operations
// only (the FP64 pipe is narrow): positive doubles order like their bits, and
// the draws of a regular segment are (A + k R) u with u = 2^(e-23) the float
// ulp of its binade, A = u_start / u, R = delta / u, so the count of those
// below s is ceil((ceil(s / u) - A) / R), clamped to [0, n].
__device__ __forceinline__ long long count_below_fx(const Segment* seg, int ns, long long c_fx)
{
    constexpr unsigned long long kM52 = (1ull << 52) - 1ull;
    long long sb = 0;   // bits of the double c_fx 2^-52 (exact)
    if (c_fx > 0) {
        const int lz = __clzll(c_fx);   // at least 11
        sb = ((long long)(63 - lz - 52 + 1023) << 52) | (long long)(((unsigned long long)c_fx << (lz - 11)) & kM52);
    }
    int lo = 0, hi = ns;   // first segment with u_start >= s
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (__double_as_longlong(seg[mid].u_start) < sb) lo = mid + 1;
        else hi = mid;
    }
    if (lo == 0) return 0;
    const Segment& g = seg[lo - 1];
    const unsigned long long db = (unsigned long long)__double_as_longlong(g.delta);
    if (db == 0ull) return g.j0 + 1;
    const unsigned long long ub = (unsigned long long)__double_as_longlong(g.u_start);
    const int e = (int)((ub >> 52) & 0x7ff) - 1023, ed = (int)((db >> 52) & 0x7ff) - 1023;
    const unsigned long long A = ((ub & kM52) | (1ull << 52)) >> 29;
    const unsigned long long R = ((db & kM52) | (1ull << 52)) >> (e + 29 - ed);
    const unsigned long long L = A + (unsigned long long)g.n * R;   // the segment's end, below 2^50
    const int t = -29 - e;   // s / u = c_fx 2^t
    unsigned long long S;    // ceil(s / u), or L when it is at least L
    if (t >= 0) {
        S = (t >= 50 || ((unsigned long long)c_fx >> (63 - t)) != 0ull) ? L : (unsigned long long)c_fx << t;
        if (S > L) S = L;
    } else {
        const int n = -t;
        S = n >= 63 ? 1ull : ((unsigned long long)c_fx + (1ull << n) - 1ull) >> n;
    }
    if (S >= L) return g.j0 + g.n;
    if (S <= A) return g.j0;
    return g.j0 + (long long)((S - A + R - 1ull) / R);
}

// Copies particle m (7 floats) to the output rows [lo, hi) below cap, or writes
// its index there.
__device__ __forceinline__ void copy_rows(const float* particles, int m, long long lo, long long hi, long long cap,
                                          float* out, uint32_t* idx_out)
{
    for (long long j = lo; j < hi && j < cap; ++j) {
        if (idx_out) idx_out[j] = (uint32_t)m;
        if (out) {
            const float* src = particles + 7 * (size_t)m;
            float* dst = out + 7 * (size_t)j;
            for (int k = 0; k < 7; ++k) dst[k] = src[k];
        }
    }
}

// Particle m receives the draws in [cdf_{m-1}, cdf_m) (novel_resampling.h:52-68):
// writes their indices and, when asked, copies of the particle.
__device__ __forceinline__ void assign_block(const float* particles, int M, float* out, uint32_t* idx_out,
                                             long long cap, uint32_t* count_out, const ResampleWs& ws, int32_t* status,
                                             Segment* seg, int per)
{
    const int ns = *ws.nseg;
    for (int k = threadIdx.x; k < ns; k += blockDim.x) seg[k] = ws.segs[k];
    __syncthreads();
    const int m = (int)blockIdx.x * per + (int)threadIdx.x;
    if ((int)threadIdx.x >= per || m >= M) return;
    const long long c_hi_fx = ws.cdf[m] + ws.tile_off[m / kScanTile];
    long long c_lo_fx = 0;
    if (m > 0) c_lo_fx = ws.cdf[m - 1] + ws.tile_off[(m - 1) / kScanTile];
    long long lo = count_below_fx(seg, ns, c_lo_fx);
    long long hi = count_below_fx(seg, ns, c_hi_fx);
    if (m == M - 1) {
        *count_out = (uint32_t)hi;
        if (hi > cap) atomicExch(status, TSDFL_ERR_CAPACITY);
    }
    copy_rows(particles, m, lo, hi, cap, out, idx_out);
}

constexpr int kChainTile = 2048;

// Fallback of the parallel systematic path for weights that are not exact
// multiples of 2^-52 (tiny or huge) but non-negative and finite: the serial
// double sums s_m = s_{m-1} + w_m of the reference loop (novel_resampling.h:
// 53-56), formed in parallel.  While the sum stays in one binade [2^b, 2^(b+1))
// every result is a multiple of u = 2^(b-52), so s_k = s_{k-1} + r_k u with
// r_k = floor(w_k / u) + [frac > 1/2] -- independent of s -- except at ties
// (frac == 1/2), which round to the even multiple.  The sum after a tie is
// always even, so the parity before a tie is that of the last tie (or the
// binade's start) XOR the low bits of the increments since: a segmented XOR
// scan.  Where the exact sum leaves the binade (or a weight reaches 2^(b+1))
// one ordinary double addition is made and the scan restarts; that happens
// about once per binade.
// The weights are cut into chunks of kSumsChunk.  Approximate double sums of
// the scan tiles tell which chunks keep every serial sum they touch inside one
// binade with a margin far above the sums' rounding (all but a few: a chunk
// per binade the running sum crosses).  Such a chunk's increment depends on
// the sum before it only through that sum's parity, at the chunk's first tie,
// so it is formed for both parities by one block per chunk
// (chunk_transfer_block); the last block to finish then chains the chunks'
// starts, walking the others weight by weight (serial_sums_block), after which one
// block per chunk forms the chained chunks' sums and gives every particle its
// draws (resample_finish_kernel).
// The chain verifies each transfer it applies (the start in the chunk's binade,
// the end below the binade's top), so the margin only decides speed, never the
// result.  Negative or non-finite weights set *ws.serial: only the literal loop
// reproduces them.  With s monotone, the draws each particle emits then follow
// from the draw segments in parallel.
// One weight in units u = 2^(b-52) of the running sum's binade [2^b, 2^(b+1)),
// from the float's bits alone (integer shifts, no FP64 operation): q =
// floor(w / u), whether the remainder is exactly half a unit (a tie) or above
// it, and whether w >= 2^(b+1).
struct FloatSplit {
    unsigned long long q;
    bool tie, above, big;
};

__device__ __forceinline__ FloatSplit split_weight(float w, int b)
{
    FloatSplit o{0ull, false, false, false};
    const uint32_t bits = __float_as_uint(w);
    int ex = (int)((bits >> 23) & 0xffu);
    unsigned long long man = bits & 0x7fffffu;
    if (man == 0ull && ex == 0) return o;   // +0
    if (ex) man |= 0x800000ull;
    else ex = 1;                            // subnormal: man * 2^-149
    // w = man * 2^(ex - 150); big: w >= 2^(b+1)
    if (man >= 0x800000ull) {
        o.big = ex - 127 >= b + 1;
    } else {
        const int k = b + 1 + 149;          // man >= 2^k
        o.big = k <= 0 ? true : (k >= 23 ? false : man >= (1ull << k));
    }
    if (o.big) return o;
    const int sh = ex - 150 + 52 - b;       // w / u = man * 2^sh
    if (sh >= 0) {
        o.q = man << sh;                    // below 2^53: w < 2^(b+1)
    } else {
        const int n = -sh;
        if (n >= 64) return o;              // far below half a unit
        o.q = n >= 32 ? 0ull : man >> n;
        const unsigned long long rem = n >= 32 ? man : man & ((1ull << n) - 1ull);
        const unsigned long long half = 1ull << (n - 1);
        o.tie = rem == half;
        o.above = rem > half;
    }
    return o;
}


// The binade of a positive normal double, and its value in units 2^(b-52).
__device__ __forceinline__ int binade_of(double s)
{
    return (int)((__double_as_longlong(s) >> 52) & 0x7ff) - 1023;
}
__device__ __forceinline__ unsigned long long binade_units(double s)
{
    return ((unsigned long long)__double_as_longlong(s) & ((1ull << 52) - 1ull)) | (1ull << 52);
}

struct ParityPrefix {   // segmented XOR: the parity state after a run of items
    uint32_t reset;     // a tie occurred in the run: the parity restarted at 0 there
    uint32_t x;         // XOR of the increments' low bits since the start or the last tie
};

__device__ __forceinline__ ParityPrefix parity_combine(ParityPrefix a, ParityPrefix b)
{
    return b.reset ? b : ParityPrefix{a.reset, a.x ^ b.x};
}

// The increments of the staged weights sw[pos, t) in units 2^(b-52) for a
// running sum of parity p0 before item pos.  Thread k of the block's
// kSumsThreads takes items pos + kSumsItems k + j; incl[j] is the sum of the
// increments up to and including its item j.  Increments of weights that
// reach 2^(b+1) are 0 (big set); increments are clamped at 2^53 (where the
// sum leaves the binade anyway).  The block's threads all call it; red_par and
// red_sum are read after the call returns, so the caller synchronises before
// calling again.
struct BinadeRun {
    unsigned long long q[kSumsItems], r[kSumsItems], incl[kSumsItems];
    bool tie[kSumsItems], big[kSumsItems], valid[kSumsItems];
};

__device__ __forceinline__ void binade_increments(const float* sw, int pos, int t, int b, uint32_t p0, BinadeRun& x,
                                                  ParityPrefix* red_par, unsigned long long* red_sum)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned long long LIM = 1ull << 53;
    ParityPrefix agg{0u, 0u};
    for (int j = 0; j < kSumsItems; ++j) {
        const int i = pos + kSumsItems * tid + j;
        x.valid[j] = i < t;
        x.q[j] = 0;
        x.r[j] = 0;
        x.tie[j] = false;
        x.big[j] = false;
        if (x.valid[j]) {
            const FloatSplit f = split_weight(sw[i], b);
            x.big[j] = f.big;
            if (!f.big) {
                x.q[j] = f.q;
                x.tie[j] = f.tie;
                x.r[j] = f.q + (f.above ? 1ull : 0ull);
            }
        }
        agg = parity_combine(agg, x.tie[j] ? ParityPrefix{1u, 0u} : ParityPrefix{0u, (uint32_t)(x.r[j] & 1)});
    }
    // exclusive segmented-XOR scan of the threads' aggregates
    ParityPrefix px = agg;
    for (int o = 1; o < 32; o <<= 1) {
        ParityPrefix y{__shfl_up_sync(0xffffffffu, px.reset, o), __shfl_up_sync(0xffffffffu, px.x, o)};
        if (lane >= o) px = parity_combine(y, px);
    }
    if (lane == 31) red_par[warp] = px;
    __syncthreads();
    // the warps' aggregates before this warp: every warp scans the 32 of them
    ParityPrefix wx = red_par[lane];
    for (int o = 1; o < 32; o <<= 1) {
        ParityPrefix y{__shfl_up_sync(0xffffffffu, wx.reset, o), __shfl_up_sync(0xffffffffu, wx.x, o)};
        if (lane >= o) wx = parity_combine(y, wx);
    }
    ParityPrefix before{__shfl_sync(0xffffffffu, wx.reset, (warp + 31) & 31),
                        __shfl_sync(0xffffffffu, wx.x, (warp + 31) & 31)};
    if (warp == 0) before = ParityPrefix{0u, 0u};
    {
        ParityPrefix y{__shfl_up_sync(0xffffffffu, px.reset, 1), __shfl_up_sync(0xffffffffu, px.x, 1)};
        if (lane > 0) before = parity_combine(before, y);
    }
    uint32_t par = before.reset ? before.x : (p0 & 1u) ^ before.x;   // parity before the first item
    unsigned long long tsum = 0;
    for (int j = 0; j < kSumsItems; ++j) {
        if (x.tie[j]) {   // round half to even: +1 when the sum before plus q is odd
            x.r[j] = x.q[j] + ((par ^ (uint32_t)(x.q[j] & 1)) & 1u);
            par = 0u;
        } else {
            par ^= (uint32_t)(x.r[j] & 1);
        }
        if (x.r[j] > LIM) x.r[j] = LIM;
        tsum += x.r[j];
    }
    // exclusive sum scan of the threads' increments
    unsigned long long xs = tsum;
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, xs, o);
        if (lane >= o) xs += y;
    }
    if (lane == 31) red_sum[warp] = xs;
    __syncthreads();
    unsigned long long ws_ = red_sum[lane];
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, ws_, o);
        if (lane >= o) ws_ += y;
    }
    const unsigned long long wbefore = __shfl_sync(0xffffffffu, ws_, (warp + 31) & 31);
    unsigned long long run = xs - tsum + (warp ? wbefore : 0ull);
    for (int j = 0; j < kSumsItems; ++j) {
        run += x.r[j];
        x.incl[j] = run;
    }
}

__device__ __forceinline__ double block_sum_d(double v, double* red)
{
    v = warp_sum_d(v);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = 0.0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) t += red[k];
    __syncthreads();
    return t;
}

struct SumsShared {   // binade_increments' reductions
    unsigned long long sum[kSumsThreads / 32];
    ParityPrefix par[kSumsThreads / 32];
};

// Stages chunk c's weights in shared memory; returns its length.
__device__ __forceinline__ int stage_chunk(const float* __restrict__ w, int stride, int M, int c, float* sw)
{
    const int c0 = c * kSumsChunk, t = min(kSumsChunk, M - c0);
    for (int i = threadIdx.x; i < t; i += blockDim.x) sw[i] = w[(size_t)(c0 + i) * stride];
    return t;
}

// One block per chunk: the chunk's binade (the serial sums' bounds from the
// tiles' double sums, widened by far more than their rounding), and for a
// chunk inside one binade its increment R0 from an even start and the change
// delta for an odd one.
__device__ __forceinline__ void chunk_transfer_block(const float* __restrict__ w, int stride, int M,
                                                     const ResampleWs& ws, float* sw, SumsShared& sh)
{
    __shared__ double red_d[kSumsThreads / 32];
    __shared__ int s_b, s_first, s_big;
    const int c = blockIdx.x, tid = threadIdx.x;
    constexpr int kTilesPerChunk = kSumsChunk / kScanTile;
    const int tiles = (M + kScanTile - 1) / kScanTile;
    const int t0 = c * kTilesPerChunk, t1 = min(t0 + kTilesPerChunk, tiles);
    double a = 0.0, e = 0.0;
    for (int i = tid; i < t0; i += kSumsThreads) a += ws.tile_dsum[i];
    for (int i = t0 + tid; i < t1; i += kSumsThreads) e += ws.tile_dsum[i];
    a = block_sum_d(a, red_d);
    e = block_sum_d(e, red_d);
    if (tid == 0) {
        // |serial - approximate| <= (M + tiles + 2 kScanTile) 2^-53 relative: widen by 4x that
        const double eps = ((double)M + (double)tiles + 2.0 * kScanTile) * 0x1p-51;
        const double lo = a * (1.0 - eps), hi = (a + e) * (1.0 + eps);
        int b = kNoBinade;
        if (a > 0.0 && lo > 0.0 && binade_of(lo) == binade_of(hi)) b = binade_of(lo);
        s_b = b;
        s_first = kSumsChunk;
        s_big = 0;
        SumsChunk& k = ws.chunks[c];
        k.b = b;
        k.ok = 0;
        k.par = 0;
        k.delta = 0;
        k.R0 = 0;
        k.P = 0;
        k.start = 0.0;
    }
    __syncthreads();
    const int b = s_b;
    if (b == kNoBinade) return;
    const int t = stage_chunk(w, stride, M, c, sw);
    __syncthreads();
    BinadeRun x;
    binade_increments(sw, 0, t, b, 0u, x, sh.par, sh.sum);
    bool big = false;
    for (int j = 0; j < kSumsItems; ++j) {
        big |= x.big[j];
        if (x.tie[j]) atomicMin(&s_first, kSumsItems * tid + j);
    }
    if (big) s_big = 1;
    __syncthreads();
    SumsChunk& k = ws.chunks[c];
    for (int j = 0; j < kSumsItems; ++j)   // r(odd start) - r(even start) at the first tie
        if (kSumsItems * tid + j == s_first) k.delta = x.r[j] == x.q[j] ? 1 : -1;
    if (tid == kSumsThreads - 1) {
        k.R0 = x.incl[kSumsItems - 1];
        k.ok = s_big ? 0 : 1;
    }
}

__device__ void systematic_chain_block(const float* __restrict__ w, int stride, int M, float u0,
                                       uint32_t* __restrict__ cnt, uint32_t* __restrict__ off,
                                       unsigned long long* total, int* err, unsigned char* buf);

// The chain: one block walks the chunks in order, applying the transfers of
// chunks inside one binade (thread 0, checked) and forming the others' sums
// weight by weight; then thread 0 describes the draws below the total as
// segments.  Where only the literal loop reproduces the reference (*ws.serial:
// set by the scan for negative or non-finite weights, or here when the draws
// cannot be described), the block walks that instead.
__device__ void serial_sums_block(const float* __restrict__ w, int stride, int M, float u0, const ResampleWs& ws,
                                  float* sw, SumsShared& sh)
{
    __shared__ double s_s, s_prev;
    __shared__ int s_pos, s_e, s_c;
    const int tid = threadIdx.x;
    const int chunks = (M + kSumsChunk - 1) / kSumsChunk;
    const unsigned long long LIM = 1ull << 53;
    if (tid == 0) {
        s_s = 0.0;
        s_c = 0;
    }
    __syncthreads();
    for (;;) {
        if (tid == 0) {   // chunks inside one binade: only their starts
            int c = s_c;
            double sum = s_s;
            for (; c < chunks; ++c) {
                SumsChunk& k = ws.chunks[c];   // another block's transfer: read past the L1
                const int kb = __ldcg(&k.b);
                if (kb == kNoBinade || !__ldcg(&k.ok) || !(sum > 0.0) || binade_of(sum) != kb) break;
                const unsigned long long P = binade_units(sum);
                const unsigned long long E =
                    P + __ldcg(&k.R0) + ((P & 1ull) ? (unsigned long long)(long long)__ldcg(&k.delta) : 0ull);
                if (E >= LIM) break;
                k.P = P;
                k.par = 1;
                sum = binade_value(E, kb);
            }
            s_c = c;
            s_s = sum;
            if (c < chunks) ws.chunks[c].start = sum;
        }
        __syncthreads();
        const int c = s_c;
        if (c >= chunks) break;
        const int c0 = c * kSumsChunk;
        const int t = stage_chunk(w, stride, M, c, sw);
        if (tid == 0) s_pos = 0;
        __syncthreads();
        for (int guard = 0; guard <= kSumsChunk; ++guard) {   // one pass per event: at most t + 1
            const int pos = s_pos;
            if (pos >= t) break;
            const double s = s_s;
            if (tid == 0) s_e = t;
            __syncthreads();
            if (s == 0.0) {   // leading zero weights keep the sum 0; the first positive one is the sum
                for (int i = pos + tid; i < t; i += kSumsThreads)
                    if (sw[i] > 0.0f) atomicMin(&s_e, i);
                __syncthreads();
                const int z = s_e;
                for (int i = pos + tid; i < z; i += kSumsThreads) ws.sums[c0 + i] = 0.0;
                if (tid == 0) {
                    if (z < t) {
                        s_s = (double)sw[z];
                        ws.sums[c0 + z] = s_s;
                    }
                    s_pos = z < t ? z + 1 : t;
                }
                __syncthreads();
                continue;
            }
            const int b = binade_of(s);   // s in [2^b, 2^(b+1))
            const unsigned long long P0 = binade_units(s);
            BinadeRun x;
            binade_increments(sw, pos, t, b, (uint32_t)(P0 & 1ull), x, sh.par, sh.sum);
            for (int j = 0; j < kSumsItems; ++j) {
                const int i = pos + kSumsItems * tid + j;
                const unsigned long long before = x.incl[j] - x.r[j];
                if (x.valid[j] && (x.big[j] || P0 + before + x.q[j] >= LIM)) atomicMin(&s_e, i);   // leaves the binade
            }
            __syncthreads();
            const int e = s_e;
            for (int j = 0; j < kSumsItems; ++j) {   // below e every sum stays in the binade
                const int i = pos + kSumsItems * tid + j;
                if (i < e) ws.sums[c0 + i] = binade_value(P0 + x.incl[j], b);
                if (i == e - 1) s_prev = binade_value(P0 + x.incl[j], b);
            }
            __syncthreads();
            if (tid == 0) {
                const double prev = e > pos ? s_prev : s;
                if (e < t) {
                    const double nx = prev + (double)sw[e];   // one ordinary double addition
                    ws.sums[c0 + e] = nx;
                    s_s = nx;
                    s_pos = e + 1;
                } else {
                    s_s = prev;
                    s_pos = t;
                }
            }
            __syncthreads();
        }
        if (tid == 0) s_c = c + 1;
        __syncthreads();
    }
    if (tid == 0 && !(build_segments(M, u0, s_s, ws) >= s_s)) *ws.serial = 1;   // s_s: the total
    __syncthreads();
}

// The draws' copies on the exact path (`per` particles a block); else the first part of the fallbacks: the
// chunks' transfers, then (the last block) their chain, or the literal loop.
constexpr int kAssignBytes = kMaxSegments * (int)sizeof(Segment);
static_assert(kAssignBytes >= kSumsChunk * (int)sizeof(float) && kAssignBytes >= 3 * 2048 * 4, "one buffer for all");

__global__ void __launch_bounds__(kSumsThreads) resample_assign_kernel(const float* particles,
                                                                       const float* __restrict__ w, int stride, int M,
                                                                       float u0, float* out, uint32_t* idx_out,
                                                                       long long cap, uint32_t* count_out,
                                                                       ResampleWs ws, uint32_t* cnt, uint32_t* off,
                                                                       int32_t* status, int per)
{
    chain_enter();
    __shared__ __align__(16) unsigned char buf[kAssignBytes];
    __shared__ SumsShared sh;
    if (*ws.exact_ok) {
        assign_block(particles, M, out, idx_out, cap, count_out, ws, status, reinterpret_cast<Segment*>(buf), per);
        return;
    }
    float* sw = reinterpret_cast<float*>(buf);
    if (!*ws.serial && (int)blockIdx.x < (M + kSumsChunk - 1) / kSumsChunk) chunk_transfer_block(w, stride, M, ws, sw, sh);
    if (!last_block(ws.done + 1)) return;
    if (ws.u0p) u0 = *ws.u0p;
    if (!*ws.serial) serial_sums_block(w, stride, M, u0, ws, sw, sh);
    if (*ws.serial)
        systematic_chain_block(w, stride, M, u0, cnt, off, reinterpret_cast<unsigned long long*>(ws.total), ws.err, buf);
}

__device__ void scatter_block(const float* particles, int M, const uint32_t* cnt, const uint32_t* off,
                              const unsigned long long* total, const int* err, float* out, uint32_t* idx_out,
                              long long cap, uint32_t* count_out, int32_t* status);

// The fallbacks' second part (at once over on the exact path): from the literal
// loop's counts and offsets (*ws.serial), else one block per chunk -- the chunk's
// serial double sums from the start the chain gave it, or as the chain stored
// them, and particle m receives the draws in [s_{m-1}, s_m).
__global__ void __launch_bounds__(kSumsThreads) resample_finish_kernel(const float* particles,
                                                                       const float* __restrict__ w, int stride, int M,
                                                                       float* out, uint32_t* idx_out, long long cap,
                                                                       uint32_t* count_out, ResampleWs ws,
                                                                       const uint32_t* cnt, const uint32_t* off,
                                                                       int32_t* status)
{
    chain_enter();
    __shared__ float sw[kSumsChunk];
    __shared__ SumsShared sh;
    // the counters start the next call at 0, whatever overlapping calls on one context
    // (whose results race anyway) may have left in them
    if (blockIdx.x == 0 && threadIdx.x < 2) ws.done[threadIdx.x] = 0u;
    if (*ws.exact_ok) return;
    if (*ws.serial) {
        scatter_block(particles, M, cnt, off, reinterpret_cast<const unsigned long long*>(ws.total), ws.err, out, idx_out,
                      cap, count_out, status);
        return;
    }
    const int c = blockIdx.x;
    if (c >= (M + kSumsChunk - 1) / kSumsChunk) return;
    const SumsChunk k = ws.chunks[c];
    const int c0 = c * kSumsChunk, t = min(kSumsChunk, M - c0), ns = *ws.nseg;
    double s[kSumsItems + 1];   // the sums before and after this thread's items
    if (k.par) {
        stage_chunk(w, stride, M, c, sw);
        __syncthreads();
        BinadeRun x;
        binade_increments(sw, 0, t, k.b, (uint32_t)(k.P & 1ull), x, sh.par, sh.sum);
        s[0] = binade_value(k.P + x.incl[0] - x.r[0], k.b);
        for (int j = 0; j < kSumsItems; ++j) s[j + 1] = binade_value(k.P + x.incl[j], k.b);
    } else {
        const int i = kSumsItems * (int)threadIdx.x;
        s[0] = i == 0 ? k.start : (i <= t ? ws.sums[c0 + i - 1] : 0.0);
        for (int j = 0; j < kSumsItems; ++j) s[j + 1] = i + j < t ? ws.sums[c0 + i + j] : 0.0;
    }
    const int i = kSumsItems * (int)threadIdx.x;
    long long lo = i < t ? count_below(ws.segs, ns, s[0]) : 0;
    for (int j = 0; j < kSumsItems && i + j < t; ++j) {
        const int m = c0 + i + j;
        const long long hi = count_below(ws.segs, ns, s[j + 1]);
        if (m == M - 1) {
            *count_out = (uint32_t)hi;
            if (hi > cap) atomicExch(status, TSDFL_ERR_CAPACITY);
        }
        copy_rows(particles, m, lo, hi, cap, out, idx_out);
        lo = hi;
    }
}

// SystematicResampler's loop (novel_resampling.h:41-72) literally, for the
// weights the parallel path cannot reproduce exactly (negative, tiny or huge):
// one thread walks it over tiles of weights the block stages in shared memory,
// writing every particle's count and exclusive offset; the copies are made in
// parallel afterwards.  A draw that stops advancing or a count beyond 4M + 16
// (the reference would never finish) stops the walk and sets *err.  Run by one
// block when *ws.serial is set (neither parallel form applies).
__device__ void systematic_chain_block(const float* __restrict__ w, int stride, int M, float u0,
                                       uint32_t* __restrict__ cnt, uint32_t* __restrict__ off,
                                       unsigned long long* total, int* err, unsigned char* buf)
{
    float* sw = reinterpret_cast<float*>(buf);
    uint32_t* sc = reinterpret_cast<uint32_t*>(sw + kChainTile);
    uint32_t* so = sc + kChainTile;
    __shared__ int s_stop;
    const double inv_m = 1.0 / (double)M;
    float u = u0;
    double s = 0.0;
    unsigned long long n = 0;
    if (threadIdx.x == 0) s_stop = 0;
    for (int base = 0; base < M; base += kChainTile) {
        const int t = min(kChainTile, M - base);
        for (int i = threadIdx.x; i < t; i += blockDim.x) sw[i] = w[(size_t)(base + i) * stride];
        __syncthreads();
        if (threadIdx.x == 0) {
            bool stop = false;   // kept in a register: the loop reads no shared flag
#pragma unroll 4
            for (int i = 0; i < t; ++i) {
                uint32_t k = 0;
                s += (double)sw[i];
                while (s > (double)u) {
                    ++k;
                    const float next = (float)((double)u + inv_m);
                    if (next == u || n + k > 4ull * (unsigned long long)M + 16ull) {   // would never finish
                        stop = true;
                        break;
                    }
                    u = next;
                }
                sc[i] = k;
                so[i] = (uint32_t)n;
                n += k;
                if (n >= (1ull << 31)) stop = true;   // offsets stay 32-bit
                if (stop) break;
            }
            *total = n;
            s_stop = stop ? 1 : 0;
        }
        __syncthreads();
        if (s_stop) {
            if (threadIdx.x == 0) *err = 1;
            return;
        }
        for (int i = threadIdx.x; i < t; i += blockDim.x) {
            cnt[base + i] = sc[i];
            off[base + i] = so[i];
        }
        __syncthreads();
    }
}

// Copies particle m (7 floats) to its cnt[m] output slots below cap, or writes
// its index there; thread 0 reports the count (and the chain's failure).
__device__ void scatter_block(const float* particles, int M, const uint32_t* cnt, const uint32_t* off,
                              const unsigned long long* total, const int* err, float* out, uint32_t* idx_out,
                              long long cap, uint32_t* count_out, int32_t* status)
{
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (*err) {
        if (m == 0) {
            *count_out = (uint32_t)*total;
            atomicExch(status, TSDFL_ERR_UNSUPPORTED);
        }
        return;
    }
    if (m == 0) {
        *count_out = (uint32_t)*total;
        if ((long long)*total > cap) atomicExch(status, TSDFL_ERR_CAPACITY);
    }
    if (m >= M) return;
    const long long o = off[m];
    copy_rows(particles, m, o, o + (long long)cnt[m], cap, out, idx_out);
}

// Best particle of mcl_3d.cpp:382-394: the first index with the largest weight
// above 0 (strict comparison from max_value = 0).  Keys (weight bits, ~index)
// order positive floats by value and equal weights by the lower index.
__global__ void best_particle_kernel(const float* particles, int M, unsigned long long* key)
{
    unsigned long long best = 0ull;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < M; i += gridDim.x * blockDim.x) {
        const float w = particles[7 * (size_t)i + 6];
        if (w > 0.0f) {
            const unsigned long long k = ((unsigned long long)__float_as_uint(w) << 32) | (0xffffffffu - (uint32_t)i);
            best = k > best ? k : best;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long y = __shfl_xor_sync(0xffffffffu, best, o);
        best = y > best ? y : best;
    }
    if ((threadIdx.x & 31) == 0 && best) atomicMax(key, best);
}

__global__ void best_index_kernel(const unsigned long long* key, uint32_t* index_out)
{
    const unsigned long long k = *key;
    *index_out = k ? 0xffffffffu - (uint32_t)(k & 0xffffffffu) : 0xffffffffu;
}

// ------------------------------------------------------------- map layouts

__global__ void halves_kernel(const uint16_t* codes, const float* values, const float* data, size_t n,
                              uint16_t* h16)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const float v = codes ? values[codes[i]] : data[i];
        h16[i] = __half_as_ushort(__float2half_rn(v));
    }
}

// Grid layout: output brick j of the bounding box order with skirts -- for
// j < 2 up_dim_2 brick j / 2 of the lowest layer (odd j) behind its skirt (even
// j), beyond that brick j - up_dim_2 -- copied from the code array, whose
// leading miss brick is what the skirt of the first allocated brick reads.
__global__ void grid_fill_kernel(const uint16_t* codes, const int32_t* grid_occ, uint64_t uxy, uint64_t s3,
                                 uint64_t n, uint16_t* grid)
{
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t j = i / s3, t = i - j * s3;
        const bool low = j < 2 * uxy;
        const uint64_t up = low ? j >> 1 : j - uxy;
        const bool skirt = low && (j & 1) == 0;
        const int32_t base = grid_occ[up];
        grid[i] = base < 0 ? (uint16_t)kCodeMiss : codes[(int64_t)base + (int64_t)t - (skirt ? (int64_t)s3 : 0)];
    }
}

__global__ void codes_from_floats_kernel(const float* data, size_t n, const float* values, float init_value,
                                         uint16_t* codes, int32_t* fail)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        float v = data[i];
        uint32_t vb = __float_as_uint(v);
        int code = -1;
        if (vb == __float_as_uint(init_value)) {
            code = kCodeInit;
        } else {
            // likelihood values decrease with |tsdf|: binary search, then exact match
            int lo = 0, hi = kCodeInit - 1;
            while (lo < hi) {
                int mid = (lo + hi) >> 1;
                if (values[mid] > v) lo = mid + 1;
                else hi = mid;
            }
            for (int c = max(0, lo - 2); c <= min(kCodeInit - 1, lo + 2); ++c)
                if (__float_as_uint(values[c]) == vb) { code = c; break; }
        }
        if (code < 0) {
            atomicExch(fail, 1);
            code = kCodeInit;
        }
        codes[i] = (uint16_t)code;
    }
}


int check(cudaError_t e)
{
    return e == cudaSuccess ? TSDFL_OK : TSDFL_ERR_DEVICE;
}

}  // namespace

// ------------------------------------------------------------------ launchers

int launch_pose_prepare(const float* tf, const float* particles, int P, const float* points, int N, int npad,
                        float max_range_sq, float c_in, float c_out, const float* code_values, int shift, bool order,
                        const EvalBuffers& b, cudaStream_t s)
{
    Tf16 t;
    for (int k = 0; k < 16; ++k) t.v[k] = tf[k];
    const int groups = (P + kPoseSlots - 1) / kPoseSlots;   // a warp each
    const int warps = std::max(1, std::min(kPoseThreads / 32, (groups + kPoseBlocks - 1) / kPoseBlocks));
    PointParams p{points, N, npad, 32 * ((N + 63) / 64), particles, P, max_range_sq, c_in, c_out, code_values,
                  shift, order ? 1 : 0, warps};
    const unsigned blocks = (unsigned)((groups + warps - 1) / warps + kPrepBlocks - 1) / kPrepBlocks * kPrepBlocks;
    launch_chained_clusters(pose_prepare_kernel, kPrepBlocks + blocks, kPrepBlocks, kPoseThreads, s, t, p, b);
    g_launches += 1;
    return check(cudaGetLastError());
}

int launch_particle_order(const float* particles, int P, const EvalBuffers& b, cudaStream_t s)
{
    if (P <= 0) return TSDFL_OK;
    // the cell histogram was cleared by pose_prepare_kernel (or, for another order of the
    // same poses, by the caller): the scatter leaves the cells' ends in it
    const unsigned blocks = (unsigned)std::min((P + 255) / 256, 4096);
    launch_chained(particle_cells_kernel, blocks, 256, 0, s, particles, P, b);
    launch_chained(particle_scan_kernel, 1, kCellScanThreads, 0, s, b);
    launch_chained(particle_scatter_kernel, blocks, 256, 0, s, P, b);
    g_launches += 3;
    return check(cudaGetLastError());
}

size_t eval_smem_bytes(bool serial, int n)
{
    int npad = (n + 3) & ~3;
    return serial ? (size_t)kLutFBytes + 4ull * npad * 4 : (size_t)kLutBytes + 3ull * npad * 4;
}

using TiledKernel = void (*)(TiledParams);

// The wide and the debug kernels come without the shortcut for a min corner at the
// origin, and the debug ones wide only: sums and hits are the same.
template <int LAY, bool TWO>
TiledKernel pick_tiled_2(bool dbg, bool min0, bool packed)
{
    if (dbg) return eval_tiled_kernel<LAY, TWO, true, false, false>;
    if (!packed) return eval_tiled_kernel<LAY, TWO, false, false, false>;
    return min0 ? eval_tiled_kernel<LAY, TWO, false, true, true> : eval_tiled_kernel<LAY, TWO, false, false, true>;
}

template <int LAY>
TiledKernel pick_tiled_1(bool two, bool dbg, bool min0, bool packed)
{
    return two ? pick_tiled_2<LAY, true>(dbg, min0, packed) : pick_tiled_2<LAY, false>(dbg, min0, packed);
}

TiledKernel pick_tiled(int lay, bool two, bool dbg, bool min0, bool packed)
{
    switch (lay) {
    case kLayBitmap: return pick_tiled_1<kLayBitmap>(two, dbg, min0, packed);
    case kLayHash: return pick_tiled_1<kLayHash>(two, dbg, min0, packed);
    case kLayGrid: return pick_tiled_1<kLayGrid>(two, dbg, min0, packed);
    default: return pick_tiled_1<kLayTable>(two, dbg, min0, packed);
    }
}

using SpreadKernel = void (*)(SpreadParams);

template <int LAY, bool TWO>
SpreadKernel pick_spread_2(bool min0, bool packed)
{
    if (!packed) return eval_spread_kernel<LAY, TWO, false, false>;
    return min0 ? eval_spread_kernel<LAY, TWO, true, true> : eval_spread_kernel<LAY, TWO, false, true>;
}

template <int LAY>
SpreadKernel pick_spread_1(bool two, bool min0, bool packed)
{
    return two ? pick_spread_2<LAY, true>(min0, packed) : pick_spread_2<LAY, false>(min0, packed);
}

SpreadKernel pick_spread(int lay, bool two, bool min0, bool packed)
{
    switch (lay) {
    case kLayBitmap: return pick_spread_1<kLayBitmap>(two, min0, packed);
    case kLayHash: return pick_spread_1<kLayHash>(two, min0, packed);
    case kLayGrid: return pick_spread_1<kLayGrid>(two, min0, packed);
    default: return pick_spread_1<kLayTable>(two, min0, packed);
    }
}

size_t tiled_smem_bytes(const MapView& m, bool dense, int n)
{
    return (size_t)kLutTableBytes + (dense ? (size_t)m.occ_bytes : 0) + (size_t)(32 * ((n + 63) / 64)) * 24 +
           sizeof(float4) * kRing * kTiledWarps;
}

int tiled_warps_per_cta() { return kTiledWarps; }

int tiled_pass_points(const MapView& m, bool dense)
{
    const size_t budget = kMaxDynamicSmem;
    size_t fixed = tiled_smem_bytes(m, dense, 0);
    if (fixed >= budget) return 0;
    size_t pts = (budget - fixed) / 12 / 64 * 64;
    return (int)(pts < (size_t)kMaxPassPoints ? pts : (size_t)kMaxPassPoints);
}

int launch_eval_pass(const MapView& m, float a_hit, int P, int n0, int n1, int n_total, bool first, bool serial,
                     bool dense, bool generic, const EvalBuffers& b, double* sum_f64, int sm_count, cudaStream_t s)
{
    EvalParams p;
    p.m = m;
    p.pose12 = b.pose12;
    p.xs = b.xs; p.ys = b.ys; p.zs = b.zs; p.cs = b.cs;
    p.pxy = b.pxy; p.pz = b.pz; p.perm = b.perm;
    p.lut_fx = b.lut_fx;
    p.lut_f = b.lut_f;
    p.sum_fx = b.sum_fx;
    p.sum_f64 = sum_f64;
    p.raw = b.raw;
    p.hits = b.hits;
    p.dbg = b.dbg_index;
    p.order = b.order;
    p.sched = b.counts + 2;
    p.status = b.status;
    p.P = P; p.n0 = n0; p.n1 = n1; p.n_total = n_total; p.first_pass = first ? 1 : 0;
    p.a_hit = a_hit;
    size_t smem = eval_smem_bytes(serial, n1 - n0);
    const bool f32 = m.storage != 0;   // value slots (float or half) rather than codes
    if (serial) {
        auto k = f32 ? eval_serial_kernel<true> : eval_serial_kernel<false>;
        if (allow_smem(k, kMaxDynamicSmem) != cudaSuccess) return TSDFL_ERR_DEVICE;
        k<<<(P + 255) / 256, 256, smem, s>>>(p);
        g_launches += 1;
    } else if (!f32 && m.tiled && !generic) {
        // one launch covers the whole scan; sums are accumulated with atomics
        TiledParams tp;
        tp.e = p;
        tp.work = b.work;
        // as many chunks as kTiledChunk makes, of equal length
        const int parts = (n1 - n0 + kTiledChunk - 1) / kTiledChunk;
        tp.chunk = ((n1 - n0 + parts - 1) / parts + 63) / 64 * 64;
        tp.group = kTiledGroup;
        // small filters: smaller work items (fewer particles, then fewer points)
        // until the grid has about two per warp; the sums are exact integers,
        // so the shape changes no result
        auto items_of = [&](int chunk, int group) {
            return (long long)((n1 - n0 + chunk - 1) / chunk) * (long long)((P + group - 1) / group);
        };
        const long long want = 2ll * sm_count * kTiledWarps;
        // mid-size filters: fewer particles an item until there are about sixteen
        // per warp, so that the last items to finish are short (20,000 particles x
        // 4,099 points: 334 -> 316 us)
        while (tp.group > 1 && items_of(tp.chunk, tp.group) < 8 * want) tp.group /= 2;
        while (items_of(tp.chunk, tp.group) < want && (tp.group > 1 || tp.chunk > 256)) {
            if (tp.group > 1) tp.group /= 2;
            else tp.chunk = (tp.chunk / 2 + 63) / 64 * 64;
        }
        tp.groups = (P + tp.group - 1) / tp.group;
        tp.items = ((n1 - n0 + tp.chunk - 1) / tp.chunk) * tp.groups;
        // sub_fast 2: floor(s * sub_inv) is the sub-voxel index; 1: the two-term multiplier
        const bool two = m.sub_fast == 1, dbg = p.dbg != nullptr;
        // the slot: from the brick index alone on the grid layout; else the brick
        // rank from the shared-memory bitmap, the sparse brick hash when the map
        // has one, or the brick table
        const int lay = m.grid_b ? kLayGrid : (dense ? kLayBitmap : (m.hash ? kLayHash : kLayTable));
        size_t tsmem = tiled_smem_bytes(m, dense, n1 - n0);
        // pose_prepare_kernel cleared sum_fx and hits before the first pass
        int blocks = sm_count;
        int need = (tp.items + kTiledWarps - 1) / kTiledWarps;
        if (need < blocks) blocks = need > 0 ? need : 1;
        auto k = pick_tiled(lay, two, dbg, m.min0 != 0, b.packed != 0);
        if (allow_smem(k, kMaxDynamicSmem) != cudaSuccess) return TSDFL_ERR_DEVICE;
        launch_chained(k, (unsigned)blocks, kTiledThreads, tsmem, s, tp);
        g_launches += 1;
        // the debug kernel scores either kind of cloud; otherwise the one of the
        // two kernels that the staging kernel's choice is not meant for returns at
        // once.  The spread one takes the whole scan, beside the first pass.
        if (!dbg && first && order_particles((size_t)P, (size_t)n_total)) {
            SpreadParams sp;
            sp.e = p;
            sp.work = b.work + 2;
            sp.chunks = (n_total + 64 * kSpreadBlocks - 1) / (64 * kSpreadBlocks);
            sp.groups = (P + kSpreadGroup - 1) / kSpreadGroup;
            sp.items = (unsigned long long)sp.chunks * (unsigned long long)sp.groups;
            const size_t ssmem = spread_smem_bytes(lay == kLayBitmap ? m.occ_bytes : 0u);
            auto ks = pick_spread(lay, two, m.min0 != 0, b.packed != 0);
            if (allow_smem(ks, kMaxDynamicSmem) != cudaSuccess) return TSDFL_ERR_DEVICE;
            launch_chained(ks, (unsigned)sm_count, kSpreadThreads, ssmem, s, sp);
            g_launches += 1;
        }
    } else {
        auto k = dense && !f32 ? eval_exact_kernel<true, 0>
                               : (m.storage == 2 ? eval_exact_kernel<false, 2>
                                                 : (f32 ? eval_exact_kernel<false, 1> : eval_exact_kernel<false, 0>));
        if (allow_smem(k, kMaxDynamicSmem) != cudaSuccess) return TSDFL_ERR_DEVICE;
        int blocks = sm_count;
        int need = (P + 31) / 32;
        if (need < blocks) blocks = need > 0 ? need : 1;
        k<<<blocks, 1024, smem, s>>>(p);
        g_launches += 1;
    }
    return check(cudaGetLastError());
}

using SubKernel = void (*)(SubParams);

template <bool DENSE, bool TWO, bool STAGED>
SubKernel pick_sub_2(bool min0, bool packed)
{
    if (!packed) return eval_subsample_kernel<DENSE, TWO, false, STAGED, false>;
    return min0 ? eval_subsample_kernel<DENSE, TWO, true, STAGED, true>
                : eval_subsample_kernel<DENSE, TWO, false, STAGED, true>;
}

template <bool DENSE, bool STAGED>
SubKernel pick_sub(bool two, bool min0, bool packed)
{
    return two ? pick_sub_2<DENSE, true, STAGED>(min0, packed) : pick_sub_2<DENSE, false, STAGED>(min0, packed);
}

int launch_eval_subsample(const MapView& m, float a_hit, int P, int N, int K, unsigned long long seed, float c_in,
                          const EvalBuffers& b, int sm_count, cudaStream_t s)
{
    if (!m.tiled || m.storage != 0) return TSDFL_ERR_UNSUPPORTED;
    SubParams sp;
    EvalParams& p = sp.e;
    p = EvalParams{};
    p.m = m;
    p.pose12 = b.pose12;
    p.xs = b.xs; p.ys = b.ys; p.zs = b.zs; p.cs = b.cs;
    p.lut_fx = b.lut_fx;
    p.sum_fx = b.sum_fx;
    p.hits = b.hits;
    p.order = b.order;
    p.sched = b.counts + 2;
    p.status = b.status;
    p.P = P; p.n0 = 0; p.n1 = N; p.n_total = N; p.first_pass = 1;
    p.a_hit = a_hit;
    sp.K = K;
    sp.seed = seed;
    sp.nin = b.nin;
    sp.c_in = c_in;
    const bool dense = m.occ_bytes != 0, two = m.sub_fast == 1;
    const int threads = sub_threads(dense), warps_cta = threads / 32;
    size_t smem = (size_t)kLutTableBytes + (dense ? (size_t)m.occ_bytes : 0) + sizeof(float4) * kRing * warps_cta;
    // the scan beside no bitmap, where it fits: 150,000 x 200 of 5,500 points, warehouse,
    // brick table 329 us, 348 from the SoA arrays
    const bool staged = !dense && smem + sizeof(float4) * (size_t)N <= kMaxDynamicSmem;
    if (staged) smem += sizeof(float4) * (size_t)N;
    const bool min0 = m.min0 != 0, packed = b.packed != 0;
    const SubKernel k = dense    ? pick_sub<true, false>(two, min0, packed)
                        : staged ? pick_sub<false, true>(two, min0, packed)
                                 : pick_sub<false, false>(two, min0, packed);
    if (allow_smem(k, kMaxDynamicSmem) != cudaSuccess) return TSDFL_ERR_DEVICE;
    int blocks = sm_count;
    const int need = (P + warps_cta - 1) / warps_cta;
    if (need < blocks) blocks = need > 0 ? need : 1;
    sp.work = b.work;
    sp.group = P >= 32 * blocks * warps_cta ? 2 : 1;   // 300,000 x 256, building, compact: 791 us, 806 singly, 800 in fours
    sp.items = (P + sp.group - 1) / sp.group;
    k<<<blocks, threads, smem, s>>>(sp);
    g_launches += 1;
    return check(cudaGetLastError());
}

size_t batch_seg_bytes() { return sizeof(BatchSeg); }

uint32_t build_batch_segs(const BatchSegSpec* specs, int nseg, int chunk, int group, void* host_out,
                          BatchKinds* kinds)
{
    BatchSeg* out = static_cast<BatchSeg*>(host_out);
    // within a kind, the segments of one map follow each other, so that the L2
    // holds one map's footprint at a time
    std::vector<int> order(nseg);
    for (int i = 0; i < nseg; ++i) order[i] = i;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
        return reinterpret_cast<uintptr_t>(specs[a].m.codes) < reinterpret_cast<uintptr_t>(specs[b].m.codes);
    });
    uint32_t total = 0;
    int o = 0;
    for (int kind = 0; kind < kBatchKinds; ++kind) {
        kinds->first[kind] = o;
        kinds->count[kind] = 0;
        uint32_t batches = 0, items = 0;
        for (int oi = 0; oi < nseg; ++oi) {
            const BatchSegSpec& sp = specs[order[oi]];
            const int k = (!sp.b.packed ? 8 : (sp.m.min0 ? 4 : 0)) + (sp.dense ? 2 : 0) + (sp.m.sub_fast == 1 ? 1 : 0);
            if (k != kind) continue;
            const EvalBuffers& b = sp.b;
            BatchSeg g{};
            EvalParams& p = g.e;
            p.m = sp.m;
            p.pose12 = b.pose12;
            p.xs = b.xs; p.ys = b.ys; p.zs = b.zs; p.cs = b.cs;
            p.pxy = b.pxy; p.pz = b.pz; p.perm = b.perm;
            p.lut_fx = b.lut_fx;
            p.lut_f = b.lut_f;
            p.sum_fx = b.sum_fx;
            p.hits = b.hits;
            p.status = b.status;
            p.P = sp.P; p.n0 = sp.n0; p.n1 = sp.n1; p.n_total = sp.n_total; p.first_pass = sp.n0 == 0 ? 1 : 0;
            p.a_hit = sp.a_hit;
            g.chunk = chunk;
            g.group = group;
            g.groups = (sp.P + group - 1) / group;
            g.items = ((sp.n1 - sp.n0 + chunk - 1) / chunk) * g.groups;
            g.first_item = items;
            items += (uint32_t)g.items;
            batches += (uint32_t)((g.items + kBatchItems - 1) / kBatchItems);
            out[o++] = g;
            kinds->count[kind]++;
        }
        kinds->items[kind] = items;
        total += batches;
    }
    return total;
}

// 24 filters (1,000-10,000 particles, 1,000-7,500 points, three maps), scoring and
// all other kernels of an update: 2.36 ms with one queue of batches of 8 items a
// warp and barriers around each, 1.94 with batches of 2 or 1, 1.75-1.78 with a
// counter a segment and no barriers.  The kinds' launches follow one another: side by side on
// streams of their own the update took 1.87 ms.
int launch_eval_batch(void* d_segs, const BatchKinds& kinds, int32_t* status, int sm_count, cudaStream_t s)
{
    BatchSeg* segs = static_cast<BatchSeg*>(d_segs);
    const size_t smem = kMaxDynamicSmem;
    using BatchKernel = void (*)(BatchSeg*, int, uint32_t, int32_t*);
    static const BatchKernel kKinds[kBatchKinds] = {
        eval_batch_kernel<false, false, false, true>,  eval_batch_kernel<false, true, false, true>,
        eval_batch_kernel<true, false, false, true>,   eval_batch_kernel<true, true, false, true>,
        eval_batch_kernel<false, false, true, true>,   eval_batch_kernel<false, true, true, true>,
        eval_batch_kernel<true, false, true, true>,    eval_batch_kernel<true, true, true, true>,
        eval_batch_kernel<false, false, false, false>, eval_batch_kernel<false, true, false, false>,
        eval_batch_kernel<true, false, false, false>,  eval_batch_kernel<true, true, false, false>};
    int nseg = 0;
    for (int kind = 0; kind < kBatchKinds; ++kind) nseg += kinds.count[kind];
    if (nseg == 0) return TSDFL_OK;
    cudaMemset2DAsync(&segs->next, sizeof(BatchSeg), 0, sizeof(uint32_t), (size_t)nseg, s);   // the items' counters
    for (int kind = 0; kind < kBatchKinds; ++kind) {
        if (kinds.items[kind] == 0) continue;
        auto k = kKinds[kind];
        if (allow_smem(k, kMaxDynamicSmem) != cudaSuccess) return TSDFL_ERR_DEVICE;
        // no more CTAs than give every warp an item
        const unsigned blocks =
            std::min((unsigned)sm_count, (kinds.items[kind] + (unsigned)kTiledWarps - 1u) / (unsigned)kTiledWarps);
        k<<<blocks, kTiledThreads, smem, s>>>(segs + kinds.first[kind], kinds.count[kind], kinds.items[kind], status);
        g_launches += 1;
    }
    return check(cudaGetLastError());
}

int launch_norm(int P, int mode, int shift, double a_hit, double c_in, double c_out, int n_points,
                const double* sum_f64, float* particles_out, float* pose_out, const EvalBuffers& b, cudaStream_t s,
                int32_t* sticky, const uint32_t* nin, bool log_domain)
{
    // one block per kNormThreads particles, at most kNormBlocks: the block count
    // depends on P alone, so the sums' order does too
    const int nb = std::max(1, std::min(kNormBlocks, (P + kNormThreads - 1) / kNormThreads));
    NormParams q{P, mode, shift, a_hit, c_in, c_out, n_points, nin};
    launch_chained(norm_partial_kernel, (unsigned)nb, kNormThreads, 0, s, q, b, sum_f64);
    g_launches += 1;
    if (P > 0 && log_domain) {
        launch_chained(norm_final_kernel, 1, kNormThreads, 0, s, b, pose_out, nb);
        cudaMemsetAsync(b.counts + 1, 0, sizeof(int32_t), s);
        log_max_kernel<<<kNormBlocks, kNormThreads, 0, s>>>(P, b);
        log_sum_kernel<<<kNormBlocks, kNormThreads, 0, s>>>(P, b);
        log_final_kernel<<<1, kNormBlocks, 0, s>>>(b);
        normalize_log_kernel<<<(P + 255) / 256, 256, 0, s>>>(P, b, particles_out, sticky);
        g_launches += 5;
    } else {
        // at most a few blocks an SM: each adds the weight sum's partials once
        const unsigned blocks = (unsigned)std::min((P + kNormThreads - 1) / kNormThreads, kNormalizeBlocks);
        launch_chained(normalize_kernel, 1u + blocks, kNormThreads, 0, s, P, b, particles_out, pose_out, nb, sticky);
        g_launches += 1;
    }
    return check(cudaGetLastError());
}

int launch_fold_status(const int32_t* status, int n, int32_t* sticky, cudaStream_t s)
{
    fold_statuses_kernel<<<1, 1, 0, s>>>(status, n, sticky);
    g_launches += 1;
    return check(cudaGetLastError());
}

size_t resample_workspace_bytes(size_t M)
{
    size_t tiles = (M + kScanTile - 1) / kScanTile + 1;
    size_t chunks = (M + kSumsChunk - 1) / kSumsChunk + 1;
    // flags: 16 + 16 + 8 + 4 + 4 <= 64
    return 8 * (M + 3 * tiles) + 4 * (tiles + 1) + sizeof(Segment) * kMaxSegments + 64 + sizeof(SumsChunk) * chunks;
}

int launch_resample_impl(const float* particles, const float* w, int stride, size_t M, float u0, float* out,
                         uint32_t* idx_out, size_t cap, uint32_t* count_out, void* workspace, uint32_t* done,
                         int32_t* status, cudaStream_t s, const float* u0p)
{
    size_t tiles = (M + kScanTile - 1) / kScanTile;
    char* p = static_cast<char*>(workspace);
    ResampleWs ws;
    ws.cdf = reinterpret_cast<long long*>(p); p += 8 * M;
    ws.tile_sums = reinterpret_cast<long long*>(p); p += 8 * (tiles + 1);
    ws.tile_off = reinterpret_cast<long long*>(p); p += 8 * (tiles + 1);
    ws.segs = reinterpret_cast<Segment*>(p); p += sizeof(Segment) * kMaxSegments;
    ws.nseg = reinterpret_cast<int*>(p); p += 16;
    ws.exact_ok = reinterpret_cast<int*>(p);
    ws.reach = reinterpret_cast<double*>(p + 8); p += 16;
    ws.total = reinterpret_cast<long long*>(p); p += 8;
    ws.err = reinterpret_cast<int*>(p); p += 4;
    ws.serial = reinterpret_cast<int*>(p); p += 4;
    ws.tile_dsum = reinterpret_cast<double*>(p); p += 8 * (tiles + 1);
    const unsigned chunks = (unsigned)((M + kSumsChunk - 1) / kSumsChunk);
    ws.chunks = reinterpret_cast<SumsChunk*>(p); p += sizeof(SumsChunk) * (chunks + 1);
    ws.tile_flag = reinterpret_cast<int*>(p);
    ws.sums = reinterpret_cast<double*>(ws.cdf);
    ws.u0p = u0p;
    ws.done = done;
    // the literal loop reuses the prefix-sum array for counts and offsets
    uint32_t* cnt = reinterpret_cast<uint32_t*>(ws.cdf);
    uint32_t* off = cnt + M;
    const unsigned blocks = (unsigned)((M + kSumsThreads - 1) / kSumsThreads);
    // small clouds' copies over more SMs
    const int per = blocks >= 128u ? kSumsThreads : (blocks >= 32u ? 256 : 64);
    // each kernel reads what the one before it wrote: none runs after a failed launch
    cudaError_t e = launch_chained(resample_scan_kernel, (unsigned)tiles + 1u, kScanThreads, 0, s, w, stride, (int)M, u0, ws);
    if (e == cudaSuccess)
        e = launch_chained(resample_assign_kernel, (unsigned)((M + per - 1) / per), kSumsThreads, 0, s, particles, w,
                           stride, (int)M, u0, out, idx_out, (long long)cap, count_out, ws, cnt, off, status, per);
    if (e == cudaSuccess)
        e = launch_chained(resample_finish_kernel, blocks, kSumsThreads, 0, s, particles, w, stride, (int)M, out,
                           idx_out, (long long)cap, count_out, ws, (const uint32_t*)cnt, (const uint32_t*)off, status);
    g_launches += 3;
    const cudaError_t last = cudaGetLastError();
    return check(e == cudaSuccess ? last : e);
}

int launch_best_particle(const float* particles, size_t M, unsigned long long* key, uint32_t* index_out, int sm_count,
                         cudaStream_t s)
{
    cudaMemsetAsync(key, 0, sizeof(unsigned long long), s);
    unsigned blocks = (unsigned)((M + 255) / 256);
    if (blocks > (unsigned)(4 * sm_count)) blocks = (unsigned)(4 * sm_count);
    if (blocks == 0) blocks = 1;
    best_particle_kernel<<<blocks, 256, 0, s>>>(particles, (int)M, key);
    best_index_kernel<<<1, 1, 0, s>>>(key, index_out);
    g_launches += 2;
    return check(cudaGetLastError());
}

int launch_codes_from_floats(const float* data, size_t n, const float* code_values, float init_value,
                             uint16_t* codes, int32_t* fail, cudaStream_t s)
{
    if (n) codes_from_floats_kernel<<<1024, 256, 0, s>>>(data, n, code_values, init_value, codes, fail);
    return check(cudaGetLastError());
}

int launch_grid_fill(const uint16_t* codes, const int32_t* grid_occ, uint64_t up_dim_2, uint64_t sub_dim_3,
                     uint64_t n, uint16_t* grid, cudaStream_t s)
{
    if (n) grid_fill_kernel<<<4096, 256, 0, s>>>(codes, grid_occ, up_dim_2, sub_dim_3, n, grid);
    return check(cudaGetLastError());
}

int launch_halves(const uint16_t* codes, const float* code_values, const float* data, size_t n, uint16_t* h16,
                  cudaStream_t s)
{
    if (n) halves_kernel<<<1024, 256, 0, s>>>(codes, code_values, data, n, h16);
    return check(cudaGetLastError());
}


}  // namespace tsdfl
