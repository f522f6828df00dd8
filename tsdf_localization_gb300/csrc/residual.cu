// ResidualSystematicResampler::resample (novel_resampling.h:76-104), mcl_3d's
// default resampler, on the device.
//
// Its draw chain carries float roundings from particle to particle:
//   c = (float)M w;  temp = c - u;  o = (size_t)(temp + 1.0);  u = (float)o - temp
// (every operation rounded to float), particle m being emitted o times.  The
// walk is four dependent float additions a particle, about 10 ns: 0.99 ms at
// 100,000 particles when one thread walks it all.
//
// The parallel form (M of kParallelFrom and more) returns the same counts bit for bit:
//
//   * In exact arithmetic u stays congruent to u0 - (c_0 + c_1 + ...) modulo 1
//     and lies in (0, 1], so prefix sums predict it anywhere; the roundings
//     move the true value a random walk away from the prediction, a few hundred
//     units of 2^-24 at 100,000 particles (measured: at most 2.7 of the
//     standard deviations bounded below, over flat, uneven and peaked weights).
//   * Behind a particle with c >= 1 the true u is a multiple of 2^-24, behind
//     one with c >= 2 of 2^(floor(log2(c - 1)) - 23): temp is one there and
//     (float)o - temp is exact.  So the weights are cut into segments that
//     start behind the largest of the first kHead weights of a tile, and the
//     few hundred floats of that grid around the prediction (4.5 standard
//     deviations to each side) are all the starts that are likely.
//   * Every candidate start of every segment is walked, one thread each, and
//     its end kept (residual_candidates_kernel): the tables are the true chain,
//     segment by segment.
//   * One thread then follows the tables from u0, one lookup a segment
//     (residual_follow_kernel).  A start that is not among its segment's
//     candidates is walked there and then, so the window decides speed only.
//   * With every segment's start known, one block a segment walks it once more
//     for the counts and copies its particles (residual_emit_kernel).
//
// Measured (a device call, us): 100,000 particles 989 -> 50, 23,457 238 -> 32,
// a million 9,800 -> 282.  Of the 50: candidates 14, following 26 (one thread,
// about 90 cycles a segment, and the tables' way into one SM), emitting 13.
//
// Counts need no walk to be placed: a segment emits sum(c) + u_end - u_start
// up to roundings that add to less than a quarter (checked; else one thread
// walks everything).
#include <stdint.h>

#include <algorithm>
#include <atomic>
#include <cmath>

#include "chain.h"
#include "tsdfl_internal.h"

namespace tsdfl {

extern std::atomic<unsigned long long> g_launches;

namespace {

constexpr int kChainTile = 2048;
constexpr int kChainThreads = 512;
constexpr int kHead = 128;            // weights of a tile among which its segment's boundary is chosen
constexpr int kMaxTile = 4096;
constexpr int kMaxSegs = 4096;        // 2^24 particles in tiles of 4,096
constexpr int kTileThreads = 256;
constexpr int kCandThreads = 256;
constexpr int kEmitThreads = 256;
constexpr int kMaxWindow = 8192;
constexpr size_t kFollowSmem = 212 * 1024;  // shared memory of the following block, beside its static part
constexpr int kEmitRows = 1024;             // output rows the emitting block places at a time

// One step of the chain for -1 <= c - u < 2^22: rounding temp + 1.5 * 2^23
// down lands on an integer (unit spacing there), so floor(temp) + 1 takes two
// exact steps.
__device__ __forceinline__ float residual_step(float c, float u, float& of)
{
    const float temp = __fsub_rn(c, u);
    of = __fsub_rn(__fadd_rd(temp, 12582912.0f), 12582911.0f);
    return __fsub_rn(of, temp);
}

// The whole chain by one thread, for weights w >= 0 with (float)M * w <
// 2^22 - 1 (others stop it with *err), over tiles of (float)M w staged in
// shared memory; the block then turns the counts into offsets with a scan.
__device__ void residual_chain_block(const float* __restrict__ w, int stride, int M, float u0,
                                     uint32_t* __restrict__ cnt, uint32_t* __restrict__ off,
                                     unsigned long long* total, int* err)
{
    static_assert(kChainTile == 4 * kChainThreads, "four counts per thread in the scan");
    __shared__ float sc[kChainTile];   // (float)M * w, then the counts
    __shared__ uint32_t warp_tot[kChainThreads / 32];
    __shared__ uint32_t s_base;
    __shared__ int s_err;
    const float Mf = (float)M;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float u = u0;
    if (threadIdx.x == 0) {
        s_base = 0u;
        s_err = 0;
        *err = 0;
    }
    for (int base = 0; base < M; base += kChainTile) {
        const int t = min(kChainTile, M - base);
        bool bad = false;
        for (int i = threadIdx.x; i < t; i += blockDim.x) {
            const float x = w[(size_t)(base + i) * stride];
            const float c = __fmul_rn(Mf, x);
            bad |= !(x >= 0.0f) || !(c < 4194303.0f);
            sc[i] = c;
        }
        if (__syncthreads_or(bad ? 1 : 0)) {
            if (threadIdx.x == 0) {
                *err = 1;
                *total = s_base;
            }
            return;
        }
        if (threadIdx.x == 0) {
            // 32 products to registers at a time, so that only the chain is serial
            int i = 0;
            for (; i + 32 <= t; i += 32) {
                float v[32];
#pragma unroll
                for (int k = 0; k < 32; ++k) v[k] = sc[i + k];
#pragma unroll
                for (int k = 0; k < 32; ++k) {
                    float of;
                    u = residual_step(v[k], u, of);
                    v[k] = of;
                }
#pragma unroll
                for (int k = 0; k < 32; ++k) sc[i + k] = v[k];
            }
            for (; i < t; ++i) {
                float of;
                u = residual_step(sc[i], u, of);
                sc[i] = of;
            }
        }
        __syncthreads();
        // exclusive offsets of this tile's counts, four per thread
        uint32_t v[4], run = 0;
        for (int k = 0; k < 4; ++k) {
            const int i = 4 * threadIdx.x + k;
            v[k] = i < t ? (uint32_t)sc[i] : 0u;
            run += v[k];
        }
        uint32_t x = run;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) warp_tot[warp] = x;
        __syncthreads();
        uint32_t woff = 0, tile_total = 0;
        for (int k = 0; k < kChainThreads / 32; ++k) {
            if (k < warp) woff += warp_tot[k];
            tile_total += warp_tot[k];
        }
        uint32_t o = s_base + woff + x - run;
        for (int k = 0; k < 4; ++k) {
            const int i = 4 * threadIdx.x + k;
            if (i < t) {
                cnt[base + i] = v[k];
                off[base + i] = o;
            }
            o += v[k];
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            s_base += tile_total;
            if (s_base >= (1u << 31)) *err = s_err = 1;   // offsets stay 32-bit
        }
        __syncthreads();
        if (s_err) {
            if (threadIdx.x == 0) *total = s_base;
            return;
        }
    }
    if (threadIdx.x == 0) *total = s_base;
}


__global__ void __launch_bounds__(kChainThreads) residual_chain_kernel(const float* __restrict__ w, int stride,
                                                                       int M, float u0, uint32_t* cnt, uint32_t* off,
                                                                       unsigned long long* total, int* err)
{
    chain_enter();
    residual_chain_block(w, stride, M, u0, cnt, off, total, err);
}

// ------------------------------------------------------------- parallel form

struct TileSums {
    unsigned long long isum, fsum;     // sum of floor(c); of its fractions in units of 2^-48
    unsigned long long h_isum, h_fsum; // the same up to the boundary
    float var, h_var;                  // bound on the roundings' variance, units of 2^-24 squared
    float err;                         // bound on the sum of the roundings, units of 2^-24
    float c_max;                       // c of the particle before the boundary
    int head;                          // the boundary: particles of the tile before it
    int bad;                           // a weight the chain does not take
};

struct Seg {
    uint32_t woff;   // first table entry, a multiple of 4
    uint32_t lo;     // grid index of the first candidate
    uint32_t wk;     // candidates | grid shift << 16
    uint32_t begin;  // first particle
};

struct ResidualWs {
    TileSums* tiles;            // S
    Seg* segs;                  // S + 1 (the last: total entries, M)
    double* sums;               // S: sum of c over the segment
    uint32_t* table;            // ends: u 2^24, or kOffGrid | float bits
    float* start;               // S + 1
    uint32_t* base;             // S + 1: outputs before the segment
    int* mode;                  // 0: parallel, 1: one thread walks the chain
    uint32_t* cnt;              // M, mode 1
    uint32_t* off;              // M, mode 1
    unsigned long long* total;
    int* err;
    int S, tile, window;        // segments, particles a tile, most candidates a segment
    uint32_t staged;            // table entries the following block holds at a time, a multiple of 4
};

constexpr uint32_t kOffGrid = 0x80000000u;

// u in (0, 1] as a multiple of 2^-24, else its bits marked as off that grid.
__device__ __forceinline__ uint32_t grid_value(float u)
{
    const float v = u * 16777216.0f;   // exact
    const uint32_t n = (uint32_t)v;    // at most 2^24
    return (float)n == v ? n : kOffGrid | __float_as_uint(u);
}
__device__ __forceinline__ float grid_float(uint32_t v)
{
    return v & kOffGrid ? __uint_as_float(v & ~kOffGrid) : (float)v * 0x1p-24f;
}

template <typename T>
__device__ __forceinline__ T warp_add(T v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sums of a tile and its boundary.  One pass over the weights: memory-bound in
// principle (28 B a particle), a few microseconds of latency in practice.
__global__ void __launch_bounds__(kTileThreads) residual_tiles_kernel(const float* __restrict__ w, int stride, int M,
                                                                      ResidualWs ws)
{
    chain_enter();
    __shared__ unsigned long long red_i[2][kTileThreads / 32], red_f[2][kTileThreads / 32];
    __shared__ float red_v[3][kTileThreads / 32];
    __shared__ unsigned long long red_key[kHead / 32];
    __shared__ int s_head;
    const int s = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int t0 = s * ws.tile, t = min(ws.tile, M - t0);
    const float Mf = (float)M;
    unsigned long long isum = 0, fsum = 0, i0 = 0, f0 = 0;
    float var = 0.0f, err = 0.0f, v0 = 0.0f, c0 = 0.0f;
    bool bad = false;
    for (int i = tid; i < t; i += kTileThreads) {
        const float x = w[(size_t)(t0 + i) * stride];
        const float c = __fmul_rn(Mf, x);
        const bool b = !(x >= 0.0f) || !(c < 4194303.0f);
        bad |= b;
        if (b) continue;
        const float fl = floorf(c);
        const unsigned long long iv = (unsigned long long)(uint32_t)fl;
        const unsigned long long fv = __float2ull_rz((c - fl) * 281474976710656.0f);   // both exact to 2^-48
        // ulp(temp) <= e units of 2^-24, u's rounding is at most one
        const int ex = (int)(__float_as_uint(c) >> 23) - 127;
        const float e = ex < 0 ? 1.0f : __uint_as_float((uint32_t)(ex + 1 + 127) << 23);
        const float v = (e * e + 1.0f) * (1.0f / 12.0f);
        isum += iv;
        fsum += fv;
        var += v;
        err += 0.5f * (e + 1.0f);
        if (i < kHead) {   // the thread's first element
            i0 = iv;
            f0 = fv;
            v0 = v;
            c0 = c;
        }
    }
    if (warp < kHead / 32) {   // the largest c of the first kHead, the first of equals
        unsigned long long key = 0;
        if (tid < t) key = ((unsigned long long)__float_as_uint(c0) << 32) | (0xffffffffu - (uint32_t)tid);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long y = __shfl_xor_sync(0xffffffffu, key, o);
            key = y > key ? y : key;
        }
        if (lane == 0) red_key[warp] = key;
    }
    __syncthreads();
    if (tid == 0) {
        unsigned long long key = 0;
        for (int k = 0; k < kHead / 32; ++k) key = red_key[k] > key ? red_key[k] : key;
        s_head = s == 0 ? 0 : (int)(0xffffffffu - (uint32_t)key) + 1;
        ws.tiles[s].c_max = __uint_as_float((uint32_t)(key >> 32));
    }
    const int any_bad = __syncthreads_or(bad ? 1 : 0);
    const int head = s_head;
    const bool in_head = tid < head;
    const unsigned long long a = warp_add(isum), b = warp_add(fsum);
    const unsigned long long ha = warp_add(in_head ? i0 : 0ull), hb = warp_add(in_head ? f0 : 0ull);
    const float va = warp_add(var), vb = warp_add(in_head ? v0 : 0.0f), vc = warp_add(err);
    if (lane == 0) {
        red_i[0][warp] = a;
        red_i[1][warp] = ha;
        red_f[0][warp] = b;
        red_f[1][warp] = hb;
        red_v[0][warp] = va;
        red_v[1][warp] = vb;
        red_v[2][warp] = vc;
    }
    __syncthreads();
    if (tid == 0) {
        TileSums& o = ws.tiles[s];
        unsigned long long si = 0, sf = 0, hi = 0, hf = 0;
        float sv = 0.0f, hv = 0.0f, se = 0.0f;
        for (int k = 0; k < kTileThreads / 32; ++k) {
            si += red_i[0][k];
            hi += red_i[1][k];
            sf += red_f[0][k];
            hf += red_f[1][k];
            sv += red_v[0][k];
            hv += red_v[1][k];
            se += red_v[2][k];
        }
        o.isum = si;
        o.fsum = sf;
        o.h_isum = hi;
        o.h_fsum = hf;
        o.var = sv;
        o.h_var = hv;
        o.err = se;
        o.head = head;
        o.bad = any_bad;
    }
}

constexpr int kPlanThreads = 1024;
constexpr int kPlanItems = kMaxSegs / kPlanThreads;

// Predicts every segment's start and lays out its candidates: one block, a
// scan over the tiles' sums (four tiles a thread) and one over the windows.
__global__ void __launch_bounds__(kPlanThreads) residual_plan_kernel(int M, float u0, ResidualWs ws)
{
    chain_enter();
    __shared__ unsigned long long red_f[kPlanThreads / 32];
    __shared__ float red_v[kPlanThreads / 32];
    __shared__ uint32_t red_w[kPlanThreads / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int first = tid * kPlanItems;
    // exclusive prefixes of the fractions (modulo 1 in units of 2^-64) and variances
    unsigned long long f = 0;
    float v = 0.0f;
    int bad = 0;
    for (int k = 0; k < kPlanItems; ++k) {
        const int s = first + k;
        if (s >= ws.S) break;
        const TileSums& t = ws.tiles[s];
        f += t.fsum << 16;
        v += t.var;
        // two tiles meet in a segment: each below an eighth
        if (t.bad || !(t.err < 2097152.0f)) bad = 1;
    }
    unsigned long long fx = f;
    float vx = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, fx, o);
        const float z = __shfl_up_sync(0xffffffffu, vx, o);
        if (lane >= o) {
            fx += y;
            vx += z;
        }
    }
    if (lane == 31) {
        red_f[warp] = fx;
        red_v[warp] = vx;
    }
    bad = __syncthreads_or(bad);
    if (tid == 0) {
        *ws.mode = bad;
        *ws.err = 0;
    }
    if (bad) return;
    unsigned long long fb = fx - f;
    float vb = vx - v;
    for (int k = 0; k < warp; ++k) {
        fb += red_f[k];
        vb += red_v[k];
    }
    Seg seg[kPlanItems];
    uint32_t wsum = 0;
    const unsigned long long u64 = __float2ull_rz(u0 * 9223372036854775808.0f) << 1;   // u0 in [0, 1)
    for (int k = 0; k < kPlanItems; ++k) {
        const int s = first + k;
        if (s >= ws.S) break;
        const TileSums t = ws.tiles[s];
        Seg g;
        g.begin = (uint32_t)(s * ws.tile + t.head);
        // behind c >= 2, u is a multiple of 2^shift units of 2^-24
        uint32_t shift = 0;
        if (t.c_max >= 2.0f) shift = (__float_as_uint(t.c_max - 1.0f) >> 23) - 126u;
        shift = min(shift, 20u);
        const uint32_t G = 1u << (24u - shift);
        const unsigned long long pred = u64 - (fb + (t.h_fsum << 16));
        const uint32_t centre = (uint32_t)((pred + (1ull << (39 + shift))) >> (40 + shift));
        const float half = 4.5f * sqrtf(fmaxf(vb + t.h_var, 0.0f)) * __uint_as_float((127u - shift) << 23) + 2.0f;
        uint32_t W = s == 0 ? 1u : (uint32_t)fminf(2.0f * half + 1.0f, (float)ws.window);
        W = min(W, G);
        g.lo = centre - W / 2;   // modulo G
        g.wk = W | (shift << 16);
        g.woff = wsum;
        wsum += (W + 3u) & ~3u;
        seg[k] = g;
        // sum of c over [boundary, next boundary): exact integers, then one rounding
        long long si = (long long)(t.isum - t.h_isum);
        long long sf = (long long)(t.fsum - t.h_fsum);
        if (s + 1 < ws.S) {
            si += (long long)ws.tiles[s + 1].h_isum;
            sf += (long long)ws.tiles[s + 1].h_fsum;
        }
        ws.sums[s] = (double)si + (double)sf * 0x1p-48;
        fb += t.fsum << 16;
        vb += t.var;
    }
    uint32_t wx = wsum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, wx, o);
        if (lane >= o) wx += y;
    }
    if (lane == 31) red_w[warp] = wx;
    __syncthreads();
    uint32_t wb = wx - wsum;
    for (int k = 0; k < warp; ++k) wb += red_w[k];
    for (int k = 0; k < kPlanItems; ++k) {
        const int s = first + k;
        if (s >= ws.S) break;
        seg[k].woff += wb;
        ws.segs[s] = seg[k];
        if (s == ws.S - 1) ws.segs[ws.S] = Seg{wb + wsum, 0u, 0u, (uint32_t)M};
    }
}

// Stages (float)M w of particles [b0, b1) in shared memory, padded to a
// multiple of four.
__device__ __forceinline__ void stage_products(const float* __restrict__ w, int stride, float Mf, int b0, int n,
                                               float* sc)
{
    for (int i = threadIdx.x; i < n; i += blockDim.x) sc[i] = __fmul_rn(Mf, w[(size_t)(b0 + i) * stride]);
}

// Walks n staged products from u; the weights are read as float4 broadcasts.
__device__ __forceinline__ float walk(const float* sc, int n, float u)
{
    float of;
    int i = 0;
    for (; i + 4 <= n; i += 4) {
        const float4 c = *reinterpret_cast<const float4*>(sc + i);
        u = residual_step(c.x, u, of);
        u = residual_step(c.y, u, of);
        u = residual_step(c.z, u, of);
        u = residual_step(c.w, u, of);
    }
    for (; i < n; ++i) u = residual_step(sc[i], u, of);
    return u;
}

// Every candidate start of segment blockIdx.x (kCandThreads of them a block):
// four dependent float additions a particle and thread.  Bound by their latency at
// 100,000 particles (512 steps of 16 cycles), by FP32 issue at a million.
__global__ void __launch_bounds__(kCandThreads) residual_candidates_kernel(const float* __restrict__ w, int stride,
                                                                           int M, float u0, ResidualWs ws)
{
    chain_enter();
    extern __shared__ __align__(16) float sc[];
    if (*ws.mode) return;
    const int s = blockIdx.x;
    const Seg g = ws.segs[s];
    const uint32_t W = g.wk & 0xffffu, shift = g.wk >> 16;
    if (blockIdx.y * kCandThreads >= W) return;
    const int n = (int)(ws.segs[s + 1].begin - g.begin);
    stage_products(w, stride, (float)M, (int)g.begin, n, sc);
    __syncthreads();
    const uint32_t j = blockIdx.y * kCandThreads + threadIdx.x;
    if (j >= W) return;
    const uint32_t G = 1u << (24u - shift);
    const uint32_t idx = ((g.lo + j - 1u) & (G - 1u)) + 1u;   // 1 .. G
    const float u = s == 0 ? u0 : (float)(idx << shift) * 0x1p-24f;
    ws.table[g.woff + j] = grid_value(walk(sc, n, u));
}

// Follows the tables from u0: the starts of all segments, then the outputs
// before each.  One block; the tables come through shared memory, so that the
// dependent lookups of one thread take a shared-memory latency each.
__global__ void __launch_bounds__(kChainThreads) residual_follow_kernel(const float* __restrict__ w, int stride,
                                                                        int M, float u0, ResidualWs ws)
{
    chain_enter();
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_seg, s_need;
    __shared__ uint32_t red[kChainThreads / 32];
    __shared__ unsigned long long s_run;
    const int tid = threadIdx.x, S = ws.S;
    Seg* segs = reinterpret_cast<Seg*>(smem);                       // S + 1
    uint32_t* start = reinterpret_cast<uint32_t*>(segs + S + 1);    // S + 1, as grid values
    uint32_t* tab = start + ((S + 1 + 3) & ~3);                     // ws.staged
    if (!*ws.mode) {
        for (int i = tid; i <= S; i += kChainThreads) segs[i] = ws.segs[i];
        if (tid == 0) {
            s_seg = 0;
            s_need = 0;
        }
        __syncthreads();
        for (;;) {
            const int s0 = s_seg;
            if (s0 >= S) break;
            const uint32_t first = segs[s0].woff;
            const uint32_t n = min(ws.staged, segs[S].woff - first);
            const uint4* from = reinterpret_cast<const uint4*>(ws.table + first);
#pragma unroll 8
            for (uint32_t i = tid; i < n / 4; i += kChainThreads) reinterpret_cast<uint4*>(tab)[i] = from[i];
            __syncthreads();
            if (tid == 0) {
                int s = s0;
                uint32_t v = s ? start[s] : 0u;
                Seg g = segs[s];
                while (s < S) {
                    const uint32_t next = segs[s + 1].woff;
                    if (next - first > n) break;   // not staged yet
                    const uint32_t shift = g.wk >> 16, W = g.wk & 0xffffu;
                    const uint32_t j = ((v >> shift) - g.lo) & ((1u << (24u - shift)) - 1u);
                    // off the grid, or outside the window: walked below
                    const bool miss = (v & kOffGrid) || (v & ((1u << shift) - 1u)) || j >= W;
                    if (s > 0 && miss) {
                        s_need = 1;
                        break;
                    }
                    v = tab[g.woff - first + (s ? j : 0u)];
                    ++s;
                    start[s] = v;
                    g = segs[s];
                }
                s_seg = s;
            }
            __syncthreads();
            if (s_need) {   // one segment walked by one thread
                const int s = s_seg;
                const int b0 = (int)segs[s].begin, len = (int)(segs[s + 1].begin - segs[s].begin);
                float* sc = reinterpret_cast<float*>(tab);
                stage_products(w, stride, (float)M, b0, len, sc);
                __syncthreads();
                if (tid == 0) {
                    start[s + 1] = grid_value(walk(sc, len, grid_float(start[s])));
                    s_seg = s + 1;
                    s_need = 0;
                }
                __syncthreads();
            }
        }
        // outputs of every segment: sum(c) + u_end - u_start, a whole number up to roundings
        const int lane = tid & 31, warp = tid >> 5;
        if (tid == 0) s_run = 0;
        for (int b = 0; b < S; b += kChainThreads) {
            const int s = b + tid;
            uint32_t n = 0;
            if (s < S) {
                const float us = s ? grid_float(start[s]) : u0;
                n = (uint32_t)__double2ull_rn(ws.sums[s] + ((double)grid_float(start[s + 1]) - (double)us));
                ws.start[s] = us;
            }
            uint32_t x = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            if (lane == 31) red[warp] = x;
            __syncthreads();
            unsigned long long before = s_run, all = 0;
            for (int k = 0; k < kChainThreads / 32; ++k) {
                if (k < warp) before += red[k];
                all += red[k];
            }
            if (s < S) ws.base[s] = (uint32_t)(before + x - n);
            __syncthreads();
            if (tid == 0) s_run += all;
            __syncthreads();
        }
        if (tid == 0) {
            *ws.total = s_run;
            ws.base[S] = (uint32_t)s_run;
            if (s_run >= (1ull << 31)) *ws.mode = 1;   // the walk reports it
        }
        __syncthreads();
    }
    if (*ws.mode) residual_chain_block(w, stride, M, u0, ws.cnt, ws.off, ws.total, ws.err);
}

// Copies of the particles [m0, m0 + n): particle m0 + i goes to cnt[i] rows from
// row off[i] on (both in shared memory), or its index does.  The rows are
// placed kEmitRows at a time and written element by element, so that a warp's
// stores are consecutive.
__device__ __forceinline__ void emit_rows(const float* particles, uint32_t m0, int n, const uint32_t* off,
                                          uint32_t rows, uint32_t row0, float* out, uint32_t* idx_out, long long cap,
                                          uint32_t* src)
{
    for (uint32_t r0 = 0; r0 < rows; r0 += kEmitRows) {
        const uint32_t r1 = min(rows, r0 + (uint32_t)kEmitRows);
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            const uint32_t a = max(off[i], r0), b = min(i + 1 < n ? off[i + 1] : rows, r1);
            for (uint32_t r = a; r < b; ++r) src[r - r0] = m0 + (uint32_t)i;
        }
        __syncthreads();
        const long long g0 = (long long)row0 + r0;
        const int k = (int)max(0ll, min((long long)(r1 - r0), cap - g0));
        if (idx_out)
            for (int i = threadIdx.x; i < k; i += blockDim.x) idx_out[g0 + i] = src[i];
        if (out)
            for (int i = threadIdx.x; i < 7 * k; i += blockDim.x) {
                const int r = i / 7;
                out[7 * g0 + i] = particles[7 * (size_t)src[r] + (size_t)(i - 7 * r)];
            }
        __syncthreads();
    }
}

__device__ __forceinline__ void report(const unsigned long long* total, const int* err, long long cap,
                                       uint32_t* count_out, int32_t* status)
{
    *count_out = (uint32_t)*total;
    if (*err) atomicExch(status, TSDFL_ERR_UNSUPPORTED);
    else if ((long long)*total > cap) atomicExch(status, TSDFL_ERR_CAPACITY);
}

// One block a segment: the segment walked from its start for the counts (one
// thread, the products staged), offsets by a scan, the copies.
__global__ void __launch_bounds__(kEmitThreads) residual_emit_kernel(const float* particles,
                                                                     const float* __restrict__ w, int stride, int M,
                                                                     float* out, uint32_t* idx_out, long long cap,
                                                                     uint32_t* count_out, ResidualWs ws,
                                                                     int32_t* status)
{
    chain_enter();
    extern __shared__ __align__(16) float sc[];   // the products, then the offsets
    __shared__ uint32_t src[kEmitRows];
    __shared__ uint32_t red[kEmitThreads / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (blockIdx.x == 0 && tid == 0) report(ws.total, ws.err, cap, count_out, status);
    if (*ws.mode) {   // counts and offsets from the one-thread walk
        if (*ws.err) return;
        const int t0 = (int)blockIdx.x * ws.tile, t1 = min(M, t0 + ws.tile);
        for (int m = t0 + tid; m < t1; m += kEmitThreads) {
            const long long o = ws.off[m];
            for (long long j = o; j < o + (long long)ws.cnt[m] && j < cap; ++j) {
                if (idx_out) idx_out[j] = (uint32_t)m;
                if (out)
                    for (int k = 0; k < 7; ++k) out[7 * j + k] = particles[7 * (size_t)m + k];
            }
        }
        return;
    }
    const int s = blockIdx.x;
    const uint32_t b0 = ws.segs[s].begin;
    const int n = (int)(ws.segs[s + 1].begin - b0);
    stage_products(w, stride, (float)M, (int)b0, n, sc);
    __syncthreads();
    if (tid == 0) {
        float u = ws.start[s], of;
        int i = 0;
        for (; i + 32 <= n; i += 32) {   // 32 products to registers at a time: only the chain is serial
            float v[32];
#pragma unroll
            for (int k = 0; k < 32; ++k) v[k] = sc[i + k];
#pragma unroll
            for (int k = 0; k < 32; ++k) {
                u = residual_step(v[k], u, of);
                v[k] = of;
            }
#pragma unroll
            for (int k = 0; k < 32; ++k) sc[i + k] = v[k];
        }
        for (; i < n; ++i) {
            u = residual_step(sc[i], u, of);
            sc[i] = of;
        }
    }
    __syncthreads();
    // exclusive offsets of the counts in place, a run of consecutive particles a thread
    const int per = (n + kEmitThreads - 1) / kEmitThreads, i0 = min(n, tid * per), i1 = min(n, i0 + per);
    uint32_t run = 0;
    for (int i = i0; i < i1; ++i) run += (uint32_t)sc[i];
    uint32_t x = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) red[warp] = x;
    __syncthreads();
    uint32_t o = x - run, rows = 0;
    for (int k = 0; k < kEmitThreads / 32; ++k) {
        if (k < warp) o += red[k];
        rows += red[k];
    }
    uint32_t* off = reinterpret_cast<uint32_t*>(sc);
    for (int i = i0; i < i1; ++i) {
        const uint32_t c = (uint32_t)sc[i];
        off[i] = o;
        o += c;
    }
    __syncthreads();
    emit_rows(particles, b0, n, off, rows, ws.base[s], out, idx_out, cap, src);
}

// Small clouds: the copies from the one-thread walk's counts and offsets.
__global__ void residual_scatter_kernel(const float* particles, int M, const uint32_t* cnt, const uint32_t* off,
                                        const unsigned long long* total, const int* err, float* out,
                                        uint32_t* idx_out, long long cap, uint32_t* count_out, int32_t* status)
{
    chain_enter();
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m == 0) report(total, err, cap, count_out, status);
    if (*err || m >= M) return;
    const long long o = off[m];
    for (long long j = o; j < o + (long long)cnt[m] && j < cap; ++j) {
        if (idx_out) idx_out[j] = (uint32_t)m;
        if (out)
            for (int k = 0; k < 7; ++k) out[7 * j + k] = particles[7 * (size_t)m + k];
    }
}

int check(cudaError_t e) { return e == cudaSuccess ? TSDFL_OK : TSDFL_ERR_DEVICE; }

// Below this the one-thread walk takes less time than the five launches (a
// device call at 2,048 particles: 25 against 26 us; at 2,560 30 against 26).
constexpr size_t kParallelFrom = 2560;

// Particles a tile: a short tile keeps the walks short (candidates and counts,
// about 8 ns a particle each), a long one the segments to follow few.
int tile_of(size_t M) { return M <= (1u << 18) ? 512 : (M <= (1u << 20) ? 1024 : kMaxTile); }

// Most candidates a segment: the window of weights whose c stays below 2
// (roundings of variance 5/12 a particle) on the finest grid; larger c widen the
// walk and the grid alike.
int window_of(size_t M)
{
    const int w = (int)(9.0 * std::sqrt(0.42 * (double)M)) + 64;
    return std::min(kMaxWindow, (w + kCandThreads - 1) / kCandThreads * kCandThreads);
}

size_t up(size_t v) { return (v + 255) / 256 * 256; }

// The one-thread walk's part and the parallel form's tables, each in a buffer of its own.
struct Carve {
    char* p;
    size_t at = 0;
    template <typename T>
    T* take(size_t n)
    {
        T* r = p ? reinterpret_cast<T*>(p + at) : nullptr;
        at += up(sizeof(T) * n);
        return r;
    }
};

size_t layout_walk(size_t M, void* p, ResidualWs* ws)
{
    Carve a{static_cast<char*>(p)};
    ws->total = a.take<unsigned long long>(1);
    ws->err = a.take<int>(1);
    ws->mode = a.take<int>(1);
    ws->cnt = a.take<uint32_t>(M);
    ws->off = a.take<uint32_t>(M);
    return a.at;
}

size_t layout_tables(size_t M, void* p, ResidualWs* ws)
{
    Carve a{static_cast<char*>(p)};
    ws->tile = tile_of(M);
    ws->window = window_of(M);
    ws->S = (int)((M + (size_t)ws->tile - 1) / (size_t)ws->tile);
    const size_t S = (size_t)ws->S;
    ws->tiles = a.take<TileSums>(S);
    ws->segs = a.take<Seg>(S + 1);
    ws->sums = a.take<double>(S);
    ws->start = a.take<float>(S + 1);
    ws->base = a.take<uint32_t>(S + 1);
    ws->table = a.take<uint32_t>(S * (size_t)ws->window);
    return a.at;
}

}  // namespace

size_t residual_workspace_bytes(size_t M)
{
    ResidualWs ws{};
    return layout_walk(M, nullptr, &ws);
}

size_t residual_tables_bytes(size_t M)
{
    ResidualWs ws{};
    return M < kParallelFrom ? 0 : layout_tables(M, nullptr, &ws);
}

int launch_resample_residual(const float* particles, const float* w, int stride, size_t M, float u0, float* out,
                             uint32_t* idx_out, size_t cap, uint32_t* count_out, void* workspace, void* tables,
                             int32_t* status, cudaStream_t s)
{
    ResidualWs ws{};
    layout_walk(M, workspace, &ws);
    const int m = (int)M;
    const long long c = (long long)cap;
    // a draw outside [0, 1) is walked literally
    if (M < kParallelFrom || !tables || !(u0 >= 0.0f) || !(u0 < 1.0f)) {
        cudaError_t e = launch_chained(residual_chain_kernel, 1, kChainThreads, 0, s, w, stride, m, u0, ws.cnt, ws.off,
                                       ws.total, ws.err);
        if (e == cudaSuccess)
            e = launch_chained(residual_scatter_kernel, (unsigned)((M + 255) / 256), 256, 0, s, particles, m,
                               (const uint32_t*)ws.cnt, (const uint32_t*)ws.off,
                               (const unsigned long long*)ws.total, (const int*)ws.err, out, idx_out, c, count_out,
                               status);
        g_launches += 2;
        const cudaError_t last = cudaGetLastError();
        return check(e == cudaSuccess ? last : e);
    }
    layout_tables(M, tables, &ws);
    const size_t seg_smem = sizeof(float) * ((size_t)ws.tile + kHead + 4);
    const size_t follow_fixed = sizeof(Seg) * (ws.S + 1) + 4 * (((size_t)ws.S + 1 + 3) / 4 * 4);
    const size_t follow_smem = std::min(kFollowSmem, follow_fixed + 4 * (size_t)ws.S * ws.window);
    ws.staged = (uint32_t)((follow_smem - follow_fixed) / 16 * 4);
    if (allow_smem(residual_follow_kernel, kFollowSmem) != cudaSuccess) return TSDFL_ERR_DEVICE;
    // each kernel reads what the one before it wrote: none runs after a failed launch
    cudaError_t e = launch_chained(residual_tiles_kernel, (unsigned)ws.S, kTileThreads, 0, s, w, stride, m, ws);
    if (e == cudaSuccess) e = launch_chained(residual_plan_kernel, 1, kPlanThreads, 0, s, m, u0, ws);
    if (e == cudaSuccess)
        e = launch_chained_2d(residual_candidates_kernel, dim3((unsigned)ws.S, (unsigned)(ws.window / kCandThreads)),
                              kCandThreads, seg_smem, s, w, stride, m, u0, ws);
    if (e == cudaSuccess)
        e = launch_chained(residual_follow_kernel, 1, kChainThreads, follow_smem, s, w, stride, m, u0, ws);
    if (e == cudaSuccess)
        e = launch_chained(residual_emit_kernel, (unsigned)ws.S, kEmitThreads, seg_smem, s, particles, w, stride, m,
                           out, idx_out, c, count_out, ws, status);
    g_launches += 5;
    const cudaError_t last = cudaGetLastError();
    return check(e == cudaSuccess ? last : e);
}

}  // namespace tsdfl
