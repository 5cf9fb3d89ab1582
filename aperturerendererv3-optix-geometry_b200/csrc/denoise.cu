// denoise.cu -- the screen-space denoiser's bilateral filter and frame
// recording from caller-supplied primary hits.
//
// k_dn_bilateral replaces denoise::Bilateral16x16<7>
// (core/denoise/denoise.cuh:359-443).  A CTA handles a 32 x 8 tile in two
// phases over the same shared-memory window of 46 x 22 pixels (radius 7,
// coordinates clamped at the borders), staged as per-pixel terms, one warp per
// tile row, so a warp's 32 lanes read 32 consecutive words.  Phase 1 evaluates
// the skewness-corrected Welch t-test of all 225 taps from the pixels' halves
// of ComputeTStatistic / ComputeWelchNu (12 words per staged pixel) into a
// 225-bit mask per pixel in shared memory.  Phase 2 stages log(1 + c) and the
// guide values (14 words) and sums the taps whose bit is set, in the
// reference's order; a failing tap has weight 0 and costs nothing.  Every
// weight is computed with the reference's expressions and order of operations,
// so it is the reference's (with the fixed exp/log of detmath.h); the guide
// weight's half-precision differences round to half as the reference's device
// code does (__hsub).
//
// Bound: instruction issue (81 % of the slots, DRAM 1 %).  The 675 channel
// tests per pixel are decided as the reference's float expressions decide
// them, but without their three divisions (tap_passes) and, for all taps
// outside a narrow band of shares, without the degrees of freedom at all; two
// channels share packed two-lane arithmetic and a tap's terms come in 128-bit
// loads.  At 1920x1080 (8 recorded frames of a sphere field): 5.45 ms with the
// divisions and two kernels that passed the mask through memory, 4.62 ms as
// one kernel without divisions, 3.46 ms with packed arithmetic and wide loads,
// 2.54 ms with the band.  One kernel also needs no scratch allocation.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <atomic>
#include <string>

#include "../../include/aperture_b200.h"
#include "denoise.cuh"
#include "detmath.h"
#include "t_quantile_table.h"

namespace ar {

ar_status set_error(ar_status st, const std::string& msg);

namespace {

constexpr int kDnRadius = 7;
constexpr int kTileX = 32, kTileY = 8;
constexpr int kWinX = kTileX + 2 * kDnRadius, kWinY = kTileY + 2 * kDnRadius;
constexpr int kWin = kWinX * kWinY;
constexpr int kTaps = (2 * kDnRadius + 1) * (2 * kDnRadius + 1);

// FilterParams (denoise.cuh:13-32), the same float expressions
constexpr float kInvAlbedo = 1.0f / (2.0f * 1.0f * 1.0f);
constexpr float kInvNormal = 1.0f / (2.0f * 0.5f * 0.5f);
constexpr float kInvDepth = 1.0f / (2.0f * 0.25f * 0.25f);
constexpr float kInvMetallic = 1.0f / (2.0f * 0.5f * 0.5f);
constexpr float kInvRough = 1.0f / (2.0f * 0.5f * 0.5f);
constexpr float kInvShading = 1.0f / (2.0f * 0.1f * 0.1f);
constexpr float kInvSpatial = 1.0f / (2.0f * 2.0f * 2.0f);
constexpr float kCenterEps = 1.0e-6f;

// Shared-memory windows.  A pixel's words lie in 16-byte groups (group g of
// pixel p at float4 [g * kWin + p]), so a warp's 32 consecutive pixels load one
// group as one conflict-free 128-bit access.  Phase 1 stages the terms of
// ComputeTStatistic and ComputeWelchNu (denoise.cuh:278-339): theta,
// varianceThetaHat, s^2 / n (Welch numerator term) and (s^2 / n)^2 / max(n - 1, 1),
// the first two channels side by side for two-lane arithmetic:
//   group 0: theta 0, theta 1, vth 0, vth 1;  group 1: u 0, u 1, l 0, l 1;
//   then 8 bytes per pixel: theta 2, vth 2;  then 8: u 2, l 2.
// Phase 2 stages log(1 + c) and the guide values (half pairs as bits):
//   group 0: log 0-2, depth;  group 1: albedo 0-2, normal x;
//   group 2: normal y, z, metallic | roughness, model shares 0 | 1;
//   then 8 bytes per pixel: model shares 2 | 3, 4.
constexpr int kSide = 2 * kDnRadius + 1;       // taps per row
constexpr int kMaskWords = (kSide + 1) / 2;    // two rows of tap bits per word
constexpr int kWinFloats = 14 * kWin;          // the larger of the two windows
// the window of either phase, then the threshold table (phase 1) or the taps'
// spatial weights and offsets (phase 2), then the masks: 68.9 KB, 3 CTAs per SM
constexpr size_t kDnSmem = (static_cast<size_t>(kWinFloats) + kTQuantiles + kMaskWords * kTileX * kTileY) * sizeof(float);

// a - b of both half pairs, rounded to half as __hsub rounds each
__device__ __forceinline__ float2 hsub2_f(float a, float b)
{
    const __half2 x = *reinterpret_cast<const __half2*>(&a), y = *reinterpret_cast<const __half2*>(&b);
    return __half22float2(__hsub2(x, y));
}

// Two float lanes in one register pair: the packed add and fused multiply-add
// of sm_100; each lane rounds like the scalar instruction.  Products are two
// scalar multiplications: a packed product whose result feeds a packed add is
// contracted with it to one rounding, also under --fmad=false (and an fma with
// an addend of -0 counts as a product).
using f2 = unsigned long long;
__device__ __forceinline__ f2 pack2(float x, float y)
{
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float2 unpack2(f2 a)
{
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
    return r;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b)
{
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c)
{
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b)
{
    const float2 x = unpack2(a), y = unpack2(b);
    return pack2(__fmul_rn(x.x, y.x), __fmul_rn(x.y, y.y));
}

// LookupTQuantile005(floorToInt(nu)) (t_quantile.cuh:15-27) with the device's
// saturating float-to-int conversion (NaN -> 0)
__device__ __forceinline__ int t_index(float nu)
{
    if (!(nu >= 1.0f)) return 0;
    if (nu >= 1024.0f) return kTQuantiles - 1;
    return static_cast<int>(floorf(nu)) - 1;
}

__device__ __forceinline__ int64_t window_pixel(int p, int gx0, int gy0, int width, int height)
{
    const int gx = min(max(gx0 + p % kWinX, 0), width - 1);
    const int gy = min(max(gy0 + p / kWinX, 0), height - 1);
    return static_cast<int64_t>(gy) * width + gx;
}

// ComputeTStatistic (denoise.cuh:278-302) and the per-pixel quotients of
// ComputeWelchNu (denoise.cuh:326-339); counts in 32-bit unsigned arithmetic
__device__ uint32_t stage_tstat(float4* w, int p, const ar_screen_stats* st, int64_t idx)
{
    const ar_screen_stats s = st[idx];
    const double num = static_cast<double>(s.num);
    const double invNm1 = 1.0 / static_cast<double>(max(s.num - 1u, 1u));
    const float fnum = static_cast<float>(s.num);
    const float fnm1 = static_cast<float>(max(s.num - 1u, 1u));
    float th[3], vth[3], u[3], l[3];
    bool plain = true;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const float vb = static_cast<float>(static_cast<double>(s.m2_div_n[c]) * num * invNm1);
        vth[c] = static_cast<float>(static_cast<double>(vb) / num);
        th[c] = s.mean[c] + s.m3_div_n[c] / 6.0f / vb;
        u[c] = vb / fnum;
        l[c] = u[c] * u[c] / fnm1;
        plain &= vb == 0.0f || (u[c] >= 1.0e-15f && u[c] <= 1.0e15f);
    }
    w[p] = make_float4(th[0], th[1], vth[0], vth[1]);
    w[kWin + p] = make_float4(u[0], u[1], l[0], l[1]);
    reinterpret_cast<float2*>(w + 2 * kWin)[p] = make_float2(th[2], vth[2]);
    reinterpret_cast<float2*>(w + 2 * kWin)[kWin + p] = make_float2(u[2], l[2]);
    // sample count for the tile's bounds of nu; 0 where their derivation does
    // not hold: a variance so small or large that its square leaves the float
    // range, or so small that its quotient u is zero, when a pair's nu may be
    // 0 / 0.  A variance of exactly zero makes theta infinite or NaN, so its
    // taps fail whatever nu is.
    return plain ? s.num : 0u;
}

__device__ __forceinline__ float half_pair(uint32_t lo, uint32_t hi) { return __uint_as_float(lo | (hi << 16)); }

__device__ void stage_guide(float4* w, int p, const float* hdr, const ar_screen_gbuffer* gb, int64_t idx)
{
    const ar_screen_gbuffer g = gb[idx];
    // SeparateSample (denoise.cuh:250-259)
    w[p] = make_float4(log_det(hdr[3 * idx] + 1.0f), log_det(hdr[3 * idx + 1] + 1.0f), log_det(hdr[3 * idx + 2] + 1.0f),
                       g.depth);
    const f3 n = normalize(mk(h2f(g.normal[0]), h2f(g.normal[1]), h2f(g.normal[2])));
    w[kWin + p] = make_float4(h2f(g.albedo[0]), h2f(g.albedo[1]), h2f(g.albedo[2]), n.x);
    w[2 * kWin + p] = make_float4(n.y, n.z, half_pair(g.metallic, g.roughness),
                                  half_pair(g.shading_model[0], g.shading_model[1]));
    reinterpret_cast<float2*>(w + 3 * kWin)[p] = make_float2(half_pair(g.shading_model[2], g.shading_model[3]),
                                                             half_pair(g.shading_model[4], 0u));
}

__device__ __forceinline__ float rcp_approx(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// floor(nu) clamped to [1, 1024] in the low mantissa bits of the returned
// float (a round-down add of 2^23), and the distance of the clamped value from
// the middle between two integers.
__device__ __forceinline__ float floor_bits(float nu, float& off_middle)
{
    const float c = fminf(fmaxf(nu, 1.0f), 1024.5f);
    const float f = __fadd_rd(c, 8388608.0f);
    off_middle = fabsf((c - (f - 8388608.0f)) - 0.5f);
    return f;
}
constexpr int kFloorBase = 0x4B000001;         // bits of 2^23 + 1: index 0
constexpr float kOffMiddle = 0.5f - 0x1p-10f;  // farther: an integer within 2^-10

// ComputeTStatisticFinal (denoise.cuh:341-356) of one tap: whether for all
// three channels
//     W = N / D,  x = 0.5 / (1 - W) - 1,  nu = P / Q,  !(x < 0) && sqrt(x) < t[floor(nu)]
// holds in the float expressions of the reference, without dividing.
//  * x grows monotonically with W in every float step, so the condition is
//    kShareLeast <= W < kShareThreshold[index] (t_quantile_table.h).
//  * fl(N / D) < c holds exactly when N / D lies below the midpoint under c,
//    c - u with u half the float spacing below c (2^-25 for the thresholds,
//    which lie in (0.5, 1); 2^-26 for kShareLeast; a quotient of floats is
//    never such a midpoint).  fma(-c, D, N) is exact near that border and
//    rounds monotonically away from it, so comparing it with -u D decides.
//    D >= 1e-6 keeps both sides normal.  NaN or infinite N or D fail.
//  * the index needs floor(nu) only: nu by an approximate reciprocal is off by
//    less than 2^-11 below 1024, so it decides unless an integer lies within
//    2^-10 or Q is near the ends of the float range; then (and for NaN, which
//    the clamp turns into 1) the IEEE quotients are taken.
// Channels 0 and 1 go through two-lane arithmetic.
struct TapCenter {
    f2 th, vth, u, l;
    float th2, vth2, u2, l2;
};
// N, D and u D of a tap: channels 0 and 1 packed, channel 2
struct TapShare {
    f2 n, d, u;
    float n2, d2, u2;
};
__device__ __forceinline__ bool tap_share(const TapCenter& a, float4 b0, float2 b2, TapShare& s)
{
    const f2 vb = pack2(b0.z, b0.w);
    const f2 t = fma2(pack2(b0.x, b0.y), pack2(-1.0f, -1.0f), a.th);
    const f2 tt = mul2(t, t);
    s.n = add2(tt, vb);
    const float2 ds = unpack2(add2(add2(tt, a.vth), vb));
    s.d = pack2(fmaxf(ds.x, 1.0e-6f), fmaxf(ds.y, 1.0e-6f));
    s.u = mul2(s.d, pack2(0x1p-25f, 0x1p-25f));
    const float tz = a.th2 - b2.x, ttz = tz * tz;
    s.n2 = ttz + b2.y;
    s.d2 = fmaxf(ttz + a.vth2 + b2.y, 1.0e-6f);
    s.u2 = s.d2 * 0x1p-25f;
    // kShareLeast <= W in every channel
    const float2 r = unpack2(fma2(s.d, pack2(-kShareLeast, -kShareLeast), s.n));
    const float2 h = unpack2(mul2(s.u, pack2(-0.5f, -0.5f)));
    return (r.x >= h.x) & (r.y >= h.y) & (fmaf(-kShareLeast, s.d2, s.n2) >= -0.5f * s.u2);
}

// Whether N < c D in every channel (the sign of a fused multiply-add is exact).
__device__ __forceinline__ bool share_below(const TapShare& s, float c)
{
    const float2 r = unpack2(fma2(s.d, pack2(-c, -c), s.n));
    return (r.x < 0.0f) & (r.y < 0.0f) & (fmaf(-c, s.d2, s.n2) < 0.0f);
}

__device__ __noinline__ bool tap_passes(const TapCenter& a, float4 b0, float2 b2, float4 b1, float2 b3, const float* thr)
{
    TapShare s;
    const bool least = tap_share(a, b0, b2, s);
    const f2 up = add2(a.u, pack2(b1.x, b1.y));
    const float2 q = unpack2(add2(a.l, pack2(b1.z, b1.w)));
    const float2 p = unpack2(mul2(up, up));
    const float upz = a.u2 + b3.x, qz = a.l2 + b3.y, pz = upz * upz;
    float o0, o1, o2;
    const float f0 = floor_bits(p.x * rcp_approx(q.x), o0), f1 = floor_bits(p.y * rcp_approx(q.y), o1);
    const float f2z = floor_bits(pz * rcp_approx(qz), o2);
    int k0 = __float_as_int(f0) - kFloorBase, k1 = __float_as_int(f1) - kFloorBase, k2 = __float_as_int(f2z) - kFloorBase;
    const float qlo = fminf(fminf(q.x, q.y), qz), qhi = fmaxf(fmaxf(q.x, q.y), qz);
    if (least && (fmaxf(fmaxf(o0, o1), o2) > kOffMiddle || !(qlo > 0x1p-100f && qhi < 0x1p100f))) {
        k0 = t_index(p.x / q.x);
        k1 = t_index(p.y / q.y);
        k2 = t_index(pz / qz);
    }
    const float2 rt = unpack2(fma2(s.d, pack2(-thr[k0], -thr[k1]), s.n)), us = unpack2(s.u);
    return least & (rt.x < -us.x) & (rt.y < -us.y) & (fmaf(-thr[k2], s.d2, s.n2) < -s.u2);
}

__global__ void __launch_bounds__(kTileX * kTileY, 3)
k_dn_bilateral(const float* __restrict__ hdr, float* __restrict__ out, const ar_screen_gbuffer* __restrict__ gb,
               const ar_screen_stats* __restrict__ st, int width, int height)
{
    extern __shared__ __align__(16) float sm[];
    float4* w = reinterpret_cast<float4*>(sm);
    float* thr = sm + kWinFloats;
    uint32_t* mask = reinterpret_cast<uint32_t*>(thr + kTQuantiles);   // word k of thread t at [k * 256 + t]
    const int tid = threadIdx.y * kTileX + threadIdx.x;
    const int gx0 = blockIdx.x * kTileX - kDnRadius, gy0 = blockIdx.y * kTileY - kDnRadius;
    const int ox = blockIdx.x * kTileX + threadIdx.x, oy = blockIdx.y * kTileY + threadIdx.y;
    const bool inside = ox < width && oy < height;
    const int c = (threadIdx.y + kDnRadius) * kWinX + threadIdx.x + kDnRadius;
    // phase 1: the t-test of every tap, center = A
    __shared__ uint32_t countMin, countMax;
    if (tid == 0) {
        countMin = 0xFFFFFFFFu;
        countMax = 0u;
    }
    for (int k = tid; k < kTQuantiles; k += kTileX * kTileY) thr[k] = kShareThreshold[k];
    __syncthreads();
    {
        uint32_t lo = 0xFFFFFFFFu, hi = 0u;
        for (int p = tid; p < kWin; p += kTileX * kTileY) {
            const uint32_t m = stage_tstat(w, p, st, window_pixel(p, gx0, gy0, width, height));
            lo = min(lo, m);
            hi = max(hi, m);
        }
        lo = __reduce_min_sync(0xFFFFFFFFu, lo);
        hi = __reduce_max_sync(0xFFFFFFFFu, hi);
        if (threadIdx.x == 0) {
            atomicMin(&countMin, lo);
            atomicMax(&countMax, hi);
        }
    }
    __syncthreads();
    const float2* w2 = reinterpret_cast<const float2*>(w + 2 * kWin);
    if (inside) {
        // Welch's nu of two pixels lies in [min(n) - 1, n_A + n_B - 2]: a share
        // below the threshold of the tile's largest nu passes whatever nu is,
        // one above that of its smallest fails, both with an index (and 2^-20)
        // to spare for rounding; only the shares between them need their nu.
        const bool bounds = countMin >= 3u;
        const float below = bounds ? thr[min(2u * min(countMax, 600u) - 2u, 1023u)] * (1.0f - 0x1p-20f) : 0.0f;
        const float above = bounds ? thr[min(countMin - 3u, 1023u)] * (1.0f + 0x1p-20f) : 2.0f;
        const float4 c0 = w[c], c1 = w[kWin + c];
        const float2 c2 = w2[c], c3 = w2[kWin + c];
        const TapCenter a = {pack2(c0.x, c0.y), pack2(c0.z, c0.w), pack2(c1.x, c1.y), pack2(c1.z, c1.w), c2.x, c2.y, c3.x, c3.y};
#pragma unroll 1
        for (int k = 0; k < kMaskWords; ++k) {
            uint32_t bits = 0, open = 0;   // bit 15 r + i: tap i of row 2 k + r passes, needs its nu
            const int q0 = c + (2 * k - kDnRadius) * kWinX - kDnRadius;
#pragma unroll 1
            for (int r = 0; r < (k == kMaskWords - 1 ? 1 : 2); ++r) {
                const int q = q0 + r * kWinX;
                uint32_t yes = 0, may = 0;
#pragma unroll
                for (int i = 0; i < kSide; ++i) {
                    TapShare s;
                    const bool least = tap_share(a, w[q + i], w2[q + i], s);
                    yes |= static_cast<uint32_t>(least & share_below(s, below)) << i;
                    may |= static_cast<uint32_t>(least & share_below(s, above)) << i;
                }
                bits |= yes << (kSide * r);
                open |= (may & ~yes) << (kSide * r);
            }
            while (open) {
                const int tap = __ffs(open) - 1;
                open &= open - 1u;
                const int q = q0 + (tap >= kSide ? kWinX - kSide : 0) + tap;
                if (tap_passes(a, w[q], w2[q], w[kWin + q], w2[kWin + q], thr)) bits |= 1u << tap;
            }
            mask[k * (kTileX * kTileY) + tid] = bits;
        }
    }
    __syncthreads();
    // phase 2: the weighted mean of Bilateral16x16 (denoise.cuh:359-443) over
    // the taps that passed, in the reference's order (rows, then columns)
    float2* taps = reinterpret_cast<float2*>(thr);   // spatial weight, window offset (int bits)
    for (int k = tid; k < kTaps; k += kTileX * kTileY) {
        const int j = k / (2 * kDnRadius + 1) - kDnRadius, i = k % (2 * kDnRadius + 1) - kDnRadius;
        taps[k] = make_float2(exp_det(static_cast<float>(-(i * i + j * j)) * kInvSpatial), __int_as_float(j * kWinX + i));
    }
    for (int p = tid; p < kWin; p += kTileX * kTileY)
        stage_guide(w, p, hdr, gb, window_pixel(p, gx0, gy0, width, height));
    __syncthreads();
    if (!inside) return;
    const int64_t pix = static_cast<int64_t>(oy) * width + ox;
    const float2* w3 = reinterpret_cast<const float2*>(w + 3 * kWin);
    const float4 a0 = w[c], a1 = w[kWin + c], a2 = w[2 * kWin + c];
    const float2 a3 = w3[c];
    float acc0 = 0.0f + a0.x * kCenterEps, acc1 = 0.0f + a0.y * kCenterEps, acc2 = 0.0f + a0.z * kCenterEps;
    float wsum = 0.0f + kCenterEps;
#pragma unroll 1
    for (int k = 0; k < kMaskWords; ++k) {
        uint32_t m = mask[k * (kTileX * kTileY) + tid];
        while (m) {   // passing taps in increasing order: rows, then columns
            const float2 tp = taps[2 * kSide * k + __ffs(m) - 1];
            m &= m - 1u;
            const int q = c + __float_as_int(tp.y);
            const float4 b0 = w[q], b1 = w[kWin + q], b2 = w[2 * kWin + q];
            const float2 b3 = w3[q];
            // ComputeSVGFWeight (denoise.cuh:185-245)
            float wt = 0.0f;
            {
                const float d0 = a1.x - b1.x, d1 = a1.y - b1.y, d2 = a1.z - b1.z;
                wt += (d0 * d0 + d1 * d1 + d2 * d2) * kInvAlbedo;
            }
            {
                const float dv = a1.w * b1.w + a2.x * b2.x + a2.y * b2.y;
                const float d = 1.0f - dv;
                wt += d * d * kInvNormal;
            }
            {
                const float denom = fmaxf(fmaxf(a0.w, b0.w), 1.0e-6f);
                const float d = (a0.w - b0.w) / denom;
                wt += d * d * kInvDepth;
            }
            const float2 mr = hsub2_f(a2.z, b2.z);
            wt += mr.x * mr.x * kInvMetallic;
            wt += mr.y * mr.y * kInvRough;
            {
                const float2 m01 = hsub2_f(a2.w, b2.w), m23 = hsub2_f(a3.x, b3.x), m4 = hsub2_f(a3.y, b3.y);
                float l1 = 0.0f;
                l1 += fabsf(m01.x);
                l1 += fabsf(m01.y);
                l1 += fabsf(m23.x);
                l1 += fabsf(m23.y);
                l1 += fabsf(m4.x);
                const float tv = 0.5f * l1;
                wt += tv * tv * kInvShading;
            }
            float weight = exp_det(-wt) * tp.x;
            if (isnan_(weight)) weight = 0.0f;  // zero normal of a pixel that never hit a surface
            if (weight == 0.0f) continue;
            acc0 = acc0 + b0.x * weight;
            acc1 = acc1 + b0.y * weight;
            acc2 = acc2 + b0.z * weight;
            wsum = wsum + weight;
        }
    }
    // CompositeSample (denoise.cuh:261-270)
    float* o = out + 3 * pix;
    o[0] = fmaxf(exp_det(acc0 / wsum) - 1.0f, 0.0f);
    o[1] = fmaxf(exp_det(acc1 / wsum) - 1.0f, 0.0f);
    o[2] = fmaxf(exp_det(acc2 / wsum) - 1.0f, 0.0f);
}

__global__ void k_dn_record(const float* __restrict__ hits, const float* __restrict__ samples, int64_t n,
                            ar_screen_gbuffer* gb, ar_screen_stats* st)
{
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        if (gb) {
            const float* h = hits + 12 * i;
            const int model = min(max(static_cast<int>(h[9]), 0), kDnModels - 2);
            record_gbuffer(gb + i, h[10] != 0.0f, mk(h[0], h[1], h[2]), mk(h[3], h[4], h[5]), h[6], h[7], h[8], model);
        }
        if (st) record_stats(st + i, mk(samples[3 * i], samples[3 * i + 1], samples[3 * i + 2]));
    }
}

ar_status dn_cuda_fail(cudaError_t e, const char* where)
{
    cudaGetLastError();
    return set_error(AR_ERR_CUDA, std::string(where) + ": " + cudaGetErrorString(e));
}

bool have_device()
{
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess || count == 0) {
        cudaGetLastError();
        return false;
    }
    return true;
}

}  // namespace

cudaError_t launch_dn_record(const float* hits, const float* samples, int64_t n, ar_screen_gbuffer* gb,
                             ar_screen_stats* st, cudaStream_t stream)
{
    if (n == 0) return cudaSuccess;
    const int64_t want = (n + 255) / 256;
    const int grid = static_cast<int>(want < 148 * 16 ? want : 148 * 16);
    k_dn_record<<<grid, 256, 0, stream>>>(hits, samples, n, gb, st);
    return cudaGetLastError();
}

}  // namespace ar

extern "C" ar_status ar_denoise_record(const float* hits, const float* samples, size_t n, ar_screen_gbuffer* gbuffer,
                                       ar_screen_stats* stats, void* stream)
{
    using namespace ar;
    if (n == 0) return AR_OK;
    if (!gbuffer && !stats) return set_error(AR_ERR_INVALID_ARGUMENT, "gbuffer and stats are both NULL");
    if (gbuffer && !hits) return set_error(AR_ERR_INVALID_ARGUMENT, "hits is NULL");
    if (stats && !samples) return set_error(AR_ERR_INVALID_ARGUMENT, "samples is NULL");
    if (!have_device()) return set_error(AR_ERR_NO_DEVICE, "no CUDA device available");
    const cudaError_t e = launch_dn_record(hits, samples, static_cast<int64_t>(n), gbuffer, stats,
                                           static_cast<cudaStream_t>(stream));
    return e == cudaSuccess ? AR_OK : dn_cuda_fail(e, "k_dn_record launch");
}

extern "C" ar_status ar_denoise_bilateral(const float* hdr_in, float* hdr_out, const ar_screen_gbuffer* gbuffer,
                                          const ar_screen_stats* stats, int32_t width, int32_t height, void* stream)
{
    using namespace ar;
    if (!hdr_in || !hdr_out || !gbuffer || !stats) return set_error(AR_ERR_INVALID_ARGUMENT, "NULL buffer");
    if (width <= 0 || height <= 0) return set_error(AR_ERR_INVALID_ARGUMENT, "width and height must be positive");
    if (hdr_in == hdr_out) return set_error(AR_ERR_INVALID_ARGUMENT, "hdr_out must not alias hdr_in");
    if (!have_device()) return set_error(AR_ERR_NO_DEVICE, "no CUDA device available");
    // the shared-memory opt-in is a per-device attribute of the kernel
    static std::atomic<uint64_t> attr_set{0};
    cudaError_t e;
    int dev = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return dn_cuda_fail(e, "cudaGetDevice");
    const uint64_t bit = dev < 64 ? (uint64_t{1} << dev) : 0;
    if (!bit || !(attr_set.load() & bit)) {
        if ((e = cudaFuncSetAttribute(k_dn_bilateral, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      static_cast<int>(kDnSmem))) != cudaSuccess)
            return dn_cuda_fail(e, "cudaFuncSetAttribute");
        attr_set.fetch_or(bit);
    }
    const dim3 block(kTileX, kTileY);
    const dim3 grid((width + kTileX - 1) / kTileX, (height + kTileY - 1) / kTileY);
    k_dn_bilateral<<<grid, block, kDnSmem, static_cast<cudaStream_t>(stream)>>>(hdr_in, hdr_out, gbuffer, stats, width,
                                                                               height);
    if ((e = cudaGetLastError()) != cudaSuccess) return dn_cuda_fail(e, "k_dn_bilateral launch");
    return AR_OK;
}
