// spectral_tc.cu -- the RGB lookup table of the spectral mode built on the
// 5th-generation tensor cores (PrecomputeRGBLUTKernel,
// core/spectrum/spectrum_lut.cuh:12-38, evaluates the reference's RGB
// spectrum-basis network -- 32 sin/cos input features, an input layer and 7
// residual blocks of width 32 with ReLU, a 4-wide output -- at every voxel
// centre of the unit colour cube; 512^3 voxels in the reference).
//
// A tile is 128 voxels, one per thread; every layer is one 128 x 32 x 32
// matrix product on tcgen05.mma (kind::f16) with fp32 accumulators in tensor
// memory.  The MMA takes bf16 operands, so fp32 accuracy comes from splitting
// both operands into three bf16 terms, x = x0 + x1 + x2 (x0 = bf16(x),
// x1 = bf16(x - x0), x2 = bf16(x - x0 - x1): 24 significant bits), and adding the
// six products whose order is at most 2: x0 w0; x1 w0, x0 w1; x2 w0, x1 w1,
// x0 w2.  The weight splits lie one below the other in one operand, so each
// activation split is one product with as many of them as it needs, and the
// products of one order meet in one of three accumulators; the epilogue adds
// these, smallest first.  The activations stay fp32 in the registers of the row's
// thread between layers (bias, ReLU, residual sum from tcgen05.ld); only the next
// layer's split operand goes back to shared memory.  Entries differ from the SIMT
// build (one thread per voxel, fmaf in input order) by the summation order and
// the dropped products of order 3 and above: a few fp32 ulps, measured by
// ar_spectral_rgb_lut.
//
// A CTA of 640 threads runs five tiles side by side, one CTA per SM (registers,
// and 480 of the 512 tensor-memory columns).  Bound: the latency of a layer's
// chain (operand to shared memory, MMA, commit, accumulator back) and the issue
// slots of its fp32 part.  160^3 table: 1212 us with two tiles per CTA and two
// CTAs per SM, twelve 32-column MMAs per layer and scalar conversions; 1063 us
// with six tiles in one CTA; 960 us with packed conversions; 850 us with
// six MMAs per layer and five tiles.
//
// Every wait is bounded; a CTA whose MMA does not complete within the limit
// sets the error word, waits once more for its commit, frees its tensor
// memory and returns.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "render_kernels.h"
#include "spectral.cuh"
#include "tcgen05.cuh"

namespace ar {

namespace {

constexpr int kLutRows = 128;                                 // voxels per CTA tile (M)
constexpr int kLutLayers = 2 + kSpecBlocks;                   // input, 7 blocks, output
constexpr int kLutN = 32;                                     // width of the hidden layers
constexpr int kLutNOut = 32;                                  // output layer N (4 used, the others' weights are 0)
constexpr int kLutK = 32;
constexpr int kLutWLayer = kLutN * kLutK * 2;                 // bytes of one bf16 weight split (hidden)
constexpr int kLutWOut = kLutNOut * kLutK * 2;
constexpr int kLutWBytes = 3 * ((kLutLayers - 1) * kLutWLayer + kLutWOut);   // three splits
constexpr int kLutABytes = kLutRows * kLutK * 2;              // one bf16 split of the activations
constexpr int kLutTiles = 5;                                  // tiles side by side in a CTA
constexpr int kLutBarriers = kLutWBytes + kLutTiles * 3 * kLutABytes;   // offset of the mbarriers
constexpr int kLutBias = kLutBarriers + 128;                 // offset of the hidden layers' biases (fp32)
constexpr int kLutSmem = kLutBias + (kLutLayers - 1) * kLutN * 4;   // weights, the tiles' A operands, barriers, biases
constexpr int kLutCols = 3 * kLutN;                          // TMEM columns of a tile (three fp32 accumulators)
constexpr int kLutAllocCols = 512;
constexpr uint32_t kLutSpinLimit = 1u << 22;

// byte offset of layer l's weights: the three splits' rows one after the other, a
// B operand of 3 N rows
__host__ __device__ constexpr int lut_w_offset(int l) { return 3 * l * kLutWLayer; }

__device__ __forceinline__ void split3(float x, __nv_bfloat16* t)
{
    t[0] = __float2bfloat16_rn(x);
    const float r1 = x - __bfloat162float(t[0]);
    t[1] = __float2bfloat16_rn(r1);
    t[2] = __float2bfloat16_rn(r1 - __bfloat162float(t[1]));
}

// The three bf16 terms of two values at once, as packed pairs (a in the low
// half).  The packed conversion does not go through the conversion unit that the
// scalar one occupies (56 % busy, the kernel's busiest pipe).
__device__ __forceinline__ uint32_t pack_bf16x2(float a, float b)
{
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ void split3_pair(float a, float b, uint32_t* t)
{
    t[0] = pack_bf16x2(a, b);
    const float a1 = a - __uint_as_float(t[0] << 16), b1 = b - __uint_as_float(t[0] & 0xFFFF0000u);
    t[1] = pack_bf16x2(a1, b1);
    t[2] = pack_bf16x2(a1 - __uint_as_float(t[1] << 16), b1 - __uint_as_float(t[1] & 0xFFFF0000u));
}

// row t's 32 fp32 values as the three bf16 splits of the A operand
__device__ __forceinline__ void store_row(unsigned char* sA, int t, const float* h)
{
#pragma unroll
    for (int kc = 0; kc < kLutK / 8; ++kc) {
        uint32_t v[3][4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            uint32_t s3[3];
            split3_pair(h[8 * kc + 2 * e], h[8 * kc + 2 * e + 1], s3);
            v[0][e] = s3[0];
            v[1][e] = s3[1];
            v[2][e] = s3[2];
        }
#pragma unroll
        for (int j = 0; j < 3; ++j)
            *reinterpret_cast<uint4*>(sA + j * kLutABytes + tc_chunk_offset(kLutRows, t, kc)) =
                make_uint4(v[j][0], v[j][1], v[j][2], v[j][3]);
    }
}

}  // namespace

namespace {

// Groups of 128 threads run the tiles side by side: each group has its own A
// operand, mbarrier and 96 tensor-memory columns and synchronises on a named
// barrier of its own, so one group's epilogue (tcgen05.ld, bias, ReLU, split,
// store) overlaps the others' MMAs.  The weights are shared.
__global__ void __launch_bounds__(kLutTiles * kLutRows, 1) k_lut_rgb_tc(const float* __restrict__ tab, int res,
                                                             float4* __restrict__ lut, int* err)
{
    extern __shared__ __align__(128) unsigned char smem[];
    unsigned char* sW = smem;
    const int half = threadIdx.x >> 7;                 // which tile of the CTA
    const int t = threadIdx.x & (kLutRows - 1);        // row within the tile
    const int warp = threadIdx.x >> 5;
    unsigned char* sA = smem + kLutWBytes + half * 3 * kLutABytes;
    uint64_t* mbar = reinterpret_cast<uint64_t*>(smem + kLutBarriers) + half;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + kLutBarriers + 64);

    // weights [out][in] of every layer as three bf16 splits, B operands (N rows x K)
    for (int e = threadIdx.x; e < kLutLayers * kLutN * kLutK; e += kLutTiles * kLutRows) {
        const int l = e / (kLutN * kLutK), rem = e - l * (kLutN * kLutK);
        const int n = rem / kLutK, k = rem - n * kLutK;
        const int R = l == kLutLayers - 1 ? kLutNOut : kLutN;
        if (n >= R) continue;
        float w;
        if (l == 0) w = tab[kTabRgbInW + n * kLutK + k];
        else if (l < kLutLayers - 1) w = tab[kTabRgbBlkW + (l - 1) * 1024 + n * kLutK + k];
        else w = n < kSpecKernel ? tab[kTabRgbOutW + n * kLutK + k] : 0.0f;
        __nv_bfloat16 s3[3];
        split3(w, s3);
        for (int j = 0; j < 3; ++j)
            *reinterpret_cast<__nv_bfloat16*>(sW + lut_w_offset(l) + tc_chunk_offset(3 * R, j * R + n, k / 8) + (k % 8) * 2) =
                s3[j];
    }
    float* sBias = reinterpret_cast<float*>(smem + kLutBias);
    for (int e = threadIdx.x; e < (kLutLayers - 1) * kLutN; e += kLutTiles * kLutRows)
        sBias[e] = e < kLutN ? tab[kTabRgbInB + e] : tab[kTabRgbBlkB + e - kLutN];
    if (t == 0) {   // thread 0 of each group: its mbarrier
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" : : "r"(smem_addr(mbar)), "r"(1) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     : : "r"(smem_addr(tmem_slot)), "r"(kLutAllocCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot + static_cast<uint32_t>(half * kLutCols);   // this group's columns
    const uint32_t taddr = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);  // lanes of this warp's rows
    const uint32_t aBase = smem_addr(sA), wBase = smem_addr(sW), mb = smem_addr(mbar);
    uint32_t phase = 0;
    bool failed = false;
    const int64_t total = static_cast<int64_t>(res) * res * res;
    const float invRes = 1.0f / static_cast<float>(res);
    for (int64_t tile = kLutTiles * static_cast<int64_t>(blockIdx.x) + half; tile * kLutRows < total && !failed;
         tile += kLutTiles * static_cast<int64_t>(gridDim.x)) {
        const int64_t vx = tile * kLutRows + t;
        const bool valid = vx < total;
        const int64_t v = valid ? vx : total - 1;
        const int x = static_cast<int>(v % res), y = static_cast<int>((v / res) % res);
        const int z = static_cast<int>(v / (static_cast<int64_t>(res) * res));
        // RGBEncode's input features (spectrum_basis.cuh:2273-2300), as rgb_encode
        const float in[3] = {(static_cast<float>(x) + 0.5f) * invRes, (static_cast<float>(y) + 0.5f) * invRes,
                             (static_cast<float>(z) + 0.5f) * invRes};
        const float scale = fmaxf(fmaxf(in[0], in[1]), in[2]);
        const float inv = 1.0f / (scale + 0.001f);
        float h[kLutK];
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int k = 0; k < 4; ++k)
                sincos_det(in[c] * inv * kSpecPi * static_cast<float>(k + 1), &h[8 * c + k], &h[8 * c + k + 4]);
#pragma unroll
        for (int k = 0; k < 4; ++k) sincos_det(scale * kSpecPi * static_cast<float>(k + 1), &h[24 + k], &h[28 + k]);
        float out[kSpecKernel] = {0.0f, 0.0f, 0.0f, 0.0f};
        for (int l = 0; l < kLutLayers && !failed; ++l) {
            const int N = l == kLutLayers - 1 ? kLutNOut : kLutN;
            store_row(sA, t, h);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            half_sync(half);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (t == 0) {
                // activation split p times the weight splits 0 .. 2 - p, as one product
                // of (3 - p) N columns whose accumulators start at p N: accumulator o
                // collects the products of order o
#pragma unroll
                for (int p = 0; p < 3; ++p)
#pragma unroll
                    for (int ks = 0; ks < kLutK / 16; ++ks) {
                        const uint64_t da = tc_desc(aBase + static_cast<uint32_t>(p * kLutABytes + 2 * ks * kLutRows * 16),
                                                    kLutRows * 16, 128);
                        const uint64_t db = tc_desc(wBase + static_cast<uint32_t>(lut_w_offset(l) + 2 * ks * 3 * N * 16),
                                                    static_cast<uint32_t>(3 * N * 16), 128);
                        tc_mma(tmem + static_cast<uint32_t>(p * N), da, db, tc_idesc(kLutRows, (3 - p) * N), (ks > 0 || p > 0) ? 1u : 0u);
                    }
                tc_commit(mb);
            }
            uint32_t spins = 0;
            bool late = false;
            while (!mbar_try_wait(mb, phase)) {
                if (++spins >= kLutSpinLimit) { late = true; break; }
            }
            phase ^= 1u;
            failed = half_sync_or(half, late);   // the same decision in every thread of the group
            if (failed) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            // the accumulators in two halves of 16: registers for all tiles
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                if (c == 1 && l == kLutLayers - 1) break;
                uint32_t acc[16], acc1[16], acc2[16];
                tc_ld16x3(taddr + 16 * c, static_cast<uint32_t>(N), acc, acc1, acc2);
#pragma unroll
                for (int i = 0; i < 16; ++i)   // smallest first
                    acc[i] = __float_as_uint((__uint_as_float(acc2[i]) + __uint_as_float(acc1[i])) + __uint_as_float(acc[i]));
                if (l < kLutLayers - 1) {
                    const float4* B = reinterpret_cast<const float4*>(sBias + l * kLutN + 16 * c);
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const float4 b = B[q];
                        const float z[4] = {__uint_as_float(acc[4 * q]) + b.x, __uint_as_float(acc[4 * q + 1]) + b.y,
                                            __uint_as_float(acc[4 * q + 2]) + b.z, __uint_as_float(acc[4 * q + 3]) + b.w};
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const int i = 16 * c + 4 * q + e;
                            h[i] = (l == 0 ? 0.0f : h[i]) + fmaxf(z[e], 0.0f);
                        }
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < kSpecKernel; ++i) out[i] = __uint_as_float(acc[i]) * scale;
                }
            }
        }
        if (failed) break;
        if (valid) lut[vx] = make_float4(out[0], out[1], out[2], out[3]);
    }
    if (failed) {   // the timed-out MMAs may still write tensor memory: wait for their commit once more
        uint32_t spins = 0;
        while (!mbar_try_wait(mb, phase ^ 1u) && ++spins < 4u * kLutSpinLimit) {
        }
        atomicOr(err, 1);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" : : "r"(*tmem_slot), "r"(kLutAllocCols) : "memory");
}

}  // namespace

// Scratch of ar_spectral_rgb_lut, held by every device that loads the library:
// its table block, the lambda table it does not return, an error word (86 KB).
static __device__ __align__(256) float g_lut_tables[kTabFloats];
static __device__ __align__(256) float4 g_lut_lambda[kLambdaLutRes];
static __device__ int g_lut_error;

cudaError_t spectral_scratch(float** tables, float4** lambda, int** err)
{
    cudaError_t e = cudaGetSymbolAddress(reinterpret_cast<void**>(tables), g_lut_tables);
    if (e == cudaSuccess) e = cudaGetSymbolAddress(reinterpret_cast<void**>(lambda), g_lut_lambda);
    if (e == cudaSuccess) e = cudaGetSymbolAddress(reinterpret_cast<void**>(err), g_lut_error);
    return e;
}

cudaError_t launch_spectral_rgb_lut_tc(const float* tab, int res, float4* lut, int* err, int sm_count,
                                       cudaStream_t st)
{
    cudaError_t e = cudaFuncSetAttribute(k_lut_rgb_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, kLutSmem);
    if (e != cudaSuccess) return e;
    const int64_t total = static_cast<int64_t>(res) * res * res;
    const int64_t tiles = (total + kLutRows - 1) / kLutRows;
    const int grid = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>((tiles + kLutTiles - 1) / kLutTiles, sm_count)));
    k_lut_rgb_tc<<<grid, kLutTiles * kLutRows, kLutSmem, st>>>(tab, res, lut, err);
    return cudaGetLastError();
}

}  // namespace ar
