// render.cu -- sm_100a kernels of the wavefront path tracer and the ray queries.
//
// Built with --fmad=false: every floating-point expression rounds exactly as
// the reference's source reads (see detmath.h); fused multiply-adds appear only
// where written as fmaf (the BVH box planes and the sampling polynomials).
#include "path_stages.cuh"
#include "xorwow_jump.h"

#include <algorithm>
#include <cstring>
#include <mutex>
#include <vector>

namespace ar {

cudaError_t set_intersect_eps(const float* tab9)
{
    return cudaMemcpyToSymbol(c_eps_tab, tab9, 9 * sizeof(float));
}

// ------------------------------------------------------------------ ray queries
template <bool kSdf>
struct RaysIO {
    const float4* rays;
    int32_t* out_obj;
    float* out_t;
    int any;
    __device__ __forceinline__ int load(const SceneView&, int k, RayState& r)
    {
        const float4 a = rays[2 * static_cast<int64_t>(k)], b = rays[2 * static_cast<int64_t>(k) + 1];
        ray_begin(r, mk(a.x, a.y, a.z), mk(b.x, b.y, b.z), a.w, b.w);
        return k;
    }
    __device__ __forceinline__ void store(const SceneView& s, int k, const RayState& r)
    {
        int32_t obj = r.best.obj;
        float t = r.best.t;
        if (kSdf && s.num_sdf > 0) {  // standalone queries use the depth-0 tolerance
            if (!any) sdf_closest(s, r.o, r.d, r.tmin, kEpsDepth0, &t, &obj);
            else if (obj < 0) obj = sdf_any(s, r.o, r.d, r.tmin, t, kEpsDepth0);
        }
        out_obj[k] = obj;
        if (out_t) out_t[k] = t;
    }
};

template <bool kAny, bool kSdf>
__global__ void __launch_bounds__(kTraceBlock, kTraceMinBlocks) k_trace_rays(SceneView s, RaysIO<kSdf> io, int n, PoolCtl* ctl,
                                                            uint32_t* ovf, int* err)
{
    extern __shared__ uint32_t smem[];
    traverse_queue<kAny>(s, io, n, &ctl->fetch_rays, lane_stack(smem), thread_overflow(ovf), err, nullptr);
}

// ------------------------------------------------------------------ RNG
// A uniform jump by the whole warp: lane c looks up chunk c (and c + 32), the
// contributions meet in a warp-wide XOR.
__device__ __forceinline__ void xorwow_jump_warp(uint32_t v[5], const uint32_t* __restrict__ table)
{
    uint32_t r[5] = {0, 0, 0, 0, 0};
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int c = static_cast<int>(lane_id()) + 32 * h;
        if (c < kJumpChunks) {
            const uint32_t word = h ? v[4] : (c < 8 ? v[0] : c < 16 ? v[1] : c < 24 ? v[2] : v[3]);
            const uint32_t* row = table + c * 80 + ((word >> (4 * (c & 7))) & 15u);
#pragma unroll
            for (int k = 0; k < 5; ++k) r[k] ^= __ldg(row + 16 * k);
        }
    }
#pragma unroll
    for (int k = 0; k < 5; ++k) v[k] = __reduce_xor_sync(0xFFFFFFFFu, r[k]);
}

// Every pixel's state of InitRand (random.cuh:35-38): curand_init(GLOBAL_SEED, s,
// frame0 * 2^32) with s its reference pixel index.  The seed's state comes from
// curand_init without a skip; frame0 and s are then jumps of the register (the
// Weyl counter moves by 362437 * 2^32 or 2^67 = 0 mod 2^32) along their bits.  A
// warp takes 8 consecutive 8x4 pixel blocks, i.e. 256 consecutive s: the bits
// they share are jumped by the warp together, then each lane takes one row of 8
// pixels of one block: its row's and block's jumps, and one jump per pixel.
// Bound: latency of the chain of jumps for small images, shared-memory lookups
// (200 per jump, conflict-free) for large ones.  With one thread per block, its
// curand_init and 31 jumps one after the other, a 160x120 image took 103 us and
// 1920x1080 260 us; this takes 14 us and
// 137 us.
constexpr int kInitBlock = 128;
constexpr size_t kInitSmem = static_cast<size_t>(kInitLaneTables) * kJumpWords * 4;
__global__ void __launch_bounds__(kInitBlock) k_rng_init(FrameParams fp, uint4* base0, uint2* base1,
                                                         const uint32_t* __restrict__ tables)
{
    extern __shared__ __align__(16) uint32_t jt[];
    const uint32_t* frame_t = tables;
    const uint32_t* lane_t = tables + kInitFrameBits * kJumpWords;
    const uint32_t* group_t = lane_t + kInitLaneTables * kJumpWords;
    for (int k = threadIdx.x; k < kInitLaneTables * kJumpWords / 4; k += kInitBlock)
        reinterpret_cast<uint4*>(jt)[k] = __ldg(reinterpret_cast<const uint4*>(lane_t) + k);
    __syncthreads();
    const int nblk = fp.grid_x * ((fp.height + 3) / 4);
    const int groups = (nblk + 7) / 8;
    const int lane = static_cast<int>(lane_id()), row = lane & 3;
    for (int w = blockIdx.x * (kInitBlock / 32) + (threadIdx.x >> 5); w < groups; w += gridDim.x * (kInitBlock / 32)) {
        curandStateXORWOW_t st;
        curand_init(fp.seed, 0, 0, &st);
        uint32_t v[5] = {st.v[0], st.v[1], st.v[2], st.v[3], st.v[4]};
        for (uint32_t f = static_cast<uint32_t>(fp.frame0); f; f &= f - 1u)
            xorwow_jump_warp(v, frame_t + (__ffs(f) - 1) * kJumpWords);
        for (uint32_t b = static_cast<uint32_t>(w); b; b &= b - 1u)
            xorwow_jump_warp(v, group_t + (__ffs(b) - 1) * kJumpWords);
#pragma unroll 1
        for (int k = 0; k < 5; ++k)   // rows 1 and 2 of 4, then blocks 1, 2 and 4 of 8
            if ((lane >> k) & 1) xorwow_jump(v, jt + (1 + k) * kJumpWords);
        const int b = 8 * w + (lane >> 2);
        const int bx = b % fp.grid_x, j = 4 * (b / fp.grid_x) + row;
#pragma unroll 1
        for (int x = 0; x < 8; ++x) {
            if (x) xorwow_jump(v, jt);
            const int i = 8 * bx + x;
            if (b < nblk && i < fp.width && j < fp.height) {
                const int p = j * fp.width + i;
                base0[p] = make_uint4(st.d, v[0], v[1], v[2]);
                base1[p] = make_uint2(v[3], v[4]);
            }
        }
    }
}

// out[(s * npix + p) * per_path + k] = k-th uniform of pixel p at sample s
__global__ void k_rng_tape(FrameParams fp, int spp, int per_path, float* out)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= fp.npix) return;
    const int i = p % fp.width, j = p / fp.width;
    for (int s = 0; s < spp; ++s) {
        curandStateXORWOW_t st;
        curand_init(fp.seed, ref_pixel_index(i, j, fp.grid_x), (fp.frame0 + static_cast<uint64_t>(s)) << 32, &st);
        float* o = out + (static_cast<int64_t>(s) * fp.npix + p) * per_path;
        for (int k = 0; k < per_path; ++k) o[k] = curand_uniform(&st);
    }
}

// ------------------------------------------------------------------ path pool
__device__ __forceinline__ void pool_init(PoolCtl* ctl, int64_t total)
{
    ctl->count[0] = 0;
    ctl->count[1] = 0;
    for (int b = 0; b < 8; ++b) ctl->shade_count[b] = 0;
    ctl->shadow_count = 0;
    ctl->retire_count = 0;
    ctl->fetch_ext = 0;
    ctl->fetch_shadow = 0;
    ctl->fetch_rays = 0;
    ctl->plan_new = 0;
    ctl->plan_base = 0;
    ctl->tail_done = 0;
    ctl->gen_next = 0;
    ctl->plan_first = 0;
    ctl->retired = 0;
    ctl->total = total;
}

// Start of a render: empty pool, zero sums, counters and error words.
__global__ void k_render_init(PoolCtl* ctl, int64_t total, double2* accum, int64_t pairs, unsigned long long* stats, int* err)
{
    const int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    for (int64_t i = t; i < pairs; i += static_cast<int64_t>(gridDim.x) * blockDim.x) accum[i] = make_double2(0.0, 0.0);
    if (t < 8) stats[t] = 0;
    if (t < 16) err[t] = 0;
    if (t == 0) pool_init(ctl, total);
}

// Start of an iteration: the current pool holds the paths that survived the
// previous one; top it up with new samples (the next ones in sample-major
// order, several of a pixel where the pool has room) and reset the queues this
// iteration fills.
__global__ void k_plan(PoolCtl* ctl, int cur, int capacity)
{
    const int64_t remaining = ctl->total - ctl->gen_next;
    const int ncont = ctl->count[cur];
    int n = capacity - ncont;
    if (static_cast<int64_t>(n) > remaining) n = static_cast<int>(remaining);
    ctl->plan_new = n;
    ctl->plan_base = ncont;
    ctl->count[cur] = ncont + n;
    ctl->plan_first = ctl->gen_next;
    ctl->gen_next += n;
    ctl->count[1 - cur] = 0;
    for (int b = 0; b < 8; ++b) ctl->shade_count[b] = 0;
    ctl->shadow_count = 0;
    ctl->retire_count = 0;
    ctl->fetch_ext = 0;
    ctl->fetch_shadow = 0;
}

// shared memory of the kernels that exchange path records between their lanes
constexpr size_t kStageSmem = static_cast<size_t>(kShadeBlock) * sizeof(PathRec);

// RenderCamera (scene.cu:213-230) + CalculateRadiance prologue (render.cuh:520-539)
// for the planned samples g = s * npix + p, written to the current pool behind
// the survivors.  A thread makes all of a pixel's samples, in sample order: the
// per-pixel random state goes from frame to frame by a jump.  (One sample per
// pixel and iteration kept small images from filling the GPU: the 256x256,
// 16-sample box took 32 iterations of at most 65,536 paths, 3.98 ms.)
__global__ void k_regen(FrameParams fp, PathBuffers B, PoolCtl* ctl, int cur, uint4* base0, uint2* base1,
                        const uint32_t* __restrict__ jump_table, ar_path_record* rec)
{
    __shared__ uint32_t jt[kJumpWords];
    for (int k = threadIdx.x; k < kJumpWords; k += blockDim.x) jt[k] = jump_table[k];
    __syncthreads();
    const int n = ctl->plan_new;
    const int base = ctl->plan_base;
    const int64_t first = ctl->plan_first;
    PathRec* pool = pool_of(B, cur);
    // A record is one 128-byte line and a warp makes 32 consecutive ones: they are
    // exchanged through shared memory (16-byte pieces, rotated by the record so
    // that neither side has bank conflicts) and leave as whole lines, 8 lanes to a
    // record.  One record per lane meant 32 lines for each of the 8 stores, which
    // kept L1 94 % busy: 7.3 ms of the 64-sample 1080p render, now 5.2.
    extern __shared__ __align__(16) uint4 stage_all[];
    uint4* stage = stage_all + (threadIdx.x >> 5) * (32 * 8);
    const int lane = static_cast<int>(lane_id());
    const int lanes = min(n, fp.npix);
    for (int i0 = blockIdx.x * blockDim.x + threadIdx.x - lane; i0 < lanes; i0 += gridDim.x * blockDim.x) {
        const int i = min(i0 + lane, lanes - 1);   // lanes past the end repeat the last pixel and store nothing
        const bool mine = i0 + lane < lanes;
        int sidx = static_cast<int>((first + i) / fp.npix);
        const int p = static_cast<int>(first + i - static_cast<int64_t>(sidx) * fp.npix);
        const int px = p % fp.width, py = p / fp.width;
        uint4 a = base0[p];
        uint2 b = base1[p];
        for (int k0 = i0; k0 < n; k0 += fp.npix, ++sidx) {
            const int k = k0 + lane;
            const bool live = mine && k < n;
            const int64_t g = first + k;
            Rng r;
            rng_from(r, a, make_uint4(b.x, b.y, 0u, 0u));
            if (live) {   // advance the per-pixel state to the next frame: offset + 2^32
                uint32_t nv[5] = {a.y, a.z, a.w, b.x, b.y};
                xorwow_jump(nv, jt);
                a = make_uint4(a.x, nv[0], nv[1], nv[2]);
                b = make_uint2(nv[3], nv[4]);
            }
            const float jx = r.next();
            const float jy = r.next();
            const float u = (static_cast<float>(px) + jx) / static_cast<float>(fp.width);
            const float v = (static_cast<float>(py) + jy) / static_cast<float>(fp.height);
            const float ndcx = u * 2.0f - 1.0f;
            const float ndcy = static_cast<float>((1.0 - static_cast<double>(v)) * 2.0 - 1.0);
            const float sx = ndcx * fp.tan_half_x;
            const float sy = ndcy * fp.tan_half_y;
            const f3 cd = mk(fp.cam_d[0], fp.cam_d[1], fp.cam_d[2]);
            const f3 right = mk(fp.right[0], fp.right[1], fp.right[2]);
            const f3 up = mk(fp.up[0], fp.up[1], fp.up[2]);
            const f3 dir0 = normalize(cd + right * sx + up * sy);
            const f3 dir = normalize(dir0);  // CalculateRadiance: rayDirection = normalize(rayDirection)
            const f3 o = mk(fp.cam_o[0], fp.cam_o[1], fp.cam_o[2]);
            if (rec && live) {
#pragma unroll
                for (int h = 0; h < AR_DEBUG_MAX_HITS; ++h) rec[g].hit_object[h] = -1;
            }
            PathRec pr;
            pr.o = f4(o, fbits(0));
            pr.d = f4(dir, fbits(fp.camera_inside ? kFlagInside : 0));
            pr.mask = make_float4(1.0f, 1.0f, 1.0f, fbits(p));
            if (fp.spectral) {  // CalculateRadiance starts with SampleCIE1931(Rand3(seed)) (render.cuh:467)
                const float r0 = r.next(), r1 = r.next(), r2 = r.next();
                const LambdaSample ls = sample_cie1931(r0, r1, r2);
                if (fp.spectral == 4) {   // hero wavelength + 3 rotations: throughputs 1, hero in the side record
                    pr.mask = make_float4(1.0f, 1.0f, 1.0f, fbits(p));
                    if (live) aux_of(B, cur)[base + k] = make_float4(1.0f, 0.0f, ls.lambda, 0.0f);
                } else {
                    pr.mask = make_float4(1.0f, ls.lambda, ls.pdf, fbits(p));
                }
            }
            pr.rad = make_float4(0.0f, 0.0f, 0.0f, fbits(sidx));
            pr.rng0 = make_uint4(r.st.d, r.st.v[0], r.st.v[1], r.st.v[2]);
            pr.rng1 = make_uint4(r.st.v[3], r.st.v[4], static_cast<uint32_t>(-1), static_cast<uint32_t>(r.used));
            pr.prev = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            pr.vloc = make_float4(o.x, o.y, o.z, 0.0f);
            uint4* own = stage + lane * 8;
            const int rot = lane & 7;
            own[0 ^ rot] = *reinterpret_cast<const uint4*>(&pr.o);
            own[1 ^ rot] = *reinterpret_cast<const uint4*>(&pr.d);
            own[2 ^ rot] = *reinterpret_cast<const uint4*>(&pr.mask);
            own[3 ^ rot] = *reinterpret_cast<const uint4*>(&pr.rad);
            own[4 ^ rot] = pr.rng0;
            own[5 ^ rot] = pr.rng1;
            own[6 ^ rot] = *reinterpret_cast<const uint4*>(&pr.prev);
            own[7 ^ rot] = *reinterpret_cast<const uint4*>(&pr.vloc);
            __syncwarp();
            uint4* out = reinterpret_cast<uint4*>(pool + base + k0);
            const int count = min(32, min(lanes - i0, n - k0));   // records of the warp
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int rr = 4 * q + (lane >> 3), c = lane & 7;
                if (rr < count) out[rr * 8 + c] = stage[rr * 8 + (c ^ (rr & 7))];
            }
            __syncwarp();
        }
        if (mine) {
            base0[p] = a;
            base1[p] = b;
        }
    }
}

// ------------------------------------------------------------------ extend
// Scenes with SDF objects or a medium (kExt): this kernel leaves the BVH's hit,
// k_extend_finish does the rest.
template <bool kExt>
struct ExtendIO {
    const PathRec* pool;
    int4* hit;
    int32_t* shade_count;
    int32_t* qsh;
    int cap;
    // queue the path for shading, bucketed by what it hit (render.cuh:97-118)
    __device__ __forceinline__ void to_shade(const SceneView& s, int k, const int4& h)
    {
        hit[k] = h;
        bucket_append(shade_count, qsh, cap, hit_model(s, h.x) + 1, k);
    }
    __device__ __forceinline__ int load(const SceneView& s, int k, RayState& r)
    {
        if (kExt) {
            const float4 o4 = pool[k].o, d4 = pool[k].d;
            if (extend_solo(s, d4, pool[k].rng1)) return -1;
            ray_begin(r, xyz(o4), xyz(d4), c_eps_tab[min(ibits(o4.w) >> 16, 8)], INFINITY);
            return k;
        }
        int4 h;
        if (extend_begin<false>(s, pool[k].o, pool[k].d, pool[k].rng1, r, h)) return k;
        to_shade(s, k, h);
        return -1;
    }
    __device__ __forceinline__ void store(const SceneView& s, int k, const RayState& r)
    {
        if (kExt) hit[k] = make_int4(r.best.obj, r.best.prim, ibits(r.best.t), 0);
        else to_shade(s, k, extend_end<false>(s, pool[k], r, 0u));
    }
};

// Trace's closest-hit query (render.cuh:86-99) for every path of the pool.
template <bool kExt>
__global__ void __launch_bounds__(kTraceBlock, kTraceMinBlocks) k_extend(SceneView s, PathBuffers B, int cur, PoolCtl* ctl,
                                                        unsigned long long* stats, uint32_t* ovf, int* err)
{
    extern __shared__ uint32_t smem[];
    ExtendIO<kExt> io;
    io.pool = pool_of(B, cur);
    io.hit = B.hit;
    io.shade_count = ctl->shade_count;
    io.qsh = B.qsh;
    io.cap = B.capacity;
    const int n = ctl->count[cur];
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&stats[0], static_cast<unsigned long long>(n));
    traverse_queue<false>(s, io, n, &ctl->fetch_ext, lane_stack(smem), thread_overflow(ovf), err, &stats[2]);
}

// The rest of Trace in scenes with SDF objects or a medium: solo traces, SDF
// objects, free-flight sampling, shading buckets.  A kernel of its own because
// these loops (sphere tracing, delta tracking) are long and run here with all
// lanes of a warp; at the refill point of the traversal only the 8 or so lanes
// whose rays had just finished ran them while the others waited (1280x720, 16
// samples, four wavelengths: 21.4 ms in k_extend, now 2.3 + 10.9 ms; the shadow
// queries 12.4, now 1.8 + 7.4 ms).  A queue of the rays that meet an object's box,
// marched with lane refill, measured the same: the longest marches (512 steps)
// and the extra pass over the paths cost what it saved.
__global__ void __launch_bounds__(kTraceBlock) k_extend_finish(SceneView s, PathBuffers B, int cur, PoolCtl* ctl, uint32_t medium_key)
{
    const PathRec* pool = pool_of(B, cur);
    const int n = ctl->count[cur];
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const PathRec pr = pool[k];
        RayState r;
        int4 h;
        if (extend_begin<true>(s, pr.o, pr.d, pr.rng1, r, h)) {
            const int4 b = B.hit[k];
            r.best.obj = b.x;
            r.best.prim = b.y;
            r.best.t = fbits(b.z);
            h = extend_end<true>(s, pr, r, medium_key);
        }
        B.hit[k] = h;
        bucket_append(ctl->shade_count, B.qsh, B.capacity, hit_model(s, h.x) + 1, k);
    }
}

// ------------------------------------------------------------------ shade
// One iteration of the loop body for every path of bucket kModel + 1; kModel
// is the shading model of every path of the launch, -1 = miss.
template <int kModel, bool kExt, int kSpec, bool kNrc, bool kGuide>
__global__ void __launch_bounds__(kShadeBlock) k_shade(SceneView s, FrameParams fp, PathBuffers B, int cur,
                                                       PoolCtl* ctl, ar_path_record* rec)
{
    const int bucket = kModel + 1;
    const int n = ctl->shade_count[bucket];
    const int32_t* q = B.qsh + static_cast<int64_t>(bucket) * B.capacity;
    const uint4* pool = reinterpret_cast<const uint4*>(pool_of(B, cur));
    uint4* next_pool = reinterpret_cast<uint4*>(pool_of(B, 1 - cur));
    // records go through shared memory in both directions, 8 lanes to a record's
    // line (see k_regen); these kernels wait on memory, and the shorter queue at
    // L1 takes the 64-sample 1080p render from 123.1 to 121.7 ms
    extern __shared__ __align__(16) uint4 stage_all[];
    uint4* stage = stage_all + (threadIdx.x >> 5) * (32 * 8);
    const int lane = static_cast<int>(lane_id()), piece = lane & 7, rot = lane & 7;
    for (int q0 = blockIdx.x * blockDim.x + threadIdx.x - lane; q0 < n; q0 += gridDim.x * blockDim.x) {
        const bool live = q0 + lane < n;
        const int k = live ? q[q0 + lane] : 0;
        uint4 in[8];
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            const int kk = __shfl_sync(0xFFFFFFFFu, k, 4 * m + (lane >> 3));
            in[m] = pool[static_cast<int64_t>(kk) * 8 + piece];
        }
        __syncwarp();
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            const int rr = 4 * m + (lane >> 3);
            stage[rr * 8 + (piece ^ (rr & 7))] = in[m];
        }
        __syncwarp();
        ShadeResult R;
        R.cont = R.shadow = R.nrc_query = false;
        if (live) {
            PathRec pr;
            const uint4* own = stage + lane * 8;
            *reinterpret_cast<uint4*>(&pr.o) = own[0 ^ rot];
            *reinterpret_cast<uint4*>(&pr.d) = own[1 ^ rot];
            *reinterpret_cast<uint4*>(&pr.mask) = own[2 ^ rot];
            *reinterpret_cast<uint4*>(&pr.rad) = own[3 ^ rot];
            pr.rng0 = own[4 ^ rot];
            pr.rng1 = own[5 ^ rot];
            *reinterpret_cast<uint4*>(&pr.prev) = own[6 ^ rot];
            *reinterpret_cast<uint4*>(&pr.vloc) = own[7 ^ rot];
            shade_path<kModel, kExt, kSpec, kNrc, kGuide>(s, fp, pr, kSpec == 4 ? aux_of(B, cur)[k] : make_float4(0.0f, 0.0f, 0.0f, 0.0f),
                                                          B.hit[k], kModel, rec, R);
        }
        __syncwarp();
        int target = 0;
        const int j = warp_alloc(&ctl->count[1 - cur], live && R.cont);
        const int r = warp_alloc(&ctl->retire_count, live && !R.cont);
        if (kNrc) {
            const int ni = warp_alloc(fp.nrc.query_count, live && R.nrc_query);
            if (live && R.nrc_query && ni < fp.nrc.query_cap) fp.nrc.queries[ni] = query_record<kSpec>(R);
        }
        const unsigned conts = __ballot_sync(0xFFFFFFFFu, live && R.cont);
        if (live && R.cont) {
            if (kSpec == 4) aux_of(B, 1 - cur)[j] = make_float4(R.mask3, R.rad3, R.lambda, 0.0f);
            const PathRec out = next_record<kSpec, kNrc>(R);
            const int slot = __popc(conts & lanes_below()), srot = slot & 7;
            uint4* own = stage + slot * 8;
            own[0 ^ srot] = *reinterpret_cast<const uint4*>(&out.o);
            own[1 ^ srot] = *reinterpret_cast<const uint4*>(&out.d);
            own[2 ^ srot] = *reinterpret_cast<const uint4*>(&out.mask);
            own[3 ^ srot] = *reinterpret_cast<const uint4*>(&out.rad);
            own[4 ^ srot] = out.rng0;
            own[5 ^ srot] = out.rng1;
            own[6 ^ srot] = *reinterpret_cast<const uint4*>(&out.prev);
            own[7 ^ srot] = *reinterpret_cast<const uint4*>(&out.vloc);
            target = j;
        } else if (live) {
            B.retire[r] = retire_record<kSpec>(R);
            target = ~r;
        }
        const int m = warp_alloc(&ctl->shadow_count, live && R.shadow);
        if (live && R.shadow) {
            if (kSpec == 4) B.shadow3[m] = R.pend3;
            B.shadow[m] = shadow_record(R, target);
        }
        if (conts) {
            const int j0 = __shfl_sync(0xFFFFFFFFu, j, __ffs(conts) - 1), count = __popc(conts);
            __syncwarp();
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const int rr = 4 * c + (lane >> 3);
                if (rr < count) next_pool[static_cast<int64_t>(j0 + rr) * 8 + piece] = stage[rr * 8 + (piece ^ (rr & 7))];
            }
        }
        __syncwarp();
    }
}

// ------------------------------------------------------------------ shadow
// SegmentTrace -> AnyHitSegmentBVH (render.cuh:167-183, intersection.cuh:372-397)
// and the remainder of NEE (render.cuh:242-343): the pending term is added when
// the segment is unoccluded, and previousDidNEE_ becomes "occluded or cos > 0".
template <bool kExt>
struct ShadowIO {
    const ShadowRec* rec;
    PathRec* next_pool;
    RetireRec* retire;
    float4* next_aux;         // four-wavelength mode: side records of the next pool
    const float* pend3;       // four-wavelength mode: pending radiance of wavelength 3
    int spec4;
    unsigned long long traced;
    int32_t* state;           // kExt: per segment 0 open, 1 blocked, 2 too short, for k_shadow_finish
    __device__ __forceinline__ void finish(int m, bool occ, float tr = 1.0f)
    {
        const float4 dst = rec[m].dst;
        float4 nee = rec[m].nee;
        const int target = ibits(dst.w);
        const bool cosOK = (ibits(nee.w) & 1) != 0;
        const bool add = !occ && cosOK;
        if (kExt) { nee.x *= tr; nee.y *= tr; nee.z *= tr; }  // medium transmittance
        if (target >= 0) {
            PathRec& p = next_pool[target];
            if (add) {
                const float4 r = p.rad;
                p.rad = make_float4(r.x + nee.x, r.y + nee.y, r.z + nee.z, r.w);
                if (spec4) next_aux[target].y += pend3[m] * (kExt ? tr : 1.0f);
            }
            if (occ || cosOK) {
                const float4 d = p.d;
                p.d = make_float4(d.x, d.y, d.z, fbits(ibits(d.w) | kFlagPrevNEE));
            }
        } else if (add) {
            RetireRec& p = retire[~target];
            const float4 r = p.rad;
            p.rad = make_float4(r.x + nee.x, r.y + nee.y, r.z + nee.z, r.w);
            if (spec4) p.meta.w = __float_as_int(__int_as_float(p.meta.w) + pend3[m] * (kExt ? tr : 1.0f));
        }
    }
    __device__ __forceinline__ int load(const SceneView&, int m, RayState& r)
    {
        if (shadow_begin(rec[m].src, xyz(rec[m].dst), r)) {
            ++traced;
            return m;
        }
        if (kExt) state[m] = 2;
        else finish(m, false);
        return -1;
    }
    __device__ __forceinline__ void store(const SceneView&, int m, const RayState& r)
    {
        if (kExt) state[m] = r.best.obj >= 0 ? 1 : 0;
        else finish(m, r.best.obj >= 0);
    }
};

template <bool kExt>
__device__ __forceinline__ ShadowIO<kExt> shadow_io(const PathBuffers& B, int cur, int spec4)
{
    ShadowIO<kExt> io;
    io.rec = B.shadow;
    io.next_pool = pool_of(B, 1 - cur);
    io.retire = B.retire;
    io.next_aux = aux_of(B, 1 - cur);
    io.pend3 = B.shadow3;
    io.spec4 = spec4;
    io.traced = 0;
    io.state = B.qsh;   // the shading queues are free by now
    return io;
}

template <bool kExt>
__global__ void __launch_bounds__(kTraceBlock, kTraceMinBlocks) k_shadow(SceneView s, PathBuffers B, int cur, PoolCtl* ctl,
                                                        unsigned long long* stats, uint32_t* ovf, int* err, int spec4)
{
    extern __shared__ uint32_t smem[];
    const int n = ctl->shadow_count;
    ShadowIO<kExt> io = shadow_io<kExt>(B, cur, spec4);
    traverse_queue<true>(s, io, n, &ctl->fetch_shadow, lane_stack(smem), thread_overflow(ovf), err, &stats[4]);
    unsigned long long c = io.traced;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xFFFFFFFFu, c, o);
    if (lane_id() == 0 && c) atomicAdd(&stats[1], c);
}

// The rest of a shadow query in scenes with SDF objects or a medium: SDF
// objects, transmittance, and the light sample's term (see k_extend_finish).
__global__ void __launch_bounds__(kTraceBlock) k_shadow_finish(SceneView s, PathBuffers B, int cur, PoolCtl* ctl, int spec4)
{
    ShadowIO<true> io = shadow_io<true>(B, cur, spec4);
    const int n = ctl->shadow_count;
    for (int m = blockIdx.x * blockDim.x + threadIdx.x; m < n; m += gridDim.x * blockDim.x) {
        const int st = B.qsh[m];
        bool occ = st == 1;
        float tr = 1.0f;
        if (st == 0) {
            RayState r;
            const float4 src = B.shadow[m].src;
            shadow_begin(src, xyz(B.shadow[m].dst), r);
            occ = shadow_end<true>(s, r, src.w, static_cast<uint32_t>(ibits(B.shadow[m].nee.w)), tr);
        }
        io.finish(m, occ, tr);
    }
}

// ------------------------------------------------------------------ retire
__global__ void k_retire(FrameParams fp, PathBuffers B, PoolCtl* ctl, double* accum, ar_path_record* rec)
{
    const int n = ctl->retire_count;
    if (blockIdx.x == 0 && threadIdx.x == 0) ctl->retired += n;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        retire_path(fp, B.retire[i], accum, rec);
}

__global__ void k_mean(const double* accum, int64_t n, double inv, float* out)
{
    const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (i < n) out[i] = static_cast<float>(accum[i] * inv);
}

__global__ void k_add(const double* src, int64_t n, double* dst)
{
    const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (i < n) dst[i] += src[i];
}

// ------------------------------------------------------------------ launchers
constexpr size_t kTraceSmem = static_cast<size_t>(kStackShared) * kTraceBlock * 4;

int trace_grid(int sm_count)
{
    static int blocks = 0;
    if (blocks == 0) {
        int b0 = 1, b1 = 1, b2 = 1, b3 = 1;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b0, k_extend<false>, kTraceBlock, kTraceSmem);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b1, k_shadow<false>, kTraceBlock, kTraceSmem);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b2, k_trace_rays<false, false>, kTraceBlock, kTraceSmem);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b3, k_trace_rays<true, false>, kTraceBlock, kTraceSmem);
        cudaGetLastError();
        blocks = max(1, max(max(b0, b1), max(b2, b3)));
    }
    return blocks * sm_count;
}

cudaError_t launch_trace_rays(const SceneView& s, const float4* rays, int n, int any, int32_t* obj, float* t,
                              PoolCtl* ctl, uint32_t* ovf, int* err, int grid, cudaStream_t st)
{
    if (s.num_sdf > 0) {
        RaysIO<true> io;
        io.rays = rays;
        io.out_obj = obj;
        io.out_t = t;
        io.any = any ? 1 : 0;
        if (any) k_trace_rays<true, true><<<grid, kTraceBlock, kTraceSmem, st>>>(s, io, n, ctl, ovf, err);
        else k_trace_rays<false, true><<<grid, kTraceBlock, kTraceSmem, st>>>(s, io, n, ctl, ovf, err);
    } else {
        RaysIO<false> io;
        io.rays = rays;
        io.out_obj = obj;
        io.out_t = t;
        io.any = any ? 1 : 0;
        if (any) k_trace_rays<true, false><<<grid, kTraceBlock, kTraceSmem, st>>>(s, io, n, ctl, ovf, err);
        else k_trace_rays<false, false><<<grid, kTraceBlock, kTraceSmem, st>>>(s, io, n, ctl, ovf, err);
    }
    return cudaGetLastError();
}

// The generator's jump tables (0.77 MB), constants that every scene of a device
// shares.  A copy per scene took 0.04 of the 0.23 ms that a small scene takes to
// create.  The last words tell whether they are there: a device that was reset
// has lost them.
static __device__ __align__(16) uint32_t g_rng_tables[kInitTables * kJumpWords];
cudaError_t rng_tables(const uint32_t** tables)
{
    static std::mutex* lock = new std::mutex;   // never destroyed: scenes may be created during process exit
    static const auto* host = new std::vector<uint32_t>(xorwow_init_tables());
    constexpr size_t kTail = 80;
    const uint32_t* tail = host->data() + host->size() - kTail;
    std::lock_guard<std::mutex> g(*lock);
    void* p = nullptr;
    uint32_t have[kTail];
    cudaError_t e = cudaGetSymbolAddress(&p, g_rng_tables);
    if (e == cudaSuccess) e = cudaMemcpyFromSymbol(have, g_rng_tables, sizeof(have), sizeof(g_rng_tables) - sizeof(have));
    if (e == cudaSuccess && std::memcmp(have, tail, sizeof(have)) != 0)
        e = cudaMemcpyToSymbol(g_rng_tables, host->data(), sizeof(g_rng_tables));
    *tables = static_cast<const uint32_t*>(p);
    return e;
}

cudaError_t launch_rng_init(const FrameParams& fp, uint4* b0, uint2* b1, const uint32_t* tables, int sm_count, cudaStream_t st)
{
    const cudaError_t e = cudaFuncSetAttribute(k_rng_init, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kInitSmem));
    if (e != cudaSuccess) return e;
    const int groups = (fp.grid_x * ((fp.height + 3) / 4) + 7) / 8;
    const int grid = std::min((groups + kInitBlock / 32 - 1) / (kInitBlock / 32), 2 * sm_count);
    k_rng_init<<<grid, kInitBlock, kInitSmem, st>>>(fp, b0, b1, tables);
    return cudaGetLastError();
}

cudaError_t launch_rng_tape(const FrameParams& fp, int spp, int per_path, float* out, cudaStream_t st)
{
    k_rng_tape<<<(fp.npix + 127) / 128, 128, 0, st>>>(fp, spp, per_path, out);
    return cudaGetLastError();
}

cudaError_t launch_render_init(PoolCtl* ctl, int64_t total, double* accum, int64_t npix, unsigned long long* stats, int* err,
                               int sm_count, cudaStream_t st)
{
    const int64_t pairs = (3 * npix + 1) / 2;   // the sums are allocated in multiples of 256 bytes
    const int grid = static_cast<int>(std::min<int64_t>((pairs + 255) / 256, static_cast<int64_t>(sm_count) * 8));
    k_render_init<<<grid, 256, 0, st>>>(ctl, total, reinterpret_cast<double2*>(accum), pairs, stats, err);
    return cudaGetLastError();
}

cudaError_t launch_generate(const FrameParams& fp, const PathBuffers& B, PoolCtl* ctl, uint4* b0, uint2* b1,
                            const uint32_t* jump_table, ar_path_record* rec, int cur, int grid_other, cudaStream_t st)
{
    k_plan<<<1, 1, 0, st>>>(ctl, cur, B.capacity);
    k_regen<<<grid_other, kShadeBlock, kStageSmem, st>>>(fp, B, ctl, cur, b0, b1, jump_table, rec);
    return cudaGetLastError();
}

// The five per-material shading launches of one iteration.
template <bool kExt, int kSpec, bool kNrc, bool kGuide = false>
void launch_shade(const SceneView& s, const FrameParams& fp, const PathBuffers& B, int c, PoolCtl* ctl,
                  ar_path_record* rec, int grid, cudaStream_t st)
{
    k_shade<-1, kExt, kSpec, kNrc, kGuide><<<grid, kShadeBlock, kStageSmem, st>>>(s, fp, B, c, ctl, rec);
    k_shade<AR_MAT_DIFFUSE, kExt, kSpec, kNrc, kGuide><<<grid, kShadeBlock, kStageSmem, st>>>(s, fp, B, c, ctl, rec);
    k_shade<AR_MAT_LIGHT, kExt, kSpec, kNrc, kGuide><<<grid, kShadeBlock, kStageSmem, st>>>(s, fp, B, c, ctl, rec);
    k_shade<AR_MAT_GLASS, kExt, kSpec, kNrc, kGuide><<<grid, kShadeBlock, kStageSmem, st>>>(s, fp, B, c, ctl, rec);
    k_shade<AR_MAT_GGX, kExt, kSpec, kNrc, kGuide><<<grid, kShadeBlock, kStageSmem, st>>>(s, fp, B, c, ctl, rec);
    if (kExt && s.has_medium)
        k_shade<kModelMedium, kExt, kSpec, kNrc, kGuide><<<grid, kShadeBlock, kStageSmem, st>>>(s, fp, B, c, ctl, rec);
}

cudaError_t launch_iterations(const SceneView& s, const FrameParams& fp, const PathBuffers& B, PoolCtl* ctl,
                              uint4* b0, uint2* b1, const uint32_t* jump_table, unsigned long long* stats,
                              uint32_t* ovf, int* err, double* accum, ar_path_record* rec, int iterations, int* cur,
                              int grid_trace, int grid_other, cudaStream_t st, int64_t* launches, LaunchTimers* tm)
{
    const bool ext = s.num_sdf > 0 || s.has_medium;
    for (int it = 0; it < iterations; ++it) {
        const int c = *cur;
        launch_generate(fp, B, ctl, b0, b1, jump_table, rec, c, grid_other, st);
        const bool te = tm && tm->n_extend < tm->cap;
        if (te) cudaEventRecord(tm->extend_ev[2 * tm->n_extend], st);
        if (ext) {
            k_extend<true><<<grid_trace, kTraceBlock, kTraceSmem, st>>>(s, B, c, ctl, stats, ovf, err);
            k_extend_finish<<<grid_trace, kTraceBlock, 0, st>>>(s, B, c, ctl, fp.medium_key);
        } else {
            k_extend<false><<<grid_trace, kTraceBlock, kTraceSmem, st>>>(s, B, c, ctl, stats, ovf, err);
        }
        if (te) cudaEventRecord(tm->extend_ev[2 * tm->n_extend++ + 1], st);
        if (fp.spectral == 4 && fp.nrc.enabled) {
            if (ext) launch_shade<true, 4, true>(s, fp, B, c, ctl, rec, grid_other, st);
            else launch_shade<false, 4, true>(s, fp, B, c, ctl, rec, grid_other, st);
        } else if (fp.spectral == 4) {
            if (ext) launch_shade<true, 4, false>(s, fp, B, c, ctl, rec, grid_other, st);
            else launch_shade<false, 4, false>(s, fp, B, c, ctl, rec, grid_other, st);
        } else if (fp.spectral) {
            if (ext) launch_shade<true, 1, false>(s, fp, B, c, ctl, rec, grid_other, st);
            else launch_shade<false, 1, false>(s, fp, B, c, ctl, rec, grid_other, st);
        } else if (fp.guiding) {
            if (ext) launch_shade<true, 0, false, true>(s, fp, B, c, ctl, rec, grid_other, st);
            else launch_shade<false, 0, false, true>(s, fp, B, c, ctl, rec, grid_other, st);
        } else if (fp.nrc.enabled) {
            if (ext) launch_shade<true, 0, true>(s, fp, B, c, ctl, rec, grid_other, st);
            else launch_shade<false, 0, true>(s, fp, B, c, ctl, rec, grid_other, st);
        } else {
            if (ext) launch_shade<true, 0, false>(s, fp, B, c, ctl, rec, grid_other, st);
            else launch_shade<false, 0, false>(s, fp, B, c, ctl, rec, grid_other, st);
        }
        const bool ts = tm && tm->n_shadow < tm->cap;
        if (ts) cudaEventRecord(tm->shadow_ev[2 * tm->n_shadow], st);
        const int spec4 = fp.spectral == 4 ? 1 : 0;
        if (ext) {
            k_shadow<true><<<grid_trace, kTraceBlock, kTraceSmem, st>>>(s, B, c, ctl, stats, ovf, err, spec4);
            k_shadow_finish<<<grid_trace, kTraceBlock, 0, st>>>(s, B, c, ctl, spec4);
        } else k_shadow<false><<<grid_trace, kTraceBlock, kTraceSmem, st>>>(s, B, c, ctl, stats, ovf, err, spec4);
        if (ts) cudaEventRecord(tm->shadow_ev[2 * tm->n_shadow++ + 1], st);
        k_retire<<<grid_other, kShadeBlock, 0, st>>>(fp, B, ctl, accum, rec);
        *launches += 10 + (ext ? 2 : 0) + (s.has_medium ? 1 : 0);
        *cur = 1 - c;
    }
    return cudaGetLastError();
}

cudaError_t launch_mean(const double* accum, int64_t n, double inv, float* out, cudaStream_t st)
{
    k_mean<<<static_cast<unsigned>((n + 255) / 256), 256, 0, st>>>(accum, n, inv, out);
    return cudaGetLastError();
}

cudaError_t launch_add(const double* src, int64_t n, double* dst, cudaStream_t st)
{
    k_add<<<static_cast<unsigned>((n + 255) / 256), 256, 0, st>>>(src, n, dst);
    return cudaGetLastError();
}

}  // namespace ar
