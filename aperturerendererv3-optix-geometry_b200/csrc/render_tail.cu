// render_tail.cu -- the last paths of a render, each run to its end by one lane.
//
// An iteration of the wavefront (render.cu) is ten dependent launches, 30-40 us
// however few paths it advances.  When the remaining paths no longer fill the
// GPU that latency is all the time there is: a 160x120 preview spent 1.1 ms in
// 16 iterations that held 0.2 ms of work.  k_tail takes over there: a lane keeps
// its path in registers and runs closest hit, shading, shadow query and
// retirement until the path ends, with no launch and no memory round trip
// between them.  The device functions are the wavefront's own (path_stages.cuh),
// so every path is the same bit for bit.
//
// Bound: instruction fetch and the latency of one path after the other (ncu on
// the 160x120 preview, 19,200 paths: issue slots 17 % busy, half of a warp's wait
// for instructions, 61 % of the fetches hit).  So one block of 8 warps per SM,
// whose warps advance segment by segment together, and few paths spread over all
// warps, 16 to 32 each.  That preview: 272 us with three blocks of 4 warps that
// run free, 240 with the warps of a block together, 206 with one block.
#include "path_stages.cuh"

#include <algorithm>

namespace ar {

namespace {

constexpr size_t kTailSmem = static_cast<size_t>(kStackShared) * kTailBlock * 4;

template <bool kAny>
__device__ __forceinline__ void traverse_one(const SceneView& s, RayState& r, uint32_t* stack, uint32_t* ovf, int* err)
{
    if (s.num_nodes == 0) return;
    while (!ray_step<kAny, false>(s, r, stack, ovf, err)) {
    }
}

template <bool kExt, int kSpec, bool kNrc, bool kGuide>
__global__ void __launch_bounds__(kTailBlock, 1)
k_tail(SceneView s, FrameParams fp, PathBuffers B, int cur, PoolCtl* ctl, unsigned long long* stats, uint32_t* ovf_base,
       int* err, double* accum, ar_path_record* rec, int limit)
{
    extern __shared__ uint32_t smem[];
    const int n = ctl->count[cur];
    // the last block to finish changes these words, after every block has read them
    if (n == 0 || n > limit || ctl->gen_next < ctl->total) return;
    uint32_t* stack = lane_stack(smem);
    uint32_t* ovf = thread_overflow(ovf_base);
    const PathRec* pool = pool_of(B, cur);
    const int warps = gridDim.x * (kTailBlock / 32);
    const int lanes = min(32, max(16, (n + warps - 1) / warps));   // paths per warp
    // warps of consecutive index on different SMs
    const int warp = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    unsigned long long ext = 0, shd = 0;
    for (int first = 0; first < n; first += warps * lanes) {
        const int k = first + warp * lanes + static_cast<int>(lane_id());
        bool live = static_cast<int>(lane_id()) < lanes && k < n;
        PathRec pr;
        float4 aux = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (live) {
            pr = pool[k];
            if (kSpec == 4) aux = aux_of(B, cur)[k];
        }
        // the block's warps go from segment to segment together: the loop body is
        // larger than the instruction cache, and warps at different places of it
        // evict each other's code
        while (__syncthreads_or(live)) {
            if (live) {
                RayState r;
                int4 hr;
                ++ext;
                if (extend_begin<kExt>(s, pr.o, pr.d, pr.rng1, r, hr)) {
                    traverse_one<false>(s, r, stack, ovf, err);
                    hr = extend_end<kExt>(s, pr, r, fp.medium_key);
                }
                ShadeResult R;
                shade_path<kModelAny, kExt, kSpec, kNrc, kGuide>(s, fp, pr, aux, hr, hit_model(s, hr.x), rec, R);
                if (kNrc && R.nrc_query) {
                    const int q = atomicAdd(fp.nrc.query_count, 1);
                    if (q < fp.nrc.query_cap) fp.nrc.queries[q] = query_record<kSpec>(R);
                }
                if (R.shadow) {   // the rest of NEE (render.cuh:242-343), as ShadowIO::finish
                    const ShadowRec sr = shadow_record(R, 0);
                    bool occ = false;
                    float tr = 1.0f;
                    if (shadow_begin(sr.src, R.light, r)) {
                        ++shd;
                        traverse_one<true>(s, r, stack, ovf, err);
                        occ = shadow_end<kExt>(s, r, sr.src.w, static_cast<uint32_t>(ibits(sr.nee.w)), tr);
                    }
                    if (!occ && R.cos_ok) {
                        f3 nee = R.pending;
                        if (kExt) nee = mk(nee.x * tr, nee.y * tr, nee.z * tr);
                        R.radiance = R.radiance + nee;
                        if (kSpec == 4) R.rad3 += R.pend3 * (kExt ? tr : 1.0f);
                    }
                    if (occ || R.cos_ok) R.flags |= kFlagPrevNEE;
                }
                live = R.cont;
                if (R.cont) {
                    pr = next_record<kSpec, kNrc>(R);
                    if (kSpec == 4) aux = make_float4(R.mask3, R.rad3, R.lambda, 0.0f);
                } else {
                    retire_path(fp, retire_record<kSpec>(R), accum, rec);
                }
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        ext += __shfl_xor_sync(0xFFFFFFFFu, ext, o);
        shd += __shfl_xor_sync(0xFFFFFFFFu, shd, o);
    }
    if (lane_id() == 0 && ext) {
        atomicAdd(&stats[0], ext);
        if (shd) atomicAdd(&stats[1], shd);
    }
    __syncthreads();
    if (threadIdx.x == 0 && atomicAdd(&ctl->tail_done, 1) == static_cast<int>(gridDim.x) - 1) {
        ctl->tail_done = 0;
        ctl->count[cur] = 0;
        ctl->retired += n;
    }
}

}  // namespace

cudaError_t set_intersect_eps_tail(const float* tab9)
{
    return cudaMemcpyToSymbol(c_eps_tab, tab9, 9 * sizeof(float));
}

cudaError_t launch_tail(const SceneView& s, const FrameParams& fp, const PathBuffers& B, PoolCtl* ctl,
                        unsigned long long* stats, uint32_t* ovf, int* err, double* accum, ar_path_record* rec, int cur,
                        int limit, int sm_count, cudaStream_t st)
{
    const bool ext = s.num_sdf > 0 || s.has_medium;
    const int grid = sm_count;
    auto go = [&](auto kernel) {
        kernel<<<grid, kTailBlock, kTailSmem, st>>>(s, fp, B, cur, ctl, stats, ovf, err, accum, rec, limit);
    };
    if (fp.spectral == 4 && fp.nrc.enabled) ext ? go(k_tail<true, 4, true, false>) : go(k_tail<false, 4, true, false>);
    else if (fp.spectral == 4) ext ? go(k_tail<true, 4, false, false>) : go(k_tail<false, 4, false, false>);
    else if (fp.spectral) ext ? go(k_tail<true, 1, false, false>) : go(k_tail<false, 1, false, false>);
    else if (fp.guiding) ext ? go(k_tail<true, 0, false, true>) : go(k_tail<false, 0, false, true>);
    else if (fp.nrc.enabled) ext ? go(k_tail<true, 0, true, false>) : go(k_tail<false, 0, true, false>);
    else ext ? go(k_tail<true, 0, false, false>) : go(k_tail<false, 0, false, false>);
    return cudaGetLastError();
}

}  // namespace ar
