// path_stages.cuh -- the stages of the path loop as device functions, shared by
// the wavefront kernels (render.cu) and the kernel that runs the last paths of a
// render to their end (render_tail.cu).
//
// Built with --fmad=false: every floating-point expression rounds exactly as
// the reference's source reads (see detmath.h); fused multiply-adds appear only
// where written as fmaf (the BVH box planes and the sampling polynomials).
#pragma once

#include <curand_kernel.h>

#include "render_kernels.h"
#include "shading.cuh"
#include "wavefront.cuh"

namespace ar {

// ------------------------------------------------------------------ warp helpers
__device__ __forceinline__ unsigned lane_id() { return threadIdx.x & 31u; }
__device__ __forceinline__ unsigned lanes_below() { return (1u << lane_id()) - 1u; }

// Warp-aggregated allocation, called by all 32 lanes together: one atomic per
// warp, so the indices given out are consecutive, ordered by lane.  Returns the
// caller's index, or -1 when pred is false.  (The mask is the whole warp, not
// __activemask(), which may see only part of a warp that a branch has split:
// k_shade stores the warp's records as one run of slots.)
__device__ __forceinline__ int warp_alloc(int32_t* counter, bool pred)
{
    const unsigned m = __ballot_sync(0xFFFFFFFFu, pred);
    if (m == 0) return -1;
    const int leader = __ffs(m) - 1;
    int base = 0;
    if (static_cast<int>(lane_id()) == leader) base = atomicAdd(counter, __popc(m));
    base = __shfl_sync(0xFFFFFFFFu, base, leader);
    return pred ? base + __popc(m & lanes_below()) : -1;
}

// Append `value` to bucket `bucket` of a bucketed queue (data[bucket * cap + i]);
// lanes of a warp with the same bucket share one atomic (__match_any_sync).
__device__ __forceinline__ void bucket_append(int32_t* counts, int32_t* data, int cap, int bucket, int32_t value)
{
    const unsigned active = __activemask();
    const unsigned same = __match_any_sync(active, bucket);
    const int leader = __ffs(same) - 1;
    int base = 0;
    if (static_cast<int>(lane_id()) == leader) base = atomicAdd(&counts[bucket], __popc(same));
    base = __shfl_sync(same, base, leader);
    data[static_cast<int64_t>(bucket) * cap + base + __popc(same & lanes_below())] = value;
}

// reference pixel index of InitRand (random.cuh:31-39) for 8x4 blocks
__device__ __forceinline__ unsigned long long ref_pixel_index(int i, int j, int grid_x)
{
    const int tx = i & 7, ty = j & 3, bxi = i >> 3, byi = j >> 2;
    return static_cast<unsigned long long>(tx + ty * 8) + 32ull * static_cast<unsigned long long>(bxi + byi * grid_x);
}

__device__ __forceinline__ uint32_t* lane_stack(uint32_t* smem)
{
    return smem + (threadIdx.x >> 5) * (kStackShared * 32) + lane_id();
}
__device__ __forceinline__ uint32_t* thread_overflow(uint32_t* base)
{
    return base + (static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x) * kStackOverflow;
}

__device__ __forceinline__ int ibits(float f) { return __float_as_int(f); }
// pool buffer `c` without dynamic indexing of the kernel-parameter array
__device__ __forceinline__ PathRec* pool_of(const PathBuffers& B, int c) { return c ? B.pool[1] : B.pool[0]; }
__device__ __forceinline__ float4* aux_of(const PathBuffers& B, int c) { return c ? B.aux[1] : B.aux[0]; }
__device__ __forceinline__ float fbits(int i) { return __int_as_float(i); }

// ------------------------------------------------------------------ RNG
__device__ __forceinline__ void rng_from(Rng& r, uint4 a, uint4 b)
{
    r.st.d = a.x; r.st.v[0] = a.y; r.st.v[1] = a.z; r.st.v[2] = a.w; r.st.v[3] = b.x; r.st.v[4] = b.y;
    r.st.boxmuller_flag = 0; r.st.boxmuller_flag_double = 0;
    r.st.boxmuller_extra = 0.0f; r.st.boxmuller_extra_double = 0.0;
    r.used = 0;
}

// ------------------------------------------------------------------ extend
// Free-flight sampling in the medium along the extension segment [0, tmax):
// the distance of the first real collision, or -1 (out of line: only scenes
// with a medium reach it).
static __device__ __noinline__ float medium_collision(const SceneView& s, const PathRec& pr, f3 o, f3 d, float tmax,
                                               uint32_t key)
{
    HashRng h;
    h.seed = medium_seed(key, static_cast<uint32_t>(ibits(pr.rad.w)), static_cast<uint32_t>(ibits(pr.mask.w)),
                         static_cast<uint32_t>(ibits(pr.o.w) & 0xFFFF), 0u);
    h.n = 0;
    return delta_track(s.medium, o, d, tmax, h);
}

// Whether a path's closest-hit query is the solo trace of the medium's object
// (render.cuh:91-94).
__device__ __forceinline__ bool extend_solo(const SceneView& s, float4 d4, const uint4& rng1)
{
    const int mobj = static_cast<int>(rng1.z);
    return (ibits(d4.w) & kFlagInside) && mobj >= 0 && s.objects[mobj].type != AR_OBJ_TRIANGLE;
}

// The start of a path's closest-hit query (Trace, render.cuh:86-99): true when
// the BVH has to be traversed with r, false when the query was the solo trace
// of the medium's object (render.cuh:91-94, intersection.cuh:185-193), whose
// result is `hit` (object, primitive slot, t bits).
template <bool kExt>
__device__ __forceinline__ bool extend_begin(const SceneView& s, float4 o4, float4 d4, const uint4& rng1, RayState& r, int4& hit)
{
    const f3 o = xyz(o4), d = xyz(d4);
    const float e = c_eps_tab[min(ibits(o4.w) >> 16, 8)];
    if (extend_solo(s, d4, rng1)) {
        const int mobj = static_cast<int>(rng1.z);
        const float t = (kExt && s.objects[mobj].type == AR_OBJ_SDF) ? sdf_solo_t(s, mobj, o, d, e)
                                                                     : isect_analytic_t(s, mobj, o, d);
        hit = t >= 0.0f && !(t < e) ? make_int4(mobj, -1, ibits(t), 0) : make_int4(-1, -1, 0, 0);
        return false;
    }
    ray_begin(r, o, d, e, INFINITY);
    return true;
}

// The result of a traversed closest-hit query: the BVH's hit, then SDF objects
// and free-flight sampling in the participating medium.
template <bool kExt>
__device__ __forceinline__ int4 extend_end(const SceneView& s, const PathRec& pr, const RayState& r, uint32_t medium_key)
{
    int32_t obj = r.best.obj, prim = r.best.prim;
    float t = r.best.t;
    if (kExt && s.num_sdf > 0) {
        const int32_t before = obj;
        sdf_closest(s, r.o, r.d, r.tmin, c_eps_tab[min(ibits(pr.o.w) >> 16, 8)], &t, &obj);
        if (obj != before) prim = -1;
    }
    if (kExt && s.has_medium && !(ibits(pr.d.w) & kFlagInside)) {
        const float tc = medium_collision(s, pr, r.o, r.d, obj >= 0 ? t : INFINITY, medium_key);
        if (tc >= 0.0f) { obj = kHitMedium; prim = -1; t = tc; }
    }
    return obj >= 0 || obj == kHitMedium ? make_int4(obj, prim, ibits(t), 0) : make_int4(-1, -1, 0, 0);
}

// Shading model of a hit (render.cuh:97-118): -1 = miss.
__device__ __forceinline__ int hit_model(const SceneView& s, int obj)
{
    return obj >= 0 ? s.materials[s.objects[obj].material].model : (obj == kHitMedium ? kModelMedium : -1);
}

// ------------------------------------------------------------------ shade
// G-buffer of an RGB material at one wavelength (EvaluateMaterial, spectral).
__device__ __forceinline__ GB gb_at(const GB& rgb, const MaterialBasis& mb, const float4& lk, float lambda)
{
    GB g = rgb;
    const float a = interact(mb.albedo, lk);
    const float e = interact(mb.emissive, lk);
    g.albedo = mk(a, a, a);
    g.emissive = mk(e, e, e);
    g.ior = ior_abbe(lambda, rgb.ior, rgb.abbe);
    g.sigma_a = sigma_tilt(rgb.sigma_a, lambda, rgb.tilt);
    g.spectral = true;
    return g;
}

// What one loop body leaves behind, unpacked: the state of the path's next
// record or, when it ended, of its result, and the shadow segment and cache
// query it may have issued.  next_record() and the functions after it pack them.
struct ShadeResult {
    bool cont, shadow, nrc_query, cos_ok;
    int depth, non_delta, flags, mdepth, mobj, pixel, sample;
    uint32_t used;
    f3 pos, next, mask, radiance, vloc;
    float4 prev;
    float lambda, lpdf;             // one wavelength
    float mask3, rad3, pend3;       // wavelength 3 of four
    float nrc_spread, nrc_a0;       // cache mode
    f3 pending, light;              // shadow segment: contribution, end point
    uint32_t medium_seed;
    NrcVertex vertex;               // nrc_query
    Rng g;
};

template <int kSpec, bool kNrc>
__device__ __forceinline__ PathRec next_record(const ShadeResult& r)
{
    PathRec out;
    out.o = f4(r.pos, fbits((r.depth + 1) | (r.non_delta << 16)));
    out.d = f4(r.next, fbits(r.flags | (r.mdepth << 8)));
    out.mask = kSpec == 1 ? make_float4(r.mask.x, r.lambda, r.lpdf, fbits(r.pixel)) : f4(r.mask, fbits(r.pixel));
    out.rad = kSpec == 1 ? make_float4(r.radiance.x, 0.0f, 0.0f, fbits(r.sample)) : f4(r.radiance, fbits(r.sample));
    out.rng0 = make_uint4(r.g.st.d, r.g.st.v[0], r.g.st.v[1], r.g.st.v[2]);
    out.rng1 = make_uint4(r.g.st.v[3], r.g.st.v[4], static_cast<uint32_t>(r.mobj), kNrc ? __float_as_uint(r.nrc_spread) : r.used);
    out.prev = r.prev;
    out.vloc = f4(r.vloc, kNrc ? r.nrc_a0 : 0.0f);
    return out;
}
template <int kSpec>
__device__ __forceinline__ RetireRec retire_record(const ShadeResult& r)
{
    RetireRec out;
    out.rad = f4(r.radiance, fbits(r.pixel));
    out.meta = make_int4(r.sample, static_cast<int>(r.used), ibits(r.lambda), ibits(kSpec == 4 ? r.rad3 : r.lpdf));
    return out;
}
__device__ __forceinline__ ShadowRec shadow_record(const ShadeResult& r, int target)
{
    ShadowRec out;
    out.src = f4(r.pos, c_eps_tab[min(r.depth, 8)]);
    out.dst = f4(r.light, fbits(target));
    out.nee = f4(r.pending, fbits(static_cast<int>(r.medium_seed | (r.cos_ok ? 1u : 0u))));
    return out;
}
template <int kSpec>
__device__ __forceinline__ NrcQuery query_record(const ShadeResult& r)   // the path ends; the cache supplies the rest
{
    NrcQuery out;
    out.v = r.vertex;
    out.t = f4(r.mask, kSpec == 4 ? r.mask3 : 0.0f);
    return out;
}

constexpr int kModelAny = -2;   // shade_path: the model is the run-time argument

// One iteration of the CalculateRadiance loop body (render.cuh:541-908) up to
// the shadow query: Trace's material evaluation and hit offset, emission with
// MIS, light sampling for NEE, throughput and Russian roulette.  kModel is the
// shading model of the hit, -1 = miss (kModelAny: rt_model).
template <int kModel, bool kExt, int kSpec, bool kNrc, bool kGuide>
__device__ __forceinline__ void shade_path(const SceneView& s, const FrameParams& fp, const PathRec& pr, float4 aux, int4 hr,
                                           int rt_model, ar_path_record* rec, ShadeResult& R)
{
    const int model = kModel == kModelAny ? rt_model : kModel;
    const int depth = ibits(pr.o.w) & 0xFFFF;
    int nonDelta = ibits(pr.o.w) >> 16;
    int flags = ibits(pr.d.w) & 0xFF;
    const int mdepth = ibits(pr.d.w) >> 8;
    const int pixel = ibits(pr.mask.w);
    const int sidx = ibits(pr.rad.w);
    const int64_t ri = static_cast<int64_t>(sidx) * fp.npix + pixel;
    const f3 crd = xyz(pr.d);
    const f3 cro = xyz(pr.o);
    f3 mask = xyz(pr.mask);
    f3 radiance = xyz(pr.rad);
    // spectral: scalar throughput and radiance broadcast to the three lanes
    // of the RGB arithmetic, the wavelength's basis and D65 weight
    float lambda = 0.0f, lpdf = 0.0f, d65 = 1.0f;
    float4 lk = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (kSpec == 1) {
        lambda = pr.mask.y;
        lpdf = pr.mask.z;
        mask = mk(pr.mask.x, pr.mask.x, pr.mask.x);
        radiance = mk(pr.rad.x, pr.rad.x, pr.rad.x);
        lk = query_lambda(fp.spec.lut_lam, lambda);
        d65 = d65_norm(fp.spec.tables, lambda);
    }
    f3 d65v = mk(d65, d65, d65);
    // four wavelengths (extension): lanes x, y, z of the RGB arithmetic carry
    // wavelengths 0-2, the *3 scalars wavelength 3; directions follow the hero (0)
    float mask3 = 0.0f, rad3 = 0.0f, d65_3 = 0.0f;
    float lam4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    float4 lk4[4];
    if (kSpec == 4) {
        const float4 ax = aux;
        lambda = ax.z;
        mask3 = ax.x;
        rad3 = ax.y;
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            lam4[w] = rotate_lambda(lambda, w);
            lk4[w] = query_lambda(fp.spec.lut_lam, lam4[w]);
        }
        lk = lk4[0];
        d65v = mk(d65_norm(fp.spec.tables, lam4[0]), d65_norm(fp.spec.tables, lam4[1]), d65_norm(fp.spec.tables, lam4[2]));
        d65_3 = d65_norm(fp.spec.tables, lam4[3]);
    }
    const bool inside = (flags & kFlagInside) != 0;
    const f3 vloc = xyz(pr.vloc);
    const f3 maskIn = mask, radIn = radiance;   // path guiding: values at arrival
    const bool med = model == kModelMedium;  // collisions in the participating medium
    const bool hit = model >= 0 && !med;
    const float eps = c_eps_tab[min(nonDelta, 8)];
    Rng g;
    rng_from(g, pr.rng0, pr.rng1);
    if (rec && depth < AR_DEBUG_MAX_HITS) rec[ri].hit_object[depth] = hit || med ? hr.x : -1;
    if (rec) rec[ri].segments = depth + 1;
    // ---- intersection details (re-run of the accepted test)
    f3 pos = mk(0.0f, 0.0f, 0.0f), nrm = mk(0.0f, 0.0f, 0.0f);
    GB gb, gbr;
    MaterialBasis mb;   // spectral: of the hit's material
    int light = -1;
    if (hit) {
        const ObjInfo oi = s.objects[hr.x];
        gb = load_gb(s.materials[oi.material]);
        gbr = gb;
        if (kSpec) {  // EvaluateMaterial / SampleBSDF at the path's wavelength (material.cuh)
            mb = material_basis(fp.spec.basis, oi.material);
            gb = gb_at(gbr, mb, lk, lambda);
        }
        light = oi.light;
        if (oi.type == AR_OBJ_TRIANGLE) {
            const PrimRec& prim = s.prims[hr.y];
            const f3 v0 = mk(prim.v0[0], prim.v0[1], prim.v0[2]);
            const f3 e1 = mk(prim.e1[0], prim.e1[1], prim.e1[2]);
            const f3 e2 = mk(prim.e2[0], prim.e2[1], prim.e2[2]);
            const f3 h = cross(crd, e2);
            const float a = dot(e1, h);
            const float f = __frcp_rn(a);
            const f3 sv = cro - v0;
            const float u = f * dot(sv, h);
            const f3 qv = cross(sv, e1);
            const float v = f * dot(crd, qv);
            const float t = fbits(hr.z);
            pos = cro + crd * t;
            const float w = 1.0f - u - v;
            const TriShade& ts = s.trishade[oi.aux];
            const f3 n0 = mk(ts.n0[0], ts.n0[1], ts.n0[2]);
            const f3 n1 = mk(ts.n1[0], ts.n1[1], ts.n1[2]);
            const f3 n2 = mk(ts.n2[0], ts.n2[1], ts.n2[2]);
            const f3 ni = normalize(n0 * w + n1 * u + n2 * v);
            nrm = dot(crd, ni) > 0.0f ? -ni : ni;
        } else if (oi.type == AR_OBJ_CUBE) {
            isect_cube<true>(s.analytic[oi.aux], cro, crd, &pos, &nrm);
        } else if (kExt && oi.type == AR_OBJ_SDF) {
            sdf_surface_of(s, oi.aux, cro, crd, fbits(hr.z), eps, &pos, &nrm);
        } else {
            isect_sphere<true>(s.analytic[oi.aux], cro, crd, &pos, &nrm);
        }
    }
    if (med) pos = cro + crd * fbits(hr.z);  // no surface: the normal stays zero
    // denoiser guide buffer: the primary hit (RecordScreenGBuffer at depth 0, render.cuh:640-643)
    if (fp.dn.gbuf && depth == 0) {
        if (hit) record_gbuffer(fp.dn.gbuf + pixel, true, gb.albedo, nrm, gb.metallic, gb.roughness, fbits(hr.z), model);
        else record_gbuffer(fp.dn.gbuf + pixel, false, nrm, nrm, 0.0f, 0.0f, 0.0f, 0);
    }
    // ---- learned radiance cache (extension): path spread (Mueller et al. 2021,
    // a = (sum_i sqrt(|x_i-1 - x_i|^2 / (p_i |cos_i|)))^2 against
    // a0 = |x_0 - x_1|^2 / (4 pi |cos_1|)), training vertices, termination
    bool nrcQuery = false;
    float nrcS = 0.0f, nrcA = 0.0f;
    NrcVertex nv;
    if (kNrc) {
        nrcS = __uint_as_float(pr.rng1.w);
        nrcA = pr.vloc.w;
        if (hit && !inside && model != AR_MAT_LIGHT && model != AR_MAT_GLASS) {
            const float tt = fbits(hr.z);
            const float cosT = fmaxf(fabsf(dot(nrm, crd)), 1e-4f);
            if (depth == 0) {
                nrcA = tt / sqrtf(4.0f * kPi * cosT);
                nrcS = 0.0f;
            } else {
                nrcS = nrcS + tt / sqrtf(fmaxf(pr.prev.w, 1e-12f) * cosT);
            }
            nv.p = make_float4(pos.x, pos.y, pos.z, fbits(pixel));
            nv.d = make_float4(-crd.x, -crd.y, -crd.z, model == AR_MAT_GGX ? gb.roughness : 1.0f);
            // four wavelengths: the hero wavelength rides in n.w, the features
            // keep the material's RGB albedo
            nv.n = make_float4(nrm.x, nrm.y, nrm.z, kSpec == 4 ? lambda : 0.0f);
            const f3 alb = kSpec ? gbr.albedo : gb.albedo;
            nv.a = make_float4(alb.x, alb.y, alb.z, 0.0f);
            int slot;
            if (sidx == 0 && nrc_train_slot(fp.nrc, pixel, &slot)) {   // sample 0 of a training pixel
                const int kv = fp.nrc.slot_count[slot];
                if (kv < fp.nrc.max_train_vertices) {
                    NrcTrainVertex tv;
                    tv.v = nv;
                    tv.t = f4(mask, kSpec == 4 ? mask3 : 0.0f);
                    tv.lb = f4(radiance, kSpec == 4 ? rad3 : 0.0f);
                    fp.nrc.train_vertices[static_cast<int64_t>(slot) * fp.nrc.max_train_vertices + kv] = tv;
                    fp.nrc.slot_count[slot] = kv + 1;
                }
            } else if (depth >= 1 && nrcS > sqrtf(fp.nrc.spread_c) * nrcA) {
                nrcQuery = true;
            }
        }
    }
    // ---- SampleContext (material.cuh:19-37, 177-330, 389-425)
    f3 next = mk(0.0f, 0.0f, 0.0f), emis = mk(0.0f, 0.0f, 0.0f), brdf = mk(0.0f, 0.0f, 0.0f);
    float pdf = 1.0f;
    bool terminate = false, delta = false, missThin = false;
    bool nInside = false;
    f3 nvloc = mk(0.0f, 0.0f, 0.0f);
    int nmobj = -1, nmdepth = 0;
    f3 malb = mk(0.0f, 0.0f, 0.0f);  // medium: single-scatter albedo
    float emis3 = 0.0f, brdf3 = 0.0f, malb3 = 0.0f;  // wavelength 3 (four-wavelength mode)
    bool dispersed = false;
    if (!hit && !med && inside) {
        missThin = true;
        nvloc = cro;
    }
    if (hit) {
        const f3 N = nrm;
        if (model == AR_MAT_DIFFUSE) {
            const float e0 = g.next(), e1 = g.next(), e2 = g.next();
            next = sample_cosine(e0, e1, e2, N, pdf);
            emis = gb.emissive;
            nInside = inside; nvloc = pos;
        } else if (model == AR_MAT_LIGHT) {
            pdf = 1.0f; emis = gb.emissive; terminate = true;
        } else if (model == AR_MAT_GLASS) {
            delta = true;
            const float eta = inside ? gb.ior : 1.0f / gb.ior;
            const f3 nIn = (dot(N, crd) > 0.0f) ? -N : N;
            const float cosI = -dot(nIn, crd);
            const float sin2I = fmaxf(0.0f, 1.0f - cosI * cosI);
            const float kk = 1.0f - sin2I * (eta * eta);
            if (kk <= 0.0f) {
                if (mdepth < 1024) { next = reflect(crd, nIn); nInside = inside; }
                else { next = crd; nInside = !inside; }
                pdf = 1.0f; nvloc = pos;
            } else {
                const float cosT = sqrtf(kk);
                const float Fr = fresnel_exact(cosI, cosT, eta);
                if (g.next() < Fr) { next = reflect(crd, nIn); pdf = Fr; nInside = inside; }
                else { next = refract(crd, nIn, eta); pdf = 1.0f - Fr; nInside = !inside; }
                nvloc = pos;
            }
        } else if (model == AR_MAT_GGX) {
            emis = gb.emissive;
            const f3 V = -crd;
            const float NoV = fmaxf(0.0f, dot(N, V));
            if (NoV <= 0.0f) {
                terminate = true;
            } else {
                float alpha, kD;
                f3 F0;
                ggx_params(gb, alpha, kD, F0);
                const float pSpec = ggx_pspec(gb, F0);
                const float uu = g.next();
                const float e0 = g.next(), e1 = g.next(), e2 = g.next();
                if (uu < pSpec) {
                    float ps;
                    const f3 L = sample_ggx_vndf(V, N, alpha, e0, e1, e2, ps);
                    const float NoL = fmaxf(0.0f, dot(N, L));
                    if (NoL <= 0.0f) {
                        terminate = true;
                    } else {
                        next = L; pdf = pSpec * ps + (1.0f - pSpec) * (NoL / kPi);
                        nInside = inside; nvloc = pos;
                    }
                } else {
                    float pd;
                    const f3 L = sample_cosine(e0, e1, e2, N, pd);
                    const float pspec = ggx_vndf_pdf(V, N, L, alpha);
                    next = L; pdf = pSpec * pspec + (1.0f - pSpec) * pd;
                    nInside = inside; nvloc = pos;
                }
            }
        }
        nmobj = hr.x;
        nmdepth = mdepth + 1;
        brdf = eval_bsdf_cos(model, crd, next, N, pos, gb, inside, vloc);
        if (kSpec == 4) {
            if (model != AR_MAT_GLASS) {
                emis = mk(interact(mb.emissive, lk4[0]), interact(mb.emissive, lk4[1]), interact(mb.emissive, lk4[2]));
                emis3 = interact(mb.emissive, lk4[3]);
            }
            if (model == AR_MAT_GLASS && gbr.abbe > 0.0f && !(flags & kFlagHeroOnly)) {
                // dispersive glass: the other wavelengths cannot follow the hero's
                // direction; the path continues with the hero alone (its weight
                // becomes that of a single-wavelength sample)
                dispersed = true;
            } else if (model != AR_MAT_LIGHT && !(flags & kFlagHeroOnly)) {
                const float b1 = eval_bsdf_cos(model, crd, next, N, pos, gb_at(gbr, mb, lk4[1], lam4[1]), inside, vloc).x;
                const float b2 = eval_bsdf_cos(model, crd, next, N, pos, gb_at(gbr, mb, lk4[2], lam4[2]), inside, vloc).x;
                brdf3 = eval_bsdf_cos(model, crd, next, N, pos, gb_at(gbr, mb, lk4[3], lam4[3]), inside, vloc).x;
                brdf = mk(brdf.x, b1, b2);
            }
        }
    } else if (med) {
        // Henyey-Greenstein scattering; phase / pdf = 1, throughput weight = albedo
        const float u1 = g.next(), u2 = g.next();
        next = hg_sample(crd, s.medium.g, u1, u2);
        pdf = hg_phase(s.medium.g, dot(crd, next));
        malb = mk(s.medium.albedo[0], s.medium.albedo[1], s.medium.albedo[2]);
        if (kSpec == 4) {
            const RgbBasis ab = material_basis(fp.spec.basis, fp.spec.materials).albedo;
            malb = mk(interact(ab, lk4[0]), interact(ab, lk4[1]), interact(ab, lk4[2]));
            malb3 = interact(ab, lk4[3]);
            brdf3 = malb3 * pdf;
        } else if (kSpec) {
            const float a = interact(material_basis(fp.spec.basis, fp.spec.materials).albedo, lk);
            malb = mk(a, a, a);
        }
        brdf = malb * pdf;
        nInside = false;
        nvloc = pos;
        nmobj = static_cast<int>(pr.rng1.z);
        nmdepth = mdepth;
    } else {
        brdf = mk(1.0f, 1.0f, 1.0f);
        next = crd;
        pdf = 1.0f;
        emis = sky_lighting(crd, fp.sky);
        if (kSpec == 4) {
            const RgbBasis eb = rgb_basis(fp.spec.lut_rgb, fp.spec.res, emis);
            emis = mk(interact(eb, lk4[0]), interact(eb, lk4[1]), interact(eb, lk4[2]));
            emis3 = interact(eb, lk4[3]);
            brdf3 = 1.0f;
        } else if (kSpec) {
            const float e = interact(rgb_basis(fp.spec.lut_rgb, fp.spec.res, emis), lk);
            emis = mk(e, e, e);
        }
        nInside = false;
    }
    // ---- path guiding (render.cuh:555-640): mix the probe's hemisphere
    // density into the BSDF's, or sample the probe with probability alpha
    int gProbe = -1;
    bool guidable = false;
    f3 gq = mk(0.0f, 0.0f, 0.0f);
    uint64_t gKey = 0;
    if (kGuide && hit && (model == AR_MAT_DIFFUSE || model == AR_MAT_GGX) && !inside && !terminate) {
        guidable = true;
        gKey = pg_key(pos, reflect(crd, nrm), fp.guide.faces);
        gProbe = pg_lookup(fp.guide, gKey);
        if (gProbe >= 0) {
            const f3 mq = vmaxs(mask, 1.0e-6f);
            gq = mq / (mq.x + mq.y + mq.z + 1.0e-6f);
            const float4* P = fp.guide.probes + static_cast<int64_t>(gProbe) * kPgStride;
            const float pP = pg_hemi_pdf(P, next, nrm, gq);
            const float a = fp.guide.alpha;
            if (pdf > 1.0e-12f && pP > 1.0e-12f) {
                if (g.next() < a) {
                    float u[5];
#pragma unroll
                    for (int t = 0; t < 5; ++t) u[t] = g.next();
                    float pg;
                    const f3 w = pg_sample_hemi(P, nrm, gq, u, &pg);
                    if (dot(w, nrm) > 1.0e-12f) {
                        const float pBs = bsdf_pdf(model, gb, nrm, crd, w);
                        next = w;
                        brdf = eval_bsdf_cos(model, crd, w, nrm, pos, gb, inside, vloc);
                        pdf = (1.0f - a) * fmaxf(pBs, 1.0e-12f) + a * pg;
                    } else {
                        gProbe = -1;
                    }
                } else {
                    pdf = (1.0f - a) * pdf + a * pP;
                }
            } else {
                gProbe = -1;
            }
        }
    }
    if (!med) {   // hit offset, always one uniform (render.cuh:156-160)
        const float offEps = eps * fmaxf(1.0f, length(pos));
        const float sg = signf(dot(nrm, next));
        const float r = g.next();
        pos = pos + ((nrm * sg) * offEps) * (r + 0.5f);
    }
    const bool mInside = nInside;  // media state after this segment
    // ---- emission (render.cuh:648-723)
    if (!hit && !med) {
        if (!missThin) {
            radiance = radiance + (mask * emis) * d65v;
            if (kSpec == 4) rad3 = rad3 + (mask3 * emis3) * d65_3;
        }
    } else if (hit && light >= 0 && !nrcQuery) {
        float misW = 1.0f;
        if (fp.use_nee && depth > 0 && (flags & kFlagPrevNEE)) {
            const float pB = fmaxf(pr.prev.w, 0.0f);
            const float pL = pdf_light_from_hit(s, hr.x, xyz(pr.prev), pos, nrm, fp.tri_light_nee != 0);
            if (pL >= 0.0f && pB > 0.0f) misW = power_heuristic(pB, pL);
        }
        radiance = radiance + ((mask * emis) * d65v) * misW;
        if (kSpec == 4) rad3 = rad3 + ((mask3 * emis3) * d65_3) * misW;
    }
    const bool brk = (!hit && !med && !missThin) || terminate || nrcQuery;
    bool cont = false, shadow = false, cosOK = false;
    f3 pending = mk(0.0f, 0.0f, 0.0f), lightP = mk(0.0f, 0.0f, 0.0f);
    float pend3 = 0.0f;
    float4 prevOut = pr.prev;
    if (!brk) {
        // ---- NEE (render.cuh:766-827)
        if (!missThin) {
            const float lum = kSpec == 4 ? 0.25f * (mask.x + mask.y + mask.z + mask3)
                                         : (kSpec ? mask.x : luminance(mask));
            const float rate = sqrtf(saturate(lum));
            if (fp.use_nee && nonDelta < 10 && !delta && !mInside && g.next() < rate) {
                LightSample ls = sample_light(s, pos, g, fp.tri_light_nee != 0);
                RgbBasis lb;   // spectral: of the light's emission
                if (kSpec && ls.valid) {
                    lb = material_basis(fp.spec.basis, ls.material).emissive;
                    const float e = interact(lb, lk);
                    ls.emis = mk(e, e, e);
                }
                if (ls.valid) {
                    const float pATotal = fmaxf(1e-20f, ls.pA * ls.pFacet);
                    const f3 lu = ls.p - pos;
                    const float d2 = fmaxf(dot(lu, lu), 1.0e-12f);
                    const f3 ld = lu * rsqrt_ieee(d2);
                    const float cosX = med ? 1.0f : fmaxf(0.0f, dot(nrm, ld));
                    const float cosY = fmaxf(0.0f, dot(ls.n, -ld));
                    if (cosX > 0.0f && cosY > 0.0f) {
                        cosOK = true;
                        const f3 fcos = med ? malb * hg_phase(s.medium.g, dot(crd, ld))
                                             : eval_bsdf_cos(model, crd, ld, nrm, pos, gb, false, mk(0.0f, 0.0f, 0.0f));
                        const float G = cosY / d2;
                        const f3 contrib = (fcos * ls.emis) * (G / pATotal);
                        const float pL = area_to_solid_angle(pos, ls.p, ls.n, ls.pFacet * ls.pA);
                        float pB = med ? hg_phase(s.medium.g, dot(crd, ld))
                                        : fmaxf(bsdf_pdf(model, gb, nrm, crd, ld), 0.0f);
                        if (kGuide && gProbe >= 0) {
                            const float a = fp.guide.alpha;
                            pB = (1.0f - a) * pB +
                                 a * pg_hemi_pdf(fp.guide.probes + static_cast<int64_t>(gProbe) * kPgStride, ld, nrm, gq);
                        }
                        const float wmis = power_heuristic(pL, pB);
                        pending = (mask * (contrib * wmis)) * d65v;
                        if (kSpec == 4) {
                            const float G4 = G / pATotal;
                            float f1, f2, f3v;
                            if (med) {
                                const float ph = hg_phase(s.medium.g, dot(crd, ld));
                                f1 = malb.y * ph; f2 = malb.z * ph; f3v = malb3 * ph;
                            } else {
                                const f3 z0 = mk(0.0f, 0.0f, 0.0f);
                                f1 = eval_bsdf_cos(model, crd, ld, nrm, pos, gb_at(gbr, mb, lk4[1], lam4[1]), false, z0).x;
                                f2 = eval_bsdf_cos(model, crd, ld, nrm, pos, gb_at(gbr, mb, lk4[2], lam4[2]), false, z0).x;
                                f3v = eval_bsdf_cos(model, crd, ld, nrm, pos, gb_at(gbr, mb, lk4[3], lam4[3]), false, z0).x;
                            }
                            const f3 c3 = mk(contrib.x,
                                             (f1 * interact(lb, lk4[1])) * G4,
                                             (f2 * interact(lb, lk4[2])) * G4);
                            pending = (mask * (c3 * wmis)) * d65v;
                            pend3 = (mask3 * (((f3v * interact(lb, lk4[3])) * G4) * wmis)) * d65_3;
                        }
                    }
                    shadow = true;
                    lightP = ls.p;
                    if (rec) {
                        rec[ri].nee_rays += 1;
                        if (depth < 32) rec[ri].nee_depth_mask |= static_cast<int32_t>(1u << depth);
                    }
                }
            }
            // previousDidNEE_ is decided by the shadow query when one is cast
            flags &= ~kFlagPrevNEE;
            prevOut = f4(pos, (kNrc && delta) ? INFINITY : pdf);
        }
        // ---- throughput and Russian roulette (render.cuh:829-907)
        const f3 contrib = mk(brdf.x / fmaxf(pdf, 1e-12f), brdf.y / fmaxf(pdf, 1e-12f), brdf.z / fmaxf(pdf, 1e-12f));
        float qrr = 1.0f;
        bool survived = true;
        if (nonDelta >= fp.rr_depth) {
            const float lum = kSpec == 4 ? 0.25f * (mask.x + mask.y + mask.z + mask3)
                                         : (kSpec ? mask.x : luminance(mask));
            const float mx = kSpec == 4 ? fmaxf(max3(mask), mask3) : (kSpec ? mask.x : max3(mask));
            const float basic = clampf(lum * 0.5f + mx * 0.5f, 0.05f, 0.95f);
            qrr = lerpf(basic, 1.0f, mInside ? 0.99f : 0.0f);
            if (g.next() > qrr) survived = false;
        }
        if (survived) {
            mask = mask * contrib;
            mask = mask / qrr;
            if (kSpec == 4) {
                mask3 = (mask3 * (brdf3 / fmaxf(pdf, 1e-12f))) / qrr;
                if (dispersed) {   // hero alone from here: weight sum_j p(lambda_j) / p(lambda_0)
                    const float ps = pdf_cie1931(lam4[0]) + pdf_cie1931(lam4[1]) + pdf_cie1931(lam4[2]) + pdf_cie1931(lam4[3]);
                    mask = mk(mask.x * (ps / pdf_cie1931(lam4[0])), 0.0f, 0.0f);
                    mask3 = 0.0f;
                    flags |= kFlagHeroOnly;
                }
            }
            if (!delta) nonDelta++;
            cont = depth + 1 < fp.max_depth;
        }
    }
    flags = (flags & ~kFlagInside) | (mInside ? kFlagInside : 0);
    if (kGuide) {   // this event of the pixel's path, for the probes' samples at retirement
        const int ne = fp.guide.event_count[pixel];
        if (ne < kPgEvents) {
            float4* ev = fp.guide.events + (static_cast<int64_t>(pixel) * kPgEvents + ne) * 3;
            ev[0] = make_float4(__uint_as_float(static_cast<uint32_t>(gKey)), __uint_as_float(static_cast<uint32_t>(gKey >> 32)),
                                (guidable && cont) ? 1.0f : 0.0f, 0.0f);
            ev[1] = f4(next, 0.0f);
            ev[2] = f4(maskIn, 0.0f);
            fp.guide.event_lb[static_cast<int64_t>(pixel) * kPgEvents + ne] = f4(radIn, 0.0f);
            fp.guide.event_count[pixel] = ne + 1;
        }
    }
    const uint32_t used = pr.rng1.w + static_cast<uint32_t>(g.used);
    R.cont = cont; R.shadow = shadow; R.nrc_query = nrcQuery; R.cos_ok = cosOK;
    R.depth = depth; R.non_delta = nonDelta; R.flags = flags; R.mdepth = nmdepth; R.mobj = nmobj;
    R.pixel = pixel; R.sample = sidx; R.used = used;
    R.pos = pos; R.next = next; R.mask = mask; R.radiance = radiance; R.vloc = nvloc; R.prev = prevOut;
    R.lambda = lambda; R.lpdf = lpdf; R.mask3 = mask3; R.rad3 = rad3; R.pend3 = pend3;
    R.nrc_spread = nrcS; R.nrc_a0 = nrcA;
    R.pending = pending; R.light = lightP;
    R.medium_seed = kExt && s.has_medium
        ? medium_seed(fp.medium_key, static_cast<uint32_t>(sidx), static_cast<uint32_t>(pixel), static_cast<uint32_t>(depth), 1u) & ~1u
        : 0u;
    R.vertex = nv;
    R.g = g;
}

// ------------------------------------------------------------------ shadow
// Transmittance of the medium along an unoccluded shadow segment (out of line).
static __device__ __noinline__ float shadow_transmittance(const SceneView& s, f3 o, f3 d, float tmax, uint32_t seed)
{
    HashRng h;
    h.seed = seed;
    h.n = 0;
    return ratio_track(s.medium, o, d, tmax, h);
}

// SegmentTrace (render.cuh:167-183): the any-hit query of a shadow segment;
// false when it is too short to be blocked.
__device__ __forceinline__ bool shadow_begin(float4 a, f3 dst, RayState& r)
{
    const f3 src = xyz(a);
    f3 dir = dst - src;
    const float dist = length(dir);
    if (!(dist > 0.0f)) return false;
    dir = dir / dist;
    const float eps = a.w * fmaxf(1.0f, fmaxf(length(src), length(dst)));
    const float tMax = fmaxf(0.0f, dist - eps);
    if (!(tMax > 0.0f)) return false;
    ray_begin(r, src, dir, 0.0f, tMax);
    return true;
}

// Whether the segment is blocked, and the medium's transmittance when not.
template <bool kExt>
__device__ __forceinline__ bool shadow_end(const SceneView& s, const RayState& r, float eps, uint32_t medium_seed_bits, float& tr)
{
    bool occ = r.best.obj >= 0;
    tr = 1.0f;
    if (kExt && !occ && s.num_sdf > 0) occ = sdf_any(s, r.o, r.d, 0.0f, r.best.t, eps) >= 0;
    if (kExt && !occ && s.has_medium) tr = shadow_transmittance(s, r.o, r.d, r.best.t, medium_seed_bits & ~1u);
    return occ;
}

// ------------------------------------------------------------------ retire
// checkNanInf + clamp (render.cuh:969), max(0, .) (scene.cu:238), FP64 sum.
__device__ __forceinline__ float fix_nan_inf(float x)
{
    if (isnan_(x)) return 0.0f;
    if (isinf_(x)) return x > 0.0f ? 0.0f : -0.0f;
    return x;
}

// A finished path: its clamped sample into the FP64 sums, the denoiser's
// moments, the cache's training targets, the probes' samples, the debug record.
__device__ __forceinline__ void retire_path(const FrameParams& fp, const RetireRec& rr, double* accum, ar_path_record* rec)
{
    f3 v = xyz(rr.rad);
    if (fp.spectral == 4) {
        // four wavelengths: sum_i XYZ(lambda_i) L_i / sum_j p(lambda_j), the
        // one-sample estimator of the rotation set (balance heuristic over
        // which member was the hero)
        const float h = fbits(rr.meta.z);
        const float L[4] = {fix_nan_inf(rr.rad.x), fix_nan_inf(rr.rad.y), fix_nan_inf(rr.rad.z), fix_nan_inf(fbits(rr.meta.w))};
        float ps = 0.0f;
        f3 acc = mk(0.0f, 0.0f, 0.0f);
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            const float lw = rotate_lambda(h, w);
            ps += pdf_cie1931(lw);
            acc = acc + cmf_xyz(fp.spec.tables, lw) * L[w];
        }
        v = acc / ps;
    } else if (fp.spectral) {  // lambdaXYZ * radiance / pdf (render.cuh:966), linear CIE XYZ
        const float lam = fbits(rr.meta.z), lpdf = fbits(rr.meta.w);
        const float r = fix_nan_inf(rr.rad.x);
        const f3 c = cmf_xyz(fp.spec.tables, lam);
        v = mk((c.x * r) / lpdf, (c.y * r) / lpdf, (c.z * r) / lpdf);
    } else {
        v = mk(fix_nan_inf(v.x), fix_nan_inf(v.y), fix_nan_inf(v.z));
    }
    const float x = fmaxf(clampf(v.x, 0.0f, 1.0e3f), 0.0f);
    const float y = fmaxf(clampf(v.y, 0.0f, 1.0e3f), 0.0f);
    const float z = fmaxf(clampf(v.z, 0.0f, 1.0e3f), 0.0f);
    const int pixel = ibits(rr.rad.w);
    // denoiser moments of the clamped sample (RecordScreenStatisticBuffer, render.cuh:988-991)
    if (fp.dn.stat) record_stats(fp.dn.stat + pixel, mk(x, y, z));
    int slot;
    if (fp.nrc.enabled && rr.meta.x == 0 && nrc_train_slot(fp.nrc, pixel, &slot)) {
        // training targets: radiance gathered after each recorded vertex,
        // divided by the throughput that reached it
        const int nvtx = fp.nrc.slot_count[slot];
        const f3 L = mk(fix_nan_inf(rr.rad.x), fix_nan_inf(rr.rad.y), fix_nan_inf(rr.rad.z));
        if (fp.nrc.spectral == 4) {
            // four wavelengths: a target per wavelength, negative (left out of the
            // loss) where no throughput reached the vertex (hero-only after dispersion),
            const float L3 = fix_nan_inf(fbits(rr.meta.w));
            for (int k = 0; k < nvtx; ++k) {
                const NrcTrainVertex tv = fp.nrc.train_vertices[static_cast<int64_t>(slot) * fp.nrc.max_train_vertices + k];
                if (!nrc_vertex_finite(tv.v)) continue;   // a non-finite input would poison the whole step
                const float Lw[4] = {L.x, L.y, L.z, L3};
                const float T[4] = {tv.t.x, tv.t.y, tv.t.z, tv.t.w};
                const float B4[4] = {tv.lb.x, tv.lb.y, tv.lb.z, tv.lb.w};
                // relative to the D65 weight of the wavelength (the cache's output scale)
                float tg[4];
#pragma unroll
                for (int w = 0; w < 4; ++w)
                    tg[w] = T[w] > 1e-6f ? fminf(fmaxf(((Lw[w] - B4[w]) / T[w]) /
                                                           d65_norm(fp.spec.tables, rotate_lambda(tv.v.n.w, w)),
                                                       0.0f),
                                                 1.0e3f)
                                         : -1.0f;
                const int si = atomicAdd(fp.nrc.sample_count, 1);
                if (si < fp.nrc.sample_cap) {
                    NrcSample sm;
                    sm.v = tv.v;
                    sm.v.p.w = tg[0];
                    sm.v.n.w = tg[1];
                    sm.v.a.w = tg[2];
                    sm.x = make_float4(tg[3], tv.v.n.w, 0.0f, 0.0f);
                    fp.nrc.samples[si] = sm;
                }
            }
        }
        for (int k = 0; k < (fp.nrc.spectral == 4 ? 0 : nvtx); ++k) {
            const NrcTrainVertex tv = fp.nrc.train_vertices[static_cast<int64_t>(slot) * fp.nrc.max_train_vertices + k];
            if (!nrc_vertex_finite(tv.v)) continue;
            const f3 tgt = mk(tv.t.x > 1e-6f ? (L.x - tv.lb.x) / tv.t.x : 0.0f,
                              tv.t.y > 1e-6f ? (L.y - tv.lb.y) / tv.t.y : 0.0f,
                              tv.t.z > 1e-6f ? (L.z - tv.lb.z) / tv.t.z : 0.0f);
            const int si = atomicAdd(fp.nrc.sample_count, 1);
            if (si < fp.nrc.sample_cap) {
                NrcSample sm;
                sm.v = tv.v;
                sm.v.p.w = fminf(fmaxf(tgt.x, 0.0f), 1.0e3f);
                sm.v.n.w = fminf(fmaxf(tgt.y, 0.0f), 1.0e3f);
                sm.v.a.w = fminf(fmaxf(tgt.z, 0.0f), 1.0e3f);
                sm.x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                fp.nrc.samples[si] = sm;
            }
        }
    }
    if (fp.guiding) {
        // incident radiance along each guidable vertex's sampled direction:
        // radiance gathered from the next event on over the throughput that reached it
        const int ne = fp.guide.event_count[pixel];
        const f3 L = mk(fix_nan_inf(rr.rad.x), fix_nan_inf(rr.rad.y), fix_nan_inf(rr.rad.z));
        for (int e = 0; e + 1 < ne; ++e) {
            const float4* ev = fp.guide.events + (static_cast<int64_t>(pixel) * kPgEvents + e) * 3;
            const float4 h = ev[0];
            if (h.z == 0.0f) continue;
            const float4 tn = fp.guide.events[(static_cast<int64_t>(pixel) * kPgEvents + e + 1) * 3 + 2];
            const float4 lb = fp.guide.event_lb[static_cast<int64_t>(pixel) * kPgEvents + e + 1];
            const f3 inc = mk(tn.x > 1e-8f ? fmaxf((L.x - lb.x) / tn.x, 0.0f) : 0.0f,
                              tn.y > 1e-8f ? fmaxf((L.y - lb.y) / tn.y, 0.0f) : 0.0f,
                              tn.z > 1e-8f ? fmaxf((L.z - lb.z) / tn.z, 0.0f) : 0.0f);
            const float strength = fminf(luminance(inc), kPgMaxBrightness);
            if (!(strength >= kPgMinBrightness)) continue;
            const int si = atomicAdd(&fp.guide.counters[2], 1);
            if (si < fp.guide.sample_cap) {
                float4* o = fp.guide.samples + 3 * static_cast<int64_t>(si);
                o[0] = make_float4(h.x, h.y, 0.0f, 0.0f);
                o[1] = ev[1];
                o[2] = f4(inc, 0.0f);
            }
        }
        fp.guide.event_count[pixel] = 0;
    }
    double* a = accum + 3 * static_cast<int64_t>(pixel);
    atomicAdd(a + 0, static_cast<double>(x));
    atomicAdd(a + 1, static_cast<double>(y));
    atomicAdd(a + 2, static_cast<double>(z));
    if (rec) {
        const int64_t ri = static_cast<int64_t>(rr.meta.x) * fp.npix + pixel;
        rec[ri].radiance[0] = x; rec[ri].radiance[1] = y; rec[ri].radiance[2] = z;
        rec[ri].uniforms = rr.meta.y;
    }
}

}  // namespace ar
