"""Timed cases of the path-tracing framework, through its public Python binding.

Each case is one call a user's program makes on data it already holds: an
offline or preview render, a batch of renders, ray queries, the denoiser's
filter, the radiance cache (a frame and a training gradient), the spectral
lookup table.  Sizes are those of the framework's own benchmark
configurations, tests and examples, or plain image and batch sizes of the same
ranges; scenes come from its seeded generators.  The spectral mode's data files
are not part of the repository, so its cases use tables of the same layout:
published Gaussian fits of the colour matching functions, a smooth daylight
curve and random-init network weights with a plausible response.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "aperturerendererv3-optix-geometry_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import aperture_b200 as ab  # noqa: E402
import scenes  # noqa: E402

TRIS_PER_SPHERE = 1280


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest render: a viewport preview while a user moves the camera (one sample per pixel)
        dict(name="preview_box_160x120", kind="render", scene="box", width=160, height=120, spp=1, depth=8, nee=1,
             spectral=0, host=0),
        # benchmark configuration 1: the box at 256x256, 16 samples, image returned in host memory
        dict(name="box_256_16spp_host", kind="render", scene="box", width=256, height=256, spp=16, depth=8, nee=1,
             spectral=0, host=1),
        # benchmark configuration 2, the headline: 1,024,002 triangles at 1080p, 64 samples, depth 12
        dict(name="spheres_1m_1080p_64spp", kind="render", scene="spheres", spheres=800, width=1920, height=1080,
             spp=64, depth=12, nee=1, spectral=0, host=0),
        # benchmark configuration 3 (SDF tori, scattering medium, four wavelengths) at 720p with a draft sample count
        dict(name="sdf_medium_4wl_720p_16spp", kind="render", scene="medium", width=1280, height=720, spp=16,
             depth=16, nee=1, spectral=4, host=0),
        # benchmark configuration 5 in small: a queue of uneven thumbnails and stills rendered as one batch
        dict(name="batch_12_jobs", kind="batch", jobs=12, spheres=60, size=224, spp=16, depth=8),
        # ray queries as a physics or visibility program issues them: incoherent closest hits on the 1M-triangle scene
        dict(name="closest_1m_rays_1m_tris", kind="trace", spheres=800, rays=1 << 20, any=0, static=0),
        # occlusion tests between points and lights, an odd count
        dict(name="occlusion_300k_rays", kind="trace", spheres=120, rays=300007, any=1, static=0),
        # a handful of picking / probe rays from a real-time thread (the call that does not allocate)
        dict(name="closest_777_rays_static", kind="trace", spheres=20, rays=777, any=0, static=1),
        # the denoiser's bilateral filter on an interactive 1080p frame after 8 recorded frames
        dict(name="denoise_1080p", kind="denoise", spheres=60, width=1920, height=1080, frames=8),
        # a radiance-cache frame of a fly-through (configuration 4 at half resolution): trace, query, infer, resolve
        dict(name="cache_frame_960x540", kind="cache_frame", spheres=200, width=960, height=540, spp=1, depth=12,
             log2=19),
        # one training batch of the radiance cache: forward, loss, backward, all gradients returned
        dict(name="cache_gradients_16384", kind="cache_grad", samples=16384, log2=14),
        # the spectral mode's RGB table at a preview resolution, built on the tensor cores at scene load
        dict(name="rgb_table_160", kind="table", res=160),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["render", "render", "render", "render", "batch", "trace", "trace", "trace", "denoise",
                       "cache_frame", "cache_grad", "table"])
    if kind == "render":
        scene = rng.choice(["box", "spheres", "medium"])
        w = _log_int(rng, 97, 1920)
        h = max(64, min(1080, int(w * rng.uniform(0.5, 1.1))))
        most = 1.2e8 if scene == "spheres" else 1.5e7 if scene == "medium" else 4e7
        spp = max(1, min(_log_int(rng, 1, 64), int(most / (w * h))))
        c = dict(kind=kind, scene=scene, width=w, height=h, spp=spp, depth=rng.choice([4, 8, 12, 16]),
                 nee=rng.choice([1, 1, 1, 0]), spectral=0, host=rng.choice([0, 0, 1]))
        if scene == "spheres":
            c["spheres"] = _log_int(rng, 20, 800)
        if scene == "medium":
            c["spectral"] = rng.choice([0, 1, 4])
        return c
    if kind == "batch":
        return dict(kind=kind, jobs=rng.randint(3, 24), spheres=_log_int(rng, 10, 200), size=rng.randint(96, 400),
                    spp=_log_int(rng, 1, 32), depth=rng.choice([6, 8, 12]))
    if kind == "trace":
        static = rng.choice([0, 0, 1])
        return dict(kind=kind, spheres=_log_int(rng, 10, 800), rays=_log_int(rng, 100, 1 << 21), any=rng.choice([0, 1]),
                    static=static)
    if kind == "denoise":
        w = _log_int(rng, 127, 1920)
        return dict(kind=kind, spheres=_log_int(rng, 10, 120), width=w, height=max(65, int(w * rng.uniform(0.5, 0.6))),
                    frames=rng.randint(2, 16))
    if kind == "cache_frame":
        w = _log_int(rng, 200, 1920)
        return dict(kind=kind, spheres=_log_int(rng, 20, 400), width=w, height=max(100, int(w * rng.uniform(0.5, 0.6))),
                    spp=rng.choice([1, 1, 2, 4]), depth=rng.choice([8, 12]), log2=rng.choice([16, 19]))
    if kind == "cache_grad":
        return dict(kind=kind, samples=_log_int(rng, 500, 16384), log2=rng.randint(12, 16))
    return dict(kind=kind, res=rng.randint(33, 256))


# ------------------------------------------------------------------ inputs
def _box_size(n_spheres):
    return 100.0 * (n_spheres / 800.0) ** (1.0 / 3.0)   # the benchmark scene's sphere density


def _sphere_objects(case, seed):
    return scenes.spheres_scene(seed=scenes.SEED_BASE + 1000 + seed, n_spheres=case["spheres"],
                                n_lights=max(4, min(16, case["spheres"] // 8)), box=_box_size(case["spheres"]))


def _sphere_camera(case, width, height):
    k = _box_size(case["spheres"]) / 100.0
    d = np.array([0.0, -40.0, 150.0])
    return ab.make_camera((0.0, 30.0 * k, -150.0 * k), d / np.linalg.norm(d), 60.0, width, height)


def _tables(seed):
    """A spectral table block in the layout ar_scene_set_spectral takes: colour
    matching functions (Wyman, Sloan and Shirley 2013), a daylight-like curve,
    random-init networks whose response is close to the colour's brightness."""
    rng = np.random.default_rng(seed)
    lam = np.arange(360.0, 781.0)

    def g(mu, s1, s2):
        return np.exp(-0.5 * ((lam - mu) / np.where(lam < mu, s1, s2)) ** 2)

    x = 1.056 * g(599.8, 37.9, 31.0) + 0.362 * g(442.0, 16.0, 26.7) - 0.065 * g(501.1, 20.4, 26.2)
    y = 0.821 * g(568.8, 46.9, 40.5) + 0.286 * g(530.9, 16.3, 31.1)
    z = 1.217 * g(437.0, 11.8, 36.0) + 0.681 * g(459.0, 26.0, 13.8)
    d65 = 100.0 * (560.0 / lam) ** 5 * np.expm1(1.4388e7 / (560.0 * 6504.0)) / np.expm1(1.4388e7 / (lam * 6504.0))

    def blocks():
        return [rng.normal(0.0, 0.03, 7 * 1024), rng.uniform(0.05, 0.15, 7 * 32)]

    parts = [np.stack([x, y, z], 1).ravel(), d65, rng.normal(0.0, 0.05, 1024), rng.uniform(0.9, 1.1, 32)]
    parts += blocks() + [rng.uniform(0.8, 1.2, 128) * (0.5 / (32.0 * 1.7))]
    parts += blocks() + [rng.uniform(0.8, 1.2, 128) * (0.42 / (32.0 * 0.9))]
    return np.concatenate(parts).astype(np.float32)


def _pixels(width, height):
    return torch.empty((height, width, 3), dtype=torch.float32, device="cuda")


def _rays(case, objects, seed):
    """Bounce-like queries: origins spread through the scene's box, directions
    uniform; occlusion queries run from such a point to a point on a light."""
    g = torch.Generator(device="cuda").manual_seed(977 + seed)
    n, box = case["rays"], _box_size(case["spheres"])
    o = (torch.rand((n, 3), generator=g, device="cuda") * 2.0 - 1.0) * box
    d = torch.nn.functional.normalize(torch.randn((n, 3), generator=g, device="cuda"), dim=1)
    tmax = torch.full((n, 1), 4.0 * box, device="cuda")
    if case["any"]:
        L = objects[objects["type"] == ab.OBJ_SPHERE]
        c = torch.from_numpy(np.stack([L["center"][k] for k in "xyz"], 1)).cuda()
        r = torch.from_numpy(np.ascontiguousarray(L["extent"]["x"])).cuda()
        i = torch.randint(0, len(L), (n,), generator=g, device="cuda")
        to = c[i] + d * r[i, None] * 1.01 - o
        tmax = to.norm(dim=1, keepdim=True)
        d = to / tmax
    return torch.cat([o, torch.full((n, 1), 1.0e-3, device="cuda"), d, tmax], 1).float().contiguous()


def _cache_samples(case, seed):
    """Training samples as rows of 20 floats: vertices in the unit box, outgoing
    directions, normals, albedos and radiance targets."""
    g = torch.Generator().manual_seed(31 + seed)
    n = case["samples"]
    s = torch.zeros((n, 20))
    p = torch.rand((n, 3), generator=g) - 0.5
    wall = torch.randint(0, 3, (n,), generator=g)
    p[torch.arange(n), wall] = torch.where(torch.rand(n, generator=g) < 0.5, -0.5, 0.5)   # surfaces of the box
    s[:, 0:3] = p
    s[:, 4:7] = torch.nn.functional.normalize(torch.randn((n, 3), generator=g), dim=1)
    s[:, 7] = torch.where(torch.rand(n, generator=g) < 0.7, 1.0, 0.3)
    s[torch.arange(n), 8 + wall] = -torch.sign(p[torch.arange(n), wall])
    s[:, 12:15] = torch.rand((n, 3), generator=g) * 0.85 + 0.05
    light = torch.exp(-4.0 * ((p[:, 0:1]) ** 2 + (p[:, 1:2] - 0.5) ** 2 + p[:, 2:3] ** 2))
    target = light * torch.tensor([[1.7, 1.2, 0.4]]) * s[:, 12:15] * (0.5 + torch.rand((n, 3), generator=g))
    s[:, 3], s[:, 11], s[:, 15] = target[:, 0], target[:, 1], target[:, 2]
    return s.numpy()


def _cache_config(case, **kw):
    return ab.nrc_config(log2_entries=case["log2"], **kw)


def prepare(case, seed):
    k = case["kind"]
    st = dict(case=case)
    if k == "render":
        volumes, medium = None, None
        if case["scene"] == "box":
            objects = scenes.box_scene(seed=scenes.SEED_BASE + 1 + seed)
            cam = scenes.box_camera(case["width"], case["height"])
        elif case["scene"] == "spheres":
            objects = _sphere_objects(case, seed)
            cam = _sphere_camera(case, case["width"], case["height"])
        else:
            objects, volumes, medium = scenes.medium_box_scene(seed=scenes.SEED_BASE + 3 + seed, grid=128,
                                                               medium_grid=64)
            cam = scenes.box_camera(case["width"], case["height"])
        st["scene"] = ab.Scene(objects, volumes=volumes)
        if case["spectral"]:
            st["scene"].set_spectral(64, _tables(seed))
        if medium:
            st["scene"].set_medium(**medium)
        st["cam"] = cam
        st["params"] = ab.make_params(spp=case["spp"], max_depth=case["depth"], use_nee=case["nee"],
                                      spectral=case["spectral"], seed=ab.REFERENCE_SEED + seed)
        if case["host"]:
            st["out"] = torch.empty((case["height"], case["width"], 3), dtype=torch.float32, pin_memory=True).numpy()
        else:
            st["out"] = _pixels(case["width"], case["height"])
    elif k == "batch":
        small = dict(case, spheres=max(4, case["spheres"] // 4))
        made = [(ab.Scene(scenes.box_scene(seed=scenes.SEED_BASE + 1 + seed)), None),
                (ab.Scene(_sphere_objects(case, seed)), case), (ab.Scene(_sphere_objects(small, seed)), small)]
        rng = np.random.default_rng(17)   # the mix of sizes is part of the case, not of the seed
        st["scenes"], st["jobs"], st["out"] = made, [], []
        for j in range(case["jobs"]):
            scene, of = made[j % 3]
            w = max(32, int(case["size"] * rng.uniform(0.5, 1.5)))
            h = max(32, int(case["size"] * rng.uniform(0.5, 1.5)))
            cam = scenes.box_camera(w, h) if of is None else _sphere_camera(of, w, h)
            par = ab.make_params(spp=max(1, int(case["spp"] * rng.uniform(0.25, 2.0))), max_depth=case["depth"],
                                 seed=ab.REFERENCE_SEED + 64 * seed + j)
            out = _pixels(w, h)
            st["out"].append(out)
            st["jobs"].append((scene, cam, par, out.data_ptr(), None))
    elif k == "trace":
        objects = _sphere_objects(case, seed)
        st["scene"] = ab.Scene(objects)
        st["rays"] = _rays(case, objects, seed)
        st["hit"] = torch.empty(case["rays"], dtype=torch.int32, device="cuda")
        st["t"] = torch.empty(case["rays"], dtype=torch.float32, device="cuda")
    elif k == "denoise":
        w, h = case["width"], case["height"]
        scene = ab.Scene(_sphere_objects(case, seed))
        cam = _sphere_camera(case, w, h)
        st["hdr"], st["out"] = _pixels(w, h), _pixels(w, h)
        st["gbuffer"] = torch.zeros(w * h * ab.GBUFFER_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
        st["stats"] = torch.zeros(w * h * ab.STATS_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
        acc = torch.zeros((h, w, 3), dtype=torch.float64, device="cuda")
        for f in range(case["frames"]):
            ab.render_frame_denoise(scene, cam, ab.make_params(spp=1, max_depth=8, frame_offset=f,
                                                               seed=ab.REFERENCE_SEED + seed),
                                    st["hdr"], acc, st["gbuffer"], st["stats"])
        st["hdr"].copy_(acc / case["frames"])
    elif k == "cache_frame":
        st["scene"] = ab.Scene(_sphere_objects(case, seed))
        st["cache"] = ab.RadianceCache(st["scene"], _cache_config(case, seed=1 + seed))
        st["cam"] = _sphere_camera(case, case["width"], case["height"])
        st["params"] = ab.make_params(spp=case["spp"], max_depth=case["depth"], seed=ab.REFERENCE_SEED + seed)
        st["out"] = _pixels(case["width"], case["height"])
    elif k == "cache_grad":
        st["scene"] = ab.Scene(scenes.box_scene())
        st["cache"] = ab.RadianceCache(st["scene"], _cache_config(case, seed=1 + seed, train_paths=1024,
                                                                  max_resolution=512,
                                                                  bounds=((-0.5,) * 3, (0.5,) * 3)))
        st["samples"] = _cache_samples(case, seed)
    else:
        st["tables"] = _tables(seed)
        st["out"] = torch.empty(case["res"] ** 3 * 4, dtype=torch.float32, device="cuda")
    return st


# ------------------------------------------------------------------ one pass
def run(st):
    case = st["case"]
    k = case["kind"]
    if k == "render":
        if case["host"]:
            return st["scene"].render(st["cam"], st["params"], out=st["out"])[0]
        st["scene"].render_device(st["cam"], st["params"], st["out"].data_ptr())
        return st["out"]
    if k == "batch":
        ab.render_batch(st["jobs"])
        return st["out"]
    if k == "trace":
        call = st["scene"].trace_rays_static if case["static"] else st["scene"].trace_rays_device
        call(st["rays"].data_ptr(), case["rays"], bool(case["any"]), st["hit"].data_ptr(), st["t"].data_ptr())
        if case["any"]:
            return st["hit"] >= 0   # an occlusion query says whether something blocks, not which of the blockers
        return {"object": st["hit"], "t": st["t"]}
    if k == "denoise":
        ab.denoise_bilateral(st["hdr"], st["out"], st["gbuffer"], st["stats"], case["width"], case["height"])
        return st["out"]
    if k == "cache_frame":
        st["cache"].render_frame(st["cam"], st["params"], st["out"].data_ptr(), None, train=False)
        return st["out"]
    if k == "cache_grad":
        table, weights, loss = st["cache"].gradients(st["samples"])
        return {"table": table, "weights": weights, "loss": np.float32(loss)}
    ab.spectral_rgb_lut(case["res"], ab.LUT_TENSOR, st["tables"], st["out"])
    return st["out"]


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    """Bytes: inputs read once, outputs written once (for a render the scene's
    triangles at 48 bytes and the image).  Operations: per ray query a descent
    through the node boxes (about 10 nodes of 8 boxes) and a few triangle
    tests; the networks' products; the filter's 225 taps."""
    k = case["kind"]
    query = 1100.0
    if k in ("render", "cache_frame"):
        paths = case["width"] * case["height"] * case["spp"]
        per = 2.6 if case.get("spheres") else 6.0
        tris = case.get("spheres", 0) * TRIS_PER_SPHERE + 40
        return {"bytes": 48.0 * tris + 12.0 * case["width"] * case["height"], "flops": paths * per * query}
    if k == "batch":
        px = case["jobs"] * case["size"] ** 2
        return {"bytes": 48.0 * 1.25 * case["spheres"] * TRIS_PER_SPHERE + 12.0 * px,
                "flops": px * case["spp"] * 1.1 * 4.0 * query}
    if k == "trace":
        out = 4.0 if case["any"] else 8.0
        return {"bytes": case["rays"] * (32.0 + out) + 48.0 * case["spheres"] * TRIS_PER_SPHERE,
                "flops": case["rays"] * query}
    if k == "denoise":
        px = case["width"] * case["height"]
        return {"bytes": px * (12.0 + 48.0 + 48.0 + 12.0), "flops": px * 225.0 * 60.0}
    if k == "cache_grad":
        params = 16 * 2 * 2 ** case["log2"] + ab.NRC_PARAMS
        return {"bytes": case["samples"] * 80.0 + 8.0 * params, "flops": 6.0 * case["samples"] * ab.NRC_PARAMS}
    return {"bytes": case["res"] ** 3 * 16.0, "flops": case["res"] ** 3 * 2.0 * (8 * 32 * 32 + 32 * 4)}


# ------------------------------------------------------------------ the same in 64 bits
def exact(case, seed):
    """Ray distances, the filtered image, the cache's gradients and the lookup
    table in double precision.  Images of path tracing have no such value: a
    path's direction depends on every rounding before it."""
    k = case["kind"]
    if k == "trace" and not case["any"]:
        objects = _sphere_objects(case, seed)
        return {"object": None, "t": _exact_distances(objects, _rays(case, objects, seed).double())}
    if k == "denoise":
        st = prepare(case, seed)
        return _exact_bilateral(st["hdr"].double(), st["gbuffer"], st["stats"], case["width"], case["height"])
    if k == "cache_grad":
        st = prepare(case, seed)
        return _exact_gradients(st["cache"], torch.from_numpy(st["samples"]).cuda().double())
    if k == "table":
        return _exact_table(torch.from_numpy(_tables(seed)).cuda().double(), case["res"])
    return None


def _vec(field):
    return torch.from_numpy(np.stack([field[k] for k in "xyz"], -1).astype(np.float32)).cuda().double()


def _exact_distances(objects, rays):
    """Nearest distance in [tmin, tmax), tmax where nothing is hit: every ray
    against the spheres' hulls, then against the triangles of the hulls it meets."""
    o, tmin, d, best = rays[:, 0:3], rays[:, 3], rays[:, 4:7], rays[:, 7].clone()

    def hull(c, r):
        oc = o - c
        b = (oc * d).sum(1)
        cc = (oc * oc).sum(1) - r * r
        disc = b * b - cc
        s = disc.clamp(min=0).sqrt()
        return disc >= 0, -b - s, -b + s

    tri = objects[objects["type"] == ab.OBJ_TRIANGLE]
    pos = _vec(tri["tri"]["position"])
    center = _vec(tri["center"])
    v = (pos.float() + center.float()[:, None, :]).double()
    groups = [(i, i + TRIS_PER_SPHERE) for i in range(0, len(tri) - 2, TRIS_PER_SPHERE)] + [(len(tri) - 2, len(tri))]
    for lo, hi in groups:
        if hi - lo == 2:
            idx = torch.arange(len(o), device=o.device)
        else:
            ok, t0, t1 = hull(center[lo], pos[lo].norm(dim=1).max() * 1.0001)
            idx = torch.nonzero(ok & (t1 > 0) & (t0 < best)).flatten()
        e1, e2 = v[lo:hi, 1] - v[lo:hi, 0], v[lo:hi, 2] - v[lo:hi, 0]
        for part in idx.split(1 << 15):
            oo, dd = o[part][:, None, :], d[part][:, None, :]
            h = torch.linalg.cross(dd.expand(-1, hi - lo, -1), e2.expand(len(part), -1, -1))
            a = (e1 * h).sum(2)
            s = oo - v[lo:hi, 0]
            u = (s * h).sum(2) / a
            q = torch.linalg.cross(s, e1.expand(len(part), -1, -1))
            w = (dd * q).sum(2) / a
            t = (e2 * q).sum(2) / a
            ok = (a.abs() >= 1e-6) & (u >= 0) & (w >= 0) & (u + w <= 1) & (t > 1e-5) & (t >= tmin[part][:, None])
            t = torch.where(ok, t, torch.inf).amin(1)
            best[part] = torch.minimum(best[part], t)
    for s in objects[objects["type"] == ab.OBJ_SPHERE]:
        c = torch.tensor([float(s["center"][k]) for k in "xyz"], device=o.device, dtype=torch.float64)
        ok, t0, t1 = hull(c, float(s["extent"]["x"]))
        t = torch.where(t0 > 0, t0, t1)
        best = torch.where(ok & (t > 0) & (t >= tmin), torch.minimum(best, t), best)
    return best


def _t_quantiles():
    """Student t quantiles at 0.9975 for 1..1024 degrees of freedom, by bisection
    on the finite series of the distribution function (Abramowitz and Stegun 26.7.3/4)."""
    n = np.arange(1, 1025)
    lo, hi = np.zeros(1024), np.full(1024, 200.0)
    for _ in range(60):
        mid = 0.5 * (lo + hi)
        th = np.arctan(mid / np.sqrt(n))
        c2 = np.cos(th) ** 2
        term = np.where(n % 2 == 1, np.cos(th), 1.0)
        acc = np.where((n % 2 == 1) & (n == 1), 0.0, term)
        for k in range(1, 512):
            term = term * c2 * np.where(n % 2 == 1, 2.0 * k / (2.0 * k + 1.0), (2.0 * k - 1.0) / (2.0 * k))
            more = np.where(n % 2 == 1, 2 * k + 1 <= n - 2, 2 * k <= n - 2)
            acc = acc + np.where(more, term, 0.0)
        inside = np.where(n % 2 == 1, 2.0 / np.pi * (th + np.sin(th) * acc), np.sin(th) * acc)
        low = 0.5 + 0.5 * inside < 0.9975
        lo, hi = np.where(low, mid, lo), np.where(low, hi, mid)
    return torch.from_numpy(0.5 * (lo + hi)).cuda()


def _exact_bilateral(hdr, gbuffer, stats, width, height):
    n = width * height
    gb = gbuffer.view(n, ab.GBUFFER_DTYPE.itemsize)

    def field(raw, dtype, name, kind):
        f, off = dtype.fields[name][:2]
        x = raw[:, off:off + f.itemsize].contiguous().view(kind)
        return x.double().view(height, width, -1)

    def halves(name):
        return field(gb, ab.GBUFFER_DTYPE, name, torch.float16)

    raw = stats.view(n, ab.STATS_DTYPE.itemsize)
    num = field(raw, ab.STATS_DTYPE, "num", torch.int32)
    mean, m2, m3 = (field(raw, ab.STATS_DTYPE, k, torch.float32) for k in ("mean", "m2_div_n", "m3_div_n"))
    less = (num - 1).clamp(min=1)
    vb = m2 * num / less
    vth, theta, u = vb / num, mean + m3 / 6.0 / vb, vb / num
    low = u * u / less
    normal = torch.nn.functional.normalize(halves("normal"), dim=2, eps=0.0)
    guide = [halves("albedo"), normal, field(gb, ab.GBUFFER_DTYPE, "depth", torch.float32), halves("metallic"),
             halves("roughness"), halves("shading_model")[:, :, :5]]
    s = torch.log1p(hdr)
    quant = _t_quantiles()
    acc, wsum = s * 1.0e-6, torch.full((height, width, 1), 1.0e-6, dtype=torch.float64, device=hdr.device)
    ys, xs = torch.arange(height, device=hdr.device), torch.arange(width, device=hdr.device)
    for j in range(-7, 8):
        yy = (ys + j).clamp(0, height - 1)
        for i in range(-7, 8):
            xx = (xs + i).clamp(0, width - 1)

            def at(a):
                return a[yy][:, xx]

            t2 = (theta - at(theta)) ** 2
            share = (t2 + at(vth)) / (t2 + vth + at(vth)).clamp(min=1.0e-6)
            x = 0.5 / (1.0 - share) - 1.0
            nu = (u + at(u)) ** 2 / (low + at(low))
            q = quant[torch.nan_to_num(nu, nan=1.0).clamp(1, 1024).floor().long() - 1]
            ok = (~(x < 0) & (x < q * q)).all(2, keepdim=True)
            a, nrm, dep, met, rough, model = [at(g) for g in guide]
            w = ((guide[0] - a) ** 2).sum(2, keepdim=True) / 2.0
            w = w + (1.0 - (guide[1] * nrm).sum(2, keepdim=True)) ** 2 * 2.0
            w = w + ((guide[2] - dep) / torch.maximum(guide[2], dep).clamp(min=1.0e-6)) ** 2 * 8.0
            w = w + (guide[3] - met) ** 2 * 2.0 + (guide[4] - rough) ** 2 * 2.0
            w = w + (0.5 * (guide[5] - model).abs().sum(2, keepdim=True)) ** 2 * 50.0
            w = torch.nan_to_num(torch.exp(-w) * math.exp(-(i * i + j * j) / 8.0), nan=0.0) * ok
            acc, wsum = acc + at(s) * w, wsum + w
    return torch.expm1(acc / wsum).clamp(min=0.0)


def _sh16(d):
    x, y, z = d[:, 0], d[:, 1], d[:, 2]
    c = (0.28209479177387814, 0.48860251190291987, 1.0925484305920792, 0.94617469575755997, 0.31539156525251999,
         0.54627421529603959, 0.59004358992664352, 2.8906114426405538, 0.45704579946446572, 0.3731763325901154,
         1.4453057213202769)
    o = [torch.full_like(x, c[0]), -c[1] * y, c[1] * z, -c[1] * x, c[2] * x * y, -c[2] * y * z, c[3] * z * z - c[4],
         -c[2] * x * z, c[5] * (x * x - y * y), c[6] * y * (-3 * x * x + y * y), c[7] * x * y * z,
         c[8] * y * (1 - 5 * z * z), c[9] * z * (5 * z * z - 3), c[8] * x * (1 - 5 * z * z),
         c[10] * z * (x * x - y * y), c[6] * x * (-x * x + 3 * y * y)]
    return torch.stack(o, 1)


def _exact_gradients(cache, s):
    """Loss and gradients of the cache's network (hash grid, spherical harmonics,
    5 hidden layers of 64) on its own parameters, without the 16-bit roundings."""
    c = cache.config
    tab, W = cache.params()
    entries = 1 << c.log2_entries
    table = torch.from_numpy(tab).cuda().double().view(c.levels * entries, 2).requires_grad_()
    W = torch.from_numpy(W).cuda().double().requires_grad_()
    lo = torch.tensor([float(v) for v in c.bounds_min], device=s.device, dtype=torch.float64)
    hi = torch.tensor([float(v) for v in c.bounds_max], device=s.device, dtype=torch.float64)
    p = ((s[:, 0:3] - lo) / (hi - lo)).clamp(0.0, 1.0)
    grow = math.exp((math.log(c.max_resolution) - math.log(c.base_resolution)) / max(c.levels - 1, 1))
    feats = []
    for lv in range(c.levels):
        r = int(math.floor(c.base_resolution * grow ** lv + 1e-6))
        f = (p.float() * r)   # cell choice as in 32 bits, weights in 64
        i = f.floor().long().clamp(0, r - 1)
        t = (p * r - i).clamp(0.0, 1.0)
        sum2 = 0.0
        for corner in range(8):
            b = [(corner >> a) & 1 for a in range(3)]
            q = [i[:, a] + b[a] for a in range(3)]
            if (r + 1) ** 3 <= entries:
                h = q[0] + q[1] * (r + 1) + q[2] * (r + 1) ** 2
            else:
                h = q[0] ^ (q[1] * 2654435761) ^ (q[2] * 805459861)
            h = (h & (entries - 1)) + lv * entries
            w = torch.ones_like(p[:, 0])
            for a in range(3):
                w = w * (t[:, a] if b[a] else 1.0 - t[:, a])
            sum2 = sum2 + w[:, None] * table[h]
        feats.append(sum2)
    X = torch.cat(feats + [torch.zeros((len(s), 32 - 2 * c.levels), device=s.device, dtype=torch.float64), _sh16(s[:, 4:7]),
                           s[:, 7:8], s[:, 12:15], s[:, 8:11] * 0.5 + 0.5, torch.ones_like(s[:, :1]),
                           torch.zeros((len(s), 8), device=s.device, dtype=torch.float64)], 1)
    for lv in range(5):
        X = torch.relu(X @ W[lv * 4096:(lv + 1) * 4096].view(64, 64).T)
    pred = torch.exp((X @ W[5 * 4096:].view(16, 64).T)[:, :3].clamp(max=15.0))
    target = s[:, [3, 11, 15]]
    loss = ((pred - target) ** 2 / (pred.detach() ** 2 + 0.01)).mean()
    loss.backward()
    return {"table": table.grad.reshape(-1), "weights": W.grad, "loss": loss.detach()}


def _exact_table(tab, res):
    off = 421 * 4
    w_in, b_in = tab[off:off + 1024].view(32, 32), tab[off + 1024:off + 1056]
    w_blk, b_blk = tab[off + 1056:off + 1056 + 7168].view(7, 32, 32), tab[off + 8224:off + 8448].view(7, 32)
    w_out = tab[off + 8448:off + 8576].view(4, 32)
    c = (torch.arange(res, device=tab.device, dtype=torch.float64) + 0.5) / res
    k = torch.arange(1, 5, device=tab.device, dtype=torch.float64) * math.pi
    out = []
    for z in range(res):
        rgb = torch.stack([c.repeat(res), c.repeat_interleave(res), c[z].expand(res * res)], 1)
        scale = rgb.amax(1, keepdim=True)
        a = (rgb / (scale + 0.001))[:, :, None] * k
        s = torch.cat([torch.sin(a), torch.cos(a)], 2).flatten(1)
        s = torch.cat([s, torch.sin(scale * k), torch.cos(scale * k)], 1)
        h = torch.relu(s @ w_in.T + b_in)
        for b in range(7):
            h = h + torch.relu(h @ w_blk[b].T + b_blk[b])
        out.append((h @ w_out.T) * scale)
    return torch.cat(out).reshape(-1)
