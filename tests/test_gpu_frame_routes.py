"""Cache, guided and denoiser frames by the two routes a frame can take: alone on
the kernel of the last paths (frames below its limit), and through the wavefront
(fewer paths in flight than pixels), whose shading kernels for these modes no
small frame reaches otherwise."""
import numpy as np
import pytest

import aperture_b200 as ab
from aperture_b200 import PathGuide, RadianceCache, make_params, nrc_config
from test_gpu_tail import scene_of, tables

W, H = 64, 48


def setup(kind):
    scene, camera = scene_of(kind)
    if kind != "medium":
        scene.set_spectral(8, tables())
    cam = camera(W, H)
    if kind == "spheres":
        cam.position.z, cam.position.y = -45.0, 8.0
    return scene, cam


def params(wave, **more):
    return make_params(spp=1, max_depth=8, wave_paths=wave, **more)


WAVES = [W * H // 8, W * H - 1]


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["spheres", "medium", "box"])
@pytest.mark.parametrize("spectral", [0, 4])
def test_cache_frames(kind, spectral):
    """The same queries and training samples, and the same image of the untrained
    cache: per pixel its path's light and one prediction, added in either order."""
    import torch
    scene, cam = setup(kind)

    def frame(wave):
        cache = RadianceCache(scene, nrc_config(log2_entries=10, train_paths=300, train_batch=64, train_steps=2))
        cache.set_spectral(spectral)
        out = torch.zeros(W * H * 3, device="cuda")
        st = cache.render_frame(cam, params(wave, spectral=spectral), out.data_ptr(), None, train=True, stats=True)
        torch.cuda.synchronize()
        return out.cpu().numpy(), st
    ref, rs = frame(0)
    assert rs.queries > 100 and rs.train_samples > 100
    for wave in WAVES:
        got, st = frame(wave)
        assert (st.queries, st.train_samples, st.extension_rays, st.shadow_rays) == \
               (rs.queries, rs.train_samples, rs.extension_rays, rs.shadow_rays)
        np.testing.assert_allclose(got, ref, rtol=1e-6, atol=1e-7)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["spheres", "medium", "box"])
def test_guided_frames(kind):
    """The first frame is the same, and so are the samples it hands the probes; the
    probes add them up in another order, after which a few later choices may fall
    differently."""
    import torch
    scene, cam = setup(kind)

    def frames(wave):
        guide = PathGuide(scene, log2_table=14)
        out = torch.zeros(W * H * 3, device="cuda")
        imgs = []
        for f in range(3):
            guide.render_frame(cam, params(wave, frame_offset=f), out.data_ptr(), None)
            torch.cuda.synchronize()
            imgs.append(out.cpu().numpy().reshape(-1, 3))
            if f == 0:
                first = guide.stats()
        return imgs, (first.probes, first.samples, first.dropped)
    ref, rs = frames(0)
    assert rs[0] > 10 and rs[1] > 100
    for wave in WAVES:
        got, st = frames(wave)
        assert st == rs
        assert np.array_equal(got[0], ref[0])
        for a, b in zip(got[1:], ref[1:]):
            assert np.mean(np.abs(a - b).max(1) <= 1e-3 * (np.abs(b).max(1) + 1e-3)) > 0.95


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["spheres", "medium", "box"])
def test_denoiser_frames(kind):
    import torch
    scene, cam = setup(kind)

    def frames(wave):
        acc = torch.zeros(W * H * 3, dtype=torch.float64, device="cuda")
        gbuf = torch.zeros(W * H * ab.GBUFFER_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
        stat = torch.zeros(W * H * ab.STATS_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
        for f in range(3):
            ab.render_frame_denoise(scene, cam, params(wave, frame_offset=f), None, acc, gbuf, stat)
        torch.cuda.synchronize()
        return [x.cpu().numpy() for x in (acc, gbuf, stat)]
    ref = frames(0)
    assert ref[0].max() > 0
    for wave in WAVES:
        for a, b in zip(frames(wave), ref):
            assert np.array_equal(a, b)
