"""The kernel that runs the last paths of a render to their end against the
wavefront: the same paths, record by record.  A render that fits into one wave
below the kernel's limit uses it alone; with fewer paths in flight than samples
(wave_paths) the wavefront traces them, and only the last ones change over."""
import numpy as np
import pytest

import scenes
from aperture_b200 import Scene, make_params

LANES, PER_LANE = 256, 4   # lanes per SM of the kernel, and paths per lane up to which it is used


def tables(seed=3):
    """A spectral table block of random-init networks (layout of ar_scene_set_spectral)."""
    rng = np.random.default_rng(seed)
    lam = np.arange(360.0, 781.0)
    cmf = [np.exp(-0.5 * ((lam - m) / s) ** 2) for m, s in ((600, 35), (555, 45), (450, 22))]
    block = lambda: [rng.normal(0.0, 0.03, 7 * 1024), rng.uniform(0.05, 0.15, 7 * 32)]   # noqa: E731
    parts = [np.stack(cmf, 1).ravel(), 100.0 + 0 * lam, rng.normal(0.0, 0.05, 1024), rng.uniform(0.9, 1.1, 32)]
    parts += block() + [rng.uniform(0.8, 1.2, 128) * 0.01] + block() + [rng.uniform(0.8, 1.2, 128) * 0.015]
    return np.concatenate(parts).astype(np.float32)


def scene_of(kind):
    if kind == "spheres":
        return Scene(scenes.spheres_scene(n_spheres=40, n_lights=4, box=20.0)), scenes.spheres_camera
    if kind == "box":
        return Scene(scenes.box_scene()), scenes.box_camera
    objects, volumes, medium = scenes.medium_box_scene(grid=24, medium_grid=16)
    s = Scene(objects, volumes=volumes)
    s.set_medium(**medium)
    s.set_spectral(8, tables())
    return s, scenes.box_camera


def same(a, b):
    for f in a.dtype.names:
        assert np.array_equal(a[f], b[f]), f


@pytest.mark.gpu
@pytest.mark.parametrize("kind,spectral,nee", [("box", 0, 1), ("box", 0, 0), ("spheres", 0, 1), ("medium", 0, 1),
                                               ("medium", 1, 1), ("medium", 4, 1)])
def test_tail_traces_the_wavefronts_paths(kind, spectral, nee):
    scene, camera = scene_of(kind)
    cam = camera(47, 31)
    if kind == "spheres":
        cam.position.z, cam.position.y = -45.0, 8.0
    par = dict(spp=3, max_depth=9, use_nee=nee, spectral=spectral)
    tail = scene.debug_paths(cam, make_params(**par))
    assert (tail["segments"] > 1).mean() > 0.2
    for wave in (1000, 47 * 31 * 3 - 1):
        same(tail, scene.debug_paths(cam, make_params(wave_paths=wave, **par)))


@pytest.mark.gpu
@pytest.mark.parametrize("total", [1, 31, 33, "limit", "limit+1"])
def test_path_counts_around_the_limit(total):
    scene, camera = scene_of("box")
    sms = __import__("torch").cuda.get_device_properties(0).multi_processor_count
    limit = LANES * PER_LANE * sms
    n = {"limit": limit, "limit+1": limit + 1}.get(total, total)
    cam = camera(n, 1)
    one = scene.debug_paths(cam, make_params(spp=1, max_depth=6))
    same(one, scene.debug_paths(cam, make_params(spp=1, max_depth=6, wave_paths=max(1, n // 2))))
    img, st = scene.render(cam, make_params(spp=1, max_depth=6))
    assert st.paths == n and st.extension_rays == one["segments"].sum()
    np.testing.assert_array_equal(img.reshape(-1, 3), one["radiance"])


@pytest.mark.gpu
@pytest.mark.parametrize("w,h,spp,wave", [(3, 2, 500, 0), (3, 2, 500, 7), (16, 9, 400, 40000), (5, 1, 3, 4)])
def test_samples_of_a_pixel_started_together(w, h, spp, wave):
    """Waves that hold many samples of each pixel, whole or in part, trace the
    samples of renders of one sample each."""
    scene, camera = scene_of("box")
    cam = camera(w, h)
    got = scene.debug_paths(cam, make_params(spp=spp, max_depth=5, frame_offset=7, wave_paths=wave)).reshape(spp, w * h)
    for k in (0, 1, 2, spp // 2, spp - 1):
        same(got[k], scene.debug_paths(cam, make_params(spp=1, max_depth=5, frame_offset=7 + k)))
