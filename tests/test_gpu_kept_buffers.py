"""Buffers kept between calls: batches of growing and shrinking size, cache calls
of changing size, lookup tables from two threads at once, each equal to its own
result alone.  (A scene and its cache are used by one thread at a time.)"""
import threading

import numpy as np
import pytest

import scenes
from aperture_b200 import LUT_TENSOR, RadianceCache, Scene, make_params, nrc_config, render_batch, spectral_rgb_lut
from test_gpu_tail import tables


def together(*calls):
    """Runs the calls in threads of their own; their results in order."""
    got, errors = [None] * len(calls), []

    def run(k, f):
        try:
            got[k] = f()
        except Exception as e:   # noqa: BLE001
            errors.append(e)
    threads = [threading.Thread(target=run, args=(k, f)) for k, f in enumerate(calls)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not errors, errors
    return got


def batch_images(scene, sizes):
    import torch
    outs, jobs = [], []
    for k, (w, h, spp) in enumerate(sizes):
        o = torch.zeros(h * w * 3, dtype=torch.float32, device="cuda")
        outs.append(o)
        jobs.append((scene, scenes.box_camera(w, h), make_params(spp=spp, max_depth=6, frame_offset=k), o.data_ptr(), None))
    render_batch(jobs)
    torch.cuda.synchronize()
    return [o.cpu().numpy().reshape(h, w, 3) for o, (w, h, _) in zip(outs, sizes)]


SMALL, LARGE = [(20, 15, 2), (9, 31, 5)], [(64, 48, 9), (33, 17, 40), (128, 100, 3), (50, 2, 1)]


@pytest.mark.gpu
def test_batches_of_changing_size(box_objects):
    scene = Scene(box_objects)
    ref = {id(s): [scene.render(scenes.box_camera(w, h), make_params(spp=spp, max_depth=6, frame_offset=k))[0]
                   for k, (w, h, spp) in enumerate(s)] for s in (SMALL, LARGE)}

    def check(got, sizes):
        for a, b in zip(got, ref[id(sizes)]):
            np.testing.assert_allclose(a, b, rtol=1e-6, atol=1e-7)
    for sizes in (SMALL, LARGE, SMALL, LARGE):
        check(batch_images(scene, sizes), sizes)


@pytest.mark.gpu
def test_cache_inference_of_changing_size(box_objects):
    cache = RadianceCache(Scene(box_objects), nrc_config(log2_entries=10, train_paths=64, bounds=((-0.5,) * 3, (0.5,) * 3)))
    rng = np.random.default_rng(4)
    v = (rng.random((5000, 16)) - 0.5).astype(np.float32)
    whole = cache.infer(v)
    for n in (1, 700, 3, 5000, 129):
        assert np.array_equal(cache.infer(v[:n]), whole[:n])


@pytest.mark.gpu
def test_lookup_tables_in_two_threads():
    ta, tb = tables(1), tables(2)
    a, b = spectral_rgb_lut(24, LUT_TENSOR, ta)[0].cpu(), spectral_rgb_lut(40, LUT_TENSOR, tb)[0].cpu()
    assert not bool((a == 0).all())
    for _ in range(4):
        x, y = together(lambda: spectral_rgb_lut(24, LUT_TENSOR, ta)[0].cpu(), lambda: spectral_rgb_lut(40, LUT_TENSOR, tb)[0].cpu())
        assert bool((x == a).all()) and bool((y == b).all())


@pytest.mark.gpu
def test_scenes_share_the_path_state_of_large_renders(box_objects, small_spheres_objects):
    """Renders above the size a scene keeps for itself: two scenes in turn, growing
    and shrinking, and both at once from two threads."""
    box, sph = Scene(box_objects), Scene(small_spheres_objects)
    cam = scenes.spheres_camera(400, 300)
    cam.position.z, cam.position.y = -45.0, 8.0
    work = [(box, scenes.box_camera(300, 300), 4), (sph, cam, 3), (box, scenes.box_camera(700, 500), 2), (sph, cam, 9),
            (box, scenes.box_camera(30, 20), 2)]

    def image(w):
        scene, c, spp = w
        return scene.render(c, make_params(spp=spp, max_depth=5))[0]
    ref = [image(w) for w in work]
    for k in (3, 0, 4, 1, 2, 3):
        np.testing.assert_allclose(image(work[k]), ref[k], rtol=1e-6, atol=1e-7)
    for _ in range(3):
        a, b = together(lambda: image(work[2]), lambda: image(work[3]))
        np.testing.assert_allclose(a, ref[2], rtol=1e-6, atol=1e-7)
        np.testing.assert_allclose(b, ref[3], rtol=1e-6, atol=1e-7)
    box.close()   # the other scene still renders, and a new one after the last has gone
    np.testing.assert_allclose(image(work[1]), ref[1], rtol=1e-6, atol=1e-7)
    sph.close()
    again = Scene(box_objects)
    np.testing.assert_allclose(image((again,) + work[0][1:]), ref[0], rtol=1e-6, atol=1e-7)
