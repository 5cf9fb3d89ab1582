"""Calls where little device memory is left: what earlier calls kept gives way,
and batches run with fewer paths in flight, as single renders do."""
import numpy as np
import pytest

import scenes
from aperture_b200 import ArError, PathGuide, RadianceCache, Scene, make_params, nrc_config, render_batch

GIB = 1 << 30


class Short:
    """All but `leave` bytes of the device's free memory, held while inside."""
    def __init__(self, leave):
        self.leave = int(leave)

    def __enter__(self):
        import torch
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        free, _ = torch.cuda.mem_get_info()
        self.held = torch.empty(free - self.leave, dtype=torch.uint8, device="cuda")

    def __exit__(self, *exc):
        import torch
        del self.held
        torch.cuda.empty_cache()


def device_image(scene, cam, out, **par):
    import torch
    scene.render_device(cam, make_params(**par), out.data_ptr())
    torch.cuda.synchronize()
    return out.cpu().numpy()


@pytest.mark.gpu
def test_batch_with_little_memory(box_objects):
    """8.4 million paths: the default share of paths in flight takes 3.7 GB."""
    import torch
    scene = Scene(box_objects)
    outs = [torch.zeros(700 * 500 * 3, device="cuda") for _ in range(3)]
    jobs = [(scene, scenes.box_camera(700, 500), make_params(spp=8, max_depth=4, frame_offset=8 * k), o.data_ptr(), None)
            for k, o in enumerate(outs)]
    render_batch(jobs, path_budget=1 << 16)
    torch.cuda.synchronize()
    ref = [o.cpu().numpy() for o in outs]
    [o.zero_() for o in outs]
    with Short(2.5 * GIB):
        st = render_batch(jobs)
        torch.cuda.synchronize()
    assert st.paths == 3 * 700 * 500 * 8
    for o, r in zip(outs, ref):
        np.testing.assert_allclose(o.cpu().numpy(), r, rtol=1e-6, atol=1e-7)


@pytest.mark.gpu
def test_kept_memory_gives_way(box_objects):
    """A large render leaves its path state (3.6 GB) behind; a larger image in
    another scene needs that room."""
    import torch
    first, second = Scene(box_objects), Scene(box_objects)
    small, large = torch.zeros(1920 * 1080 * 3, device="cuda"), torch.zeros(4096 * 4096 * 3, device="cuda")
    ref = device_image(first, scenes.box_camera(4096, 4096), large, spp=1, max_depth=3)
    first.close()
    first = Scene(box_objects)
    device_image(first, scenes.box_camera(1920, 1080), small, spp=5, max_depth=3)
    large.zero_()
    with Short(0.8 * GIB):
        got = device_image(second, scenes.box_camera(4096, 4096), large, spp=1, max_depth=3)
    assert np.array_equal(got, ref)


@pytest.mark.gpu
def test_scene_after_an_image_that_did_not_fit(box_objects):
    """A render whose per-pixel state (8 GB) finds no room; the scene's ray
    queries and renders go on."""
    import torch
    scene = Scene(box_objects)
    out = torch.zeros(64 * 48 * 3, device="cuda")
    ref = device_image(scene, scenes.box_camera(64, 48), out, spp=2, max_depth=5)
    rng = np.random.default_rng(6)
    rays = np.zeros((500, 8), np.float32)
    rays[:, :3] = rng.uniform(-0.4, 0.4, (500, 3))
    rays[:, 4:7] = rng.normal(size=(500, 3))
    rays[:, 4:7] /= np.linalg.norm(rays[:, 4:7], axis=1, keepdims=True)
    rays[:, 7] = 1e30
    hits, t = scene.trace_rays(rays)
    huge = torch.zeros(16384 * 8192 * 3, device="cuda")
    with Short(1.5 * GIB):
        with pytest.raises(ArError, match="OUT_OF_MEMORY"):
            scene.render_device(scenes.box_camera(16384, 8192), make_params(spp=1, max_depth=2), huge.data_ptr())
        again, ta = scene.trace_rays(rays)
        out.zero_()
        img = device_image(scene, scenes.box_camera(64, 48), out, spp=2, max_depth=5)
    assert np.array_equal(again, hits) and np.array_equal(ta, t)
    np.testing.assert_allclose(img, ref, rtol=1e-6, atol=1e-7)


@pytest.mark.gpu
@pytest.mark.parametrize("what", ["cache", "guide"])
def test_frames_after_one_that_did_not_fit(box_objects, what):
    """A cache's queries (10 GB) and a guide's events (more) find no room; the next
    frames are those of an object of the same history without that frame."""
    import torch
    scene = Scene(box_objects)
    out, huge = torch.zeros(64 * 48 * 3, device="cuda"), torch.zeros(16384 * 8192 * 3, device="cuda")

    def frame(on, w, h, f, to):
        par = make_params(spp=1, max_depth=5, frame_offset=f)
        if what == "cache":
            on.render_frame(scenes.box_camera(w, h), par, to.data_ptr(), None, train=False)
        else:
            on.render_frame(scenes.box_camera(w, h), par, to.data_ptr(), None)
        torch.cuda.synchronize()
        return to[:w * h * 3].cpu().numpy()

    def start():   # a first frame, so that there is something to outgrow
        on = RadianceCache(scene, nrc_config(log2_entries=10, train_paths=64)) if what == "cache" else PathGuide(scene)
        frame(on, 64, 48, 9, out)
        return on
    ref = frame(start(), 64, 48, 0, out)
    on = start()
    with Short(1.5 * GIB):
        with pytest.raises(ArError, match="OUT_OF_MEMORY"):
            frame(on, 16384, 8192, 0, huge)
        got = frame(on, 64, 48, 0, out)
    if what == "cache":
        np.testing.assert_allclose(got, ref, rtol=1e-6, atol=1e-7)
    else:   # the probes' sums depend on the order of additions
        assert abs(got.mean() / ref.mean() - 1) < 0.02
