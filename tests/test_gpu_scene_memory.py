"""What a scene holds on the device: its own data, not the constants that all
scenes of the device share (the generator's jump tables, 0.77 MB)."""
import numpy as np
import pytest

import scenes
from aperture_b200 import Scene, make_params


@pytest.mark.gpu
def test_scene_holds_no_copy_of_the_jump_tables(box_objects):
    a = Scene(box_objects)
    assert a.info().device_bytes < 100_000
    cam = scenes.box_camera(41, 7)
    par = make_params(spp=1, max_depth=3, frame_offset=12345)
    ref = a.debug_paths(cam, par)
    b = Scene(box_objects)
    a.close()
    got = b.debug_paths(cam, par)
    assert all(np.array_equal(got[f], ref[f]) for f in ref.dtype.names)


@pytest.mark.gpu
def test_workspace_of_changing_size(box_objects):
    """Images and path counts that grow and shrink, around the size up to which
    path state lies in the scene's workspace (2^18 paths), and a continued render:
    each as by a new scene."""
    shapes = [(64, 48, 1), (64, 48, 40), (300, 200, 1), (512, 512, 1), (513, 512, 1), (8, 8, 4096), (8, 8, 4097), (64, 48, 1)]

    def image(scene, w, h, spp, frame=0):
        return scene.render(scenes.box_camera(w, h), make_params(spp=spp, max_depth=4, frame_offset=frame))[0]
    one = Scene(box_objects)
    for w, h, spp in shapes:
        np.testing.assert_allclose(image(one, w, h, spp), image(Scene(box_objects), w, h, spp), rtol=1e-6, atol=1e-7)
    image(one, 31, 9, 2)
    image(one, 31, 9, 2000, 2)   # grows the path state between frames 2 and 2002
    np.testing.assert_allclose(image(one, 31, 9, 3, 2002), image(Scene(box_objects), 31, 9, 3, 2002), rtol=1e-6, atol=1e-7)
