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
