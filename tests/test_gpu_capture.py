"""Renders wait for the device, so they are refused on a stream that is being
captured into a graph.  A refused call leaves no trace: a render that continues
the one before it gets that one's generator states."""
import numpy as np
import pytest

import scenes
from aperture_b200 import ArError, Scene, make_params, render_batch


@pytest.mark.gpu
@pytest.mark.parametrize("size", [(40, 30), (640, 480)])   # one kernel for all paths; the wavefront
def test_render_on_a_capturing_stream(box_objects, size):
    import torch
    scene = Scene(box_objects)
    cam = scenes.box_camera(*size)
    out = torch.zeros(size[0] * size[1] * 3, device="cuda")

    def render(on, frame, stream=0):
        on.render_device(cam, make_params(spp=1, max_depth=5, frame_offset=frame), out.data_ptr(), stream=stream)

    def image(on, frame):
        render(on, frame)
        torch.cuda.synchronize()
        return out.cpu().numpy()
    ref = image(Scene(box_objects), 2)
    render(scene, 0)   # the next frame starts from the states that this one leaves
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        graph.capture_begin(capture_error_mode="relaxed")
        try:
            with pytest.raises(ArError, match="captur"):
                render(scene, 1, stream.cuda_stream)
            with pytest.raises(ArError, match="captur"):
                render_batch([(scene, cam, make_params(spp=1, max_depth=5), out.data_ptr(), None)], stream=stream.cuda_stream)
        finally:
            try:
                graph.capture_end()
            except RuntimeError:
                pass   # the capture was invalidated
    np.testing.assert_array_equal(image(scene, 2), ref)
    np.testing.assert_array_equal(image(scene, 1), image(Scene(box_objects), 1))
