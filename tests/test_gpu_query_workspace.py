"""Ray queries use the workspace that a render of any size left: they neither
allocate nor free, so they do not wait for other work of the device."""
import numpy as np
import pytest

import scenes
from aperture_b200 import Scene, make_params


@pytest.mark.gpu
@pytest.mark.parametrize("size", [(64, 48), (700, 500)])   # path state in the workspace; in a block of its own
def test_query_after_a_render_keeps_the_workspace(box_objects, size):
    import torch
    scene, first = Scene(box_objects), Scene(box_objects)
    rays = torch.from_numpy(np.tile(np.float32([0, 0, 0, 0, 0.3, 0.5, 0.8, 1e30]), (100, 1))).cuda()
    hits, out = torch.zeros(100, dtype=torch.int32, device="cuda"), torch.zeros(size[0] * size[1] * 3, device="cuda")
    work, side = torch.cuda.Stream(), torch.cuda.Stream()

    def query(on):
        on.trace_rays_device(rays.data_ptr(), 100, False, hits.data_ptr(), None, stream=side.cuda_stream)
    query(first)   # loads the kernel
    scene.render_device(scenes.box_camera(*size), make_params(spp=1, max_depth=4), out.data_ptr())
    with torch.cuda.stream(work):
        torch.cuda._sleep(1000)   # loads this one
    torch.cuda.synchronize()
    ended = torch.cuda.Event()
    with torch.cuda.stream(work):
        torch.cuda._sleep(1_000_000_000)   # about half a second, one thread
        ended.record()
    query(scene)   # returns when the hits are there
    waited = ended.query()
    torch.cuda.synchronize()
    assert not waited
