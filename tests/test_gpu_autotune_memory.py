"""The batch autotuner times no allocation: its first, untimed run takes the
largest workspaces of its candidates."""
import threading

import pytest

import scenes
from aperture_b200 import Scene, autotune_batch, make_params


@pytest.mark.gpu
def test_largest_workspaces_come_first(box_objects):
    """14 million probe paths: workspaces of 1.9 GB for 2^22 of them in flight, 3.8
    for 2^23.  The first must not be seen between nothing and the second."""
    import torch
    scene = Scene(box_objects)
    outs = [torch.zeros(1200 * 1000 * 3, device="cuda") for _ in range(3)]
    jobs = [(scene, scenes.box_camera(1200, 1000), make_params(spp=4, max_depth=4, frame_offset=4 * k), o.data_ptr(), None)
            for k, o in enumerate(outs)]
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    seen, stop = set(), threading.Event()

    def watch():
        while not stop.is_set():
            seen.add((before - torch.cuda.mem_get_info()[0]) >> 20)
    watcher = threading.Thread(target=watch)
    watcher.start()
    try:
        tuning = autotune_batch(jobs, probe_spp=4)
    finally:
        stop.set()
        watcher.join()
    assert tuning.candidates == 24
    assert not [m for m in seen if 1500 < m < 2800], sorted(seen)
