"""How many paths the kernel of the last paths takes over in scenes with SDF
objects or a medium: fewer per lane than elsewhere, fewest with four
wavelengths.  Around those counts both routes trace the same paths."""
import pytest

from aperture_b200 import RenderStats, make_params
from test_gpu_tail import LANES, same, scene_of


def launches(scene, cam, **par):
    import torch
    st = RenderStats()
    out = torch.zeros(cam.width * cam.height * 3, device="cuda")
    scene.render_device(cam, make_params(**par), out.data_ptr(), stats=st)
    return st.kernel_launches


@pytest.mark.gpu
@pytest.mark.parametrize("spectral,per_lane", [(0, 2), (1, 2), (4, 1)])
def test_limit_of_scenes_with_marching(spectral, per_lane):
    import torch
    limit = per_lane * LANES * torch.cuda.get_device_properties(0).multi_processor_count
    scene, camera = scene_of("medium")
    par = dict(spp=1, max_depth=4, spectral=spectral)
    alone = launches(scene, camera(40, 30), **par)
    assert launches(scene, camera(limit, 1), **par) == alone
    assert launches(scene, camera(limit + 1, 1), **par) > alone
    for n in (limit, limit + 1):
        cam = camera(n, 1)
        same(scene.debug_paths(cam, make_params(**par)), scene.debug_paths(cam, make_params(wave_paths=n // 2, **par)))


@pytest.mark.gpu
def test_limit_of_other_scenes():
    import torch
    n = 4 * LANES * torch.cuda.get_device_properties(0).multi_processor_count
    scene, camera = scene_of("box")
    alone = launches(scene, camera(40, 30), spp=1, max_depth=4)
    assert launches(scene, camera(n, 1), spp=1, max_depth=4) == alone < launches(scene, camera(n + 1, 1), spp=1, max_depth=4)
