"""The spectral bases of a scene's materials and medium, kept per material: paths
against the oracle, which evaluates the lookup table at every hit, with the
medium attached before and after the spectral tables, changed and removed, and
by the wavefront and by the tail kernel (tables of random-init networks)."""
import numpy as np
import pytest

import oracle
import scenes
from aperture_b200 import Scene, make_params, rng_tape
from test_gpu_tail import tables


def compare(g, o):
    for f in ("segments", "uniforms", "nee_rays", "nee_depth_mask", "hit_object"):
        assert np.array_equal(g[f], o[f]), f
    err = np.abs(g["radiance"] - o["radiance"]) / np.maximum(np.abs(o["radiance"]), 1e-30)
    err[(g["radiance"] == 0) & (o["radiance"] == 0)] = 0
    assert err.max() <= 1e-5


@pytest.mark.gpu
@pytest.mark.parametrize("wave", [0, 300])
@pytest.mark.parametrize("order", ["medium first", "tables first", "replaced", "removed"])
def test_paths_equal_oracle(order, wave):
    objs, vols, med = scenes.medium_box_scene(precision=16, grid=16, medium_grid=16)
    med = dict(med, albedo=(0.9, 0.5, 0.2))
    tab = tables(11)
    cam, par = scenes.box_camera(24, 20), make_params(spp=2, max_depth=9, spectral=1, wave_paths=wave)
    gs, osc = Scene(objs, volumes=vols), oracle.OracleScene(objs, volumes=vols)
    osc.set_spectral(tab, 12)
    if order == "medium first":
        gs.set_medium(**med)
        gs.set_spectral(12, tab)
    elif order == "tables first":
        gs.set_spectral(12, tab)
        gs.set_medium(**med)
    elif order == "replaced":   # other tables and another medium before
        gs.set_spectral(7, tables(12))
        gs.set_medium(**dict(med, albedo=(0.1, 0.2, 0.3)))
        gs.set_spectral(12, tab)
        gs.set_medium(**med)
    else:
        gs.set_spectral(12, tab)
        gs.set_medium(**med)
        gs.set_medium(None)
    if order != "removed":
        osc.set_medium(**med)
    g = gs.debug_paths(cam, par)
    o, overflow = osc.render_paths(cam, par, rng_tape(cam, par, 768))
    assert overflow == 0
    assert (g["radiance"] > 0).mean() > 0.3
    compare(g, o)
