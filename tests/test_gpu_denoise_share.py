"""The denoiser's filter on statistics at the edges of its t-test: whole degrees
of freedom (equal variances), shares at the quantiles, table ends, sums near the
ends of the float range, zero variance and pixels without samples."""
import numpy as np
import pytest

import aperture_b200 as ab
import oracle
from test_gpu_denoise import TQ, filter_inputs, to_dev


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["equal", "border", "scales", "counts"])
@pytest.mark.parametrize("w,h", [(33, 9), (64, 16), (31, 7)])
def test_bilateral_at_the_edges_of_the_t_test(kind, w, h):
    import torch
    img, g, s = filter_inputs(w, h, 5, 31 * w + h)
    rng = np.random.default_rng(w)
    n = w * h
    s["num"] = 8
    s["m3_div_n"] = 0.0
    if kind == "equal":      # nu = 2 (n - 1) exactly for every pair
        s["m2_div_n"] = 0.25
        s["mean"] = rng.normal(size=(n, 3)).astype(np.float32)
    elif kind == "border":   # two groups of means whose differences lie a few floats around the quantile at nu = 14
        v = (0.25 * (1 + rng.integers(-8, 9, (n, 3)) * 2.0 ** -23)).astype(np.float32)
        s["m2_div_n"] = v
        x = float(TQ[13]) ** 2
        share = 1.0 - 0.5 / (1.0 + x)
        t = np.sqrt((0.25 / 7.0) * (2.0 * share - 1.0) / (1.0 - share))
        k = rng.integers(-24, 25, (n, 1)) * 2.0 ** -23
        s["mean"] = (rng.integers(0, 2, (n, 1)) * t * (1 + k) * np.ones(3)).astype(np.float32)
    elif kind == "scales":   # variances over the whole float range, zeros among them
        s["m2_div_n"] = np.exp(rng.uniform(-95.0, 88.0, (n, 3))).astype(np.float32) * (rng.random((n, 1)) < 0.9)
        s["mean"] = (rng.normal(size=(n, 3)) * np.exp(rng.uniform(-20, 20, (n, 1)))).astype(np.float32)
    else:                    # sample counts from none to past the end of the table
        s["num"] = rng.choice([0, 1, 2, 3, 16, 511, 512, 513, 514, 4000, 1 << 20], n)
        s["m2_div_n"] = (0.25 * (1 + rng.integers(0, 3, (n, 3)))).astype(np.float32)
        s["mean"] = (0.01 * rng.normal(size=(n, 3))).astype(np.float32)
    ref = oracle.dn_bilateral(img, g, s, w, h, TQ)
    out = torch.full((n * 3,), float("nan"), dtype=torch.float32, device="cuda")
    ab.denoise_bilateral(torch.from_numpy(img.reshape(-1)).cuda(), out, to_dev(g), to_dev(s), w, h)
    got = out.cpu().numpy()
    assert np.array_equal(got.view(np.uint32), ref.view(np.uint32)), np.nanmax(np.abs(got - ref))
