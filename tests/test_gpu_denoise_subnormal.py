"""The denoiser's filter where variances are a few units of the smallest float:
their quotients by the sample count round to zero, so two such pixels have no
degrees of freedom (0 / 0, looked up as 1), while their means are ordinary."""
import numpy as np
import pytest

import aperture_b200 as ab
import oracle
from test_gpu_denoise import TQ, filter_inputs, to_dev


@pytest.mark.gpu
@pytest.mark.parametrize("share", [0.0, 0.5, 1.0])
@pytest.mark.parametrize("w,h", [(33, 9), (40, 24)])
def test_bilateral_of_subnormal_variances(w, h, share):
    """share: of the pixels whose variance is exactly zero (infinite or NaN theta)."""
    import torch
    img, g, s = filter_inputs(w, h, 5, 31 * w + h)
    rng = np.random.default_rng(w)
    n = w * h
    s["num"] = 8
    s["m3_div_n"] = 0.0
    m2 = (rng.integers(1, 4, (n, 3)).astype(np.uint32)).view(np.float32)   # 1 to 3 times 2^-149
    s["m2_div_n"] = np.where(rng.random((n, 1)) < share, np.float32(0), m2)
    # differences whose share t^2 / 1e-6 lies from below one half to one
    s["mean"] = (np.sqrt(rng.choice([0.0, 0.4e-6, 0.6e-6, 0.94e-6, 0.97e-6, 0.999e-6], (n, 1))) * np.ones(3)).astype(np.float32)
    ref = oracle.dn_bilateral(img, g, s, w, h, TQ)
    out = torch.full((n * 3,), float("nan"), dtype=torch.float32, device="cuda")
    ab.denoise_bilateral(torch.from_numpy(img.reshape(-1)).cuda(), out, to_dev(g), to_dev(s), w, h)
    got = out.cpu().numpy()
    assert np.array_equal(got.view(np.uint32), ref.view(np.uint32)), np.nanmax(np.abs(got - ref))
