"""The lookup table on the tensor cores against the SIMT build at sizes around its
tiles (128 voxels, five to a CTA, one CTA per SM), on tables of random-init
networks.  Both are fp32 evaluations of the same network: an entry may differ by
1e-5 of the largest magnitude, the bound the tensor build is held to."""
import pytest

from aperture_b200 import LUT_SIMT, LUT_TENSOR, spectral_rgb_lut
from test_gpu_tail import tables


@pytest.mark.gpu
@pytest.mark.parametrize("res", [2, 5, 8, 9, 17, 43, 46, 64])   # 8 voxels ... 94,720 = 148 CTAs of 5 tiles lie between 45^3 and 46^3
def test_tensor_table_equals_simt_table(res):
    import torch
    tab = tables(res)
    pad = torch.full((res ** 3 * 4 + 1024,), 7.0, dtype=torch.float32, device="cuda")
    a, _ = spectral_rgb_lut(res, LUT_SIMT, tab)
    b, _ = spectral_rgb_lut(res, LUT_TENSOR, tab, out=pad)
    b = pad[:res ** 3 * 4]
    assert bool((pad[res ** 3 * 4:] == 7.0).all())
    assert bool(torch.isfinite(b).all())
    assert float((a - b).abs().max()) <= 1e-5 * float(a.abs().max())
