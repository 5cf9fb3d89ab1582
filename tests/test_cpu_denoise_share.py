"""The denoiser's t-test without divisions: the share thresholds of
t_quantile_table.h, and the comparison the kernel makes with them, against the
float32 expressions they replace."""
import os
import re

import numpy as np

PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "aperturerendererv3-optix-geometry_b200")
f32 = np.float32


def header():
    text = open(os.path.join(PKG, "csrc", "t_quantile_table.h")).read()
    quant, _, share = [np.array([float.fromhex(v) for v in re.findall(r"(0x1\.[0-9a-f]+p[-+]\d+)f", part)], f32)
                    for part in text.split("static __device__ const float ")[1:]]
    least = float.fromhex(re.search(r"kShareLeast = (\S+)f;", text).group(1))
    return quant[:1024], share, f32(least)


def passes(n, d, q):
    """!(x < 0) and sqrt(x) < q for x = 0.5 / (1 - n / d) - 1, every step in float32."""
    with np.errstate(divide="ignore", invalid="ignore"):
        x = f32(0.5) / (f32(1) - n / d) - f32(1)
        return ~(x < 0) & (np.sqrt(x) < q)


def passes_shares(n, d, least, thr):
    """The kernel's form: fmaf(-c, d, n) against half the spacing below c, times d."""
    def residual(c):   # fmaf: the product of two float32 is exact in float64
        return (n.astype(np.float64) - np.float64(c) * d.astype(np.float64)).astype(f32)

    u = d * f32(2.0 ** -25)
    return (residual(least) >= f32(-0.5) * u) & (residual(thr) < -u)


def test_thresholds_are_the_first_rejected_shares():
    quant, thr, least = header()
    assert len(quant) == len(thr) == 1024
    one = np.ones_like(thr)
    assert not passes(thr, one, quant).any()
    assert passes(np.nextafter(thr, f32(0)), one, quant).all()
    assert passes(np.array([least]), f32(1), f32(2)).all()
    assert not passes(np.array([np.nextafter(least, f32(0))]), f32(1), f32(2)).any()


def test_residual_comparison_decides_like_the_divisions():
    quant, thr, least = header()
    rng = np.random.default_rng(5)
    seen = set()
    for k in list(range(40)) + [100, 511, 1022, 1023]:
        d = np.concatenate([rng.uniform(1e-6, 1e-5, 4000), rng.uniform(0.5, 2.0, 8000),
                            np.exp(rng.uniform(-13.8, 80.0, 8000))]).astype(f32)
        for c in (least, thr[k]):
            n = (d.astype(np.float64) * np.float64(c)).astype(f32)
            for step in range(-3, 4):   # the shares around each border, float by float
                m = n
                for _ in range(abs(step)):
                    m = np.nextafter(m, f32(np.inf if step > 0 else 0))
                m = np.minimum(m, d)
                a, b = passes(m, d, quant[k]), passes_shares(m, d, least, thr[k])
                assert np.array_equal(a, b)
                seen |= set(np.unique(a))
        m = (d * rng.random(len(d)).astype(f32)).astype(f32)
        assert np.array_equal(passes(m, d, quant[k]), passes_shares(m, d, least, thr[k]))
    assert seen == {False, True}
