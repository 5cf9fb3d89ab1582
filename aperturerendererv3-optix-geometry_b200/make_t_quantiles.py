"""Generates csrc/t_quantile_table.h: the 0.9975 quantile of Student's t
distribution (two-sided level 0.005) for 1..1024 degrees of freedom, rounded to
float32; for each the smallest float whose square root reaches it, and the
smallest share W at which the denoiser's Welch t-test therefore rejects -- the
table the test reads (the reference's LookupTQuantile005,
core/denoise/t_quantile.cuh:15-27, holds the same quantiles;
tests/test_cpu_denoise.py checks them against a fixture of that table).

    python make_t_quantiles.py      (needs scipy; the header is committed)
"""
import os

import numpy as np
from scipy import stats

HERE = os.path.dirname(os.path.abspath(__file__))
OUT = os.path.join(HERE, "csrc", "t_quantile_table.h")


def table() -> np.ndarray:
    return stats.t.ppf(0.9975, np.arange(1, 1025)).astype(np.float32)


def sqrt_thresholds(q: np.ndarray) -> np.ndarray:
    """For each quantile q, the smallest float32 x with sqrtf(x) >= q (IEEE
    square root, correctly rounded): for x >= 0, sqrtf(x) < q exactly when
    x < threshold."""
    out = np.empty_like(q)
    for k, t in enumerate(q):
        x = np.float32(t) * np.float32(t)
        while np.sqrt(x) >= t:
            x = np.nextafter(x, np.float32(0))
        while np.sqrt(x) < t:
            x = np.nextafter(x, np.float32(np.inf))
        out[k] = x
    return out


def statistic(w: np.ndarray) -> np.ndarray:
    """The squared statistic the test forms from a share W, in float32 and in
    its order of operations: 0.5 / (1 - W) - 1."""
    w = np.asarray(w, np.float32)
    with np.errstate(divide="ignore"):
        return np.float32(0.5) / (np.float32(1.0) - w) - np.float32(1.0)


def share_threshold(x: np.ndarray) -> np.ndarray:
    """For each x >= 0, the smallest float32 W in [0, 1] with statistic(W) >= x.
    Every float32 step of statistic() is monotone, so statistic(W) >= x exactly
    when W reaches this value; found by bisection over the float's bits."""
    x = np.asarray(x, np.float32)
    lo = np.zeros(x.shape, np.int64)                                        # statistic(0) = -0.5 < x
    hi = np.full(x.shape, int(np.float32(1.0).view(np.uint32)), np.int64)   # statistic(1) = inf
    while np.any(hi - lo > 1):
        mid = (lo + hi) // 2
        reached = statistic(mid.astype(np.uint32).view(np.float32)) >= x
        hi, lo = np.where(reached, mid, hi), np.where(reached, lo, mid)
    return hi.astype(np.uint32).view(np.float32)


def main() -> None:
    vals = table()
    thr = sqrt_thresholds(vals)
    shares = share_threshold(thr)
    least = share_threshold(np.zeros(1, np.float32))[0]
    lines = ["// Generated by make_t_quantiles.py: Student t quantile 0.9975 for nu = 1..1024 (float32).",
             "// The filter reads the shares alone; the quantiles and the thresholds they derive from",
             "// are kept for the checks against their published definition.",
             "#pragma once", "", "namespace ar {", "", "constexpr int kTQuantiles = 1024;",
             "static __device__ const float kTQuantile005[kTQuantiles] = {"]
    for k in range(0, len(vals), 6):
        lines.append("    " + " ".join(f"{float(v).hex()}f," for v in vals[k:k + 6]))
    lines += ["};", "",
              "// smallest x with sqrtf(x) >= kTQuantile005[k]: sqrtf(x) < q  <=>  0 <= x < threshold",
              "static __device__ const float kTQuantileSqrtThreshold[kTQuantiles] = {"]
    for k in range(0, len(thr), 6):
        lines.append("    " + " ".join(f"{float(v).hex()}f," for v in thr[k:k + 6]))
    lines += ["};", "",
              "// smallest share W whose statistic 0.5 / (1 - W) - 1 is not negative",
              f"static constexpr float kShareLeast = {float(least).hex()}f;",
              "// smallest share W whose statistic reaches kTQuantileSqrtThreshold[k]: the test",
              "// passes exactly when kShareLeast <= W < kShareThreshold[k]",
              "static __device__ const float kShareThreshold[kTQuantiles] = {"]
    for k in range(0, len(shares), 6):
        lines.append("    " + " ".join(f"{float(v).hex()}f," for v in shares[k:k + 6]))
    lines += ["};", "", "}  // namespace ar", ""]
    with open(OUT, "w") as f:
        f.write("\n".join(lines))


if __name__ == "__main__":
    main()
