"""The variance stabilisation's bounds on the ratio of two variances against the oracle's quotient, bit
for bit: block edges (32 x 16 pixels, two rows per thread), every compiled radius and the general one, one
to four iterations, thresholds from one that puts every ratio inside the uncertain band to one beyond
every ratio, variances on both sides of a threshold by a few ulps, and parameters that take the
general kernel (variances whose products overflow, a vanishing depth threshold).
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import B, R, assert_bitwise, small_config

pytestmark = pytest.mark.gpu


def check(gpu_ctx, cfg, s, spp):
    g, o = R.Job(gpu_ctx, cfg), B.OracleJob(cfg, threads=1)
    for job in (g, o):
        job.begin_frame()
        job.push(s, 0, cfg.image_width * cfg.image_height, spp)
        job.end_pass()
        job.recompute_sensitivity()
        job.statmc_denoise()
        job.variance_denoise()
    assert_bitwise(g.read("VARIANCE_DENOISED"), o.read("VARIANCE_DENOISED"), "VARIANCE_DENOISED")
    g.close()
    o.close()


@pytest.mark.parametrize("w,h,kw", [
    (1, 1, dict(var_window_radius=1, var_iterations=1)),
    (31, 15, dict(var_window_radius=1, var_iterations=3, var_compat_sigma=30.0)),
    (32, 16, dict(var_window_radius=2, var_iterations=1, var_compat_sigma=1e-6)),
    (33, 17, dict(var_window_radius=2, var_iterations=2, var_compat_sigma=0.5)),
    (65, 33, dict(var_window_radius=3, var_iterations=4, var_compat_sigma=3.0)),
    (64, 18, dict(var_window_radius=3, var_iterations=1, var_compat_sigma=1e6)),
    (35, 19, dict(var_window_radius=4, var_iterations=2, var_compat_sigma=2.0)),
    (35, 19, dict(var_window_radius=4, var_iterations=1, var_compat_sigma=1e-7)),
    (40, 21, dict(var_window_radius=5, var_iterations=2, var_compat_sigma=1.0)),
    (40, 21, dict(var_window_radius=5, var_iterations=1, var_compat_sigma=1.0)),
    (33, 18, dict(var_window_radius=3, var_compat_sigma=3.0, adaptive_sigma_max=1e10)),
    (33, 18, dict(var_window_radius=2, var_compat_sigma=3.0, var_depth_threshold=1e-30)),
    (33, 18, dict(var_window_radius=3, var_compat_sigma=3.0, var_depth_threshold=1e-3, var_normal_threshold=0.99)),
])
def test_matches_the_oracle(gpu_ctx, w, h, kw):
    cfg = small_config(w, h, rpf_tile_size=8, color_window_radius=1, **kw)
    s = B.synth_fill(R.synth_params(w, h, 31, miss_regions=3), 0, w * h, 4)
    if kw.get("adaptive_sigma_max", 0) > 1e6:
        s.planes["radiance"][...] *= np.float32(1e6)
    check(gpu_ctx, cfg, s, 4)


@pytest.mark.parametrize("sigma", [0.3, 1.0, 3.0, 17.0])
def test_ratios_on_the_threshold(gpu_ctx, sigma):
    w, h, spp = 64, 32, 2
    cfg = small_config(w, h, rpf_tile_size=8, color_window_radius=1, var_window_radius=3, var_compat_sigma=sigma,
                       var_normal_threshold=1e-3, var_depth_threshold=1e6)
    s = B.synth_fill(R.synth_params(w, h, 5), 0, w * h, spp)
    hi = ((np.sqrt(sigma * sigma + 4) + sigma) / 2) ** 2  # |1 - x| / sqrt(x) = sigma
    rng = np.random.default_rng(8)
    # grey samples 0 and d: a variance of d^2 / 2, the two kinds a threshold ratio apart but for some ulps
    wide = rng.random(w * h) < 0.5
    ulps = rng.integers(-12, 13, size=w * h) * 2.0**-24
    d = np.where(wide, 0.2 * np.sqrt(hi), 0.2) * (1 + ulps)
    L = s.planes["radiance"].reshape(3, w * h, spp)
    L[:, :, 0] = 0.0
    L[:, :, 1] = d.astype(np.float32)
    check(gpu_ctx, cfg, s, spp)
