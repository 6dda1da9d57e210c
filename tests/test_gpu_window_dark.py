"""The StatMC window where the degrees-of-freedom denominator falls below 1e-8 (main.cpp:1071-1075):
black and nearly black pixels, whose df is the reference's n_i + n_j - 2 instead of the quotient.

The frames' columns run from black over radiances that put the denominator on either side of 1e-8
to ordinary ones, at counts that reach each loop of the kernel: one sample (df 0, raised to 1), two,
all n - 1 <= 15, mixed counts (non-finite samples dropped), n - 1 >= 31; both t tables and the normal
quantile; the fixed radii and the generic one.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import B, R, small_config
from test_gpu_parity import check_pipeline

pytestmark = pytest.mark.gpu

CASES = [
    # w, h, spp, radius, alpha, nan_rate
    (40, 24, 1, 5, 0.05, 0.0),
    (37, 21, 2, 3, 0.01, 0.0),
    (64, 40, 4, 5, 0.01, 0.0),
    (50, 33, 16, 7, 0.05, 0.0),
    (45, 30, 17, 5, 0.05, 0.1),
    (33, 20, 24, 2, 0.01, 0.05),
    (40, 30, 15, 5, 0.1, 0.0),
    (36, 28, 18, 3, 0.2, 0.2),
    (40, 24, 40, 5, 0.01, 0.0),
]


@pytest.mark.parametrize("w,h,spp,radius,alpha,nan_rate", CASES)
def test_dark_pixels(gpu_ctx, w, h, spp, radius, alpha, nan_rate):
    cfg = small_config(w, h, color_window_radius=radius, color_compat_alpha=alpha)
    s = B.synth_fill(R.synth_params(w, h, 31 + spp, miss_regions=2, nan_rate=nan_rate), 0, w * h, spp)
    x = np.repeat(np.arange(w * h) % w, spp)
    scale = np.where(x < w // 5, 0.0, 10.0 ** (-6.0 + 7.0 * x / w)).astype(np.float32)
    s.planes["radiance"] *= scale
    g, o = R.Job(gpu_ctx, cfg), B.OracleJob(cfg, threads=1)
    for job in (g, o):
        B.run_pipeline(job, s, spp)
    check_pipeline(g, o, exact_grid=False)
    g.close()
    o.close()
