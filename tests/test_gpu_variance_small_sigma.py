"""The variance stabilisation under an adaptive_sigma_max whose square is below EPS_SMALL (1e-8), against the
oracle bit for bit: the clamp's upper bound then wins over its lower one, and the iterations of a pixel with a
primary hit raise what it leaves to EPS_SMALL again. Compiled radii and the general one; a square
just below and just above EPS_SMALL, a denormal one and one that vanishes.
"""
from __future__ import annotations

import pytest

from conftest import B, R, small_config
from test_gpu_variance_bounds import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sigma_max", [1.1e-4, 9.9e-5, 5e-5, 1e-12, 1e-21, 1e-30])
@pytest.mark.parametrize("radius,iterations", [(1, 1), (2, 2), (3, 3), (4, 2), (5, 2)])
def test_matches_the_oracle(gpu_ctx, sigma_max, radius, iterations):
    w, h = 37, 21
    cfg = small_config(w, h, rpf_tile_size=8, color_window_radius=1, var_window_radius=radius,
                       var_iterations=iterations, var_compat_sigma=3.0, adaptive_sigma_max=sigma_max)
    check(gpu_ctx, cfg, B.synth_fill(R.synth_params(w, h, 6, miss_regions=4), 0, w * h, 4), 4)
