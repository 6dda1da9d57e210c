"""The importance smoothing in pairs of singles against the double-precision instructions, bit for bit, where
its guard matters: radii around the last one it takes (3), luminances for which the sums are small or
large, a black frame, opposite normals (zero weights) and distant depths (weights down to e^-8)."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import B, R, assert_bitwise, small_config
from test_gpu_smoothing import smoothed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,radius,scale", [(65, 33, 3, 1.0), (65, 33, 4, 1.0), (50, 20, 1, 1e-7), (50, 20, 2, 1e6),
                                              (33, 9, 1, 0.0), (1, 1, 1, 1.0)])
def test_pairs_equal_double_precision(gpu_ctx, w, h, radius, scale):
    cfg = small_config(w, h, adaptive_spp=4, adaptive_base_samples=1, adaptive_importance_smoothing_radius=radius)
    s = B.synth_fill(R.synth_params(w, h, 12, miss_regions=2), 0, w * h, 4)
    s.planes["radiance"][...] *= np.float32(scale)
    n = s.planes["normal"].reshape(3, w * h, 4)
    n[:, ::5] *= np.float32(-1)
    d = s.planes["depth"].reshape(w * h, 4)
    d[::7] *= np.float32(1e4)
    imp0, c0 = smoothed(gpu_ctx, cfg, s, 4, fp64=False)
    imp1, c1 = smoothed(gpu_ctx, cfg, s, 4, fp64=True)
    assert_bitwise(imp0, imp1, "smoothed importance")
    np.testing.assert_array_equal(c0, c1)
