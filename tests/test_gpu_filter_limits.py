"""What the post-filters refuse: a joint bilateral radius above 120 (over 58,000 taps per pixel) and images of
more than 65,535 blocks of eight rows; and that they take what lies just below.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import B, R
from test_gpu_filter_tiles import images, ptrs
from test_gpu_parity import FLOOR, TOL, max_rel_err

pytestmark = pytest.mark.gpu

ERR_CUDA = 5


@pytest.mark.parametrize("sigma_p", [40.1, 1e3, 1e8, 1e30])
def test_wide_bilateral_is_refused(gpu_ctx, sigma_p):
    a = images(5, 4, False)
    with pytest.raises(R.RpdError) as e:
        gpu_ctx.joint_bilateral(*a, 0.3, 0.6, sigma_p, 0.1)
    assert e.value.status == ERR_CUDA
    gpu_ctx.joint_bilateral(*a, 0.3, 0.6, 1.0, 0.1)  # the context works on


def test_widest_bilateral(gpu_ctx):
    w, h = 9, 6
    a = images(w, h, False)
    got = gpu_ctx.joint_bilateral(*a, 0.3, 0.6, 40.0, 0.1)
    want = [np.empty_like(a[0]) for _ in range(3)]
    B.port().orc_joint_bilateral(*ptrs(*a), w, h, 0.3, 0.6, 40.0, 0.1, *ptrs(*want), 1)
    # two single-precision sums of n positive terms on either side, each within n 2^-24 of its value
    n = 241 * 241
    for x, y in zip(got, want):
        assert np.all(np.abs(x - y) <= 4 * n * 2.0**-24 * np.abs(y))


def test_tall_images(gpu_ctx):
    h = 65535 * 8
    a = [np.ascontiguousarray(np.broadcast_to(x, (h + 1, 1, 3))) for x in images(1, 1, False)]
    for call in (lambda *i: gpu_ctx.atrous(*i, 0.3, 0.2, 0.1, 3), lambda *i: gpu_ctx.joint_bilateral(*i, 0.3, 0.2, 0.3, 0.1)[0]):
        with pytest.raises(R.RpdError) as e:
            call(*a)
        assert e.value.status == ERR_CUDA
        got = call(*(x[:h] for x in a))
        assert np.allclose(got, a[0][:h], rtol=1e-5)  # a constant image stays what it is


def test_passes_beyond_the_image(gpu_ctx):
    w, h = 20, 13  # from the sixth pass on every tap but the centre's is at the border
    a = images(w, h, True)
    got = gpu_ctx.atrous(*a, 0.3, 0.6, 0.1, 28)
    want = np.empty_like(a[0])
    B.port().orc_atrous_wavelet(*ptrs(*a), w, h, 0.3, 0.6, 0.1, 28, want.ctypes.data, 1)
    assert max_rel_err(got, want, FLOOR) <= TOL  # the plain form's bar
