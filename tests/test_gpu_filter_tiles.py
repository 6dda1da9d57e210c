"""The post-filters at the edges of their launch shapes against the oracle: images smaller than a
window, widths around a block's 32 columns, heights around a thread's rows (four of them `step`
apart in the a-trous pass, two adjacent ones in the joint bilateral), passes whose step exceeds the
image, bilateral radii on both sides of the shared-memory tile's limit of 16, and normals in every
direction (angles above 90 degrees take the polynomial's other branch).

The bar is the plain form's 1e-4 of each value or of the floor. The polynomial itself is evaluated in
single precision on the CPU against the arc cosine: its rounding is at most one ulp per
operation that matters (the last product and sum: 2 ulps) over a fit of 2^-23, so 4 * 2^-24 + 2^-23.
"""
from __future__ import annotations

import re
from pathlib import Path

import numpy as np
import pytest

from conftest import B, R
from test_gpu_parity import FLOOR, TOL, max_rel_err

SOURCE = Path(R.__file__).resolve().parent / "csrc" / "k_filters.cu"


def images(w, h, signed):
    rng = np.random.default_rng(w * 1000 + h)
    raw = rng.lognormal(-1.0, 0.8, size=(h, w, 3)).astype(np.float32)
    normal = rng.uniform(-1 if signed else 0, 1, size=(h, w, 3)).astype(np.float32)
    albedo = rng.uniform(0, 1, size=(h, w, 3)).astype(np.float32)
    return raw, normal, albedo


def ptrs(*arrays):
    return [a.ctypes.data for a in arrays]


@pytest.mark.gpu
@pytest.mark.parametrize("w,h,iterations,signed", [(1, 1, 2, True), (3, 40, 6, False), (31, 7, 1, True), (32, 8, 4, False),
                                                   (33, 33, 3, True), (64, 31, 2, True), (65, 129, 6, False),
                                                   (20, 13, 31, True)])
def test_atrous_groups(gpu_ctx, w, h, iterations, signed):
    raw, normal, albedo = images(w, h, signed)
    got = gpu_ctx.atrous(raw, normal, albedo, 0.3, 0.6, 0.1, iterations)
    want = np.empty_like(raw)
    # from the image's larger side on, a step's taps are all at the border: the oracle runs the same passes
    B.port().orc_atrous_wavelet(*ptrs(raw, normal, albedo), w, h, 0.3, 0.6, 0.1, min(iterations, 28), want.ctypes.data, 1)
    if iterations > 28:
        assert np.all(np.isfinite(got))  # the oracle's int steps end there
    else:
        assert max_rel_err(got, want, FLOOR) <= TOL


@pytest.mark.gpu
@pytest.mark.parametrize("w,h,sigma_p", [(1, 1, 0.2), (32, 16, 0.3), (33, 17, 2.0), (45, 29, 2.0), (96, 64, 0.3), (77, 49, 5.2),
                                         (70, 55, 5.6), (5, 3, 2.0), (129, 48, 1.0)])
def test_bilateral_tiles(gpu_ctx, w, h, sigma_p):
    raw, normal, albedo = images(w, h, False)
    got = gpu_ctx.joint_bilateral(raw, normal, albedo, 0.3, 0.6, sigma_p, 0.1)
    want = [np.empty_like(raw) for _ in range(3)]
    B.port().orc_joint_bilateral(*ptrs(raw, normal, albedo), w, h, 0.3, 0.6, sigma_p, 0.1, *ptrs(*want), 1)
    for a, b in zip(got, want):
        assert max_rel_err(a, b, FLOOR) <= TOL


@pytest.mark.gpu
def test_non_finite_neighbours_stay_in_their_windows(gpu_ctx):
    """A NaN reaches the pixels whose windows hold it, as in the oracle, and no others."""
    w, h = 70, 40
    raw, normal, albedo = images(w, h, False)
    raw[21, 40, 1] = np.nan
    normal[8, 9, 0] = np.nan
    albedo[30, 65, 2] = np.inf
    got = gpu_ctx.joint_bilateral(raw, normal, albedo, 0.3, 0.6, 1.0, 0.1)
    want = [np.empty_like(raw) for _ in range(3)]
    B.port().orc_joint_bilateral(*ptrs(raw, normal, albedo), w, h, 0.3, 0.6, 1.0, 0.1, *ptrs(*want), 1)
    for a, b in zip(got, want):
        assert np.array_equal(np.isnan(a), np.isnan(b))
    got = gpu_ctx.atrous(raw, normal, albedo, 0.3, 0.6, 0.1, 2)
    want = np.empty_like(raw)
    B.port().orc_atrous_wavelet(*ptrs(raw, normal, albedo), w, h, 0.3, 0.6, 0.1, 2, want.ctypes.data, 1)
    assert np.array_equal(np.isnan(got), np.isnan(want))


def test_angle_polynomial():
    text = SOURCE.read_text()
    body = text[text.index("void angles_squared("):]
    body = body[:body.index("a2[k] = p")]
    coefs = [np.float32(body[body.index("float p = ") + 10:].split("f;")[0])]
    coefs += [np.float32(c) for c in re.findall(r"__fmaf_rn\(p, t, (-?[\d.]+)f\)", body)]
    assert len(coefs) == 8
    d = np.unique(np.concatenate([np.linspace(0, 1, 20001), 1 - np.logspace(-7, 0, 2001)])).astype(np.float32)
    t = (np.float32(1) - d).astype(np.float32)
    p = np.full_like(t, coefs[0])
    for c in coefs[1:]:  # a fused multiply-add: exact product, one rounding
        p = (p.astype(np.float64) * t + np.float64(c)).astype(np.float32)
    p = p * t
    keep = t > 0
    # arccos loses digits near 1: its square as 4 asin^2(sqrt(t / 2))
    want = 4 * np.arcsin(np.sqrt(t.astype(np.float64) / 2)) ** 2
    assert np.max(np.abs(p[keep] - want[keep]) / want[keep]) <= 4 * 2.0**-24 + 2.0**-23
    assert np.all(p[~keep] == 0)


@pytest.mark.gpu
@pytest.mark.parametrize("w,h", [(600_000, 1), (2, 300_000)])
def test_steps_beyond_a_thin_image(gpu_ctx, w, h):
    """Steps that pass the height of a wide image and the width of a tall one, to the extent of the other side:
    the records form against the form without records, which takes one pixel per thread (the same
    arithmetic, at the no-allocation test's 1e-6)."""
    torch = pytest.importorskip("torch")
    from test_zz_no_alloc import _run_noalloc

    raw, normal, albedo = images(w, h, True)
    want = _run_noalloc(gpu_ctx, torch.cuda.Stream(), raw, normal, albedo, (0.3, 0.6, 0.1), 21)
    got = gpu_ctx.atrous(raw, normal, albedo, 0.3, 0.6, 0.1, 21)
    err = np.max(np.abs(got.astype(np.float64) - want) / np.maximum(np.abs(want), 1e-3))
    assert err <= 1e-6
