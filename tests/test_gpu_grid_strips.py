"""The random-dimension grid pass's strip form (uniform pushes over power-of-two node steps up to 32)
against the oracle's grid, at the edges of its blocks: image widths around the 64, 96 and 128
columns a block covers and its one-cell overlap, heights around a block's last strip, steps from one
column per cell to one cell per warp, counts that take each load width (8, 4 and single samples),
environment planes (the three-segment form), samples without some dimensions, non-finite radiance,
and a pass pushed in bands (later bands add to what the grid holds). The default mode's bar: 1e-9 of
each dependency's largest entry.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import B, R, small_config
from test_gpu_parity import assert_grid_close

pytestmark = pytest.mark.gpu

PLANES = ("radiance", "normal", "depth", "pixel_albedo", "pixel_u", "lens_u", "brdf_u", "light_u", "flags", "category")
CASES = [
    # w, h, spp, tile, env
    (127, 33, 8, 16, False),
    (128, 40, 4, 16, False),
    (129, 17, 3, 16, True),
    (136, 9, 1, 16, False),
    (95, 65, 12, 8, True),
    (64, 20, 8, 8, False),
    (65, 21, 6, 4, False),
    (33, 12, 4, 2, True),
    (140, 3, 2, 2, False),
    (200, 70, 4, 32, False),
    (97, 66, 16, 32, True),
    (260, 70, 8, 64, False),
    (70, 40, 72, 64, False),  # 16-bit lane sums would not hold: the general form
    (7, 300, 4, 16, False),
    (2000, 18, 4, 16, False),
    (16, 1200, 2, 8, True),
]


def samples(w, h, spp, env, seed):
    s = R.HostSamples(w * h * spp, w * h, PLANES + (("env_u",) if env else ()))
    base = B.synth_fill(R.synth_params(w, h, seed, miss_regions=2, nan_rate=0.01), 0, w * h, spp)
    for name, a in base.planes.items():
        s.planes[name][...] = a
    rng = np.random.default_rng(seed)
    flags = s.planes["flags"]
    if env:
        s.planes["env_u"][...] = rng.random(s.planes["env_u"].shape, dtype=np.float32)
        flags[rng.random(flags.size) < 0.5] |= R.ENV_VALID
    for bit in (R.BRDF_VALID, R.LENS_VALID, R.LIGHT_VALID, R.LIGHT_SELECT_VALID, R.RR_VALID, R.PIXEL_VALID):
        flags[rng.random(flags.size) < 0.05] &= np.uint8(0xFF ^ bit)
    return s


@pytest.mark.parametrize("bands", [1, 3])
@pytest.mark.parametrize("w,h,spp,tile,env", CASES)
def test_grid_matches_the_oracle(gpu_ctx, w, h, spp, tile, env, bands):
    cfg = small_config(w, h, rpf_tile_size=tile)
    s = samples(w, h, spp, env, 3 + w)
    g, o = R.Job(gpu_ctx, cfg), B.OracleJob(cfg, threads=1)
    offsets = np.arange(w * h + 1) * spp
    cuts = [w * h * k // bands for k in range(bands + 1)]
    for job in (g, o):
        job.begin_frame()
        for p0, p1 in zip(cuts, cuts[1:]):
            job.push(s.slice_pixels(offsets, p0, p1), p0, p1 - p0, spp)
        job.end_pass()
    assert_grid_close(g.read("GRID"), o.read("GRID"))
    g.close()
    o.close()
