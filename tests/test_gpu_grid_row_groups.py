"""The random dimensions' strips on small images of many samples per pixel, where two row groups share a strip although
the blocks walk more strips: against the oracle's grid, with and without environment planes, bands of odd
cuts, sample counts that load in eights, fours and one by one.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import B, R, small_config
from test_gpu_accumulate_rows import samples
from test_gpu_parity import assert_grid_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,spp,tile,env", [(256, 256, 32, 16, False), (255, 251, 36, 16, False), (257, 200, 33, 8, False),
                                              (300, 180, 32, 8, True)])
@pytest.mark.parametrize("bands", [1, 2])
def test_grid_matches_the_oracle(gpu_ctx, w, h, spp, tile, env, bands):
    cfg = small_config(w, h, rpf_tile_size=tile)
    g, o = R.Job(gpu_ctx, cfg), B.OracleJob(cfg)
    s = samples(w, h, spp, 12, env)
    offsets = np.arange(w * h + 1) * spp
    cuts = [0, w * h] if bands == 1 else [0, w * h // 3 + 7, w * h]
    for job in (g, o):
        job.begin_frame()
        for p0, p1 in zip(cuts, cuts[1:]):
            job.push(s.slice_pixels(offsets, p0, p1), p0, p1 - p0, spp)
        job.end_pass()
    assert_grid_close(g.read("GRID"), o.read("GRID"))
    g.close()
    o.close()
