"""The grid pass's totals and screen bins in strips (supports 4 to 32, more than 512 nodes) against the
oracle's grid: screen positions at and beyond their pixel's ends, where the reference's rounding (or
the position itself) puts a sample in another bin than its pixel's; pixels of one, three and more
validity patterns, with and without the screen position; uniform pushes and per-pixel counts, bands
(later ones add to what the grid holds) and several passes; widths around the 32 columns a warp
covers. The default mode's bar: 1e-9 of each dependency's largest entry.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import B, R, small_config
from test_gpu_parity import assert_grid_close

pytestmark = pytest.mark.gpu

EDGES = np.array([0.0, 1.0, 1.0 - 2.0 ** -24, 1.0 - 2.0 ** -13, 1.0 - 2.0 ** -11, 2.0 ** -30, -2.0 ** -30, -0.25, 1.5,
                  0.25, 0.5], dtype=np.float32)
CASES = [
    # w, h, spp (0: per-pixel counts), tile, share of edge positions, share of flags changed
    (200, 200, 4, 16, 0.0, 0.0),
    (200, 197, 4, 16, 0.3, 0.0),
    (193, 200, 3, 8, 0.1, 0.02),
    (161, 161, 0, 8, 0.3, 0.1),
    (225, 230, 2, 16, 0.01, 0.3),
    (97, 64, 4, 4, 0.3, 0.05),
    (400, 400, 2, 32, 0.1, 0.05),
    (417, 384, 0, 32, 0.3, 0.3),
    (33, 9000, 1, 16, 0.1, 0.05),
]


def samples(w, h, counts, edge, change, seed):
    s = B.synth_fill(R.synth_params(w, h, seed, miss_regions=2, nan_rate=0.01), 0, w * h, 0, counts=counts,
                     start_n=np.zeros(w * h, np.int32))
    rng = np.random.default_rng(seed)
    pu, flags = s.planes["pixel_u"], s.planes["flags"]
    for c in range(2):
        at = rng.random(pu.shape[1]) < edge
        pu[c][at] = rng.choice(EDGES, int(at.sum()))
    for bit in (R.PIXEL_VALID, R.LENS_VALID, R.BRDF_VALID, R.LIGHT_VALID, R.LIGHT_SELECT_VALID, R.RR_VALID):
        flags[rng.random(flags.size) < change] &= np.uint8(0xFF ^ bit)
    return s


@pytest.mark.parametrize("bands", [1, 3])
@pytest.mark.parametrize("w,h,spp,tile,edge,change", CASES)
def test_grid_matches_the_oracle(gpu_ctx, w, h, spp, tile, edge, change, bands):
    cfg = small_config(w, h, rpf_tile_size=tile)
    rng = np.random.default_rng(w)
    g, o = R.Job(gpu_ctx, cfg), B.OracleJob(cfg, threads=1)
    cuts = [w * h * k // bands for k in range(bands + 1)]
    for job in (g, o):
        job.begin_frame()
    for p in range(2):  # two passes of one frame
        counts = (rng.integers(0, 6, w * h) if spp == 0 else np.full(w * h, spp)).astype(np.int32)
        s = samples(w, h, counts, edge, change, 11 + p)
        offsets = np.concatenate([[0], np.cumsum(counts)])
        for job in (g, o):
            for p0, p1 in zip(cuts, cuts[1:]):
                part = s.slice_pixels(offsets, p0, p1)
                if spp:
                    job.push(part, p0, p1 - p0, spp)
                else:
                    job.push(part, p0, p1 - p0, 0, counts=counts[p0:p1])
            job.end_pass()
    assert_grid_close(g.read("GRID"), o.read("GRID"))
    g.close()
    o.close()
