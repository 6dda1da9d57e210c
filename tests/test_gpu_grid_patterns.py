"""Pixels of more validity patterns than the statistics pass keeps (a tracer's samples with lights, an
environment and Russian roulette hold up to eight), in the strip form of the grid's totals and screen bins: every
pixel of that kind or a few among others; with positions in their pixel's bin, at its edges and
anywhere; with and without samples that lack the position; uniform pushes, per-pixel counts and bands.
Against the oracle's grid at the default mode's bar. And such a frame's grid pass costs a small multiple of one
with a single pattern: seven classes of one walk each, beside the bins' updates, where sample by sample
it was three hundred times as much.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import B, R, small_config
from test_gpu_grid_totals import EDGES
from test_gpu_parity import assert_grid_close

pytestmark = pytest.mark.gpu

DIMS = (R.LENS_VALID, R.BRDF_VALID, R.LIGHT_VALID, R.LIGHT_SELECT_VALID, R.RR_VALID)
PLANES = ("radiance", "normal", "depth", "pixel_u", "lens_u", "brdf_u", "light_u", "env_u", "flags", "category", "pixel_albedo")


def samples(w, h, counts, seed, pixels, edge=0.0, lost=0.0, env=True, position=True):
    """pixels: the share of pixels whose samples drop dimensions at random; edge, lost: of samples at
    edge positions and without one; position: is there a pixel_u plane?"""
    base = B.synth_fill(R.synth_params(w, h, seed, miss_regions=2, nan_rate=0.01), 0, w * h, 0, counts=counts,
                        start_n=np.zeros(w * h, np.int32))
    s = R.HostSamples(base.n_samples, w * h, tuple(p for p in PLANES if (env or p != "env_u") and (position or p != "pixel_u")))
    rng = np.random.default_rng(seed)
    for name, plane in s.planes.items():
        plane[...] = base.planes[name] if name in base.planes else rng.random(plane.shape, dtype=np.float32)
    flags = s.planes["flags"]
    some = np.repeat(rng.random(w * h) < pixels, counts)
    if env:
        flags[some & (rng.random(flags.size) < 0.5)] |= R.ENV_VALID
    for bit in DIMS:
        flags[some & (rng.random(flags.size) < 0.4)] &= np.uint8(0xFF ^ bit)
    flags[some & (rng.random(flags.size) < lost)] &= np.uint8(0xFF ^ R.PIXEL_VALID)
    if position and edge:
        for plane in s.planes["pixel_u"]:
            at = rng.random(plane.size) < edge
            plane[at] = rng.choice(EDGES, int(at.sum()))
    return s


@pytest.mark.parametrize("w,h,spp,tile,bands,kw", [
    (200, 200, 8, 16, 1, dict(pixels=1.0)),
    (193, 211, 9, 16, 2, dict(pixels=0.05)),
    (161, 161, 8, 8, 1, dict(pixels=1.0, edge=0.2)),
    (161, 163, 0, 8, 2, dict(pixels=0.5, edge=0.05)),
    (200, 200, 8, 16, 1, dict(pixels=1.0, edge=1.0, env=False)),
    (200, 200, 8, 16, 2, dict(pixels=0.5, lost=0.2)),
    (97, 64, 12, 4, 1, dict(pixels=1.0, lost=0.05, edge=0.3)),
    (400, 400, 6, 32, 1, dict(pixels=1.0, lost=0.01)),
    (417, 384, 0, 32, 2, dict(pixels=1.0, lost=0.3, edge=0.1)),
    (200, 200, 33, 16, 1, dict(pixels=0.02, lost=0.1, edge=0.02)),
    (200, 200, 64, 16, 1, dict(pixels=0.3, edge=0.02)),
    (200, 200, 8, 16, 1, dict(pixels=1.0, position=False)),
])
def test_grid_matches_the_oracle(gpu_ctx, w, h, spp, tile, bands, kw):
    cfg = small_config(w, h, rpf_tile_size=tile)
    rng = np.random.default_rng(w)
    g, o = R.Job(gpu_ctx, cfg), B.OracleJob(cfg, threads=1)
    cuts = [w * h * k // bands for k in range(bands + 1)]
    for job in (g, o):
        job.begin_frame()
    for p in range(2):  # two passes of one frame
        counts = (rng.integers(0, 12, w * h) if spp == 0 else np.full(w * h, spp)).astype(np.int32)
        s = samples(w, h, counts, 21 + p, **kw)
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


@pytest.mark.parametrize("kw", [dict(pixels=1.0), dict(pixels=1.0, edge=1e-3)])
def test_cost_of_many_patterns(gpu_ctx, kw):
    w, h, spp = 960, 540, 16
    cfg = small_config(w, h)
    job = R.Job(gpu_ctx, cfg)
    ms = []
    for k in (dict(pixels=0.0), kw):
        dev = R.DeviceSamples.from_host(gpu_ctx, samples(w, h, np.full(w * h, spp, np.int32), 3, **k))
        job.set_profiling(True)
        for run in range(4):
            if run == 1:
                job.sync()
                job.reset_kernel_times()
            job.begin_frame()
            job.push(dev, 0, w * h, spp)
            job.end_pass()
        job.sync()
        ms.append(job.kernel_times()["grid"][0])
        dev.free()
    job.close()
    assert ms[1] <= 25 * ms[0], ms
