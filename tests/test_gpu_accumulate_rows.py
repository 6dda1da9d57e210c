"""The statistics pass on staged rows (uniform pushes of 32 samples per pixel and more, a million
samples) against the oracle, bit for bit: the pixel statistics and feature sums of FP32 planes, with
albedo per sample or per pixel, environment planes, samples without a hit, non-finite radiance, mixed
validity patterns, a count of pixels that is no multiple of 32 and a second push on top of the first;
and of compact planes against the FP32 push of the decoded samples.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import B, R, assert_bitwise, small_config
from test_gpu_compact_exact import decode
from test_gpu_parity import EXACT_FIELDS, assert_grid_close

pytestmark = pytest.mark.gpu

FIELDS = [f for f in EXACT_FIELDS if f != "GRID"]
PLANES = ("radiance", "normal", "depth", "pixel_u", "lens_u", "brdf_u", "light_u", "flags", "category")


def samples(w, h, spp, seed, env=False, sample_albedo=False):
    planes = PLANES + (("env_u",) if env else ()) + (("albedo",) if sample_albedo else ("pixel_albedo",))
    s = R.HostSamples(w * h * spp, w * h, planes)
    base = B.synth_fill(R.synth_params(w, h, seed, miss_regions=3, nan_rate=0.01), 0, w * h, spp)
    for name in planes:
        if name in base.planes:
            s.planes[name][...] = base.planes[name]
    rng = np.random.default_rng(seed)
    if sample_albedo:
        s.planes["albedo"][...] = rng.random(s.planes["albedo"].shape, dtype=np.float32)
    flags = s.planes["flags"]
    if env:
        s.planes["env_u"][...] = rng.random(s.planes["env_u"].shape, dtype=np.float32)
        flags[rng.random(flags.size) < 0.3] |= R.ENV_VALID
    flags[rng.random(flags.size) < 0.2] &= np.uint8(0xFF ^ R.RR_VALID)
    flags[rng.random(flags.size) < 0.02] &= np.uint8(0xFF ^ R.HIT)
    return s


@pytest.mark.parametrize("w,h,spp,env,sample_albedo", [(183, 90, 64, False, False), (331, 100, 32, True, True),
                                                       (219, 100, 48, False, True), (150, 98, 72, True, False)])
def test_fp32_statistics_match_the_oracle(gpu_ctx, w, h, spp, env, sample_albedo):
    cfg = small_config(w, h)
    g, o = R.Job(gpu_ctx, cfg), B.OracleJob(cfg, threads=1)
    for job in (g, o):
        job.begin_frame()
    for k in range(2):  # the second push adds to the first's statistics
        s = samples(w, h, spp, 5 + k, env, sample_albedo)
        assert s.n_samples >= 1 << 20
        for job in (g, o):
            job.push(s, 0, w * h, spp)
            job.end_pass()
    for f in FIELDS:
        assert_bitwise(g.read(f), o.read(f), f)
    assert_grid_close(g.read("GRID"), o.read("GRID"))
    g.close()
    o.close()


@pytest.mark.parametrize("w,h,spp", [(183, 90, 64), (331, 100, 32)])
def test_compact_statistics_match_the_decoded_samples(gpu_ctx, w, h, spp):
    cfg = small_config(w, h)
    s = samples(w, h, spp, 9)
    dev = R.DeviceSamples.from_host(gpu_ctx, s)
    c16 = R.DeviceSamples16.encode(gpu_ctx, dev, 16.0)
    a, b = R.Job(gpu_ctx, cfg), R.Job(gpu_ctx, cfg)
    decoded = R.DeviceSamples.from_host(gpu_ctx, decode(c16))
    for job, planes in ((a, c16), (b, decoded)):
        job.begin_frame()
        job.push(planes, 0, w * h, spp)
        job.end_pass()
        job.sync()
    for f in FIELDS:
        assert_bitwise(a.read(f), b.read(f), f)
    assert_grid_close(a.read("GRID"), b.read("GRID"))
    for job in (a, b):
        job.close()
    for d in (dev, c16, decoded):
        d.free()
