"""The statistics pass where a pixel's samples are read one by one (its work split over two warps) and
where its quotients by the count come from one reciprocal, against the oracle bit for bit: pixel counts
around the 64 of a block, 1 to 6 samples per pixel and per-pixel counts with empty pixels, FP32 and
compact planes, and radiance for which a quotient's fast form does not hold: near the type's limits
(differences overflow), tiny, denormal, zero and negative zero.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import B, R, assert_bitwise, small_config
from test_gpu_accumulate_rows import FIELDS, samples
from test_gpu_compact_exact import decode

pytestmark = pytest.mark.gpu


def extreme(s, seed):
    rng = np.random.default_rng(seed)
    L = s.planes["radiance"]
    values = np.array([2e38, -2e38, 3e-39, -1e-45, 1e-21, 0.0, -0.0, 1e-30, 7.5, 1e19], np.float32)
    pick = rng.random(L.shape) < 0.5
    L[pick] = rng.choice(values, size=int(pick.sum()))
    return s


def same(a, b, name):
    if a.dtype.kind == "f":  # any NaN for any NaN
        a, b = np.where(np.isnan(a), np.float32(1), a), np.where(np.isnan(b), np.float32(1), b)
    assert_bitwise(a, b, name)


@pytest.mark.parametrize("w,h,spp,wild,sample_albedo", [(63, 1, 1, False, False), (13, 5, 2, True, True),
                                                        (64, 3, 3, False, True), (43, 29, 6, True, False),
                                                        (21, 7, 5, False, False), (33, 21, 8, True, True),
                                                        (33, 21, 16, True, False)])
def test_uniform_pushes(gpu_ctx, w, h, spp, wild, sample_albedo):
    cfg = small_config(w, h)
    g, o = R.Job(gpu_ctx, cfg), B.OracleJob(cfg, threads=1)
    for job in (g, o):
        job.begin_frame()
    for k in range(2):
        s = samples(w, h, spp, 21 + k, sample_albedo=sample_albedo)
        if wild:
            s = extreme(s, k)
        for job in (g, o):
            job.push(s, 0, w * h, spp)
            job.end_pass()
    for f in FIELDS:
        same(g.read(f), o.read(f), f)
    g.close()
    o.close()


def test_staged_rows_with_extreme_radiance(gpu_ctx):
    w, h, spp = 331, 100, 32
    cfg = small_config(w, h)
    g, o = R.Job(gpu_ctx, cfg), B.OracleJob(cfg, threads=1)
    s = extreme(samples(w, h, spp, 3), 3)
    for job in (g, o):
        job.begin_frame()
        job.push(s, 0, w * h, spp)
        job.end_pass()
    for f in FIELDS:
        same(g.read(f), o.read(f), f)
    g.close()
    o.close()


@pytest.mark.parametrize("compact", [False, True])
def test_counts(gpu_ctx, compact):
    w, h = 37, 19
    cfg = small_config(w, h)
    p = R.synth_params(w, h, 4, miss_regions=2)
    rng = np.random.default_rng(4)
    counts = rng.integers(0, 8, size=w * h).astype(np.int32)
    counts[rng.random(w * h) < 0.2] = 0
    s = B.synth_fill(p, 0, w * h, 0, counts=counts, start_n=np.zeros(w * h, np.int32))
    g = R.Job(gpu_ctx, cfg)
    planes = s
    free = []
    if compact:
        dev = R.DeviceSamples.from_host(gpu_ctx, s)
        planes = R.DeviceSamples16.encode(gpu_ctx, dev, 16.0)
        s = decode(planes)
        free = [dev, planes]
    o = B.OracleJob(cfg, threads=1)
    for job, data in ((g, planes), (o, s)):
        job.begin_frame()
        job.push(data, 0, w * h, 0, counts=counts)
        job.end_pass()
    for f in FIELDS:
        same(g.read(f), o.read(f), f)
    g.close()
    o.close()
    for d in free:
        d.free()
