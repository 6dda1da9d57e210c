"""Pushes that add to a frame's statistics, over several waves of blocks: where single samples are read a
pixel's two halves belong to two warps, both of which begin with its count. A uniform push, then
per-pixel counts (many 0 and 1: short walks, so that one warp ends long before the other begins if
nothing holds it back) in bands and a uniform push of one sample, against the oracle bit for bit,
several times over.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import B, R, assert_bitwise, small_config
from test_gpu_accumulate_rows import FIELDS, samples
from test_gpu_compact_exact import decode

pytestmark = pytest.mark.gpu

W, H = 640, 479  # 4790 blocks of 64 pixels, 152 SMs with 8 at a time


def pushes():
    """[(samples, first, count, spp, counts)]"""
    rng = np.random.default_rng(17)
    out = [(samples(W, H, 2, 3), 0, W * H, 2, None)]
    for k in range(2):
        counts = rng.choice(np.array([0, 1, 2, 7], np.int32), size=W * H, p=[0.4, 0.4, 0.15, 0.05])
        s = B.synth_fill(R.synth_params(W, H, 40 + k, miss_regions=2, nan_rate=0.01), 0, W * H, 0, counts=counts,
                         start_n=np.zeros(W * H, np.int32))
        offsets = np.concatenate([[0], np.cumsum(counts)])
        for p0, p1 in ((0, 150_001), (150_001, W * H)):
            out.append((s.slice_pixels(offsets, p0, p1), p0, p1 - p0, 0, np.ascontiguousarray(counts[p0:p1])))
    out.append((samples(W, H, 1, 4, sample_albedo=True), 0, W * H, 1, None))
    return out


def frame(job, parts):
    job.begin_frame()
    for s, first, count, spp, counts in parts:
        job.push(s, first, count, spp, counts=counts)
    job.end_pass()
    return {f: job.read(f) for f in FIELDS}


def on_device(gpu_ctx, part, compact, free):
    """The push's planes and counts in device memory, and the push a CPU reads (the decoded planes)."""
    s, first, count, spp, counts = part
    dev = R.DeviceSamples.from_host(gpu_ctx, s)
    free.append(dev)
    if compact:
        dev = R.DeviceSamples16.encode(gpu_ctx, dev, 16.0)
        free.append(dev)
        s = decode(dev)
    buf = None
    if counts is not None:
        buf = R.DeviceBuffer(gpu_ctx, counts.nbytes)
        buf.upload(counts)
        free.append(buf)
    return (dev, first, count, spp, buf), (s, first, count, spp, counts)


@pytest.mark.parametrize("compact", [False, True])
def test_pushes_added_to_a_frame(gpu_ctx, compact):
    cfg = small_config(W, H)
    parts = pushes()[:-1] if compact else pushes()  # compact planes hold no albedo per sample
    free = []
    both = [on_device(gpu_ctx, part, compact, free) for part in parts]
    o = B.OracleJob(cfg)
    want = frame(o, [host for _, host in both])
    o.close()
    g = R.Job(gpu_ctx, cfg)
    for _ in range(4):
        got = frame(g, [dev for dev, _ in both])
        for f in FIELDS:
            assert_bitwise(got[f], want[f], f)
    g.close()
    for d in free:
        d.free()
