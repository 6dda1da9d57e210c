"""Uniform compact pushes of many samples per pixel: without RPD their planes are 16 bytes per sample, and the
statistics pass must take less time than over the FP32 planes of the same samples (about 0.6 of it; 0.82
in the staged form, which is for pushes with the random dimensions). With and without RPD around the sample count
where the staged form begins, compact and decoded pushes give the same bits.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import R, assert_bitwise, small_config
from test_gpu_accumulate_rows import FIELDS, samples
from test_gpu_compact_exact import decode

pytestmark = pytest.mark.gpu


def both(gpu_ctx, w, h, spp):
    dev = R.DeviceSamples.from_host(gpu_ctx, samples(w, h, spp, 9))
    c16 = R.DeviceSamples16.encode(gpu_ctx, dev, 16.0)
    return dev, c16


@pytest.mark.parametrize("spp", [32, 40, 48])
@pytest.mark.parametrize("scale", [0.0, 1.0])
def test_same_bits(gpu_ctx, spp, scale):
    w, h = 331, 100
    cfg = small_config(w, h, rpf_shrinkage_scale=scale)
    dev, c16 = both(gpu_ctx, w, h, spp)
    decoded = R.DeviceSamples.from_host(gpu_ctx, decode(c16))
    jobs = [R.Job(gpu_ctx, cfg), R.Job(gpu_ctx, cfg)]
    for job, planes in zip(jobs, (c16, decoded)):
        job.begin_frame()
        job.push(planes, 0, w * h, spp)
        job.push(planes, 0, w * h, spp)  # and on top of statistics
        job.end_pass()
        job.sync()
    for f in FIELDS:
        assert_bitwise(jobs[0].read(f), jobs[1].read(f), f)
    for o in (*jobs, dev, c16, decoded):
        (o.close if isinstance(o, R.Job) else o.free)()


def test_compact_costs_less_without_rpd(gpu_ctx):
    w, h, spp = 640, 360, 64
    job = R.Job(gpu_ctx, small_config(w, h, rpf_shrinkage_scale=0.0))
    job.set_profiling(True)
    dev, c16 = both(gpu_ctx, w, h, spp)
    ms = []
    for planes in (dev, c16):
        for run in range(6):
            if run == 2:
                job.sync()
                job.reset_kernel_times()
            job.begin_frame()
            job.push(planes, 0, w * h, spp)
            job.end_pass()
        job.sync()
        ms.append(job.kernel_times()["accumulate_pixels"][0])
    job.close()
    dev.free()
    c16.free()
    assert ms[1] <= 0.72 * ms[0], ms
