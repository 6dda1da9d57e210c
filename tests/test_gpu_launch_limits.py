"""Launches whose shared-memory tile depends on a radius, from several threads at once: the kernel's limit is one
for all calls, so a thread with a small tile must not lower it under one with a large tile. Joint
bilaterals of radius 6, 9 and 15 on one context, variance stabilisations of radius 5, 9 and 14 on a job each;
every call gives what it gives alone.
"""
from __future__ import annotations

import threading

import numpy as np
import pytest

from conftest import B, R, small_config
from test_gpu_filter_tiles import images

pytestmark = pytest.mark.gpu


def together(calls, repeats):
    """Each call alone, then all at once on their own threads, `repeats` times each."""
    want = [call() for call in calls]
    bad = []

    def work(k):
        try:
            for _ in range(repeats):
                if not all(np.array_equal(x, y) for x, y in zip(calls[k](), want[k])):
                    bad.append((k, "differs"))
        except R.RpdError as e:
            bad.append((k, str(e)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad[:3]


def test_bilaterals_of_several_radii(gpu_ctx):
    a = images(33, 17, False)
    together([lambda s=s: gpu_ctx.joint_bilateral(*a, 0.3, 0.2, s, 0.1) for s in (2.0, 3.0, 5.0, 2.0)], 300)


def test_variances_of_several_radii(gpu_ctx):
    w, h, spp = 33, 18, 2
    s = B.synth_fill(R.synth_params(w, h, 7, miss_regions=2), 0, w * h, spp)
    jobs = []
    for radius in (5, 9, 14, 5):
        job = R.Job(gpu_ctx, small_config(w, h, color_window_radius=1, var_window_radius=radius))
        job.begin_frame()
        job.push(s, 0, w * h, spp)
        job.end_pass()
        job.recompute_sensitivity()
        jobs.append(job)

    def call(job):
        job.variance_denoise()
        return [job.read("VARIANCE_DENOISED")]

    together([lambda j=j: call(j) for j in jobs], 300)
    for job in jobs:
        job.close()
