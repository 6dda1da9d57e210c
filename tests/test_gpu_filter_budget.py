"""What a context keeps of its filters' scratch, its buffers and its jobs stay within its budget together: a
small budget bounds it from the start, a buffer that takes most of the budget makes the context give the
scratch back, and freeing the buffer lets it keep again. (Device memory is told apart to the allocator's
32 MiB granularity, twice.)
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import R
from test_gpu_filter_tiles import images

pytestmark = pytest.mark.gpu

MB = 1 << 20
SLACK = 64 * MB


def test_kept_scratch_follows_the_budget():
    torch = pytest.importorskip("torch")
    free = lambda: torch.cuda.mem_get_info(0)[0]
    small = images(64, 48, False)
    big = [np.ascontiguousarray(np.broadcast_to(x[:1, :1], (1024, 2048, 3))) for x in small]  # 200 MiB of scratch
    call = lambda ctx, a: ctx.atrous(*a, 0.3, 0.2, 0.1, 1)
    warm = R.Context()
    call(warm, small)
    warm.close()
    before = free()
    ctx = R.Context(0, 16 * MB)
    call(ctx, big)
    call(ctx, small)
    assert before - free() <= 16 * MB + SLACK
    ctx.close()
    ctx = R.Context(0, 256 * MB)
    call(ctx, big)
    assert before - free() >= 150 * MB  # kept
    buf = R.DeviceBuffer(ctx, 240 * MB)
    assert before - free() <= 256 * MB + SLACK
    call(ctx, big)
    call(ctx, small)
    assert before - free() <= 256 * MB + SLACK
    buf.free()
    call(ctx, big)
    assert 150 * MB <= before - free() <= 256 * MB + SLACK
    ctx.close()
    assert free() >= before
