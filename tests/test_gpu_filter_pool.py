"""The context's scratch pool: calls from several threads on one context give what one thread gets,
what the pool keeps between calls is bounded (512 MiB, plus the allocator's 32 MiB granularity twice)
and goes back to the device with the context."""
from __future__ import annotations

import threading

import numpy as np
import pytest

from conftest import R
from test_gpu_filter_tiles import images

pytestmark = pytest.mark.gpu


def test_threads_share_a_context(gpu_ctx):
    inputs = [images(w, h, False) for w, h in ((64, 48), (401, 97), (33, 300), (640, 360))]
    call = lambda a: [gpu_ctx.atrous(*a, 0.3, 0.2, 0.1, 3), *gpu_ctx.joint_bilateral(*a, 0.3, 0.2, 1.0, 0.1)]
    want = [call(a) for a in inputs]
    bad = []

    def work(k):
        for _ in range(5):
            for x, y in zip(call(inputs[k]), want[k]):
                if not np.array_equal(x, y):
                    bad.append(k)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(inputs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


def test_kept_memory_is_bounded_and_given_back():
    torch = pytest.importorskip("torch")
    free = lambda: torch.cuda.mem_get_info(0)[0]
    ctx = R.Context()
    a = images(64, 48, False)
    ctx.atrous(*a, 0.3, 0.2, 0.1, 1)  # modules loaded, pool in place
    before = free()
    big = [np.ascontiguousarray(np.broadcast_to(x[:1, :1], (4096, 3072, 3))) for x in a]  # 768 MiB of scratch
    ctx.atrous(*big, 0.3, 0.2, 0.1, 1)
    ctx.atrous(*a, 0.3, 0.2, 0.1, 1)
    assert before - free() <= (512 + 64) << 20
    ctx.close()
    assert free() >= before
