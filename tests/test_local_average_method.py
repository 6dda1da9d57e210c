"""The 3x3 average of the window's sqrt variances (csrc/k_statmc.cu, local_average) restated in numpy
singles and checked against the reference's nine double additions: wherever the sums of exact-error pairs
round to one float with 2^-40 added or taken away, that float is the reference's, and all but ties
do. Values spread over one, ten and thirty orders of magnitude, equal values, and values at EPS_SMALL."""
from __future__ import annotations

import numpy as np
import pytest

F = np.float32


def two_sum(a, b):
    s = a + b
    t = s - a
    return s, (a - (s - t)) + (b - t)


def fma(a, b, c):
    # a b is exact in double; the double sum's rounding to single is off only in the error terms' last bits
    return (a.astype(np.float64) * b.astype(np.float64) + c.astype(np.float64)).astype(F)


def fast(t, wsum):
    third, inv = 1.0 / 3.0, 1.0 / wsum
    th, ih = F(third), F(inv)
    tl, il = F(third - float(th)), F(inv - float(ih))
    c0, e0 = two_sum(t[0], t[2])
    c1, e1 = two_sum(t[6], t[8])
    ch, e2 = two_sum(c0, c1)
    cl = (e0 + e1) + e2
    d0, e3 = two_sum(t[1], t[7])
    d1, e4 = two_sum(t[3], t[5])
    dh, e5 = two_sum(d0, d1)
    dl = (e3 + e4) + e5
    ph = ch * th
    pl = fma(ch, np.full_like(ch, th), -ph) + fma(ch, np.full_like(ch, tl), cl * th)
    s, e6 = two_sum(ph, F(0.5) * dh)
    total, e7 = two_sum(s, t[4])
    low = ((e6 + e7) + pl) + F(0.5) * dl
    q = total * ih
    ql = fma(total, np.full_like(q, ih), -q) + fma(total, np.full_like(q, il), low * ih)
    m = F(9.094947e-13)
    return q + fma(q, np.full_like(q, m), ql), q + fma(q, np.full_like(q, -m), ql)


@pytest.mark.parametrize("decades", [0, 1, 10, 30])
def test_decided_values_are_the_references(decades):
    rng = np.random.default_rng(decades)
    n = 400_000
    if decades:
        t = (10.0 ** rng.uniform(-decades / 2, decades / 2, size=(9, n))).astype(F)
    else:
        t = np.repeat(rng.uniform(0.1, 4.0, size=(1, n)), 9, axis=0).astype(F)
        t[:, ::3] = F(1e-8)
        t[4, ::5] = F(1e-8)
    w = [1.0 / 3.0, 0.5, 1.0 / 3.0, 0.5, 1.0, 0.5, 1.0 / 3.0, 0.5, 1.0 / 3.0]
    acc, wsum = np.zeros(n), 0.0
    for k in range(9):
        acc = acc + t[k].astype(np.float64) * w[k]
        wsum += w[k]
    want = (acc / wsum).astype(F)
    up, down = fast(t, wsum)
    decided = up == down
    assert np.array_equal(up[decided], want[decided])
    # ties: the average is a sum of floats over 26, a multiple of 13 halves of an ulp one time in 13, and
    # halfway where its lowest bit is set too; fewer when the values differ in size
    assert np.mean(decided) >= 1 - 1.5 / 26 or decades == 0
