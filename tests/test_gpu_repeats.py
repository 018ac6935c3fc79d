"""Inputs of repeats: hundreds of times the hits that the sequences' sizes let one expect."""
import time

import numpy as np
import pytest

from helpers import oracle_search

pytestmark = pytest.mark.gpu
P12 = "1110100110010101111"


def satellite(rng, n, unit, divergence):
    s = np.tile(unit, n // len(unit) + 1)[:n].copy()
    at = rng.random(n) < divergence
    s[at] = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, int(at.sum()))]
    return s.tobytes()


def test_search_of_a_satellite_uses_the_device(gxy, ctx):
    # 20 kbp of a 171-base satellite against 20 kbp of it: 290,000 hits where two
    # random sequences have 700.  The same query with 4 Mbp of N after it has the same
    # hits and more to do, so it must not be the faster one (it was, 0.6 to 1.6 ms, when
    # the grids were sized by the number of windows).
    rng = np.random.default_rng(171)
    unit = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, 171)]
    t, q = satellite(rng, 20_000, unit, 0.15), satellite(rng, 20_000, unit, 0.15)
    m, sp = gxy.ScoringMatrix.hoxd70(), gxy.SearchParams()
    tab = gxy.PosTable.build(gxy.PackedSeq.from_ascii(t), P12, 1, ctx=ctx)
    found, best = [], []
    for bases in (q, q + b"N" * 4_000_000):
        dq = gxy.DeviceSeq.from_ascii(bases, ctx)
        times = []
        for _ in range(8):
            t0 = time.perf_counter()
            h = gxy.search_device(tab, dq, m, sp)
            times.append(time.perf_counter() - t0)
        found.append(h.tobytes())
        best.append(min(times[1:]))
    want, _ = oracle_search(t, q, P12, m, sp)
    assert len(want) > 100 and found[0] == found[1] == want.tobytes()
    assert best[0] < 1.5 * best[1], best
