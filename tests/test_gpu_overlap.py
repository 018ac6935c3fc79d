"""Calls on several streams of one device: one call's kernels must not wait until
another's have left every SM."""
import threading
import time

import numpy as np
import pytest

from helpers import rand_ascii

pytestmark = pytest.mark.gpu
P12 = "1110100110010101111"


def test_search_started_during_a_long_walk(gxy):
    # A gapless 1 Mbp alignment is walked by one warp, which takes most of the
    # search; the rest of the device is free for another stream's.  A second search
    # that starts when a third of the first one's time has passed takes less than 1.3
    # times what it takes alone (1.6 times, when one of its launches waits for an SM
    # that the first one's walk sits on).
    rng = np.random.default_rng(3)
    c = gxy.Context(0)
    t = np.frombuffer(rand_ascii(rng, 1_000_000, b"ACGT"), np.uint8)
    q = t.copy()
    at = rng.random(len(q)) < 0.1
    q[at] = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, int(at.sum()))]
    tab = gxy.PosTable.build(gxy.PackedSeq.from_ascii(t.tobytes()), P12, 1, ctx=c)
    dq = [gxy.DeviceSeq.from_ascii(q.tobytes(), c) for _ in range(2)]
    m, sp = gxy.ScoringMatrix.hoxd70(), gxy.SearchParams()
    found = []

    def search(k):
        t0 = time.perf_counter()
        found.append(gxy.search_device(tab, dq[k], m, sp).tobytes())
        return time.perf_counter() - t0

    def second(after):
        th = threading.Thread(target=search, args=(0,))
        th.start()
        time.sleep(after)
        dt = search(1)
        th.join()
        return dt
    second(0.0)   # both streams' buffers
    alone = min(search(0) for _ in range(7))
    beside = min(second(alone / 3) for _ in range(7))
    assert len(set(found)) == 1 and found[0]
    assert beside < 1.3 * alone, (alone, beside)


def test_free_of_a_table_with_masks(gxy):
    # A free waits for the device, which other threads' streams feel as well: once a
    # table, however many arrays it has (one wait for each of six took 24 us, 17
    # without the masks and packed bounds; 7 now).
    c = gxy.Context(0)
    t = gxy.DeviceSeq.from_ascii(rand_ascii(np.random.default_rng(8), 1_000_000, b"ACGT"), c)

    def free_time(n):
        times = []
        for _ in range(300):
            tab = gxy.PosTable.build_view(t, 0, n, P12, 1)
            t0 = time.perf_counter()
            tab.free()
            times.append(time.perf_counter() - t0)
        return sorted(times)[150]
    plain = min(free_time(30_000) for _ in range(2))
    masks = min(free_time(1_000_000) for _ in range(2))
    assert masks < 1.25 * plain, (masks, plain)
