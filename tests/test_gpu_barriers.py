"""The wait of a search's blocks for one another runs out: an error, nothing read that
was not written, and the context works on."""
import ctypes

import numpy as np
import pytest

from helpers import rand_ascii

pytestmark = pytest.mark.gpu
P12 = "1110100110010101111"


@pytest.mark.parametrize("kind", ["search", "batch", "batch graph", "records", "records graph"])
def test_barrier_that_runs_out_of_polls(gxy, kind):
    rng = np.random.default_rng(24)
    c = gxy.Context(0)
    unit = np.frombuffer(rand_ascii(rng, 171, b"ACGT"), np.uint8)
    seqs = []
    for _ in range(3):   # 20 kbp of a satellite: 290,000 candidates a pair, 71 tiles of the sort
        s = np.tile(unit, 118)[:20_000].copy()
        at = rng.random(len(s)) < 0.15
        s[at] = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, int(at.sum()))]
        seqs.append(s.tobytes())
    tab = gxy.PosTable.build(gxy.PackedSeq.from_ascii(seqs[0]), P12, 1, ctx=c)
    dq = [gxy.DeviceSeq.from_ascii(s, c) for s in seqs[1:]]
    m, sp = gxy.ScoringMatrix.hoxd70(), gxy.SearchParams()
    units = [(0, k, s) for k in (0, 1) for s in (0, 1)]
    graph = kind.endswith("graph")

    def call():
        if kind == "search":
            return gxy.search_device(tab, dq[0], m, sp).tobytes()
        if kind.startswith("batch"):
            return [h.tobytes() for h in gxy.batch_search([tab], dq, units, m, sp, use_graph=graph, ctx=c)]
        rec, off = gxy.batch_records([tab], dq, units, [(i // 2, 0) for i in range(4)], m, sp, use_graph=graph, ctx=c)
        return rec.tobytes(), np.asarray(off).tobytes()

    polls = gxy._lib.lib().gxy_ctx_set_barrier_polls
    want = call()
    assert polls(c.h, ctypes.c_uint32(1)) == 0
    for _ in range(3):
        with pytest.raises(gxy.GxyError) as e:
            call()
        assert e.value.status == gxy._lib.GXY_ETIMEDOUT
    assert polls(c.h, ctypes.c_uint32(0)) == 0
    assert call() == want
