"""Performance cases of the seed->HSP framework, each a call sequence a user's program makes.

A case is a dict of plain values; `kind` names the call sequence:

  pair       PosTable.build on a device target, the query's reverse complement, one search per strand
  resident   search() of a host query against a resident table (the reference's bench shape, the tweener's calls)
  contigs    batch_search of query contigs, both strands, against a resident table
  chunked    build_views over a target's chunks, then batch_records of every (chunk, strand) unit
  gapped     gapped_extend of the anchors a search's best HSPs give
  parse      parse_fasta / parse_2bit of a file's bytes, and the PackedSeq arrays back on the host
  consumers  choose_anchors on every HSP and best_chain_groups on each (chunk, strand) group

Sequences follow the model of the package's synthetic workloads (iid bases at 41 % GC, repeat
families, soft-masked runs, N blocks, queries evolved with Ts:Tv 2:1 substitutions and indels),
drawn with whole-array operations.  Every output is a whole number: there is nothing for exact()
to give, the outputs equal the reference's bit for bit.  Results whose number depends on the data
are copied into the state's own result buffer, as a program that collects them does, and returned
with their count.
"""
import importlib.util
import math
import os
import struct
import sys

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
P12 = "1110100110010101111"   # 12of19, the default spaced seed
M12 = "1" * 12                # match12, the reference bench's contiguous seed


def _pkg():
    if "lastz_gxy_b200" not in sys.modules:
        d = os.path.join(ROOT, "lastz-gxy_b200")
        spec = importlib.util.spec_from_file_location("lastz_gxy_b200", os.path.join(d, "__init__.py"),
                                                      submodule_search_locations=[d])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["lastz_gxy_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["lastz_gxy_b200"]


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # The smallest whole job: two 30 kbp sequences (a BAC, a virus, a test), latency and launches.
        {"name": "pair_30k", "kind": "pair", "t": 30_000, "q": 30_000, "pattern": P12, "step": 1, "transitions": 1,
         "entropy": -1, "identity": 0.80},
        # An odd-sized pair of contigs with the sensitive options: two transitions, the entropy gate.
        {"name": "pair_1m_sensitive", "kind": "pair", "t": 1_234_567, "q": 987_653, "pattern": P12, "step": 1,
         "transitions": 2, "entropy": 3000, "identity": 0.75},
        # A chromosome against a chromosome, the benchmark's shape, one thread.
        {"name": "pair_10m", "kind": "pair", "t": 10_000_000, "q": 10_000_000, "pattern": P12, "step": 1,
         "transitions": 1, "entropy": -1, "identity": 0.70},
        # The reference bench's shape: match12, no transitions, a 100 kbp host query on a resident 1 Mbp table.
        {"name": "resident_100k_match12", "kind": "resident", "t": 1_000_000, "q": 100_000, "pattern": M12, "step": 1,
         "transitions": 0, "entropy": -1, "identity": 0.85},
        # One short contig on a resident chromosome, both strands: a served request.
        {"name": "contig_20k", "kind": "contigs", "t": 20_000_000, "n": 1, "median": 20_011, "pattern": P12,
         "transitions": 1, "graph": True},
        # An assembly's contigs of uneven lengths on a chromosome, both strands, one launch.
        {"name": "contigs_300", "kind": "contigs", "t": 20_000_000, "n": 300, "median": 20_000, "pattern": P12,
         "transitions": 1, "graph": False},
        # A larger chromosome in 10 Mbp chunks, both strands, as the driver's records: the largest job.
        {"name": "chunked_33m", "kind": "chunked", "t": 33_000_000, "q": 12_000_000, "chunk": 10_000_000,
         "halo": 50_000, "pattern": P12, "transitions": 1},
        # Three anchors of one long alignment: the rows of a side are one after the other.
        {"name": "gapped_40k_3", "kind": "gapped", "t": 40_000, "segments": 0, "anchors": 3, "y_drop": 9400},
        # The gapped step of a search: many anchors of diverged segments of uneven lengths.
        {"name": "gapped_1500k_400", "kind": "gapped", "t": 1_500_000, "segments": 160, "anchors": 400,
         "y_drop": 9400},
        # A chromosome file and a file of scaffolds, 60-column lines; a 2bit file.
        {"name": "fasta_20m", "kind": "parse", "format": "fasta", "total": 20_000_003, "records": 4},
        {"name": "twobit_40m", "kind": "parse", "format": "2bit", "total": 40_000_001, "records": 3},
        # The consumers of a search's HSPs: an anchor for each, a chain for each (chunk, strand).
        {"name": "consumers_4m", "kind": "consumers", "t": 4_000_000, "chunk": 500_000, "window": 31},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pair", "pair", "resident", "contigs", "contigs", "chunked", "gapped", "gapped", "parse",
                       "consumers"])
    if kind == "pair":
        t = _log(rng, 30_000, 10_000_000)
        tr = rng.choice([0, 1, 1, 2]) if t < 1_500_000 else rng.choice([0, 1, 1])
        return {"kind": kind, "t": t, "q": min(10_000_000, max(20_000, int(t * rng.uniform(0.5, 1.5)))),
                "pattern": rng.choice([P12, P12, M12]), "step": rng.choice([1, 1, 1, 2, 3]), "transitions": tr,
                "entropy": rng.choice([-1, -1, 3000]), "identity": round(rng.uniform(0.65, 0.95), 3)}
    if kind == "resident":
        return {"kind": kind, "t": _log(rng, 200_000, 10_000_000), "q": _log(rng, 10_000, 1_000_000),
                "pattern": rng.choice([P12, M12]), "step": rng.choice([1, 1, 2]), "transitions": rng.choice([0, 1]),
                "entropy": rng.choice([-1, 3000]), "identity": round(rng.uniform(0.70, 0.95), 3)}
    if kind == "contigs":
        return {"kind": kind, "t": _log(rng, 2_000_000, 20_000_000), "n": _log(rng, 1, 300),
                "median": _log(rng, 5_000, 20_000), "pattern": P12, "transitions": rng.choice([0, 1, 1]),
                "graph": rng.random() < 0.5}
    if kind == "chunked":
        t = _log(rng, 4_000_000, 30_000_000)
        return {"kind": kind, "t": t, "q": _log(rng, 1_000_000, 12_000_000),
                "chunk": rng.choice([2_000_000, 5_000_000, 10_000_000]) if t < 16_000_000 else 10_000_000,
                "halo": rng.choice([0, 10_000, 50_000]), "pattern": P12, "transitions": rng.choice([0, 1])}
    if kind == "gapped":
        y = rng.choice([9400, 9400, 9400, 6000, 3000])
        if rng.random() < 0.3:
            return {"kind": kind, "t": _log(rng, 2_000, 40_000), "segments": 0, "anchors": rng.randint(1, 4),
                    "y_drop": y}
        t = _log(rng, 100_000, 1_500_000)
        return {"kind": kind, "t": t, "segments": max(4, t // 9400), "anchors": _log(rng, 8, 400), "y_drop": y}
    if kind == "parse":
        f = rng.choice(["fasta", "2bit"])
        return {"kind": kind, "format": f, "total": _log(rng, 100_000, 20_000_000 if f == "fasta" else 40_000_000),
                "records": rng.randint(1, 16)}
    return {"kind": kind, "t": _log(rng, 200_000, 4_000_000), "chunk": _log(rng, 100_000, 500_000),
            "window": rng.choice([1, 16, 31, 64, 201])}


# ---------------------------------------------------------------------------
# Sequences
# ---------------------------------------------------------------------------
_ACGT = np.frombuffer(b"ACGT", np.uint8)
_IID = _ACGT[np.searchsorted(np.array([75, 128, 180]), np.arange(256), side="right")]   # 41 % GC
_CODE = np.zeros(256, np.uint8)
for _k, _b in enumerate(b"ACGT"):
    _CODE[_b] = _CODE[_b + 32] = _k
_COMP = np.arange(256, dtype=np.uint8)
for _a, _b in zip(b"ACGTacgt", b"TGCAtgca"):
    _COMP[_a] = _b


def _iid(rng, n):
    return _IID[np.frombuffer(rng.bytes(n), np.uint8)]


def _substitute(rng, s, rate):
    """Substitutions at `rate`, two transitions for each transversion; N stays N, case stays."""
    k = np.flatnonzero(rng.random(len(s), dtype=np.float32) < rate)
    r = rng.integers(0, 6, len(k), dtype=np.uint8)
    x = np.array([2, 2, 2, 2, 1, 3], np.uint8)[r]
    old = s[k]
    new = _ACGT[_CODE[old] ^ x] | (old & 32)
    out = s.copy()
    out[k] = np.where((old & 95) == ord("N"), old, new)
    return out


def _evolve(rng, s, identity, indel=0.01, replace=0.0):
    out = _substitute(rng, s, 1.0 - identity)
    n = len(out)
    for _ in range(int(round(replace * n / 2750))):
        a = int(rng.integers(0, n))
        ln = min(n - a, int(rng.integers(500, 5001)))
        out[a:a + ln] = _iid(rng, ln)
    ev = int(rng.binomial(n, indel))
    pos = np.sort(rng.integers(0, n, ev))
    ln = rng.geometric(1 / 3, ev)
    ins = rng.random(ev) < 0.5
    # Each base is kept once, dropped in a deletion, or followed by an insertion.
    rep = np.ones(n, np.int64)
    dp, dl = pos[~ins], ln[~ins]
    at = np.repeat(dp, dl) + (np.arange(dl.sum()) - np.repeat(np.cumsum(dl) - dl, dl))
    rep[at[at < n]] = 0
    np.add.at(rep, pos[ins], ln[ins])
    idx = np.repeat(np.arange(n), rep)
    first = np.ones(len(idx), bool)
    first[1:] = idx[1:] != idx[:-1]
    res = out[idx]
    extra = ~first
    res[extra] = _iid(rng, int(extra.sum()))
    return res


def _chromosome(rng, n):
    """iid bases, 200 repeat families of 300 bp per Mbp in 5-50 diverged copies of either orientation,
    45 % soft-masked, two 10 kbp N blocks per Mbp from 1 Mbp on."""
    s = _iid(rng, n)
    if n >= 3_000:
        fams = max(1, n // 5_000)
        cons = _iid(rng, fams * 300).reshape(fams, 300)
        fam = np.repeat(np.arange(fams), rng.integers(5, 51, fams))
        rng.shuffle(fam)
        fam = fam[:max(1, n // 300)]
        for lo in range(0, len(fam), 16_384):
            f = fam[lo:lo + 16_384]
            c = cons[f]
            flip = rng.random(len(f)) < 0.5
            c[flip] = _COMP[c[flip][:, ::-1]]
            div = rng.uniform(0.10, 0.20, (len(f), 1)).astype(np.float32)
            c = np.where(rng.random(c.shape, dtype=np.float32) < div, _substitute(rng, c.reshape(-1), 1.0)
                         .reshape(c.shape), c)
            for a, row in zip(rng.integers(0, n - 300, len(f)), c):
                s[a:a + 300] = row
    p = int(rng.integers(0, 3_000))
    while p < n:
        ln = int(rng.integers(100, 5_001))
        s[p:p + ln] |= 32
        p += ln + int(rng.integers(1, 6_234))
    for _ in range(2 * (n // 1_000_000)):
        a = int(rng.integers(0, n - 10_000))
        s[a:a + 10_000] = ord("N")
    return s


def _planted(rng, n, segments):
    """A target and a query that share `segments` diverged segments of 500-6,000 bp."""
    t, q = _iid(rng, n), _iid(rng, n)
    for _ in range(segments):
        ln = int(round(math.exp(rng.uniform(math.log(500), math.log(6_000)))))
        a, b = int(rng.integers(0, n - ln)), int(rng.integers(0, n - ln))
        e = _evolve(rng, t[a:a + ln], rng.uniform(0.75, 0.95))[:ln]
        q[b:b + len(e)] = e
    return t, q


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
def _params(g, case):
    e = case.get("entropy", -1)
    return g.SearchParams(case.get("step", 1), g.HspParams(), case["transitions"], None if e < 0 else e)


def prepare(case, seed):
    """The inputs on the device (or in host memory where the entry point takes host data), with a result buffer."""
    state = _inputs(case, seed)
    if case["kind"] == "gapped":
        longest = case["t"] // 10 if not case["segments"] else 1_000
        state["out"] = [np.zeros(case["anchors"] * (64 + longest), np.int32)]
    elif case["kind"] == "consumers":
        rows = _most_hsps(case["t"], case["t"])
        state["out"] = [np.zeros((rows, 2), np.int32), np.zeros((rows, 4), np.int32)]
    elif case["kind"] != "parse":
        q = case["q"] if "q" in case else _contig_bases(case)
        width = 6 if case["kind"] == "chunked" else 4
        state["out"] = [np.zeros((_most_hsps(case["t"], q), width), np.int32)
                        for _ in range(2 if case["kind"] == "pair" else 1)]
    return state


def _most_hsps(t, q):
    return 4_096 + int(0.045 * (t + q))


def _contig_bases(case):
    return int(case["n"] * case["median"] * (1.0 if case["n"] == 1 else 2 * math.exp(1.3 ** 2 / 2)))


def _inputs(case, seed):
    g = _pkg()
    rng = np.random.default_rng([seed & 0xffffffff, case.get("t", case.get("total"))])
    ctx = g.Context.default(0)
    dev = lambda s: g.DeviceSeq.from_ascii(s, ctx)  # noqa: E731
    m = g.ScoringMatrix.hoxd70()
    k = case["kind"]
    if k == "pair":
        t = _chromosome(rng, case["t"])
        q = _fit(rng, _evolve(rng, t, case["identity"], replace=0.05), case["q"])
        return {"case": case, "T": dev(t), "Q": dev(q), "m": m, "sp": _params(g, case)}
    if k == "resident":
        t = _chromosome(rng, case["t"])
        a = int(rng.integers(0, max(1, len(t) - case["q"])))
        q = _fit(rng, _evolve(rng, t[a:a + case["q"]], case["identity"], 0.005), case["q"])
        T, Q = g.PackedSeq.from_ascii(t), g.PackedSeq.from_ascii(q)
        return {"case": case, "T": T, "Q": Q, "tab": g.PosTable.build(T, case["pattern"], case["step"], ctx=ctx),
                "m": m, "sp": _params(g, case)}
    if k == "contigs":
        t = _chromosome(rng, case["t"])
        n = case["n"]
        lens = [case["median"]] if n == 1 else \
            np.clip(rng.lognormal(math.log(case["median"]), 1.3, n), 1_000, 1_000_000).astype(int)
        qs = []
        for ln in lens:
            a = int(rng.integers(0, max(1, len(t) - ln)))
            qs.append(dev(_evolve(rng, t[a:a + ln], rng.uniform(0.65, 0.95), 0.005)))
        T = dev(t)
        return {"case": case, "T": T, "Q": qs, "tab": g.PosTable.build(T, case["pattern"], 1, ctx=ctx),
                "units": [(0, i, s) for i in range(n) for s in (0, 1)], "m": m, "sp": _params(g, case)}
    if k == "chunked":
        t = _chromosome(rng, case["t"])
        a = int(rng.integers(0, max(1, len(t) - case["q"])))
        q = _fit(rng, _evolve(rng, t[a:a + case["q"]], 0.70, replace=0.05), case["q"])
        chunks = g.chunk_target(len(t), case["chunk"], case["halo"])
        units = [(i, 0, s, c[2], c[3]) for s in (0, 1) for i, c in enumerate(chunks)]
        return {"case": case, "T": dev(t), "Q": dev(q), "views": [(c[0], c[1]) for c in chunks], "units": units,
                "places": [(u[2], chunks[u[0]][0]) for u in units], "m": m, "sp": _params(g, case)}
    if k == "gapped":
        if case["segments"]:
            t, q = _planted(rng, case["t"], case["segments"])
        else:
            t = _iid(rng, case["t"])
            q = _evolve(rng, t, 0.90, 0.005)
        T, Q = dev(t), dev(q)
        tab = g.PosTable.build(T, P12, 1, ctx=ctx)
        h = g.search_device(tab, Q, m, g.SearchParams())
        h = np.resize(h[np.argsort(-h["score"], kind="stable")], case["anchors"])
        return {"case": case, "T": T, "Q": Q, "anchors": g.choose_anchors(T, Q, h, m, 31, ctx), "m": m,
                "gp": g.GappedParams(case["y_drop"], 3000)}
    if k == "parse":
        s = _chromosome(rng, case["total"])
        cut = np.arange(1, case["records"]) ** 2 * len(s) // case["records"] ** 2   # uneven lengths
        recs = [("scaffold_%d" % i, x) for i, x in enumerate(np.split(s, cut))]
        return {"case": case, "bytes": _fasta(recs) if case["format"] == "fasta" else _twobit(recs)}
    t = _chromosome(rng, case["t"])
    q = _evolve(rng, t, 0.80, replace=0.05)
    T, Q = dev(t), dev(q)
    chunks = g.chunk_target(len(t), case["chunk"], 0)
    tabs = g.PosTable.build_views(T, [(c[0], c[1]) for c in chunks], P12, 1, ctx=ctx)
    groups = g.batch_search(tabs, [Q], [(i, 0, 0) for i in range(len(chunks))], m, g.SearchParams(), ctx=ctx)
    for c, h in zip(chunks, groups):
        h["t_start"] += c[0]
    return {"case": case, "T": T, "Q": Q, "groups": groups, "hsps": np.concatenate(groups), "m": m}


def _fit(rng, s, n):
    return s[:n] if len(s) >= n else np.concatenate([s, _iid(rng, n - len(s))])


def _fasta(recs):
    out = []
    for name, s in recs:
        out.append(b">%s\n" % name.encode())
        full = len(s) // 60 * 60
        out.append(np.concatenate([s[:full].reshape(-1, 60), np.full((full // 60, 1), 10, np.uint8)], 1).tobytes())
        if full < len(s):
            out.append(s[full:].tobytes() + b"\n")
    return b"".join(out)


def _runs(flags):
    d = np.flatnonzero(np.diff(np.concatenate([[0], flags.view(np.int8), [0]])))
    return d[::2], d[1::2] - d[::2]


def _twobit(recs):
    code = np.array([2, 1, 3, 0], np.uint8)   # A C G T -> the format's T C A G = 0 1 2 3
    head, body = struct.pack("<IIII", 0x1A412743, 0, len(recs), 0), []
    off = 16 + sum(5 + len(n) for n, _ in recs)
    index = b""
    for name, s in recs:
        up = s & 0xDF
        isn = up == ord("N")
        rec = struct.pack("<I", len(s))
        for flags in (isn, ((s & 32) != 0) & ~isn):
            a, ln = _runs(flags)
            rec += struct.pack("<I", len(a)) + a.astype("<u4").tobytes() + ln.astype("<u4").tobytes()
        rec += struct.pack("<I", 0)
        c = np.concatenate([np.where(isn, 0, code[_CODE[s]]), np.zeros((-len(s)) % 4, np.uint8)]).reshape(-1, 4)
        rec += (c[:, 0] << 6 | c[:, 1] << 4 | c[:, 2] << 2 | c[:, 3]).astype(np.uint8).tobytes()
        index += bytes([len(name)]) + name.encode() + struct.pack("<I", off)
        body.append(rec)
        off += len(rec)
    return head + index + b"".join(body)


def _collect(buf, arrays):
    """Copies arrays of 4-byte fields into the state's buffer, one after the other; the rows copied."""
    n = 0
    for a in arrays:
        buf[n:n + len(a)] = a.view(np.int32).reshape(len(a), *buf.shape[1:])
        n += len(a)
    return n


def run(state):
    g = _pkg()
    k = state["case"]["kind"]
    out = state.get("out")
    if k == "pair":
        tab = g.PosTable.build(state["T"], state["case"]["pattern"], state["case"]["step"])
        rc = state["Q"].reverse_complement()
        n = [_collect(o, [g.search_device(tab, x, state["m"], state["sp"])]) for o, x in zip(out, (state["Q"], rc))]
        return [*out, np.array(n)]
    if k == "resident":
        return [*out, _collect(out[0], [g.search(state["tab"], state["T"], state["Q"], state["m"], state["sp"])])]
    if k == "contigs":
        hsps = g.batch_search([state["tab"]], state["Q"], state["units"], state["m"], state["sp"],
                              use_graph=state["case"]["graph"])
        _collect(out[0], hsps)
        return [*out, np.array([len(h) for h in hsps])]
    if k == "chunked":
        tabs = g.PosTable.build_views(state["T"], state["views"], state["case"]["pattern"], 1)
        recs, offs = g.batch_records(tabs, [state["Q"]], state["units"], state["places"], state["m"], state["sp"])
        _collect(out[0], [recs])
        return [*out, offs.view(np.int64)]
    if k == "gapped":
        alns = g.gapped_extend(state["T"], state["Q"], state["anchors"], state["m"], state["gp"])
        pos = np.array([(0,) * 6 if a is None else (a.t_start, a.q_start, a.t_len, a.q_len, a.score, len(a.script))
                        for a in alns], np.int64)
        return [pos, *out, _collect(out[0], [a.script for a in alns if a is not None])]
    if k == "parse":
        parse = g.parse_fasta if state["case"]["format"] == "fasta" else g.parse_2bit
        host = [s.to_host() for _, s in parse(state["bytes"])]
        return [[p.codes, p.valid, p.mask] for p in host]
    anchors = g.choose_anchors(state["T"], state["Q"], state["hsps"], state["m"], state["case"]["window"])
    chains = g.best_chain_groups(state["groups"])
    _collect(out[0], [anchors])
    _collect(out[1], chains)
    return [*out, np.array([len(c) for c in chains])]


def exact(case, seed):
    return None


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
def _search_ops(t, q, case):
    """Integer operations of the expected raw hits: two 32-column sides and the seed's columns each."""
    n_var = {0: 1, 1: 13, 2: 79}[case["transitions"]]
    hits = 0.3 * t / case.get("step", 1) * (q / case.get("step", 1)) * n_var / 4 ** 12
    return q * n_var + hits * 2 * (64 + 19)


def work(case):
    k = case["kind"]
    if k == "pair":
        return {"bytes": 0.5 * (case["t"] + 2 * case["q"]), "flops": 2 * _search_ops(case["t"], case["q"], case)}
    if k == "resident":
        return {"bytes": 0.5 * case["q"] + 0.375 * case["t"], "flops": _search_ops(case["t"], case["q"], case)}
    if k == "contigs":
        q = _contig_bases(case) / (1 if case["n"] == 1 else 2)
        return {"bytes": 0.375 * case["t"] + q, "flops": 2 * _search_ops(case["t"], q, case)}
    if k == "chunked":
        return {"bytes": 0.5 * (case["t"] + 2 * case["q"]), "flops": 2 * _search_ops(case["t"], case["q"], case)}
    if k == "gapped":
        # Cells a side cannot do without: about 600 survive a row at y_drop 9400.
        rows = case["anchors"] * (case["t"] if not case["segments"] else 2_500)
        width = case["y_drop"] / 9400 * 600
        return {"bytes": 0.375 * 2 * case["t"] + 4.0 * rows / 20, "flops": 10.0 * rows * width}
    if k == "parse":
        return {"bytes": case["total"] * (1.017 if case["format"] == "fasta" else 0.25) + 0.5 * case["total"],
                "flops": 0.0}
    hsps = 0.02 * case["t"]
    return {"bytes": 0.75 * case["t"] + 56 * hsps, "flops": hsps * (4 * 100 + 8 * case["chunk"] * 0.02)}
