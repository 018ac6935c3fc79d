"""FASTA and 2bit parsed straight into device sequences must equal the
reference's parse followed by PackedSeq::from_ascii, bit for bit (codes, valid
and mask bytes), names included; malformed inputs fail with GxyError."""
import numpy as np
import pytest

import oracle as O
from helpers import rand_ascii, write_2bit

pytestmark = pytest.mark.gpu


def same(gxy, dev_seqs, want):
    assert [n for n, _ in dev_seqs] == [n for n, _ in want]
    for (name, d), (_, asc) in zip(dev_seqs, want):
        h = d.to_host()
        o = O.pack_ascii(asc)
        assert len(h) == o.len, name
        nb, nv = (o.len + 3) // 4, (o.len + 7) // 8
        assert bytes(h.codes[:nb]) == bytes(np.asarray(o.codes)[:nb]), name
        assert bytes(h.valid[:nv]) == bytes(np.asarray(o.valid)[:nv]), name
        assert bytes(h.mask[:nv]) == bytes(np.asarray(o.mask)[:nv]), name


FASTA_CASES = [
    b">a\n\nacgt\nACGT\n",                                   # src/sequences.rs:441-454
    b">x desc here\nACGTN\nacg\r\n>y\r\nTTTT\n\n>z\n",          # CRLF, description, empty record
    b"ACG\n>first\nTT\n",                                    # bases before the first header join it
    b">a\nAC>GT\n>b\n\tA C\x0cG\n",                          # '>' inside a line is a base; tab/FF/space skipped
    b"no header at all\n",
    b"",
]


@pytest.mark.parametrize("case", range(len(FASTA_CASES)))
def test_fasta_cases(gxy, ctx, case):
    data = FASTA_CASES[case]
    same(gxy, gxy.parse_fasta(data, ctx), O.parse_fasta(data))


def test_fasta_random_records(gxy, ctx):
    rng = np.random.default_rng(3)
    parts = []
    for r in range(40):
        seq = rand_ascii(rng, int(rng.integers(0, 30000)), b"ACGTacgtNnRY")
        width = int(rng.integers(1, 120))
        lines = [seq[i:i + width] for i in range(0, len(seq), width)]
        eol = b"\r\n" if r % 3 == 0 else b"\n"
        parts.append(b">rec%d some text%s" % (r, eol) + eol.join(lines) + eol)
    data = b"".join(parts)
    same(gxy, gxy.parse_fasta(data, ctx), O.parse_fasta(data))


def test_fasta_empty_header_fails(gxy, ctx):
    with pytest.raises(gxy.GxyError):
        gxy.parse_fasta(b">a\nACGT\n>  \nAC\n", ctx)


TWOBIT_CASES = [
    [("chr1", b"ACGTACGTACGT")],
    [("chrA", b"ACGT"), ("chrB", b"TTTT"), ("chrC", b"GATTACACATG")],
    [("chr1", b"ACGTNNNNACGT")],
    [("chr1", b"ACGTacgtACGT")],
    [("chr1", b"ACntACGT")],
    [("chr1", b"A"), ("chr2", b"AC"), ("chr3", b"ACG"), ("chr4", b"ACGT"), ("chr5", b"ACGTA")],
    [("empty", b"")],
]


@pytest.mark.parametrize("case", range(len(TWOBIT_CASES)))
@pytest.mark.parametrize("be", [False, True])
def test_2bit_cases(gxy, ctx, case, be):
    data = write_2bit(TWOBIT_CASES[case], big_endian=be)
    same(gxy, gxy.parse_2bit(data, ctx), O.parse_2bit(data))


def test_2bit_random_blocks(gxy, ctx):
    rng = np.random.default_rng(4)
    seqs = []
    for r in range(6):
        s = bytearray(rand_ascii(rng, int(rng.integers(1, 400000)), b"ACGT"))
        for _ in range(int(rng.integers(0, 60))):       # N runs and soft-masked runs, overlapping
            a = int(rng.integers(0, len(s)))
            b = min(len(s), a + int(rng.integers(1, 5000)))
            if rng.random() < 0.4:
                s[a:b] = b"N" * (b - a)
            else:
                s[a:b] = bytes(s[a:b]).lower()
        seqs.append(("s%d" % r, bytes(s)))
    data = write_2bit(seqs)
    same(gxy, gxy.parse_2bit(data, ctx), O.parse_2bit(data))


@pytest.mark.parametrize("bad", ["magic", "truncated", "version"])
def test_2bit_errors(gxy, ctx, bad):
    data = bytearray(write_2bit([("chr1", b"ACGTACGT")]))
    if bad == "magic":
        data = bytes(32)
    elif bad == "truncated":
        data = bytes(data[:-2])
    else:
        data[4] = 1
        data = bytes(data)
    with pytest.raises(gxy.GxyError):
        gxy.parse_2bit(data, ctx)


@pytest.mark.parametrize("n", [(2 << 20) - 1, 2 << 20, (2 << 20) + 1, 5 * (1 << 19), 9_000_007])
def test_large_copies(gxy, ctx, n):
    # From 2 MB on, host memory is copied in chunks of 512 KB by several threads,
    # which also look for the header lines: a FASTA file of n bytes with a header
    # around every other chunk's end and a '>' inside lines, the sequences' way back
    # and up again, and four threads at a time, of which one finds the pinned halves free.
    import threading
    rng = np.random.default_rng(n)
    buf = bytearray(rand_ascii(rng, n, b"ACGTacgtN"))
    buf[60::61] = b"\n" * len(range(60, n, 61))
    buf[:9] = b">a first\n"
    for k, c in enumerate(range(1 << 19, n - 40, 1 << 19)):
        at = c - 8 + 3 * k % 16
        buf[at:at + 16] = b"\n>r%06d x>y z\n" % k if k % 2 == 0 else b"ACGT>ACGTNNNACGT"
    data = bytes(buf)
    want = O.parse_fasta(data)
    seqs = gxy.parse_fasta(data, ctx)
    same(gxy, seqs, want)
    big = max((d for _, d in seqs), key=lambda d: d.length)
    one = gxy.DeviceSeq.from_ascii(data.replace(b"\n", b""), ctx)
    host = one.to_host()
    back = host.to_device(ctx).to_host()
    for a, b in ((host.codes, back.codes), (host.valid, back.valid), (host.mask, back.mask)):
        assert np.array_equal(a, b)
    ref = big.to_host()
    got = [None] * 4

    def work(i):
        h = host.to_device(ctx).to_host()
        got[i] = (np.array_equal(h.codes, host.codes) and np.array_equal(h.valid, host.valid)
                  and np.array_equal(h.mask, host.mask) and np.array_equal(big.to_host().codes, ref.codes))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert got == [True] * 4


@pytest.mark.parametrize("n", [1, 15, 16, 17, 4095, 4096, 4097, 8191, 12_289, 70_000])
def test_fasta_tiles(gxy, ctx, n):
    # Bases are counted and gathered in tiles of 4,096 bytes, 16 a thread: files of n
    # bytes after the first header whose further headers start or end beside the
    # tiles' and threads' edges, headers longer than a tile, and tiles full of short ones.
    rng = np.random.default_rng(n)
    for case in range(4):
        buf = bytearray(b">first\n" + rand_ascii(rng, n, b"ACGTacgtN\n\n \t\r"))
        if case == 1:
            for c in range(4096, len(buf) - 40, 4096):
                at = c - 14 + int(rng.integers(0, 28))
                buf[at:at + 9] = b"\n>h%05d\n" % (c % 99_999)
        elif case == 2 and n > 5000:
            buf[300:300 + 4500] = b"\n>long " + b"x>" * 2246 + b"\n"
        elif case == 3:
            short = b"".join(b">%d\nA%s" % (i, b"\n" * (i % 3)) if i % 3 else b">%d a\n" % i for i in range(n // 6))
            buf = bytearray(b">first\n" + short.replace(b"A>", b"A\n>") + b"\nACGT")
        data = bytes(buf)
        same(gxy, gxy.parse_fasta(data, ctx), O.parse_fasta(data))


def test_search_that_returns_early_has_read_its_pinned_query(gxy):
    # 256 MB of pinned arrays take 5 ms to the device: a search that is refused before
    # it launches anything, or has no windows, leaves no copy running.
    import time
    import torch
    c = gxy.Context(0)
    tab = gxy.PosTable.build(gxy.PackedSeq.from_ascii(b"ACGT" * 5000), "1" * 12, 1, ctx=c)
    t = gxy.PackedSeq.from_ascii(b"ACGT" * 5000)
    n = 1 << 29
    pinned = [torch.zeros(k, dtype=torch.uint8).pin_memory() for k in (n // 4, n // 8, n // 8)]
    q = gxy.PackedSeq(*(x.numpy() for x in pinned), n)
    assert q.codes.ctypes.data == pinned[0].data_ptr()
    m = gxy.ScoringMatrix.hoxd70()
    gxy.search(tab, t, gxy.PackedSeq.from_ascii(b"ACGT" * 5000), m, gxy.SearchParams())
    for _ in range(3):
        with pytest.raises(gxy.GxyError):
            gxy.search(tab, t, q, m, gxy.SearchParams(step=0))
        c.mark(0)
        t0 = time.perf_counter()
        c.elapsed_ms(0, 0)   # (waits for what the stream holds)
        assert time.perf_counter() - t0 < 1e-3


def test_to_host_in_a_loop_costs_its_copy(gxy, ctx):
    # Arrays whose memory an earlier result left: the copy's time and little more (they
    # were cleared first, which took four times as long as the copy into arrays
    # that are there).
    import time
    n = 10_000_000
    ds = gxy.DeviceSeq.from_ascii(rand_ascii(np.random.default_rng(2), n, b"ACGT"), ctx)
    held = [np.ones(n // 4, np.uint8), np.ones(n // 8, np.uint8), np.ones(n // 8, np.uint8)]

    def median(f):
        times = []
        for _ in range(30):
            t0 = time.perf_counter()
            f()
            times.append(time.perf_counter() - t0)
        return sorted(times)[15]
    into = median(lambda: gxy._lib.check(gxy._lib.lib().gxy_dseq_download(ds.h, *(x.ctypes.data for x in held))))
    loop = median(ds.to_host)
    assert loop < 3 * into, (loop, into)
    h = ds.to_host()
    assert all(np.array_equal(x, y) for x, y in zip(held, (h.codes, h.valid, h.mask)))
    empty = gxy.DeviceSeq.from_ascii(b"", ctx).to_host()
    assert len(empty) == 0 and not (empty.codes.any() or empty.valid.any() or empty.mask.any())
