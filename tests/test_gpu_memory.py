"""A table is built where only what it cannot do without fits the device's memory."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))

# (A process of its own: the memory that earlier calls' pools keep would do.)
PROGRAM = """
import sys
sys.path.insert(0, {here!r})
import conftest, torch, numpy as np
gxy = sys.modules["lastz_gxy_b200"]
length, pattern, room = {length}, {pattern!r}, {room} << 20
rng = np.random.default_rng(4)
bases = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, length)].tobytes()
c = gxy.Context(0)
ds = gxy.DeviceSeq.from_ascii(bases, c)
torch.cuda.mem_get_info()
ballast = torch.empty(torch.cuda.mem_get_info()[0] - room, dtype=torch.uint8, device="cuda:0")
few = gxy.PosTable.build_view(ds, 0, length, pattern, 1)
del ballast
torch.cuda.empty_cache()
many = gxy.PosTable.build_view(ds, 0, length, pattern, 1)
for x, y in zip(few.arrays(), many.arrays()):
    assert np.array_equal(x, y)
q = gxy.DeviceSeq.from_ascii(bases[1000:40_000], c)
m = gxy.ScoringMatrix.hoxd70()
for transitions in {transitions}:
    sp = gxy.SearchParams(transitions=transitions)
    a, b = gxy.search_device(few, q, m, sp), gxy.search_device(many, q, m, sp)
    assert len(a) and a.tobytes() == b.tobytes()
print("ok")
"""


@pytest.mark.parametrize("length,pattern,room,transitions", [
    # 256 MB of bucket starts; neighbour masks and packed bounds would be 192 MB more.
    (600_000, "1" * 13, 356, (0, 1, 2)),
    # 153 MB of positions, 88 MB of bucket lists; the partitions' windows would be 306 MB more.
    (40_000_000, "1" * 8, 310, ()),
])
def test_table_in_the_memory_that_is_left(length, pattern, room, transitions):
    code = PROGRAM.format(here=HERE, length=length, pattern=pattern, room=room, transitions=transitions)
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, CUDA_MODULE_LOADING="EAGER"))
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr


TWOBIT = """
import sys
sys.path.insert(0, {here!r})
import conftest, struct, torch, numpy as np
gxy = sys.modules["lastz_gxy_b200"]
rng = np.random.default_rng(6)
n, records = 25_000_000, 8
names = [b"r%d" % k for k in range(records)]
index, body, at = b"", [], 16 + sum(5 + len(x) for x in names)
for x in names:
    body.append(struct.pack("<4I", n, 0, 0, 0) + rng.integers(0, 256, n // 4, np.uint8).tobytes())
    index += struct.pack("<B", len(x)) + x + struct.pack("<I", at)
    at += len(body[-1])
data = struct.pack("<4I", 0x1A412743, 0, records, 0) + index + b"".join(body)
c = gxy.Context(0)
torch.cuda.mem_get_info()
ballast = torch.empty(torch.cuda.mem_get_info()[0] - ({room} << 20), dtype=torch.uint8, device="cuda:0")
few = gxy.parse_2bit(data, c)
del ballast
torch.cuda.empty_cache()
many = gxy.parse_2bit(data, c)
for (a, x), (b, y) in zip(few, many):
    x, y = x.to_host(), y.to_host()
    assert a == b and len(x) == n
    assert np.array_equal(x.codes, y.codes) and np.array_equal(x.valid, y.valid) and np.array_equal(x.mask, y.mask)
print("ok")
"""


@pytest.mark.parametrize("room", [
    # 95 MB of sequences, 48 of packed bases: none is left for the copies' streams.
    130,
    # Nor for the packed bases of all eight records at once.
    112,
])
def test_2bit_in_the_memory_that_is_left(room):
    r = subprocess.run([sys.executable, "-c", TWOBIT.format(here=HERE, room=room)], capture_output=True, text=True,
                       timeout=300, env=dict(os.environ, CUDA_MODULE_LOADING="EAGER"))
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr


GAPPED = """
import sys
sys.path.insert(0, {here!r})
import conftest, torch, numpy as np
gxy = sys.modules["lastz_gxy_b200"]
from test_gpu_gapped import both
rng = np.random.default_rng(3)
bases = np.frombuffer(b"ACGT", np.uint8)
t, q = np.full(1000, ord("N"), np.uint8), np.full(760, ord("N"), np.uint8)
t[:372] = bases[rng.integers(0, 4, 372)]
q[:102] = t[270:372]
seg = t[1:353].copy()
at = rng.choice(352, 185, replace=False)
seg[at] = bases[(np.searchsorted(bases, seg[at]) + 2) % 4]
q[291:643] = seg
c = gxy.Context(0)
c.set_tuning(gapped_pool_blocks=8)
torch.cuda.mem_get_info()
ballast = torch.empty(torch.cuda.mem_get_info()[0] - (640 << 20), dtype=torch.uint8, device="cuda:0")
g, w, st = both(gxy, c, t.tobytes(), q.tobytes(), [(0, 0)] * 400, thr=-10 ** 6)
assert g == w and st["second_pass_sides"] == 400
# (every side once, and the groups that were short of run words again)
one = st["cells"] // 400
print("ok", st["second_pass_cells"] // one)
"""


def test_gapped_second_pass_in_groups_short_of_runs():
    # 400 sides of the shape of test_gapped_second_pass_best_right_of_the_last_rows, in
    # groups that fit half of what is left: run words reserved by the last rows' ends
    # last for the first groups, a later one makes room and runs again.
    r = subprocess.run([sys.executable, "-c", GAPPED.format(here=HERE)], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, CUDA_MODULE_LOADING="EAGER"))
    assert r.returncode == 0 and r.stdout.startswith("ok "), r.stdout + r.stderr
    assert 400 < int(r.stdout.split()[1]) < 800, r.stdout
