"""One process, two devices, without a GPU: the library's own objects linked with a runtime that only notes the launches
(fake_cudart.cpp). What a function is allowed (dynamic shared memory) and what a device holds (clusters) belong to a
device: after the first has done its work, every entry point has to work on the second one too."""
import json
import subprocess
import sys

from conftest import PKG
from fakes import fake_lib  # noqa: F401

CHILD = r"""
import ctypes, json, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
import modlin, modlin._lib
modlin._lib.library_path = sys.argv[2]
L = modlin.lib()
L.fake_rejected.restype = ctypes.c_char_p
M61, P63, P31 = (1 << 61) - 1, (1 << 63) - 25, (1 << 31) - 1
PRIMES = [127, 65521, P31, M61, P63]
buf = np.zeros(1 << 23, dtype=np.uint64)
d = buf.ctypes.data
out, failed = np.zeros(64, dtype=np.int64), []

def fills():
    for kind in ("mixmax17", "mixmax240", "mixmax256", "xoroshiro128pp"):
        modlin.prng.Prng(kind, 1).fill_device(d, 1 << 22, M61)
def ranks():
    for p in PRIMES:
        for kernel in ("plain", "tc"):
            for n in (300, 641):
                modlin.fp.rank_device(p, d, n, kernel=kernel)
            modlin.fp.trailing_update_device(p, d, 640, 512, 256, d, d, 640, 64, kernel=kernel)
        modlin.fp.block_inverse_device(p, d, 64, d)
        modlin.fp.panel_pivots_device(p, d, 64, 100, 64)
def pairs():
    L.modlin_set_tc_pairs(1)
    modlin.fp.rank_device(M61, d, 641, kernel="tc")
    L.modlin_set_tc_pairs(0)
def batches():
    for ns in ([64] * 400, [512] * 3, [700] + [64] * 40):  # 256 threads, 512, teams
        modlin.fp.rank_batch_device([M61] * len(ns), [d] * len(ns), ns)
        plan = modlin.fp.BatchPlan("rank", [M61] * min(64, len(ns)), [d] * min(64, len(ns)), ns[:64], out.ctypes.data)
        plan.launch()
def complexities():
    for p in [2] + PRIMES:
        for kernel in ("block", "grid", "cluster"):
            modlin.fp.linear_complexity_device(p, d, 10000, kernel=kernel)
        modlin.fp.lc_batch_device([p] * 3, [d] * 3, [9000, 100, 20000])
        plan = modlin.fp.BatchPlan("lc", [p] * 3, [d] * 3, [9000, 100, 20000], out.ctypes.data)
        plan.launch()
        modlin._lib.check(L.modlin_linear_complexity_device_noalloc(p, d, 9000, out.ctypes.data, None))
def peaks():
    modlin.fp.plain_mac_peak(M61)
    modlin.fp.plain_mac_peak(65521)

for device in (0, 1):
    L.fake_set_device(device)
    for f in (fills, ranks, pairs, batches, complexities, peaks):
        try:
            f()
        except modlin._lib.ModlinError as e:
            failed.append([device, f.__name__, str(e)])
failed += L.fake_rejected().decode().splitlines()
print(json.dumps({"failed": failed, "teams": L.fake_launches(b"rank_team_kernel")}))
"""


def test_every_entry_point_on_the_second_device(fake_lib):
    res = subprocess.run([sys.executable, "-c", CHILD, PKG, fake_lib], capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stderr[-2000:]
    got = json.loads(res.stdout.strip().splitlines()[-1])
    assert got["failed"] == []
    assert got["teams"] > 0
