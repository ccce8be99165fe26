"""Device memory that a single linear complexity asks for: 4 bytes a residue and limb on many CTAs, and half of that on one,
which AUTO takes when memory is short. On a runtime that only notes launches (fake_cudart.cpp)."""
import json
import subprocess
import sys

import pytest

from conftest import M61, PKG
from fakes import fake_lib  # noqa: F401

N = 1 << 20
CHILD = r"""
import ctypes, json, sys
sys.path.insert(0, sys.argv[1])
import modlin, modlin._lib
modlin._lib.library_path = sys.argv[2]
L = modlin.lib()
L.fake_set_free.argtypes = [ctypes.c_size_t]
L.fake_set_free(int(sys.argv[4]))
try:
    modlin.fp.linear_complexity_device(int(sys.argv[3]), 1 << 40, 1 << 20, kernel=sys.argv[5])
    rc = 0
except modlin._lib.ModlinError as e:
    rc = e.code
print(json.dumps([rc, L.fake_launches(b"bm_long_kernel"), L.fake_launches(b"bm_block_kernel")]))
"""


@pytest.mark.parametrize("p,free,kernel,want", [
    (M61, 40 * N, "auto", [0, 1, 0]),
    (M61, 20 * N, "auto", [0, 0, 1]),
    (M61, 20 * N, "grid", [-5, 0, 0]),
    (M61, 10 * N, "auto", [-5, 0, 0]),
    (2147483647, 20 * N, "auto", [0, 1, 0]),
    (65521, 10 * N, "grid", [0, 1, 0]),
    (2, 20 * N, "auto", [0, 1, 0]),
])
def test_workspace(fake_lib, p, free, kernel, want):
    res = subprocess.run([sys.executable, "-c", CHILD, PKG, fake_lib, str(p), str(free), kernel], capture_output=True,
                         text=True, timeout=300)
    assert res.returncode == 0, res.stderr[-2000:]
    assert json.loads(res.stdout.strip().splitlines()[-1]) == want
