"""modlin_rank_batch_device_ex: the kernel option decides for sides above 8192 (include/modlin.h), which run one after
another. Seen on a runtime that only notes launches (fake_cudart.cpp): the inverse of a diagonal block belongs to the
tensor-core path alone. Memory is never touched there, so the matrices are addresses only."""
import json
import subprocess
import sys

import pytest

from conftest import PKG
from fakes import fake_lib  # noqa: F401

CHILD = r"""
import json, sys
sys.path.insert(0, sys.argv[1])
import modlin, modlin._lib
modlin._lib.library_path = sys.argv[2]
modlin.fp.rank_batch_device([65521, 65521], [1 << 40, 1 << 41], [8193, 100], kernel=sys.argv[3])
L = modlin.lib()
print(json.dumps({k: L.fake_launches(k.encode()) for k in ("block_inverse_kernel", "rank_batch_kernel")}))
"""


@pytest.mark.parametrize("kernel,blocks", [("plain", False), ("tc", True), ("auto", True)])
def test_kernel_option_reaches_large_sides(fake_lib, kernel, blocks):
    res = subprocess.run([sys.executable, "-c", CHILD, PKG, fake_lib, kernel], capture_output=True, text=True,
                         timeout=300)
    assert res.returncode == 0, res.stderr[-2000:]
    got = json.loads(res.stdout.strip().splitlines()[-1])
    assert (got["block_inverse_kernel"] > 0) == blocks
    assert got["rank_batch_kernel"] == 1
