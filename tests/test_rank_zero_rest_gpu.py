"""Panels without a pivot: the rank ends early only when everything that is left is zero. Zero column blocks before
nonzero ones, a single nonzero entry in the last column, low-rank matrices, and the small-prime field policy."""
import numpy as np
import pytest

from conftest import M61

pytestmark = pytest.mark.gpu


def matrices(O, p, n):
    rng = np.random.default_rng(n)
    base = O.gen_uniform(p, 7, n * n).reshape(n, n)
    for lo, hi in [(0, n - 1), (70, n - 3), (64, 200), (130, 131)]:
        m = base.copy()
        m[:, lo:hi] = 0
        yield m
    m = np.zeros((n, n), dtype=np.uint64)
    yield m.copy()
    m[n - 1, n - 1] = 1
    yield m
    m = base.copy()
    m[100:] = m[rng.integers(0, 100, n - 100)]  # rank <= 100
    yield m
    m = m.copy()
    m[n - 1, n - 2:] = p - 1  # and one entry more in the last columns
    yield m


@pytest.mark.parametrize("p", [2, 127, 65521, 4294967291, M61, (1 << 63) - 25])
def test_zero_blocks(M, O, p):
    n = 450
    for k, m in enumerate(matrices(O, p, n)):
        want = O.rank(p, m, n, with_pcols=True)
        for kernel in ("plain", "tc"):
            done = []
            got = M.rank(p, m, n, kernel=kernel, pivot_cols=True, progress=lambda d, t: done.append((d, t)))
            assert got == want, (p, k, kernel)
            assert done[-1][1] == n and done == sorted(done)
            if want[0] < n:
                assert done[-1][0] == n
