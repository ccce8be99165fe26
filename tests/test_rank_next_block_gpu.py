"""The block pipeline over every limb count: the next block's own product (small tensor-core products with ragged last
blocks) and the end on a zero rest after a panel with some pivots, against the oracle."""
import numpy as np
import pytest

from conftest import M61

pytestmark = pytest.mark.gpu

PRIMES = [251, 65521, 16777213, 4294967291, (1 << 40) - 87, (1 << 48) - 59, (1 << 56) - 5, M61, (1 << 63) - 25]


@pytest.mark.parametrize("p", PRIMES)
def test_next_block(M, O, p):
    for n in (129, 193, 256, 321):
        m = O.gen_uniform(p, n, n * n).reshape(n, n)
        assert M.rank(p, m, n, kernel="tc", pivot_cols=True) == O.rank(p, m, n, with_pcols=True), n


@pytest.mark.parametrize("p", PRIMES)
@pytest.mark.parametrize("r", [1, 63, 65, 200])
def test_short_panel_zero_rest(M, O, p, r):
    n = 330
    m = O.gen_uniform(p, r, n * n).reshape(n, n)
    m[r:] = m[np.arange(n - r) % r]  # rank r
    for last in (0, 1):  # 1: a single entry more in the last corner
        m[n - 1, n - 1] = (int(m[n - 1, n - 1]) + last) % p
        for kernel in ("plain", "tc"):
            assert M.rank(p, m, n, kernel=kernel, pivot_cols=True) == O.rank(p, m, n, with_pcols=True), (last, kernel)
