"""Panels whose 64-column block is singular, in the single rank: over large primes the block pipeline's chain gives up on
them without a second elimination, mod 2 and 3 no block is tried at all. Ranks and pivot columns against the oracle,
with dependent columns in the first and the second half of a 128-column block, in later steps, and in every panel."""
import numpy as np
import pytest

from conftest import M61

pytestmark = pytest.mark.gpu


def matrix(O, p, n, kind):
    m = O.gen_uniform(p, 7, n * n).reshape(n, n)
    if kind == "first":
        m[:, 40] = m[:, 3]
    elif kind == "second":
        m[:, 100] = m[:, 3]
    elif kind == "late":
        m[:, n - 70] = m[:, 0]
    elif kind == "each":
        m[:, 63::64] = m[:, :1]
    elif kind == "rows":  # the block's rows are dependent, its columns are not
        m[1] = m[0]
        m[70] = m[65]
    return m


@pytest.mark.parametrize("p", [2, 3, 5, 65521, 1048573, 2147483647, M61, (1 << 63) - 25])
@pytest.mark.parametrize("n", [128, 193, 400, 641])
def test_singular_blocks(M, O, p, n):
    for kind in ("first", "second", "late", "each", "rows", "none"):
        m = matrix(O, p, n, kind)
        assert M.rank(p, m, n, kernel="tc", pivot_cols=True) == O.rank(p, m, n, with_pcols=True), kind
