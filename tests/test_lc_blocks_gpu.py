"""Linear complexity in blocks of 32 steps (one CTA) and superblocks of 512 (many CTAs): lengths at the edges of
both, every field policy, and sequences whose discrepancies vanish for long runs (the block's matrix then has high
degrees, and the complexity jumps by more than a block). Exact against the oracle."""
import numpy as np
import pytest

from conftest import M61

pytestmark = pytest.mark.gpu

# Even; odd below 2^28; up to 2^31; up to 2^63; 2^61 - 1.
PRIMES = [2, 3, 65521, (1 << 28) - 57, (1 << 28) + 3, (1 << 31) - 1, (1 << 32) - 5, M61, (1 << 63) - 25]
LENGTHS = [1, 31, 32, 33, 64, 65, 96, 511, 512, 513, 544, 1023, 1024, 1025, 1700]


def sequences(O, p, n):
    yield O.gen_uniform(p, n, n)
    full = np.full(n, p - 1, dtype=np.uint64)  # largest residues, complexity 1
    yield full
    s = np.zeros(n, dtype=np.uint64)  # one nonzero after a run of zeros: the complexity jumps to its index + 1
    s[n * 2 // 3] = 1
    yield s
    s = np.zeros(n, dtype=np.uint64)  # sparse: runs of zero discrepancies between jumps
    s[::37] = O.gen_uniform(p, 5, len(s[::37]))
    yield s
    s = full.copy()  # constant, then one value off near the end
    s[n - 1 - n // 10] = 0
    yield s
    if n > 100:
        yield O.gen_planted(p, n // 5, 9, n)


@pytest.mark.parametrize("p", PRIMES)
def test_block_and_superblock_edges(M, O, p):
    for n in LENGTHS:
        for k, s in enumerate(sequences(O, p, n)):
            want = O.linear_complexity(p, s)
            got = {kern: M.linear_complexity(p, s, kernel=kern) for kern in ("block", "grid", "cluster")}
            assert got == dict.fromkeys(got, want), (p, n, k)


def test_batch_of_edges(M, O):
    """The same sequences as one batch: matrices of mixed primes, some in the global workspace."""
    items = [(p, s) for p in PRIMES for n in (33, 512, 1025) for s in sequences(O, p, n)]
    items += [(M61, O.gen_uniform(M61, 3, 7500)), ((1 << 31) - 1, O.gen_planted((1 << 31) - 1, 3000, 4, 14000))]
    assert M.lc_batch(items) == [O.linear_complexity(p, s) for p, s in items]


@pytest.mark.parametrize("ctas", [1, 2, 3, 9])
def test_few_ctas(M, O, ctas):
    """More chunks than CTAs, and chunks that do not fill their share."""
    for p in (65521, M61):
        for n, L in [(1500, 0), (3333, 700), (6000, 0)]:
            s = O.gen_planted(p, L, 2, n) if L else O.gen_uniform(p, 2, n)
            assert M.linear_complexity(p, s, kernel="grid", grid_ctas=ctas) == O.linear_complexity(p, s), (p, n)
