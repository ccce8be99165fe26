"""Batched rank by block steps: sides at the edges of the 64-column panels and 256-column strips, both launch shapes
(256 and 512 threads), blocks without a pivot (dependent rows and columns, zero blocks, permuted rows), and rests that
vanish, for every limb count. Exact against the oracle."""
import numpy as np
import pytest

from conftest import M61

pytestmark = pytest.mark.gpu

PRIMES = [2, 127, 251, 65521, 65537, (1 << 31) - 1, 4294967291, M61, (1 << 63) - 25]


def matrices(O, p, n):
    base = O.gen_uniform(p, n, n * n).reshape(n, n)
    yield base
    m = base.copy()
    m[:min(16, n)] = 0  # no pivot in the first 16 rows
    yield m
    m = base.copy()
    m[:, n // 3] = m[:, 0]  # a dependent column
    yield m
    m = base.copy()
    m[n // 2:] = m[:n - n // 2]  # half the rank: the rest vanishes
    yield m
    yield np.eye(n, dtype=np.uint64)[::-1].copy() * np.uint64(p - 1)
    m = np.full((n, n), p - 1, dtype=np.uint64)  # largest residues, rank 1
    yield m


def ranks(M, p, mats, n, reps):
    import torch
    a = torch.from_numpy(np.stack(mats).view(np.int64)).cuda()
    w = a.repeat(reps, 1, 1).contiguous()
    k = len(mats) * reps
    got = M.fp.rank_batch_device([p] * k, [w.data_ptr() + 8 * n * n * i for i in range(k)], [n] * k)
    return got


@pytest.mark.parametrize("p", PRIMES)
def test_edges(M, O, p):
    for n in (63, 64, 65, 127, 129, 320, 385):
        mats = list(matrices(O, p, n))
        want = [O.rank(p, m.reshape(-1), n) for m in mats]
        # Few jobs: 512 threads. More jobs than SMs: 256 threads below side 384.
        assert ranks(M, p, mats, n, 1) == want, (p, n)
        if n in (65, 320):
            assert ranks(M, p, mats, n, 26) == want * 26, (p, n)
