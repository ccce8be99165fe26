"""The batched rank's panel path (no block step: ragged, dependent or small-prime panels) against the oracle: sides
around the halves and ends of a panel, columns without a pivot at those places, rows that are zero after a few pivots,
panels that are zero from some column on, and primes at the limits of the 32-bit arithmetic. Batches of one shape run on
512 threads a CTA (few), 256 (many), and shared by teams (few, long)."""
import numpy as np
import pytest

from conftest import M61

pytestmark = pytest.mark.gpu

PRIMES = [2, 3, 5, 251, 257, 65521, 65537, 4294967291, 4294967311, M61, (1 << 63) - 25]


def matrix(O, p, n, kind, seed):
    m = O.gen_uniform(p, seed, n * n).reshape(n, n)
    if kind == "holes":  # columns without a pivot at the ends of the panel's halves
        for c in (0, 31, 32, 63, 64, n - 1):
            if c < n:
                m[:, c] = 0
    elif kind == "each":  # every panel's last column depends on the first one
        m[:, 63::64] = m[:, :1]
    elif kind == "low":
        r = max(1, n // 3)
        m[r:] = m[np.arange(n - r) % r]
    elif kind == "tail":  # zero from column 40 of every panel on, but for one late entry
        for c in range(0, n, 64):
            m[:, c + 40:c + 64] = 0
        m[n - 1, n - 1] = 1
    elif kind == "max":  # the largest residues
        m[:] = p - 1
        m[np.arange(n), (7 * np.arange(n)) % n] = p - 2 if p > 2 else 0
    return m


def check(M, O, p, shapes):
    import torch

    ms = [matrix(O, p, n, kind, s + 1) for s, (n, kind) in enumerate(shapes)]
    dev = [torch.from_numpy(m.view(np.int64).copy()).cuda() for m in ms]
    got = M.fp.rank_batch_device([p] * len(ms), [d.data_ptr() for d in dev], [m.shape[0] for m in ms])
    assert got == [O.rank(p, m, m.shape[0]) for m in ms]


KINDS = ["holes", "each", "low", "tail", "max", "full"]


@pytest.mark.parametrize("p", PRIMES)
def test_panels_few(M, O, p):
    check(M, O, p, [(n, k) for n in (1, 2, 31, 33, 63, 64, 65, 97, 129, 200) for k in KINDS])


@pytest.mark.parametrize("p", PRIMES)
def test_panels_many(M, O, p):
    check(M, O, p, [(n, k) for n in (1, 7, 32, 63, 64, 66, 127, 128, 191) for k in KINDS for _ in range(3)])


@pytest.mark.parametrize("p", [2, 3, 65521, 4294967291, M61])
def test_panels_teams(M, O, p):
    for kind in KINDS[:-1]:
        check(M, O, p, [(321, kind), (40, "full")])
