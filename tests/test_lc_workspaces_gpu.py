"""Where the one-CTA linear-complexity kernels keep their residuals: byte planes of 1, 2, 4 or 8 limbs in shared memory up
to 200 KiB, in the CTA's slice of a global workspace beyond, and single launches whose shared memory passes 48 KiB
together with the kernel's own. Against the oracle."""
import numpy as np
import pytest

from conftest import M61

pytestmark = pytest.mark.gpu

P31, P63 = (1 << 31) - 1, (1 << 63) - 25


def words(limbs, n):  # of the planes, as bm_words
    return 2 * limbs * ((n + 175) // 16 * 16) // 8


def sequences(O, jobs):
    return [O.gen_planted(p, n // 5, 3 + i, n) if i % 2 else O.gen_uniform(p, 3 + i, n) for i, (p, n) in enumerate(jobs)]


# Longest first in both kinds of memory, and slices of several CTAs at once.
JOBS = [(M61, 12700), (M61, 13001), (P63, 12649), (P31, 25500), (M61, 12600), (M61, 300), (P31, 26003), (65521, 9000),
        (2, 25500), (P63, 14003)]


@pytest.mark.parametrize("plan", [False, True])
def test_batch_beyond_shared_memory(M, O, plan):
    import torch

    cap = 200 * 1024 // 8
    beyond = [words(8 if p > 1 << 32 else 4 if p in (2, P31) else 2, n) > cap for p, n in JOBS]
    assert any(beyond) and not all(beyond)
    seqs = sequences(O, JOBS)
    dev = [torch.from_numpy(s.view(np.int64).copy()).cuda() for s in seqs]
    ps, ns, ptrs = [p for p, _ in JOBS], [n for _, n in JOBS], [d.data_ptr() for d in dev]
    want = [O.linear_complexity(p, s) for (p, _), s in zip(JOBS, seqs)]
    if plan:
        out = torch.zeros(len(JOBS), dtype=torch.int64, device="cuda")
        P = M.fp.BatchPlan("lc", ps, ptrs, ns, out.data_ptr())
        for _ in range(2):
            out.zero_()
            torch.cuda.synchronize()
            P.launch()
            torch.cuda.synchronize()
            assert out.tolist() == want
        P.free()
    else:
        assert M.fp.lc_batch_device(ps, ptrs, ns) == want


@pytest.mark.parametrize("p,limbs", [(M61, 8), (P31, 4), (127, 1)])
def test_single_around_48_kib(M, O, p, limbs):
    n0 = 48 * 1024 // (2 * limbs) - 175
    for n in (n0 - 240, n0 - 16, n0 + 1) if limbs == 1 else (n0 - 320, n0 - 240, n0 - 170, n0 - 100, n0 - 16, n0, n0 + 1):
        s = O.gen_uniform(p, n, n)
        assert M.linear_complexity(p, s, kernel="block") == O.linear_complexity(p, s), n
