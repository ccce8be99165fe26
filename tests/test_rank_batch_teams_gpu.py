"""Batches with a few long matrices: a thread-block cluster shares each of the longest (row tiles dealt to its CTAs),
the rest go one to a CTA. Ranks against the oracle: full rank, planted low rank, ragged sides, singular leading blocks
that are tried again with other rows or go through the panel path, and small primes whose blocks often fail."""
import numpy as np
import pytest

from conftest import M61

pytestmark = pytest.mark.gpu


def matrix(O, p, n, kind, seed):
    m = O.gen_uniform(p, seed, n * n).reshape(n, n)
    if kind == "low":  # rank <= n / 3
        r = n // 3
        m[r:] = m[np.arange(n - r) % r]
    elif kind == "zero":  # a zero leading block, zero columns, one late entry
        m[:64, :64] = 0
        m[:, 130:140] = 0
        m[:, n - 70:] = 0
        m[n - 1, n - 1] = 1
    elif kind == "ident":  # two singular blocks in a row: the third set of rows has the pivots
        m[:128, :64] = 0
    return m


@pytest.mark.parametrize("p", [2, 3, 127, 65521, 4294967291, M61, (1 << 63) - 25])
@pytest.mark.parametrize("few", [1, 5, 40])
def test_teams(M, O, p, few):
    import torch

    sides = [256, 257, 319, 320, 385, 448, 511]
    kinds = ["full", "low", "zero", "ident"]
    items = []
    for i in range(few):
        n = sides[i % len(sides)]
        items.append((n, kinds[(i + i // len(sides) + p) % 4], i))
    for i in range(60 if few == 40 else 0):  # shorter ones behind them
        items.append((1 + 3 * i, "full" if i < 30 else "low" if 3 * i > 8 else "full", 100 + i))
    ms = [matrix(O, p, n, kind, 10 + s) for n, kind, s in items]
    dev = [torch.from_numpy(m.view(np.int64).copy()).cuda() for m in ms]
    got = M.fp.rank_batch_device([p] * len(ms), [d.data_ptr() for d in dev], [n for n, _, _ in items])
    assert got == [O.rank(p, m, m.shape[0]) for m in ms]


@pytest.mark.parametrize("kernel", ["plan", "graph"])
def test_teams_in_a_plan(M, O, kernel):
    import torch

    p, ns = M61, [450, 320, 90, 33]
    ms = [matrix(O, p, n, k, 3) for n, k in zip(ns, ["full", "low", "full", "full"])]
    src = [torch.from_numpy(m.view(np.int64).copy()).cuda() for m in ms]
    work = [torch.empty_like(t) for t in src]
    out = torch.zeros(len(ns), dtype=torch.int64, device="cuda")
    plan = M.fp.BatchPlan("rank", [p] * len(ns), [t.data_ptr() for t in work], ns, out.data_ptr())
    want = [O.rank(p, m, m.shape[0]) for m in ms]
    st = torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    if kernel == "graph":
        with torch.cuda.graph(g, stream=st):
            for t, s in zip(work, src):
                t.copy_(s)
            plan.launch(torch.cuda.current_stream().cuda_stream)
    for _ in range(3):
        out.zero_()
        torch.cuda.synchronize()
        if kernel == "graph":
            g.replay()
        else:
            for t, s in zip(work, src):
                t.copy_(s)
            torch.cuda.synchronize()
            plan.launch(st.cuda_stream)
        torch.cuda.synchronize()
        assert out.tolist() == want
    del g
    plan.free()
