"""The work this library is used for, as timed cases: ranks, linear complexities and generator fills over F_p.

Every case goes through the public Python binding, with inputs made from a seed on the GPU. All outputs are whole
numbers (ranks, pivot columns, complexities, residues), so there is one right answer and no error to bound.
"""
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "modlin-rs_b200"))
import modlin  # noqa: E402

M61 = (1 << 61) - 1
P31 = (1 << 31) - 1
P16 = 65521
P7 = 127
P63 = (1 << 63) - 25

LISTED = [
    # The README's first rank test: one 500 x 500 matrix of MIXMAX-17 outputs (rank far below 500), generated and
    # ranked in one call; latency counts.
    {"name": "rank-prng-500", "kind": "rank_prng", "gen": "mixmax17", "p": M61, "n": 500},
    # A mid-sized singular matrix of odd side, recurrence rows: the shape a defective generator gives.
    {"name": "rank-planted-3001", "kind": "rank", "p": M61, "n": 3001, "order": 1100},
    # The small-prime test at a few thousand rows.
    {"name": "rank-6000-p16", "kind": "rank", "p": P16, "n": 6000, "order": 0},
    # The headline rank: 16384 x 16384 over 2^61 - 1, uniform residues (but for one dependent column).
    {"name": "rank-16384", "kind": "rank", "p": M61, "n": 16384, "order": 0},
    # The command line's -R loop: many repetitions of a small test.
    {"name": "rank-reps-256", "kind": "rank_reps", "gen": "xoroshiro128pp", "p": M61, "n": 256, "reps": 200},
    # A batch of uneven matrices over four primes, half of them singular.
    {"name": "rank-batch-512", "kind": "rank_batch", "count": 512, "lo": 64, "hi": 1024},
    # The smallest linear-complexity test: one short sequence in host memory.
    {"name": "lc-1500", "kind": "lc", "p": M61, "n": 1500, "order": 0, "host": True},
    # A planted recurrence found in an odd-length sequence over a 31-bit prime.
    {"name": "lc-planted-30011", "kind": "lc", "p": P31, "n": 30011, "order": 9000, "host": False},
    # The longest test: 200000 uniform residues, complexity near n / 2.
    {"name": "lc-200000", "kind": "lc", "p": M61, "n": 200000, "order": 0, "host": False},
    # Thousands of uneven sequences over three primes, half of them planted, from a plan kept by the caller.
    {"name": "lc-batch-8192", "kind": "lc_batch", "count": 8192, "lo": 256, "hi": 8192},
    # Filling a large test matrix on the device, by both generator families.
    {"name": "fill-mixmax256", "kind": "fill", "gen": "mixmax256", "p": M61, "count": 1 << 28},
    {"name": "fill-xoroshiro", "kind": "fill", "gen": "xoroshiro128pp", "p": M61, "count": 1 << 28},
]


def listed():
    return [dict(c) for c in LISTED]


def _log(rng, lo, hi):
    return min(hi, int(round(lo * (hi / lo) ** rng.random())))


def draw(rng):
    kind = rng.choice(["rank_prng", "rank", "rank", "rank_reps", "rank_batch", "lc", "lc", "lc_batch", "fill", "fill"])
    if kind == "rank_prng":
        return {"kind": kind, "gen": rng.choice(["mixmax17", "mixmax240", "mixmax256", "xoroshiro128pp"]),
                "p": rng.choice([P16, P31, M61]), "n": _log(rng, 64, 3000)}
    if kind == "rank":
        n = _log(rng, 200, 12000)
        order = rng.randint(n // 4, n) if rng.random() < 0.3 and n <= 4000 else 0
        return {"kind": kind, "p": rng.choice([P7, P16, P31, M61, M61, P63]), "n": n, "order": order}
    if kind == "rank_reps":
        n = _log(rng, 32, 600)
        return {"kind": kind, "gen": rng.choice(["mixmax17", "xoroshiro128pp"]), "p": rng.choice([P7, P16, P31, M61]),
                "n": n, "reps": _log(rng, 8, min(1000, 60_000_000 // n ** 2))}
    if kind == "rank_batch":
        return {"kind": kind, "count": _log(rng, 16, 512), "lo": 64, "hi": rng.randint(128, 1024)}
    if kind == "lc":
        n = _log(rng, 200, 200000)
        return {"kind": kind, "p": rng.choice([P7, P16, P31, M61, M61, P63]), "n": n,
                "order": rng.choice([0, rng.randint(1, n // 2)]), "host": rng.random() < 0.5}
    if kind == "lc_batch":
        return {"kind": kind, "count": _log(rng, 64, 8192), "lo": 256, "hi": rng.randint(512, 8192)}
    return {"kind": kind, "gen": rng.choice(["mixmax17", "mixmax240", "mixmax256", "xoroshiro128pp"]),
            "p": rng.choice([0, P16, P31, M61]), "count": _log(rng, 1 << 16, 1 << 28)}


def _empty(count):
    return torch.empty(count, dtype=torch.int64, device="cuda")


def _input(p, order, seed, count):
    """`count` uniform residues mod p, or an order-`order` recurrence with uniform coefficients and state."""
    t = _empty(count)
    if order:
        modlin.gen.planted_device(p, order, seed, t.data_ptr(), count)
    else:
        modlin.gen.uniform_device(p, seed, t.data_ptr(), count)
    return t


def _batch_jobs(case, primes, seed):
    """(p, n, order, seed) of every job: sides or lengths uniform in [lo, hi], half of them planted."""
    rng = np.random.default_rng(seed)
    jobs = []
    for i in range(case["count"]):
        n = int(rng.integers(case["lo"], case["hi"] + 1))
        lo, hi = (n // 4, n) if case["kind"] == "rank_batch" else (16, n // 4)
        order = int(rng.integers(lo, hi + 1)) if i % 2 else 0
        jobs.append((primes[int(rng.integers(len(primes)))], n, order, int(rng.integers(1, 1 << 62))))
    return jobs


def _batch_inputs(jobs, square):
    """All jobs' inputs in one arena; the views in it, job by job."""
    sizes = [n * n if square else n for _, n, _, _ in jobs]
    views = list(torch.split(_empty(sum(sizes)), sizes))
    planted = [i for i, j in enumerate(jobs) if j[2]]
    for i, (p, _, order, seed) in enumerate(jobs):
        if not order:
            modlin.gen.uniform_device(p, seed, views[i].data_ptr(), sizes[i])
    modlin.gen.planted_batch_device([jobs[i][0] for i in planted], [jobs[i][2] for i in planted],
                                    [jobs[i][3] for i in planted], [views[i].data_ptr() for i in planted],
                                    [sizes[i] for i in planted])
    return views


def prepare(case, seed):
    """Sides, lengths and orders are the case's less a little that the seed gives, so that every seed has an answer of
    its own; a uniform matrix gets one column that repeats the first, among its last 64, for the same reason."""
    kind = case["kind"]
    state = dict(case)
    if kind in ("rank_prng", "rank_reps"):
        state["n"] -= seed % 13
    elif kind == "lc" and not case["order"]:
        state["n"] -= seed % 61
    elif case.get("order", 0) > 61:
        state["order"] -= seed % 61
    if kind in ("rank_prng", "rank_reps", "fill"):
        state["prng"] = modlin.prng.Prng(case["gen"], seed % (1 << 31) + 1)
        state["start"] = state["prng"].get_state()
        if kind == "fill":
            state["out"] = _empty(case["count"])
    elif kind == "rank":
        n = case["n"]
        state["matrix"] = _input(case["p"], state["order"], seed, n * n)
        if not state["order"]:
            square = state["matrix"].view(n, n)
            square[:, n - 1 - seed % 64] = square[:, 0]
        state["work"] = torch.empty_like(state["matrix"])
    elif kind == "lc":
        s = _input(case["p"], state["order"], seed, state["n"])
        state["seq"] = s.cpu().numpy().view(np.uint64) if case["host"] else s
    elif kind == "rank_batch":
        jobs = _batch_jobs(case, [P7, P16, P31, M61], seed)
        views = _batch_inputs(jobs, True)
        state["matrix"] = views[0]._base
        state["work"] = torch.empty_like(state["matrix"])
        off = state["work"].data_ptr() - state["matrix"].data_ptr()
        state["ps"], state["ns"] = [j[0] for j in jobs], [j[1] for j in jobs]
        state["ptrs"] = [v.data_ptr() + off for v in views]
    elif kind == "lc_batch":
        jobs = _batch_jobs(case, [P16, P31, M61], seed)
        state["seqs"] = _batch_inputs(jobs, False)
        state["out"] = _empty(len(jobs))
        state["plan"] = modlin.fp.BatchPlan("lc", [j[0] for j in jobs], [v.data_ptr() for v in state["seqs"]],
                                            [j[1] for j in jobs], state["out"].data_ptr())
    return state


def run(state):
    kind = state["kind"]
    if kind == "rank_prng":
        state["prng"].set_state(state["start"])
        r = modlin.fp.rank_prng(state["p"], state["prng"], state["n"])
        return {"rank": r, "corank": state["n"] - r}
    if kind == "rank_reps":
        state["prng"].set_state(state["start"])
        return np.array(modlin.fp.rank_prng_batch(state["p"], state["prng"], state["n"], state["reps"]))
    if kind == "rank":
        # The call eliminates in place: it works on a copy, so that a pass can be repeated.
        state["work"].copy_(state["matrix"])
        r, cols = modlin.fp.rank_device(state["p"], state["work"].data_ptr(), state["n"], pivot_cols=True)
        profile = np.zeros(state["n"], dtype=bool)
        profile[cols] = True
        return {"rank": r, "pivot_cols": profile}
    if kind == "rank_batch":
        state["work"].copy_(state["matrix"])
        return np.array(modlin.fp.rank_batch_device(state["ps"], state["ptrs"], state["ns"]))
    if kind == "lc":
        if state["host"]:
            return modlin.linear_complexity(state["p"], state["seq"])
        return modlin.fp.linear_complexity_device(state["p"], state["seq"].data_ptr(), state["n"])
    if kind == "lc_batch":
        state["plan"].launch()
        return state["out"]
    state["prng"].set_state(state["start"])
    state["prng"].fill_device(state["out"].data_ptr(), state["count"], state["p"])
    return state["out"]


def _rank_work(n, r):
    # Elimination of r pivots: sum over k < r of (n - k)^2 multiply-adds.
    return 2.0 * (n ** 3 - (n - r) ** 3) / 3


def _lc_work(n, order):
    # The discrepancy and the update of a step take l multiply-adds each, and l grows by one half a step up to
    # the complexity; from step 2 L on there are discrepancies only.
    L = order or n // 2
    return 2.0 * (2 * L * L + max(0, n - 2 * L) * L)


def work(case):
    kind = case["kind"]
    if kind in ("rank", "rank_prng"):
        n = case["n"]
        read = 8.0 * n * n if kind == "rank" else 0.0  # a generated matrix is made on the way
        return {"bytes": read + 8, "flops": _rank_work(n, case.get("order") or n)}
    if kind == "rank_reps":
        return {"bytes": 8.0 * case["reps"], "flops": case["reps"] * _rank_work(case["n"], case["n"])}
    if kind == "lc":
        return {"bytes": 8.0 * case["n"] + 8, "flops": _lc_work(case["n"], case["order"])}
    if kind == "fill":
        return {"bytes": 8.0 * case["count"], "flops": 0.0}
    # Batches: means over the drawn sides or lengths.
    k = np.arange(case["lo"], case["hi"] + 1, dtype=np.float64)
    if kind == "rank_batch":
        flops = 0.5 * (_rank_work(k, k) + _rank_work(k, 0.625 * k)).mean()
        return {"bytes": case["count"] * (8 * (k ** 2).mean() + 8), "flops": case["count"] * flops}
    L = k / 8
    flops = 0.5 * (k ** 2 + 2 * (2 * L * L + (k - 2 * L) * L)).mean()
    return {"bytes": case["count"] * (8 * k.mean() + 8), "flops": case["count"] * flops}


def exact(case, seed):
    """Every output is a whole number: compared for equality, with nothing to measure against."""
    return None
