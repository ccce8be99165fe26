"""A long sequence on very few CTAs: a wait of the grid kernel spans a whole sweep of the outputs, which for one working
CTA and 2^24 residues takes seconds. The limit of the waits has to leave room for it: the call returns the complexity,
not a timeout. (A sequence of period 5 ends after the first sweep.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid_ctas", [2, 5])
def test_one_sweep_of_seconds(M, O, grid_ctas):
    import torch

    p, n = (1 << 63) - 25, 1 << 24
    period = torch.tensor([3, 1, 4, 1, 5], dtype=torch.int64, device="cuda")
    s = period.repeat(n // 5 + 1)[:n].contiguous()
    want = O.linear_complexity(p, s[:100].cpu().numpy().view(np.uint64))
    torch.cuda.synchronize()
    assert M.fp.linear_complexity_device(p, s.data_ptr(), n, kernel="grid", grid_ctas=grid_ctas) == want
