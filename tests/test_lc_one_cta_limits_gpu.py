"""The one-CTA linear-complexity kernel where its workspace is largest: the longest sequence of the entry point without
allocation, and planes whose offsets pass 2^31."""
import numpy as np
import pytest

from conftest import M61

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [65521, M61, (1 << 63) - 25])
def test_noalloc_longest(M, O, p):
    import torch

    out = torch.zeros(1, dtype=torch.int64, device="cuda")
    for n in (262048, 262049, 262144):
        s = torch.from_numpy(O.gen_planted(p, 40, 5, n).view(np.int64)).cuda()
        rc = M.lib().modlin_linear_complexity_device_noalloc(p, s.data_ptr(), n, out.data_ptr(), None)
        assert rc == 0
        torch.cuda.synchronize()
        assert int(out.item()) == 40, n


def test_block_planes_past_2_31_bytes(M):
    import torch

    n = (1 << 28) + 1001
    s = torch.ones(n, dtype=torch.int64, device="cuda")  # s_i = s_(i-1)
    assert M.fp.linear_complexity_device(M61, s.data_ptr(), n, kernel="block") == 1
    s[100:] = 0  # the last nonzero entry at 99
    assert M.fp.linear_complexity_device(M61, s.data_ptr(), n, kernel="block") == 100
    del s
    torch.cuda.empty_cache()
