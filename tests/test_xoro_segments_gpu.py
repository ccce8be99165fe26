"""xoroshiro128++ device fill: segments of 2^m outputs from device-side jumps. Counts around full blocks of 128
segments, longer segments, and output buffers that are not 16-byte aligned, against the host stream."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("count", [63, 64, 65, 64 * 128 - 1, 64 * 128, 64 * 128 + 1, 64 * 160 + 15, 64 * 4224,
                                   (1 << 24) + 129, 40_000_003])
def test_segments_match_host_stream(M, count, offset):
    h, d = M.prng.Prng("xoroshiro128pp", 5), M.prng.Prng("xoroshiro128pp", 5)
    t = torch.full((count + 3,), -1, dtype=torch.int64, device="cuda")
    d.fill_device(t.data_ptr() + 8 * offset, count)
    got = t.cpu().numpy()
    assert np.array_equal(got[offset:offset + count].view(np.uint64), h.fill(count))
    assert np.all(got[:offset] == -1) and np.all(got[offset + count:] == -1)
    assert np.array_equal(d.get_state(), h.get_state())
