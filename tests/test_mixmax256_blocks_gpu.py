"""MIXMAX-256 device fill with lazily reduced iterations: states planted so that an entry or sumtot is 0 mod 2^61 - 1
in the first, second or third iteration of a block (ROOT may then hold 2^61 - 1, which reaches outputs and the state
only from the third), and counts around power-of-two segments. Against the host stream."""
import numpy as np
import pytest

from mixmax_model import MIX, plant, set_mix_state
from test_prng_gpu import dev_fill

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("it", [1, 2, 3, 4, 5, 6, 61, 62, 63])
@pytest.mark.parametrize("entry", [0, 1, 2, 3, 255])
def test_planted_zero(M, it, entry):
    kind = "mixmax256"
    N = MIX[kind][0]
    if it == 1 and entry in (1, 2):
        entry = 4  # after one iteration these do not depend on the free entry v[3]
    x = plant(kind, np.random.default_rng(100 * it + entry), [(it, entry)])
    for count in (21 * (N - 1), 22 * (N - 1) + 5):
        h, d = M.prng.Prng(kind, 1), M.prng.Prng(kind, 1)
        set_mix_state(h, kind, x, N)
        set_mix_state(d, kind, x, N)
        assert np.array_equal(dev_fill(d, count), h.fill(count)), count
        assert np.array_equal(d.get_state(), h.get_state()), count


@pytest.mark.parametrize("kind", ["mixmax17", "mixmax", "mixmax256"])
def test_segment_counts(M, kind):
    n = MIX[kind][0] - 1
    for blocks in (1, 2, 31, 3551, 3552, 3553, 7200):
        h, d = M.prng.Prng(kind, 3), M.prng.Prng(kind, 3)
        count = blocks * n - 1
        assert np.array_equal(dev_fill(d, count), h.fill(count)), blocks
        assert np.array_equal(d.get_state(), h.get_state()), blocks
