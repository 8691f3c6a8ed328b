"""The order of the representatives after clustering: by segment, then by energy, as
np.lexsort has it."""
import numpy as np
import pytest

from geaxdock_gpu_b200.postmc import _by_segment_and_energy


@pytest.mark.parametrize("n,n_seg,special", [(0, 1, False), (1, 1, False), (2000, 1, True),
                                             (3000, 40, True), (9000, 70000, True)])
def test_radix_order_is_the_lexicographic_one(n, n_seg, special):
    rng = np.random.default_rng(n + n_seg)
    seg = rng.integers(0, n_seg, n)
    e = rng.normal(0, 1, n).astype(np.float32)
    if special:
        e[::7] = e[::7].round(1)  # ties keep their order
        e[rng.integers(0, n, 40)] = np.resize(
            np.array([np.nan, -np.nan, np.inf, -np.inf, 0.0, -0.0, 1e-42, -1e-42], np.float32), 40)
    assert np.array_equal(_by_segment_and_energy(seg, e), np.lexsort((e, seg)))
