"""The k-means kernels of large segments (csrc/gd_kmeans.cu: two objects and two centres at a time,
one CTA per cluster's sums) at the sizes where they can go wrong, bit for bit against the CPU
oracle: odd numbers of centres, one centre, more centres than shared memory holds, clusters of
more than a tile of members, blocks that hold the end of a large segment and small ones."""
import numpy as np
import pytest

from geaxdock_gpu_b200 import postmc
from oracle import kmeans as ok
from tests.conftest import have_gpu

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_gpu(), reason="needs a B200")]


@pytest.mark.parametrize("sizes,k", [([8193], 501), ([8200, 40, 300, 600], 7), ([8450], 1),
                                     ([8193], 1024), ([8193], 1025), ([300, 8448, 256], 2)])
def test_large_segments_match_oracle(sizes, k):
    rng = np.random.default_rng(k)
    # slowly wandering energies, as records are: many near-ties between neighbouring centres
    E = np.cumsum(rng.normal(0, 0.05, (sum(sizes), 9)), axis=0).astype(np.float32)
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
    mem, med, size, passes, base = postmc.kmeans(E, off, [k] * len(sizes), 4, max_iter=12)
    for s in range(len(sizes)):
        m_o, r_o, z_o, p_o = ok.cluster_by_kmeans(E[off[s]:off[s + 1]], k, 4, s, max_iter=12)
        cnt = min(k, sizes[s])
        assert np.array_equal(mem[off[s]:off[s + 1]], m_o), s
        got = med[base[s]:base[s] + cnt]
        assert np.array_equal(np.where(got >= 0, got - off[s], -1), r_o), s
        assert np.array_equal(size[base[s]:base[s] + cnt], z_o), s
        assert passes[s] == p_o, s
