"""k-means of one large segment (csrc/gd_kmeans.cu: bounds decide which objects a pass scans)
against the general path, which the same segment takes beside a second one: the memberships,
medoids, sizes and passes are equal, also for ties, duplicates and values that are not finite."""
import numpy as np
import pytest

from geaxdock_gpu_b200 import postmc
from tests.conftest import have_gpu

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_gpu(), reason="needs a B200")]


def _data(kind, n, rng):
    x = rng.normal(0, 1, (n, 9)).astype(np.float32)
    if kind == "clumps":  # well separated: most objects are skipped from the second pass on
        x = (rng.integers(0, 30, (n, 1)) * 3.0 + 0.2 * x).astype(np.float32)
    elif kind == "grid":  # exact ties between centres
        x = np.round(2 * x) / 2
    elif kind == "few":  # duplicates: empty clusters, centres that coincide
        x = x[rng.integers(0, 40, n)]
    elif kind == "tiny":  # squares underflow
        x = (x * np.float32(1e-20)).astype(np.float32)
    elif kind == "huge":  # squares overflow
        x = (x * np.float32(3e18)).astype(np.float32)
    elif kind == "offset":  # differences lose most of their bits
        x = (x + np.float32(3000.0)).astype(np.float32)
    elif kind == "nan":
        x[n // 2, 3] = np.nan
    elif kind == "inf":
        x[n // 3, 1] = np.inf
        x[n // 2, 4] = -np.inf
    return np.ascontiguousarray(x, np.float32)


@pytest.mark.parametrize("kind", ["normal", "clumps", "grid", "few", "tiny", "huge", "offset", "nan",
                                  "inf"])
@pytest.mark.parametrize("n,k", [(8193, 1), (8193, 2), (12000, 7), (20011, 500), (30000, 1024)])
def test_pruned_passes_are_the_general_ones(kind, n, k):
    rng = np.random.default_rng(n + k)
    x = _data(kind, n, rng)
    other = rng.normal(0, 1, (3, 9)).astype(np.float32)
    a = postmc.kmeans(x, [0, n], [k], 11, max_iter=60)
    b = postmc.kmeans(np.concatenate([x, other]), [0, n, n + 3], [k, 1], 11, max_iter=60)
    assert a[3][0] == b[3][0]  # passes
    assert np.array_equal(a[0], b[0][:n])  # memberships
    assert np.array_equal(a[1][:k], b[1][:k]) and np.array_equal(a[2][:k], b[2][:k])
