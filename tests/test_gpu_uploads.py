"""Uploads from pageable memory are ordered on the stream that reads them."""
import numpy as np
import pytest

from geaxdock_gpu_b200 import engine
from oracle import mlp as mo
from tests.conftest import have_gpu

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_gpu(), reason="needs a B200")]


def test_parameters_are_converted_after_they_arrive():
    """The 16-bit weight copies are those of the parameters just set: the gradient of each of a
    row of fresh networks agrees with the oracle's (set_params returned while the copy was on its
    way, and the conversion read the old values)."""
    rng = np.random.default_rng(5)
    x = rng.normal(0, 0.7, (64, 64)).astype(np.float32)
    t = rng.normal(0, 1, 64).astype(np.float32)
    for seed in range(6):
        net = engine.Mlp(hidden=256, n_embedding=600, seed=seed)
        theta = net.params()[rng.permutation(net.n_params)]
        net.set_params(theta)
        loss, g = net.backward(x, t, np.full(64, -1, np.int32))
        orc = mo.MlpOracle(theta, 256, 600, bf16_mode=True)
        lo, go = orc.backward(x, t, np.full(64, -1, np.int32))
        assert abs(loss - lo) <= 1e-3 * max(1.0, lo), seed
        off, size = orc.L["w2"]
        r = np.linalg.norm(g[off:off + size] - go[off:off + size]) / \
            np.linalg.norm(go[off:off + size])
        assert r <= 0.02, (seed, r)
        net.close()
