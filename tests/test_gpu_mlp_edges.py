"""Loss and gradients of the surrogate at the edges of its batch reductions (chunks of 256 rows,
tiles of 128, rows padded to 16) and of its widths, against the oracle."""
import numpy as np
import pytest

from geaxdock_gpu_b200 import engine
from oracle import mlp as mo
from tests.conftest import have_gpu

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_gpu(), reason="needs a B200")]


@pytest.mark.parametrize("hidden", [16, 64, 112, 256])
@pytest.mark.parametrize("rows", [1, 16, 17, 128, 129, 256, 257, 600])
def test_gradients_at_the_edges(hidden, rows):
    """The oracle rounds the same operands to BF16; what differs is the order of FP32 sums, and
    with it now and then one rounding (2^-9 of an operand): 2 % of a tensor's norm is some five of
    those in every element. Targets lie away from the outputs, so that dy is not a difference of
    near-equal numbers. A larger call goes first: nothing of its rows may come back."""
    n_emb = 5 if hidden != 112 else 0
    rng = np.random.default_rng(hidden + rows)
    net = engine.Mlp(hidden=hidden, n_embedding=n_emb, seed=4)
    x = rng.normal(0, 0.7, (rows, 64)).astype(np.float32)
    t = (3.0 + rng.normal(0, 0.5, rows)).astype(np.float32)
    conf = rng.integers(-1, max(n_emb, 1), rows).astype(np.int32) if n_emb else None
    big = rng.normal(0, 2.0, (rows + 300, 64)).astype(np.float32)
    net.backward(big, np.zeros(rows + 300, np.float32), None)
    loss, g = net.backward(x, t, conf)
    orc = mo.MlpOracle(net.params(), hidden, n_emb, bf16_mode=True)
    lo, go = orc.backward(x, t, np.full(rows, -1, np.int32) if conf is None else conf)
    net.close()
    assert abs(loss - lo) <= 1e-3 * max(1.0, lo)
    for name in ("w1", "b1", "w2", "b2", "w3", "b3", "w4", "b4") + (("emb",) if n_emb else ()):
        off, size = orc.L[name]
        a, b = g[off:off + size], go[off:off + size]
        assert np.linalg.norm(a - b) <= 0.02 * np.linalg.norm(b) + 1e-6, name


@pytest.mark.parametrize("hidden", [128, 256])
@pytest.mark.parametrize("rows", [1, 15, 16, 17, 31, 32, 33, 64, 65])
def test_one_kernel_forward_at_the_edges(hidden, rows):
    """Rows around the CTA's 32 and its two 16-row tiles. Each hidden unit's rounding may fall the
    other way (2^-9 of it, random signs); the output sums them with the last layer's weights, so
    1 % of the outputs' spread bounds it with room. One row alone is compared with itself among
    others: a row's sums do not depend on its neighbours."""
    rng = np.random.default_rng(hidden + rows)
    net = engine.Mlp(hidden=hidden, n_embedding=7, seed=6)
    x = rng.normal(0, 1.5, (rows + 40, 64)).astype(np.float32)
    conf = rng.integers(-1, 7, rows + 40).astype(np.int32)
    big = net.forward(x, conf)
    y = net.forward(x[:rows], conf[:rows])
    yo = mo.MlpOracle(net.params(), hidden, 7, bf16_mode=True).forward(x, conf)
    net.close()
    assert np.array_equal(y.view(np.uint32), big[:rows].view(np.uint32))
    assert np.abs(big - yo).max() <= 0.01 * yo.std() + 1e-4
