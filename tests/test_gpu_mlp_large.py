"""A batch whose partial sums do not fit together is reduced tensor by tensor: the same gradients,
in a buffer no larger than its largest tensor's partials."""
import numpy as np
import pytest

from geaxdock_gpu_b200 import engine

pytestmark = pytest.mark.gpu
H, N = 256, 131072


def _rows(rng, n, n_emb):
    x = rng.normal(0.0, 0.7, (n, 64)).astype(np.float32)
    return x, np.sin(x[:, 0]).astype(np.float32), rng.integers(0, n_emb, n).astype(np.int32)


def test_gradients_of_a_large_batch():
    """Of two halves of 2^16 rows each, reduced together: dy of the whole is half theirs, a power of
    two, so that every product is the same and only the order of FP32 additions differs (512 chunks;
    26,000 atomic additions per embedding row): 1e-5 and 1e-4 of a tensor's norm."""
    rng = np.random.default_rng(5)
    x, t, conf = _rows(rng, N, 5)
    net = engine.Mlp(H, 5, seed=3)
    loss, grad = net.backward(x, t, conf)
    half = [net.backward(x[s], t[s], conf[s]) for s in (slice(0, N // 2), slice(N // 2, N))]
    want = 0.5 * (half[0][1].astype(np.float64) + half[1][1])
    assert abs(loss - 0.5 * (half[0][0] + half[1][0])) <= 1e-6 * loss
    sizes = [64 * H, H, H * H, H, H * H, H, H, 4, 5 * 32]
    at = 0
    for k, size in enumerate(sizes):
        a, b = grad[at:at + size].astype(np.float64), want[at:at + size]
        at += size
        tol = 1e-4 if k == len(sizes) - 1 else 1e-5
        assert np.linalg.norm(a - b) <= tol * np.linalg.norm(b), k
    assert at == len(grad)


def test_memory_of_a_large_batch():
    import torch
    rng = np.random.default_rng(6)
    x, t, conf = _rows(rng, N, 5)
    net = engine.Mlp(H, 5, seed=3)
    net.forward(x, conf)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info(0)[0]
    net.backward(x, t, conf)
    # 512 chunks of a 256 x 256 gradient and the allocator's granularity
    assert before - torch.cuda.mem_get_info(0)[0] <= 512 * H * H * 4 + (8 << 20)
