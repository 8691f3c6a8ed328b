"""The device memory of a large k-means call goes back to the driver when it returns."""
import numpy as np
import pytest

from geaxdock_gpu_b200 import engine, postmc

pytestmark = pytest.mark.gpu
MB = 1 << 20


@pytest.mark.parametrize("n,held", [(20000, 40 * MB), (1500000, 40 * MB)])
def test_what_a_call_leaves_behind(n, held):
    import torch
    obj = np.random.default_rng(1).normal(0.0, 1.0, (n, 9)).astype(np.float32)
    run = lambda m: postmc.kmeans(obj[:m], np.array([0, m], np.int32), np.array([3], np.int32),
                                  seed=1, max_iter=2)
    run(1000)  # module and pool
    engine.release_memory(0)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info(0)[0]
    a = run(n)
    assert before - torch.cuda.mem_get_info(0)[0] <= held
    b = run(n)
    assert all(np.array_equal(u, v) for u, v in zip(a, b))
