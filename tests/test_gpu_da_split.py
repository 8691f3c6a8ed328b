"""The split a caller asks for is the split the delayed-acceptance exact stage runs, also on a
context whose own launches are split (few replicas)."""
import numpy as np
import pytest

from geaxdock_gpu_b200 import abi, engine, system
from tests.golden.fixtures import load_ref

pytestmark = pytest.mark.gpu


def _exact_kernels(fn):
    """Template arguments (unroll, how it splits (0: not), kind, pack) of the Monte Carlo kernels
    that ran on the GPU in fn()."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        fn()
        torch.cuda.synchronize()
    names = {e.name for e in p.events() if "gd_mc_kernel" in e.name}
    return {n.split("<")[1].split(">")[0].replace(" ", "") for n in names}


@pytest.mark.parametrize("tile", [None, (1, 512, 4, 4)])
@pytest.mark.parametrize("split", [1, 3])
def test_the_exact_stage_runs_the_split_asked_for(tile, split):
    z, _, _ = load_ref("1a07C1")
    ff = system.forcefield(abi.enepara_raw_from_array(z["enepara_raw"]), 42)
    cx = system.make_complex(np.random.default_rng(4), ff, L=28, n_lig=3, P=500, n_prt=1, n_tmp=6)
    params = abi.mc_params(steps_per_exchange=10, steps_per_dump=200, seed=5)
    states = []
    for s in (split, 0):
        with engine.Engine(ff, [cx], params) as eng:
            if tile is not None:
                eng.set_tile(*tile)
            assert eng.tile()[3] > 1
            eng.mc_init()
            sur = engine.Surrogate(eng, hidden=128, batch=256, sample_cap=1 << 14,
                                   embedding=0, fallback_accept=0.0, split=s)
            sur.collect(0, 20)
            sur.train(20)
            if s == split:
                ran = _exact_kernels(lambda: sur.run(20, 20))
                assert sur.split() == split
            else:
                sur.run(20, 20)
            eng.sync()
            states.append(eng.state())
    assert ran and all((a.split(",")[1] == "0") == (split == 1) for a in ran), ran
    # the split changes where a pair is summed, not the chains
    assert np.array_equal(states[0]["movematrix_old"], states[1]["movematrix_old"])
    assert np.array_equal(states[0]["n_accept"], states[1]["n_accept"])
