"""gd_set_tile of what gd_get_tile reports restores the tile, the automatic one of a context of few
replicas among them (its lanes exceed what a caller's tile may ask for)."""
import numpy as np
import pytest

from geaxdock_gpu_b200 import abi, engine, system
from tests.golden.fixtures import load_ref

pytestmark = pytest.mark.gpu


def _context(L, P, n_lig, n_tmp, n_prt):
    z, _, _ = load_ref("1a07C1")
    ff = system.forcefield(abi.enepara_raw_from_array(z["enepara_raw"]), 42)
    cx = system.make_complex(np.random.default_rng(L + P), ff, L=L, n_lig=n_lig, P=P,
                             n_prt=n_prt, n_tmp=n_tmp)
    return engine.Engine(ff, [cx], abi.mc_params(steps_per_exchange=10, steps_per_dump=40, seed=9))


# 128 replicas of 28 atoms (448 lanes), 252 of 34 (340), 12 of 100, and more than fill the device
@pytest.mark.parametrize("shape", [(28, 1500, 8, 16, 1), (34, 344, 7, 12, 3), (100, 700, 3, 4, 1),
                                   (20, 300, 12, 16, 12)])
def test_the_automatic_tile_comes_back(shape):
    rng = np.random.default_rng(2)
    mm = rng.normal(0.0, 1.0, (5, 6)).astype(np.float32)
    with _context(*shape) as eng, _context(*shape) as ref:
        t = eng.tile()
        eng.set_tile(*t)
        assert eng.tile() == t
        eng.set_tile(1, 512, 1, 1)  # another, and back
        assert eng.tile() == (1, 512, 1, 1, 0, 1)
        eng.set_tile(*t)
        assert eng.tile() == t
        assert eng.replicas_per_cta() == ref.replicas_per_cta()
        for e in (eng, ref):
            e.mc_init()
            e.run_fused(0, 20)
            e.sync()
        assert eng.state().tobytes() == ref.state().tobytes()
        assert eng.eval_energy(0, 0, 0, mm).tobytes() == ref.eval_energy(0, 0, 0, mm).tobytes()


def test_a_ragged_batch_gets_its_automatic_tile_back():
    z, _, _ = load_ref("1a07C1")
    ff = system.forcefield(abi.enepara_raw_from_array(z["enepara_raw"]), 42)
    rng = np.random.default_rng(6)
    cxs = [system.make_complex(rng, ff, L=L, n_lig=4, P=P, n_prt=2, n_tmp=4)
           for L, P in ((11, 400), (40, 900), (70, 350))]
    with engine.Engine(ff, cxs, abi.mc_params(steps_per_exchange=10, steps_per_dump=40)) as eng:
        t, k = eng.tile(), [eng.replicas_per_cta(i) for i in range(3)]
        eng.set_tile(1, 512, 2, 1)
        eng.set_tile(*t)
        assert eng.tile() == t and [eng.replicas_per_cta(i) for i in range(3)] == k


def test_tiles_past_a_callers_limit_are_still_refused():
    with _context(28, 1500, 8, 16, 1) as eng:
        k, chunk, unroll, split = eng.tile()[:4]
        for bad in ((k + 1, chunk, unroll, split), (k, chunk + 4, unroll, split)):
            with pytest.raises(engine.GDError) as e:
                eng.set_tile(*bad)
            assert e.value.code == abi.GD_ERR_INVALID
