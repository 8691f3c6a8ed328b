"""Split launches of the Monte Carlo kernel (the lanes of an atom in several warps, each running
some of the protein's segments): the energies are those of one lane per atom up to the order of
FP64 additions, and launches of few replicas take them by default."""
import numpy as np
import pytest

from geaxdock_gpu_b200 import abi, engine, system
from tests.golden.fixtures import load_ref

pytestmark = pytest.mark.gpu


def _system(P, L, types=None):
    z, _, _ = load_ref("1a07C1")
    raw = abi.enepara_raw_from_array(z["enepara_raw"])
    ff = system.forcefield(raw, 42)
    rng = np.random.default_rng(P + L)
    cx = system.make_complex(rng, ff, L=L, n_lig=3, P=P, n_prt=1, n_tmp=4)
    if types is not None:
        cx.prt_t = cx.prt_t % types
    return ff, cx, abi.mc_params(steps_per_exchange=10, steps_per_dump=40, seed=9)


# ligands of one warp, one atom past a warp, and several warps; more splits than segments; the
# protein in one, two (resident) and many chunks
@pytest.mark.parametrize("P,L,types,tile", [
    (300, 32, None, (1, 512, 4, 8)), (300, 33, None, (1, 512, 4, 7)),
    (700, 8, None, (2, 512, 2, 16)), (700, 8, 1, (1, 512, 1, 8)), (700, 64, 3, (2, 512, 4, 2)),
    (1100, 20, None, (3, 512, 2, 4)), (1100, 100, None, (1, 512, 4, 2))])
def test_splits_give_the_unsplit_energies(P, L, types, tile):
    ff, cx, params = _system(P, L, types)
    rng = np.random.default_rng(1)
    mm = np.concatenate([rng.normal(0, 2.0, (9, 3)), rng.uniform(-3.1, 3.1, (9, 3))],
                        1).astype(np.float32)
    out = []
    for t in ((1, 512, 2, 1), tile):
        with engine.Engine(ff, [cx], params) as eng:
            eng.set_tile(*t)
            r = eng.eval_energy(0, 0, 1, mm)
            out.append(np.concatenate([r["e"], r["cms"][:, None], r["rmsd"][:, None]], 1))
    # FP64 sums in another order, rounded to FP32 once: at most one unit in the last place
    assert np.all(np.abs(out[0] - out[1]) <= np.spacing(np.abs(out[0])))


@pytest.mark.parametrize("P,L", [(344, 34), (1500, 28)])
def test_few_replicas_are_split_by_default(P, L):
    """12 replicas: the default launch is split and its chains are those of a one-lane tile."""
    ff, cx, params = _system(P, L)
    with engine.Engine(ff, [cx], params) as a, engine.Engine(ff, [cx], params) as b:
        assert a.tile()[3] > 1
        b.set_tile(4, 512, 2, 1)
        for e in (a, b):
            e.mc_init()
            e.run_fused(0, 40)
            e.sync()
        sa, sb = a.state(), b.state()
    assert np.array_equal(sa["n_accept"], sb["n_accept"])
    assert np.array_equal(sa["movematrix_old"], sb["movematrix_old"])
    np.testing.assert_allclose(sa["energy_old"]["e"], sb["energy_old"]["e"], rtol=3e-7, atol=0)
