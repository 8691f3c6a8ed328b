"""Decisions on energies from the far fields are those of the pair loop: replica exchanges, fused into
the step launches and by the call of their own, and both kinds of delayed-acceptance steps. The
moves and temperatures make most decisions hang on the last FP32 digits."""
import numpy as np
import pytest

from geaxdock_gpu_b200 import abi, engine, system
from tests.golden.fixtures import load_ref

pytestmark = pytest.mark.gpu


def _case(floor, scale, n_tmp=6, n_lig=3, P=2300, L=24, n_prt=2):
    z, _, _ = load_ref("1a07C1")
    ff = system.forcefield(abi.enepara_raw_from_array(z["enepara_raw"]), 42)
    cx = system.make_complex(np.random.default_rng(8), ff, L=L, n_lig=n_lig, P=P, n_prt=n_prt,
                             n_tmp=n_tmp)
    cx.temp["t"] = floor * np.linspace(1.0, 4.0, n_tmp)
    cx.temp["minus_beta"] = -1.0 / cx.temp["t"]
    params = abi.mc_params(steps_per_exchange=5, steps_per_dump=200, seed=11,
                           move_scale=(scale,) * 6, move_kind=abi.MOVE_GAUSSIAN)
    return ff, cx, params


def _same(a, b):
    for f in ("movematrix_old", "n_accept", "n_exchange"):
        assert np.array_equal(a[f], b[f]), f
    assert np.array_equal(a["replica"]["idx_tmp"], b["replica"]["idx_tmp"])


@pytest.mark.parametrize("tile", [None, (2, 512, 2, 1), (4, 512, 2, 1, 0, 2), (1, 2560, 1, 1)])
@pytest.mark.parametrize("floor", [1e-6, 1e-5, 1e-3])
def test_exchanges_near_a_tie(floor, tile):
    ff, cx, params = _case(floor, 1e-5)
    states = []
    for fields in (True, False):
        for fused in (True, False):
            with engine.Engine(ff, [cx], params) as eng:
                if tile is not None:
                    eng.set_tile(*tile)
                assert eng.far_field_bytes() > 0
                if not fields:
                    eng.release_far_fields()
                eng.mc_init()
                if fused:
                    eng.run_fused(0, 100)
                else:
                    for i in range(20):
                        eng.mc_run(0, 5 * i)
                        eng.exchange(int(not (i % 2)))
                eng.sync()
                states.append(eng.state())
    assert states[0]["n_exchange"].sum() > 0
    for st in states[1:]:
        _same(states[0], st)


def test_exchanges_of_a_ragged_batch_on_several_chains():
    """Open groups of several complexes, on concurrent chains, more of them than one CTA takes."""
    z, _, _ = load_ref("1a07C1")
    ff = system.forcefield(abi.enepara_raw_from_array(z["enepara_raw"]), 42)
    rng = np.random.default_rng(3)
    cxs = []
    for i, (L, P, nt) in enumerate([(9, 2200, 5), (70, 2500, 2), (30, 400, 4), (100, 2100, 7)]):
        cx = system.make_complex(rng, ff, L=L, n_lig=2, P=P, n_prt=2, n_tmp=nt,
                                 pocket=np.array([50.0 * i, 0.0, 0.0]))
        cx.temp["t"] = 1e-6 * np.linspace(1.0, 3.0, nt)
        cx.temp["minus_beta"] = -1.0 / cx.temp["t"]
        cxs.append(cx)
    params = abi.mc_params(steps_per_exchange=5, steps_per_dump=200, seed=2,
                           move_scale=(1e-5,) * 6, move_kind=abi.MOVE_GAUSSIAN)
    states = []
    for fields in (True, False):
        for chains in (1, 3):
            with engine.Engine(ff, cxs, params) as eng:
                eng.set_concurrency(chains, 3)
                if not fields:
                    eng.release_far_fields()
                eng.mc_init()
                eng.run_fused(0, 50)
                eng.run_fused(50, 25)
                eng.sync()
                states.append(eng.state())
    for st in states[1:]:
        _same(states[0], st)


def _without_fields(eng, cx):
    """Releases the fields and takes every replica's energy again without them."""
    eng.release_far_fields()
    st = eng.state()
    pl = st["replica"]["idx_prt"] * cx.n_lig + st["replica"]["idx_lig"]
    for k in np.unique(pl):
        r = np.flatnonzero(pl == k)
        st["energy_old"][r] = eng.eval_energy(0, int(k) // cx.n_lig, int(k) % cx.n_lig,
                                              st["movematrix_old"][r])
    eng.set_state(st)


@pytest.mark.parametrize("split", [1, 3])
@pytest.mark.parametrize("floor,scale", [(1e-6, 1e-5), (1e-3, 1e-3)])
def test_delayed_acceptance_near_a_tie(floor, scale, split):
    """Given the surrogate, every decision of the exact stage and of the exchanges is the pair loop's;
    so is every collect step's."""
    ff, cx, params = _case(floor, scale)
    states, after = [], []
    for fields in (True, False):
        with engine.Engine(ff, [cx], params) as eng:
            eng.set_tile(2, 512, 2, 1)
            eng.mc_init()
            sur = engine.Surrogate(eng, hidden=128, batch=256, sample_cap=1 << 14, embedding=0,
                                   fallback_accept=0.0, split=split)
            sur.collect(0, 20)
            sur.train(30)
            if not fields:
                _without_fields(eng, cx)
            sur.run(20, 40)
            eng.sync()
            after.append(eng.state())
            sur.collect(60, 40)
            eng.sync()
            states.append(eng.state())
    _same(*after)
    _same(*states)
