"""Unsplit tiles take the ligand's atoms by distance from its centre, or replica by replica when one
replica of the tile is away from the pocket; neither order shows in an energy or a decision."""
import numpy as np
import pytest

from geaxdock_gpu_b200 import abi, engine, system
from tests.golden.fixtures import load_ref

pytestmark = pytest.mark.gpu


def _system(P, L, **kw):
    z, _, _ = load_ref("1a07C1")
    ff = system.forcefield(abi.enepara_raw_from_array(z["enepara_raw"]), 42)
    cx = system.make_complex(np.random.default_rng(P), ff, L=L, n_lig=3, P=P, n_prt=1, n_tmp=4)
    return ff, cx, abi.mc_params(steps_per_exchange=10, steps_per_dump=200, seed=9, **kw)


# proteins with and without fields, ligands below, at and past a warp, tiles with a part-filled
# last warp
@pytest.mark.parametrize("P,L", [(2100, 7), (2100, 32), (2600, 45), (600, 19)])
def test_poses_at_the_pocket_and_away_share_a_tile(P, L):
    ff, cx, params = _system(P, L)
    rng = np.random.default_rng(1)
    mm = np.concatenate([rng.normal(0, 1.0, (24, 3)), rng.uniform(-3.1, 3.1, (24, 3))],
                        1).astype(np.float32)
    mm[5, 0] = 25.0   # one far away among neighbours at the pocket
    mm[12:16, 1] -= 18.0
    mm[20, 2] = 400.0
    out = []
    for tile in ((1, 512, 2, 1), (256 // L, 512, 2, 1), (3, 512, 4, 1), (4, 512, 2, 1, 0, 2)):
        if tile[0] * L > 256:
            continue
        with engine.Engine(ff, [cx], params) as eng:
            eng.set_tile(*tile)
            out.append(eng.eval_energy(0, 0, 1, mm).tobytes())
    assert len(out) >= 3 and all(o == out[0] for o in out)


@pytest.mark.parametrize("scale", [0.1, 2.0, 6.0])
def test_chains_that_spread_do_not_depend_on_the_order(scale):
    ff, cx, params = _system(2300, 21, move_scale=(scale,) * 3 + (0.05 * scale,) * 3,
                             move_kind=abi.MOVE_GAUSSIAN)
    states = []
    for tile in ((1, 512, 2, 1), (6, 512, 2, 1), (12, 512, 4, 1)):
        with engine.Engine(ff, [cx], params) as eng:
            eng.set_tile(*tile)
            eng.mc_init()
            eng.run_fused(0, 150)
            eng.sync()
            states.append(eng.state())
    for st in states[1:]:
        assert st.tobytes() == states[0].tobytes()
