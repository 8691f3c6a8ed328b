"""A context without a tile of its own splits an atom's work over warps by how many replicas or
poses there are. Which split it takes does not show: an energy has the same bits whatever it is
computed with, alone or in a batch. The contact weights cancel so that the order of FP64 additions
would reach the FP32 results."""
import math

import numpy as np
import pytest

from geaxdock_gpu_b200 import abi, engine, system
from tests.golden.fixtures import load_ref

pytestmark = pytest.mark.gpu


def _system(P, L, n_lig=3, n_tmp=4, n_prt=1, seed=0, pocket=None):
    z, _, _ = load_ref("1a07C1")
    ff = system.forcefield(abi.enepara_raw_from_array(z["enepara_raw"]), 42)
    rng = np.random.default_rng(P + L + seed)
    cx = system.make_complex(rng, ff, L=L, n_lig=n_lig, P=P, n_prt=n_prt, n_tmp=n_tmp,
                             pocket=pocket)
    ff.b_para[2] = 0.0
    count = np.bincount(np.asarray(cx.prt_t)[0], minlength=abi.MAXTP1)
    used = np.flatnonzero(count)
    for tl in range(abi.MAXTP2):
        terms = []
        for k, tp in enumerate(used):
            v = np.float32(rng.choice([-1.0, 1.0]) * 10.0 ** rng.uniform(-3.0, 3.0))
            if k >= len(used) - 2:  # of a far pose's sum the last two leave about 1e-10
                v = np.float32(-math.fsum(terms) / count[tp])
            ff.pmf1[tl][int(tp)] = v
            terms.append(float(v) * int(count[tp]))
    return ff, cx


def _poses(rng, n):
    mm = np.concatenate([rng.normal(0, 2.0, (n, 3)), rng.uniform(-3.1, 3.1, (n, 3))], 1)
    mm[n // 2:, :3] += rng.normal(0, 1.0, (n - n // 2, 3)) + [0.0, 300.0, 0.0]  # all pairs far
    return mm.astype(np.float32)


# one block of points, several, and (9,900) a protein past four thousand points a buffer; atoms of
# one warp, of several, of the most a ligand has
@pytest.mark.parametrize("P,L", [(300, 9), (344, 34), (1500, 28), (1030, 100), (3000, 40),
                                 (6000, 64), (9900, 12), (9900, 90)])
def test_a_pose_has_the_same_energy_in_any_company(P, L):
    ff, cx = _system(P, L)
    mm = _poses(np.random.default_rng(1), 600)
    mm = mm[np.random.default_rng(2).permutation(len(mm))]
    params = abi.mc_params(steps_per_exchange=10, steps_per_dump=20)
    with engine.Engine(ff, [cx], params) as eng, engine.Engine(ff, [cx], params) as one:
        one.set_tile(1, 512, 2, 1)
        ref = one.eval_energy(0, 0, 1, mm)
        for n in (1, 3, 24, 140, 300, 600):
            got = np.concatenate([eng.eval_energy(0, 0, 1, mm[i:i + n])
                                  for i in range(0, min(600, 40 * n), n)])
            assert got.tobytes() == ref[:len(got)].tobytes(), n


def test_a_complex_alone_and_in_a_batch():
    ff, first = _system(900, 24, n_lig=2, n_tmp=4)
    cxs = [first]
    for i, (P, L) in enumerate([(400, 40), (2300, 33), (1500, 20)]):
        cxs.append(_system(P, L, n_lig=8, n_tmp=16, n_prt=4, seed=i,
                           pocket=np.array([80.0 * (i + 1), 0.0, 0.0]))[1])
    params = abi.mc_params(steps_per_exchange=10, steps_per_dump=60, seed=5,
                           move_kind=abi.MOVE_GAUSSIAN)
    with engine.Engine(ff, cxs, params) as both, engine.Engine(ff, [first], params) as alone:
        assert both.tile()[3] != alone.tile()[3]
        for e in (both, alone):
            e.mc_init()
            e.run_fused(0, 60)
            e.sync()
        assert both.state(0, first.n_rep - 1).tobytes() == alone.state().tobytes()
