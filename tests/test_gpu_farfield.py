"""The far fields of large proteins (csrc/gd_farfield.cu, far_field in gd_kernels.cu): energies of
ligands inside the tabulated cells, across their outer sphere and outside it, against the FP64
oracle, which sums every pair."""
import numpy as np
import pytest

from geaxdock_gpu_b200 import abi, engine, system
from oracle import pyoracle as po
from tests.golden.fixtures import load_ref
from tests.tolerance import rel_errors

pytestmark = pytest.mark.gpu
# relative to the sum of magnitudes: series truncation 5e-8, coefficients and their sum in FP32
# 2e-7, the near points' FP32 sums 4e-7 (the pair loop alone): 1e-6 for vdw, ele and pmf; the
# parity tolerance for the others
TOL_FAR, TOL = 1e-6, 1e-5


@pytest.fixture(scope="module", params=[(2100, 5), (3000, 40), (6000, 64)])
def case(request):
    P, L = request.param
    z, _, _ = load_ref("1a07C1")
    raw = abi.enepara_raw_from_array(z["enepara_raw"])
    ff = system.forcefield(raw, 42)
    rng = np.random.default_rng(P)
    cx = system.make_complex(rng, ff, L=L, n_lig=2, P=P, n_prt=2, n_tmp=2,
                             pocket=np.array([5.0, -31.0, 14.5]))
    params = abi.mc_params(steps_per_exchange=10, steps_per_dump=20, seed=3)
    return ff, cx, params, po.ref_map(ff, cx)


@pytest.mark.parametrize("tile", [None, (1, 512, 1, 1, 0, 2), (1, 512, 4, 2)])
@pytest.mark.parametrize("shift", [(0.0, 0.0, 0.0), (1.0, 2.0, -7.0), (15.0, 9.0, 0.0),
                                   (0.0, -60.0, 0.0)])
def test_far_fields_against_oracle(case, tile, shift):
    ff, cx, params, rm = case
    if tile is not None and tile[0] * (tile[3] or 1) * cx.lna > 256:
        pytest.skip("the tile does not hold this ligand")
    rng = np.random.default_rng(29)
    mm = np.zeros((3, 6), np.float32)
    mm[:, :3] = np.asarray(shift, np.float32)
    mm[1:, 3:] = rng.uniform(-3.1, 3.1, (2, 3))
    with engine.Engine(ff, [cx], params) as eng:
        if tile is not None:
            eng.set_tile(*tile)
        got = eng.eval_energy(0, 1, 1, mm)
    for i in range(len(mm)):
        o = po.pose_energy(ff, cx, 1, 1, mm[i], rm, 64)
        err = rel_errors(got["e"][i], o, ff)
        assert err[:3].max() <= TOL_FAR, (i, err)
        assert err.max() <= TOL, (i, err)


def test_a_shared_protein_gives_the_same_chains_as_its_own(case):
    """Complexes on one protein share a set of tables, made for all their ligands' atom types:
    a complex's chains are those it has alone."""
    ff, cx, params, _ = case
    other = cx.subset(n_lig=1)
    other.lig_t = (other.lig_t + 5) % system.N_LIG_TYPES
    with engine.Engine(ff, [cx, other], params) as both, engine.Engine(ff, [cx], params) as alone:
        for e in (both, alone):
            e.mc_init()
            e.run_fused(0, 10)
            e.sync()
        assert both.state(0, cx.n_rep - 1).tobytes() == alone.state().tobytes()
