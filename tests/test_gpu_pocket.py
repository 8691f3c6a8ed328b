"""The point lists of the pocket grid (csrc/gd_pocket.cu, short_range_lists in gd_kernels.cu):
energies of ligands inside the 40 A cube of 4 A cells, across its faces and outside it, against
the FP64 oracle, which sums every pair."""
import numpy as np
import pytest

from geaxdock_gpu_b200 import abi, engine, system
from oracle import pyoracle as po
from tests.golden.fixtures import load_ref
from tests.tolerance import rel_errors

pytestmark = pytest.mark.gpu
# each term within 1e-5 of FP64, relative to the sum of magnitudes (tests/tolerance.py); the MCC
# of exact contact counts to the rounding of its formula
TOL, TOL_CMS = 1e-5, 2e-6


@pytest.fixture(scope="module")
def system0():
    z, _, _ = load_ref("1a07C1")
    w = system.config(0, abi.enepara_raw_from_array(z["enepara_raw"]))
    return w, w.complexes[0], po.ref_map(w.ff, w.complexes[0])


@pytest.mark.parametrize("shift", [
    (0.0, 0.0, 0.0),        # centre on a cell corner
    (4.0, -4.0, 2.0),       # other cell faces
    (19.99, 0.0, 0.0),      # across the cube's +x face
    (-20.0, 20.0, 0.0),     # on an edge: most atoms outside
    (0.0, 0.0, -26.0),      # outside, inside the protein
    (45.0, 45.0, 45.0),     # outside both
])
@pytest.mark.parametrize("split", [1, 3])
def test_lists_inside_and_outside_the_cube(system0, shift, split):
    w, cx, rm = system0
    rng = np.random.default_rng(17)
    mm = np.zeros((6, 6), np.float32)
    mm[:, :3] = np.asarray(shift, np.float32)
    mm[1:, :3] += rng.normal(0.0, 0.5, (5, 3)).astype(np.float32)
    mm[1:, 3:] = rng.uniform(-3.1, 3.1, (5, 3))
    with engine.Engine(w.ff, [cx], w.params) as eng:
        if split > 1:
            eng.set_tile(2, 512, 0, split)
        got = eng.eval_energy(0, 0, 3, mm)
    for i in range(len(mm)):
        o = po.pose_energy(w.ff, cx, 0, 3, mm[i], rm, 64)
        assert rel_errors(got["e"][i], o, w.ff).max() <= TOL, (i, got["e"][i], o["e"])
        assert abs(got["cms"][i] - o["cms"]) <= TOL_CMS, (i, got["cms"][i], o["cms"])
