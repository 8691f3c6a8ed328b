"""The pocket grid's point lists are padded to whole quads with a point that no term sees, wherever
the complex lies: energies and contacts do not depend on where the origin is."""
import numpy as np
import pytest

from geaxdock_gpu_b200 import abi, engine, system
from tests.golden.fixtures import load_ref

pytestmark = pytest.mark.gpu


def _at(offset):
    """The same complex, all coordinates multiples of 1/8 A, moved by `offset`."""
    z, _, _ = load_ref("1a07C1")
    ff = system.forcefield(abi.enepara_raw_from_array(z["enepara_raw"]), 42)
    cx = system.make_complex(np.random.default_rng(3), ff, L=22, n_lig=1, P=417, n_prt=1, n_tmp=2)
    grid = lambda a: np.round(np.asarray(a, np.float64) * 8.0) / 8.0
    for axis, name in enumerate("xyz"):
        setattr(cx, "lig_" + name, grid(getattr(cx, "lig_" + name)).astype(np.float32))
        for what in ("prt_", "kde_"):
            v = grid(getattr(cx, what + name)) + offset[axis]
            setattr(cx, what + name, v.astype(np.float32))
        m = getattr(cx, "mcs_" + name)
        valid = cx.mcs_x != abi.MCS_INVALID_COORD if axis == 0 else valid
        setattr(cx, "mcs_" + name,
                np.where(valid, grid(m) + offset[axis], m).astype(np.float32))
    cx.lig_center = np.tile(np.asarray(offset, np.float32), (1, 1))
    cx.pocket_center = np.asarray(offset, np.float32)
    return ff, cx


def _energies(offset):
    ff, cx = _at(offset)
    mm = np.zeros((3, 6), np.float32)
    mm[1, :3] = 0.5, -1.25, 2.0
    mm[2, :3] = -3.0, 0.75, 1.0
    with engine.Engine(ff, [cx], abi.mc_params(steps_per_exchange=10, steps_per_dump=20)) as eng:
        return eng.eval_energy(0, 0, 0, mm)


@pytest.mark.parametrize("offset", [(1e6, 1e6, 1e6), (-1e6, 1e6, 1e6), (1e6, 1e6, 1.1e6)])
def test_energies_do_not_depend_on_the_origin(offset):
    a, b = _energies((0.0, 0.0, 0.0)), _energies(offset)
    assert np.array_equal(a["cms"], b["cms"])
    np.testing.assert_array_equal(a["e"], b["e"])
