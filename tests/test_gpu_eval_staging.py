"""Pose evaluation: calls that go through the context's page-locked buffer and calls that do not,
whose tiles come from the launch's arguments, give the same energies."""
import threading

import numpy as np
import pytest

from geaxdock_gpu_b200 import abi, engine, system
from tests.conftest import have_gpu
from tests.golden.fixtures import load_ref

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_gpu(), reason="needs a B200")]

STAGE = 256 * 1024  # bytes of the page-locked buffer, its last 4 for the error word


@pytest.fixture(scope="module")
def work():
    z, _, _ = load_ref("1a07C1")
    return system.config(0, abi.enepara_raw_from_array(z["enepara_raw"]))


def _poses(n, seed):
    rng = np.random.default_rng(seed)
    return np.concatenate([rng.normal(0, 2.0, (n, 3)), rng.uniform(-3, 3, (n, 3))],
                          1).astype(np.float32)


def _bytes(a):
    return np.ascontiguousarray(a).view(np.uint8)


def test_energies_do_not_depend_on_the_call_that_carries_the_pose(work):
    """One tile shape, so one order of additions: every pose has the same bits in calls of one
    pose, of ragged tiles and on both sides of the buffer's size."""
    edge = (STAGE - 4) // abi.ENERGY_DTYPE.itemsize
    mm = _poses(edge + 40, 1)
    with engine.Engine(work.ff, [work.complexes[0]], work.params) as eng:
        eng.set_tile(4, 512, 2, 1)
        want = eng.eval_energy(0, 0, 0, mm)
        for n in (1, 2, 7, 63, edge - 1, edge, edge + 1):
            assert np.array_equal(_bytes(eng.eval_energy(0, 0, 0, mm[:n])), _bytes(want[:n])), n
        assert np.array_equal(_bytes(eng.eval_energy(0, 0, 0, mm[100:111])),
                              _bytes(want[100:111]))
        # placed coordinates, whose buffer is filled by its inputs
        L = work.complexes[0].lna
        edge = (STAGE - 4) // (12 * L + 12)
        mm = mm[:edge + 3]
        xyz = eng.place_ligand(0, 0, mm)
        ctr = np.ascontiguousarray(mm[:, :3])
        want = eng.eval_energy_xyz(0, 0, 0, xyz, ctr)
        for n in (1, 7, edge, edge + 1):
            got = eng.eval_energy_xyz(0, 0, 0, xyz[:n], ctr[:n])
            assert np.array_equal(_bytes(got), _bytes(want[:n])), n


def test_contexts_of_several_threads_share_the_kernel_settings(work):
    """Contexts with different shapes on threads of their own: each call gets its own energies
    (the launches' attributes are kept per kernel for the whole process)."""
    mm = _poses(200, 2)
    tiles = [(1, 512, 2, 1), (4, 512, 2, 1), (4, 256, 2, 1), (8, 512, 2, 1)]
    out = [[] for _ in tiles]

    def run(i, to):
        with engine.Engine(work.ff, [work.complexes[0]], work.params) as eng:
            eng.set_tile(*tiles[i])
            for n in (200, 3, 50, 200):
                to.append(eng.eval_energy(0, 0, 0, mm[:n]))

    alone = [[] for _ in tiles]
    for i in range(len(tiles)):
        run(i, alone[i])
    ts = [threading.Thread(target=run, args=(i, out[i])) for i in range(len(tiles))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for got, want in zip(out, alone):
        assert len(got) == 4
        for g, w in zip(got, want):
            assert np.array_equal(_bytes(g), _bytes(w))
