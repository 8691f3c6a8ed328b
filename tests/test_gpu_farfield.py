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


@pytest.mark.parametrize("scale,floor", [(1e-5, 1e-6), (1e-5, 1e-3), (0.05, 0.3)])
def test_decisions_near_a_tie_are_taken_without_the_fields(scale, floor):
    """Moves so small that most decisions hang on the last FP32 digits: each is taken on the pair
    loop's energies of both poses, in whatever shape the launch has (ring, resident protein, split,
    two replicas per thread), with several tiles per CTA's ring in turn; moves of normal size
    agree too. The decisions are those of the FP64 energies wherever these are not closer to a
    tie than FP32 energies resolve."""
    z, _, _ = load_ref("1a07C1")
    ff = system.forcefield(abi.enepara_raw_from_array(z["enepara_raw"]), 42)
    rng = np.random.default_rng(8)
    cx = system.make_complex(rng, ff, L=24, n_lig=3, P=2100, n_prt=1, n_tmp=4)
    cx.temp["t"] = floor * np.array([1.0, 1.5, 2.0, 3.0])
    cx.temp["minus_beta"] = -1.0 / cx.temp["t"]
    params = abi.mc_params(steps_per_exchange=5, steps_per_dump=20, seed=11,
                           move_scale=(scale,) * 6, move_kind=abi.MOVE_GAUSSIAN)
    states, n_steps = [], 15
    for tile in (None, (2, 512, 2, 1), (1, 512, 4, 2), (4, 512, 2, 1, 0, 2), (1, 2560, 1, 1)):
        with engine.Engine(ff, [cx], params) as eng:
            if tile is not None:
                eng.set_tile(*tile)
            eng.mc_init()
            eng.trace_enable(n_steps)
            eng.run_fused(0, n_steps, exchange=False)
            eng.sync()
            states.append((tile, eng.state(), eng.trace()))
    ref = states[0]
    for tile, st, (te, ta) in states[1:-1]:
        assert np.array_equal(ta, ref[2][1]), tile
        assert st["movematrix_old"].tobytes() == ref[1]["movematrix_old"].tobytes(), tile
    # the last tile sums 2,560 points at a time: its FP32 energies, and with them its ties, differ
    if scale > 0.01:
        assert np.array_equal(states[-1][2][1], ref[2][1])
    te, ta = ref[2]
    rm = po.ref_map(ff, cx)
    close = 0
    for r in range(cx.n_rep):
        il, it = r % cx.n_lig, r // cx.n_lig
        mm = np.zeros(6, np.float32)
        e_old = po.pose_energy(ff, cx, 0, il, mm, rm, 64)["e"][9]
        for s in range(n_steps):
            delta, u = po.draw_steps(params.seed, params.move_kind, list(params.move_scale), r, s)
            new = (mm + np.asarray(delta, np.float32)).astype(np.float32)
            o = po.pose_energy(ff, cx, 0, il, new, rm, 64)
            mb = float(cx.temp["minus_beta"][it])
            # FP32 energies: 2e-6 of the weighted terms' magnitudes covers both poses' errors
            tol = 2e-6 * float(np.abs(np.asarray(o["e"])[:9] * np.array(ff.w[:9])).sum())
            lo, hi = (u < np.exp(min(0.0, mb * (o["e"][9] - e_old + d))) for d in (tol, -tol))
            if lo == hi:
                assert ta[r, s] == lo, (r, s)
            else:
                close += 1
            if ta[r, s]:
                mm, e_old = new, o["e"][9]
    # at the lowest temperature the kernel, whose margin is wider, has had ties to resolve
    assert close > 0 or floor > 1e-6
