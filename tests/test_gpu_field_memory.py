"""The far fields' tables are optional: they take no memory that the context, or a later call on it,
needs."""
import numpy as np
import pytest

from geaxdock_gpu_b200 import abi, engine, system
from tests.golden.fixtures import load_ref

pytestmark = pytest.mark.gpu
MB = 1 << 20


def _batch(n):
    """n complexes on proteins of their own, about 15 MB of tables each."""
    z, _, _ = load_ref("1a07C1")
    ff = system.forcefield(abi.enepara_raw_from_array(z["enepara_raw"]), 42)
    rng = np.random.default_rng(12)
    return ff, [system.make_complex(rng, ff, L=30, n_lig=2, P=2500, n_prt=4, n_tmp=2,
                                    pocket=np.array([60.0 * i, 0.0, 0.0])) for i in range(n)]


class _Fill:
    """Holds device memory so that `leave` bytes are free."""

    def __init__(self, leave):
        self.leave, self.held = leave, []

    def __enter__(self):
        import torch
        engine.release_memory(0)
        torch.cuda.empty_cache()
        free = torch.cuda.mem_get_info(0)[0]
        self.held = [torch.empty(free - self.leave, dtype=torch.uint8, device="cuda")]
        return self

    def __exit__(self, *a):
        import torch
        self.held = []
        torch.cuda.empty_cache()
        engine.release_memory(0)


def _steps(eng):
    eng.mc_init()
    eng.run_fused(0, 20)
    eng.sync()
    return eng.state()


def test_a_context_that_fits_without_tables_is_made():
    ff, cxs = _batch(48)
    n_rep = sum(c.n_rep for c in cxs)
    dump = 700 * MB // (n_rep * abi.RECORD_DTYPE.itemsize)
    params = abi.mc_params(steps_per_exchange=10, steps_per_dump=dump, seed=3)
    with engine.Engine(ff, cxs, params) as eng:
        tables = eng.far_field_bytes()
        ref = _steps(eng)
    assert tables > 400 * MB
    with _Fill(1100 * MB):
        with engine.Engine(ff, cxs, params) as eng:
            held = eng.far_field_bytes()
            st = _steps(eng)
    assert 0 < held <= 100 * MB
    assert np.array_equal(st["movematrix_old"], ref["movematrix_old"])
    assert np.array_equal(st["n_accept"], ref["n_accept"])
    assert np.array_equal(st["replica"]["idx_tmp"], ref["replica"]["idx_tmp"])


def test_a_later_need_takes_the_tables_memory():
    ff, cxs = _batch(20)
    n_rep = sum(c.n_rep for c in cxs)
    params = abi.mc_params(steps_per_exchange=10, steps_per_dump=40, seed=3)
    with engine.Engine(ff, cxs, params) as eng, engine.Engine(ff, cxs, params) as ref:
        tables = eng.far_field_bytes()
        assert tables > 280 * MB
        want = _steps(ref)
        got = _steps(eng)
        assert got.tobytes() == want.tobytes()
        with _Fill(128 * MB):
            eng.trace_enable(300 * MB // (8 * n_rep))
            assert eng.far_field_bytes() == 0 and ref.far_field_bytes() == tables
            for e in (eng, ref):
                e.run_fused(20, 20)
                e.sync()
            st, want = eng.state(), ref.state()
            eng.trace_enable(0)
    assert np.array_equal(st["movematrix_old"], want["movematrix_old"])
    # each side within 1e-6 of its terms' magnitudes (tests/test_gpu_farfield.py)
    e, f = st["energy_old"]["e"].astype(np.float64), want["energy_old"]["e"].astype(np.float64)
    mag = (np.abs(f[:, :9]) * np.abs(np.array(ff.w[:9]))).sum(1)
    assert np.all(np.abs(e[:, 9] - f[:, 9]) <= 2e-6 * mag)


def test_tables_are_given_back_on_request():
    ff, cxs = _batch(1)
    params = abi.mc_params(steps_per_exchange=10, steps_per_dump=40, seed=3)
    mm = np.random.default_rng(1).normal(0.0, 1.0, (40, 6)).astype(np.float32)
    with engine.Engine(ff, cxs, params) as eng:
        assert eng.far_field_bytes() > 0
        a = eng.eval_energy(0, 1, 0, mm)
        eng.release_far_fields()
        eng.release_far_fields()
        assert eng.far_field_bytes() == 0
        b = eng.eval_energy(0, 1, 0, mm)
    assert a.tobytes() != b.tobytes()
    np.testing.assert_allclose(a["e"], b["e"], rtol=2e-5, atol=1e-6)
    assert np.array_equal(a["cms"], b["cms"])
