"""Calls under a cap on the context's device memory (hjm_ctx_set_memory_limit):
what a call could do without does not make it fail."""
from __future__ import annotations

import numpy as np
import pytest

from cva_hjm_cuda_gb300.engine import HJMEngine
from cva_hjm_cuda_gb300.market import Market, RunConfig, Swap

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("room", [0, 64 * 1024])
@pytest.mark.parametrize("q", [0.975, 0.5])
def test_pfe_without_room_for_its_candidates(precision, room, q):
    """With all else held and the selection's states (4 KB) but little or no room
    for the candidates, the PFE is the same, bit for bit."""
    cfg = RunConfig(n_paths=120_001, n_steps=200, seed=8, pfe_quantile=q)
    with HJMEngine(0) as eng:
        eng.set_market(Market())
        eng.set_swap(Swap(n_periods=4, strike=0.01))
        eng.keep_exposures(True)
        eng.run(cfg, precision, pfe=False)
        held = eng.memory_in_use()
        eng.set_memory_limit(held + 4096 + room)
        v = eng.run(cfg, precision)
        assert eng.memory_in_use() <= held + 4096 + room
        eng.set_memory_limit(0)
        w = eng.run(cfg, precision)
    np.testing.assert_array_equal(v.pfe, w.pfe)
    np.testing.assert_array_equal(v.ee, w.ee)
    assert np.max(w.pfe) > 0.0


@pytest.mark.parametrize("dates,n_paths", [(4, 300), (50, 40_000)])
def test_a_small_valuation_fits_a_small_cap(dates, n_paths):
    """Partial sums (a row of dates + 3 per 64 paths at most), their column sums (2 KB) and the
    results (1.1 KB) are all that a mixed valuation on a table needs."""
    mk = Market(vol=Market().vol * (1.0 + 0.1 * np.cos(np.arange(51) / 7.0))[None, :])
    cfg = RunConfig(n_paths=n_paths, n_steps=50 * dates, seed=8)

    def run(limit):
        with HJMEngine(0) as eng:
            eng.set_market(mk)
            eng.set_swap(Swap(n_periods=dates))
            eng.set_memory_limit(limit)
            return eng.run(cfg, "mixed", pfe=False)

    v, w = run(4096 + 8 * (dates + 3) * (n_paths // 64 + 1)), run(0)
    np.testing.assert_array_equal(v.ee, w.ee)
    assert v.cva == w.cva


@pytest.mark.parametrize("scheme", ["euler", "predictor_corrector"])
@pytest.mark.parametrize("dates,n_tenor", [(2, 51), (20, 51), (34, 51), (60, 61)])
@pytest.mark.parametrize("normals", [False, True])
def test_operand_table_in_little_room(scheme, dates, n_tenor, normals):
    """An FP64 run keeps its response form while one window's operand image fits: the
    images built one at a time, and in windows of eight dates, are bit for bit those of
    the whole table, and the run convects only below that."""
    n_paths, stride = 200, 25
    mk = Market(n_tenor=n_tenor)
    mk = Market(n_tenor=n_tenor, vol=mk.vol * (1.0 + 0.1 * np.cos(np.arange(n_tenor) / 7.0))[None, :])
    sw = Swap(n_tenor=n_tenor, n_periods=dates, strike=0.01)
    cfg = RunConfig(n_paths=n_paths, n_steps=stride * dates, dt=0.02, seed=5)
    z = np.random.default_rng(dates).standard_normal((n_paths, cfg.n_steps, 3)) if normals else None

    def run(limit):
        with HJMEngine(0) as eng:
            eng.set_scheme(scheme)
            eng.set_market(mk)
            eng.set_swap(sw)
            eng.keep_exposures(True)
            eng.set_memory_limit(limit)
            v = eng.run(cfg, "fp64", pfe=False) if z is None else eng.run_with_normals(z, cfg.n_steps, cfg.dt, pfe=False)
            assert limit == 0 or eng.memory_in_use() <= limit
            x = eng.exposures() if limit == 0 else eng.exposure_paths(0, n_paths)
            return v, x, eng.remainder_form()

    # bytes of the images: a chunk of 16 steps is 3 x 5 x 32 bytes a column, two columns a date in steps of 16
    slots = min(dates - 1, 24 if normals else 32)
    chunk = lambda n: 480 * max(16, -(-2 * n // 16) * 16)  # noqa: E731
    chunks = -(-stride * (dates - 1) // 16)
    rest = 16384 + 2 * n_paths * 8 * (dates + 4) + (2 * 24 * n_paths * cfg.n_steps if normals else 0)
    want, x, form = run(0)
    assert form == "response"
    for limit in (chunks * chunk(slots) + rest, chunks * chunk(min(slots, 8)) + rest):
        got, y, form = run(limit)
        assert form == "response"
        np.testing.assert_array_equal(y, x)
        assert np.max(x) > 0.0
        np.testing.assert_allclose(got.ee, want.ee, rtol=1e-13)  # (whole or split tiles: other partial rows)
    assert dates == 2 or run(rest)[2] == "convect"  # (two dates' image fits what the rest leaves)


@pytest.mark.parametrize("dates,dt,n_paths", [(10, 0.0001, 300), (20, 0.0005, 5000), (50, 0.002, 20_000)])
def test_static_entry_with_many_steps(dates, dt, n_paths):
    """Runs whose whole operand table exceeds the static array (10y and 25y at small steps)
    equal the context's run: the same integer sums."""
    from test_zz_no_alloc import _run_static

    from cva_hjm_cuda_gb300 import _lib

    mk, sw = Market(), Swap(n_periods=dates)
    cfg = RunConfig(n_paths=n_paths, n_steps=dates * int(round(0.5 / dt)), dt=dt, seed=4)
    with HJMEngine(0) as eng:
        eng.set_market(mk)
        eng.set_swap(sw)
        ref = eng.run(cfg, "fp64", pfe=False)
    lib = _lib.load()
    st, ee, cva = _run_static(lib, mk, sw, cfg, "fp64")
    assert st == 0, lib.hjm_last_error(None)
    np.testing.assert_allclose(ee, ref.ee, rtol=1e-13, atol=0)
    assert cva[0] == pytest.approx(ref.cva, rel=1e-13)
