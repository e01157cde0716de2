"""GPU parity of the FP64 contraction kernel (hjm_contract.cu) at the sizes
where its tiling can go wrong: path counts around the 128-path tiles and the
SM count, date counts at the edges of the padded accumulator columns (8 dates
a step) and of a launch's 32 slots (24 with external normals), strides shorter
and longer than the 16-step chunks, external normals beyond the slices' range.

Tolerances (as the other FP64 tests'): per-path exposures against the all-FP64
convected step 1e-13 of the exposure scale up to 24 dates, 5e-13 beyond, where
the two FP64 orderings themselves differ by 1e-13."""
from __future__ import annotations

import numpy as np
import pytest

from cva_hjm_cuda_gb300.market import Market, RunConfig, Swap

pytestmark = pytest.mark.gpu


def _table_market(nt):
    mk = Market(n_tenor=nt)
    return Market(n_tenor=nt, vol=mk.vol * (1.0 + 0.1 * np.cos(np.arange(nt) / 7.0))[None, :])


def _both(engine, run):
    """(valuation, exposures) in the response form and convected."""
    out = []
    engine.keep_exposures(True)
    try:
        for form in ("response", "convect"):
            engine.set_remainder_form(form)
            v = run()
            assert engine.remainder_form() == form
            out.append((v, engine.exposures()))
    finally:
        engine.keep_exposures(False)
        engine.set_remainder_form("auto")
    return out


def _close(a, b, dates):
    scale = np.max(np.abs(b))
    assert np.max(np.abs(a - b)) <= (1e-13 if dates <= 24 else 5e-13) * scale


@pytest.mark.parametrize("n_paths", [1, 127, 128, 129, 152 * 128 + 1])
def test_path_counts_at_tile_edges(engine, n_paths):
    engine.set_market(_table_market(51))
    engine.set_swap(Swap(n_periods=4))
    cfg = RunConfig(n_paths=n_paths, n_steps=200, seed=5)
    (v, x), (c, xc) = _both(engine, lambda: engine.run(cfg, "fp64"))
    _close(x, xc, 4)
    np.testing.assert_allclose(v.ee[:4], c.ee[:4], rtol=1e-12, atol=1e-13 * np.max(c.ee))
    assert v.cva == pytest.approx(c.cva, rel=1e-12)


@pytest.mark.parametrize("scheme", ["euler", "predictor_corrector"])
@pytest.mark.parametrize("dates,dt", [(1, 0.01), (2, 0.01), (9, 0.01), (10, 0.02), (25, 0.02), (26, 0.02),
                                      (33, 0.02), (34, 0.02), (60, 0.02), (20, 0.25), (34, 0.125), (60, 0.1),
                                      (5, 0.00125)])
def test_date_counts_and_strides(engine, scheme, dates, dt):
    engine.set_scheme(scheme)
    try:
        engine.set_market(_table_market(61))
        engine.set_swap(Swap(n_tenor=61, n_periods=dates))
        cfg = RunConfig(n_paths=200, n_steps=dates * int(round(0.5 / dt)), dt=dt, seed=6)
        (v, x), (c, xc) = _both(engine, lambda: engine.run(cfg, "fp64"))
    finally:
        engine.set_scheme("euler")
    _close(x, xc, dates)
    np.testing.assert_allclose(v.pfe, c.pfe, rtol=0, atol=5e-13 * np.max(np.abs(xc)))


@pytest.mark.parametrize("dates", [20, 25, 26, 50])
def test_external_normals_beyond_the_slices(engine, dates):
    """FP64 normals, some paths scaled to 50 and 1e3 sigma (each path has a
    scale of its own), one path with a NaN: its exposures are zero and every
    other path equals the run without it."""
    engine.set_market(_table_market(51))
    engine.set_swap(Swap(n_periods=dates))
    z = np.random.default_rng(dates).standard_normal((140, 25 * dates, 3))
    z[3] *= 50.0
    z[135, 30:] *= 1e3
    run = lambda: engine.run_with_normals(z, 25 * dates, 0.02, "fp64")  # noqa: E731
    (_, x), (_, xc) = _both(engine, run)
    for p in range(140):  # the scaled paths on their own scale: their curves round at it
        scale = np.max(np.abs(xc[:, p])) if p in (3, 135) else np.max(np.abs(np.delete(xc, (3, 135), axis=1)))
        if np.isfinite(scale) and scale > 0:
            tol = (1e-13 if dates <= 24 else 5e-13) * (1e3 if p in (3, 135) else 1.0)
            assert np.max(np.abs(x[:, p] - xc[:, p])) <= tol * scale, p
    z[17, 40, 1] = np.nan
    engine.keep_exposures(True)
    try:
        run()
        y = engine.exposures()
    finally:
        engine.keep_exposures(False)
    assert np.all(y[:, 17] == 0.0)
    keep = np.arange(140) != 17
    np.testing.assert_array_equal(y[:, keep], x[:, keep])


@pytest.mark.parametrize("n_paths,dates", [(152 * 128 + 129, 20), (40 * 128 - 5, 50), (3 * 152 * 128 + 700, 34)])
def test_whole_waves_and_split_tiles(engine, n_paths, dates):
    """Tiles beyond the last whole wave of 152 have their steps split over the
    SMs: they must join the whole tiles' paths, exposures and partial sums."""
    engine.set_market(_table_market(51))
    engine.set_swap(Swap(n_periods=dates))
    cfg = RunConfig(n_paths=n_paths, n_steps=25 * dates, dt=0.02, seed=12)
    (v, x), (c, xc) = _both(engine, lambda: engine.run(cfg, "fp64"))
    _close(x, xc, dates)
    np.testing.assert_allclose(v.ee[:dates], c.ee[:dates], rtol=1e-12, atol=1e-13 * np.max(c.ee))
    assert v.cva == pytest.approx(c.cva, rel=1e-12) and v.cva_stderr == pytest.approx(c.cva_stderr, rel=1e-9)


def test_memory_cap_runs_whole_tiles_or_convects():
    """Under a memory cap that leaves no room for the table the run convects, as
    if asked to; with the table but without the split tiles' sums it runs its
    tiles whole (the same integer sums per path, other partial rows)."""
    from cva_hjm_cuda_gb300.engine import HJMEngine

    cfg = RunConfig(n_paths=5000, seed=3)
    with HJMEngine(0) as eng:
        eng.set_market(Market())
        eng.set_swap(Swap())
        eng.set_remainder_form("convect")
        c = eng.run(cfg, "fp64", pfe=False)
        eng.set_remainder_form("auto")
        eng.set_memory_limit(eng.memory_in_use())
        v = eng.run(cfg, "fp64", pfe=False)
        assert eng.remainder_form() == "convect"
        np.testing.assert_array_equal(v.ee, c.ee)
        eng.set_memory_limit(0)
        eng.run(RunConfig(n_paths=152 * 128, seed=3), "fp64", pfe=False)  # (one whole wave: nothing split)
        eng.set_memory_limit(eng.memory_in_use())
        w = eng.run(cfg, "fp64", pfe=False)
        assert eng.remainder_form() == "response"
        eng.set_memory_limit(0)
        s = eng.run(cfg, "fp64", pfe=False)
    np.testing.assert_allclose(w.ee, s.ee, rtol=1e-13, atol=0)
    assert w.cva == pytest.approx(s.cva, rel=1e-13) and w.cva == pytest.approx(c.cva, rel=1e-12)


@pytest.mark.parametrize("n_tenor,dates,n_paths", [(51, 50, 3000), (61, 60, 20_001), (51, 33, 152 * 128)])
def test_static_entry_in_windows(n_tenor, dates, n_paths):
    """The allocation-free entry with one and several windows, split tiles and
    none, equals the context's run (1e-13: the same integer sums)."""
    from test_zz_no_alloc import _run_static

    from cva_hjm_cuda_gb300 import _lib
    from cva_hjm_cuda_gb300.engine import HJMEngine

    mk, sw = _table_market(n_tenor), Swap(n_tenor=n_tenor, n_periods=dates)
    cfg = RunConfig(n_paths=n_paths, n_steps=25 * dates, dt=0.02, seed=4)
    with HJMEngine(0) as eng:
        eng.set_market(mk)
        eng.set_swap(sw)
        ref = eng.run(cfg, "fp64", pfe=False)
    lib = _lib.load()
    st, ee, cva = _run_static(lib, mk, sw, cfg, "fp64")
    assert st == 0, lib.hjm_last_error(None)
    np.testing.assert_allclose(ee, ref.ee, rtol=1e-13, atol=0)
    assert cva[0] == pytest.approx(ref.cva, rel=1e-13)


def test_table_of_another_market_in_the_same_shape():
    """A market change keeps the run shape's walk weights in the table: the
    second market's results equal a new context's bit for bit, also after a run
    of another shape and scheme in between."""
    from cva_hjm_cuda_gb300.engine import HJMEngine

    cfg = RunConfig(n_paths=500, n_steps=26 * 25, dt=0.02, seed=9)
    sw = Swap(n_periods=26)

    def run(eng, mk):
        eng.set_market(mk)
        eng.set_swap(sw)
        return eng.run(cfg, "fp64", pfe=False)

    with HJMEngine(0) as fresh:
        want = run(fresh, _table_market(51))
    with HJMEngine(0) as eng:
        run(eng, Market())
        got = [run(eng, _table_market(51))]
        eng.set_scheme("predictor_corrector")
        run(eng, Market())
        eng.set_scheme("euler")
        eng.set_swap(Swap(n_periods=4))
        eng.run(RunConfig(n_paths=100, n_steps=100, dt=0.02), "fp64", pfe=False)
        run(eng, Market())
        got.append(run(eng, _table_market(51)))
    for v in got:
        np.testing.assert_array_equal(v.ee, want.ee)
        assert v.cva == want.cva


@pytest.mark.parametrize("size", [1e100, 1e301])
def test_loadings_near_overflow(engine, size):
    """Volatilities whose responses come near FP64's limit: the exposures (0, inf) are
    those of the convected step, not those of a curve without noise."""
    mk = _table_market(51)
    engine.set_market(Market(vol=mk.vol * size, drift=np.zeros(51)))
    engine.set_swap(Swap(n_periods=8, strike=0.01))
    (v, x), (c, xc) = _both(engine, lambda: engine.run(RunConfig(n_paths=300, n_steps=200, dt=0.02, seed=3), "fp64"))
    np.testing.assert_array_equal(x, xc)
    assert not np.any(np.isfinite(x) & (x > 0.0))


def test_responses_that_overflow(engine):
    """Volatilities whose responses leave FP64's range give no finite positive exposure."""
    mk = _table_market(51)
    engine.set_market(Market(vol=mk.vol * 1e307, drift=np.zeros(51)))
    engine.set_swap(Swap(n_periods=30, strike=0.01))
    (v, x), _ = _both(engine, lambda: engine.run(RunConfig(n_paths=300, n_steps=750, dt=0.02, seed=3), "fp64"))
    assert not np.any(np.isfinite(x) & (x > 0.0))
