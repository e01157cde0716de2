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
