"""FP64 valuations on a caller's own normals (hjm_run_with_normals) where they
are unlike the generator's draws."""
from __future__ import annotations

import numpy as np
import pytest

from cva_hjm_cuda_gb300.market import Market, Swap

pytestmark = pytest.mark.gpu


def _exposures(engine, z, dates, dt, form):
    engine.keep_exposures(True)
    engine.set_remainder_form(form)
    try:
        engine.run_with_normals(z, z.shape[1], dt, "fp64")
        return engine.exposures()
    finally:
        engine.set_remainder_form("auto")
        engine.keep_exposures(False)


@pytest.mark.parametrize("scheme", ["euler", "predictor_corrector"])
@pytest.mark.parametrize("dates", [1, 2, 30])
@pytest.mark.parametrize("fill", [1e12, np.nan, np.inf])
def test_the_first_block_is_not_read(engine, scheme, dates, fill):
    """The first block holds the curve at spot: whatever its normals are, the
    exposures are those of the same call with zeros there, bit for bit."""
    engine.set_scheme(scheme)
    try:
        engine.set_market(Market())
        engine.set_swap(Swap(n_periods=dates))
        z = np.random.default_rng(2).standard_normal((130, 25 * dates, 3))
        z[:, :25] = 0.0
        want = _exposures(engine, z, dates, 0.02, "auto")
        z[::3, :25] = fill
        np.testing.assert_array_equal(_exposures(engine, z, dates, 0.02, "auto"), want)
        assert dates == 1 or np.max(want) > 0.0  # (one date: the swap is out of the money on every path)
    finally:
        engine.set_scheme("euler")
