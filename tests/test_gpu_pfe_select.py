"""The PFE selection's sampled bracket (hjm_pfe.cu) where it can go wrong: open
ends (the smallest and largest exposure), columns just beyond shared memory, a
median, and a column whose strided sample is nothing like the rest, so that the
bracket misses the rank and the whole column is searched.  Bit for bit numpy's
k-th smallest of the stored exposures."""
from __future__ import annotations

import numpy as np
import pytest

from cva_hjm_cuda_gb300.market import Market, RunConfig, Swap

pytestmark = pytest.mark.gpu


def _check(engine, v, q, precision):
    x = engine.exposures()
    for j in range(x.shape[0]):
        col = x[j].astype(np.float32) if precision == "mixed" else x[j]
        k = min(max(int(np.ceil(q * col.size - 1e-7)), 1), col.size)
        assert v.pfe[j] == float(np.partition(col, k - 1)[k - 1]), j


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n_paths,q", [(25_600, 0.975), (25_601, 0.975), (51_201, 0.5), (200_003, 1e-9),
                                       (200_003, 1.0 - 1e-9), (200_003, 0.5), (200_003, 0.999)])
def test_bracket_ends_and_sizes(engine, precision, n_paths, q):
    engine.set_market(Market())
    engine.set_swap(Swap(n_periods=6))
    engine.keep_exposures(True)
    try:
        _check(engine, engine.run(RunConfig(n_paths=n_paths, n_steps=300, pfe_quantile=q, seed=4), precision), q,
               precision)
    finally:
        engine.keep_exposures(False)


def test_sample_unlike_the_column(engine):
    n = 65_536  # the sample takes every fourth path
    z = np.random.default_rng(3).standard_normal((n, 100, 3)) + 1.0
    z[::4] = 0.0
    engine.set_market(Market())
    engine.set_swap(Swap(n_periods=2))
    engine.keep_exposures(True)
    try:
        for q in (0.5, 0.9):
            _check(engine, engine.run_with_normals(z, 100, 0.01, "fp64", pfe_quantile=q), q, "fp64")
    finally:
        engine.keep_exposures(False)
