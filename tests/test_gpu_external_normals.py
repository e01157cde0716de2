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


def _exact_exposures(mk, sw, z, dt):
    """Per-path exposures [date][path] of the Euler step in extended precision
    (simulation_cpu.h:37-54, 96-108, 269-296)."""
    q = np.longdouble
    n, steps, _ = z.shape
    stride = int(round(mk.dtau / dt))
    dates, dtau = steps // stride, q(mk.dtau)
    dt = q(dt)
    c = dt / dtau
    load = np.sqrt(dt) * mk.vol.astype(q)
    f = np.broadcast_to(mk.spot.astype(q), (n, mk.n_tenor)).copy()
    acc, drift = f * stride, mk.drift.astype(q) * dt
    cf = np.zeros((dates + 1, n), dtype=q)
    for i in range(1, dates + 1):
        pay = q(sw.notional) * sw.accrual.astype(q)[i] * (1 if sw.payer else -1)
        cf[i] = np.exp(-acc[:, i] * dt) * pay * ((np.exp(f[:, i] * dtau) - 1) / dtau - q(sw.strike))
        for s in range(stride * i, stride * (i + 1) if i < dates else 0):
            slope = np.concatenate([f[:, 1:] - f[:, :-1], f[:, -1:] - f[:, -2:-1]], axis=1)
            f = f + drift + c * slope + z[:, s].astype(q) @ load
            acc = acc + f
    tail = np.cumsum(cf[::-1], axis=0)[::-1]  # sum of cash flows i >= j
    return np.append(np.maximum(tail[1:], 0), np.zeros((1, n), dtype=q), axis=0).astype(float)


SHAPES = {"constant 3.65": 3.65, "constant 7.9": 7.9, "constant 0.1": 0.1, "constant 0.0039": 0.0039,
          "constant 1e-6": 1e-6, "signs": np.array([7.9, 7.9, -7.9]), "drift of 3": None, "N(0,1)": None}


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("market", ["flat-first-factor", "table"])
@pytest.mark.parametrize("dates,dt,tol", [(20, 0.01, 1e-13), (50, 0.02, 5e-13), (6, 0.0002, 1e-12)])
def test_normals_that_do_not_average_out(engine, shape, market, dates, dt, tol):
    """Normals that add up coherently (a stress path's constant shock, a drift)
    keep the accuracy of random ones against extended precision: the contraction
    holds 1e-14 of the scale, the FP64 curve and prices the rest (the bounds of
    the other FP64 tests; 12,500 additions of 2^-54 each come to 7e-13)."""
    mk = Market()
    if market == "table":
        mk = Market(vol=mk.vol * (1.0 + 0.1 * np.cos(np.arange(51) / 7.0))[None, :])
    sw = Swap(n_periods=dates, strike=0.01)
    engine.set_market(mk)
    engine.set_swap(sw)
    steps = dates * int(round(0.5 / dt))
    rng = np.random.default_rng(dates)
    z = np.full((4, steps, 3), SHAPES[shape]) if SHAPES[shape] is not None else rng.standard_normal((4, steps, 3))
    if shape == "drift of 3":
        z += 3.0
    x, want = _exposures(engine, z, dates, dt, "auto"), _exact_exposures(mk, sw, z, dt)
    scale = np.max(want)
    assert scale > 0.0
    assert np.max(np.abs(x - want)) <= tol * scale


def test_a_paths_scale_is_its_own(engine):
    """The rows of one call, 2^-30, 1 and 2^3 times standard normals, equal the
    calls with each row alone, bit for bit."""
    engine.set_market(Market())
    engine.set_swap(Swap(n_periods=6, strike=0.01))
    z = np.random.default_rng(4).standard_normal((3, 300, 3)).astype(np.float32).astype(float)
    z[0] *= 2.0**-30
    z[2] *= 2.0**3
    x = _exposures(engine, z, 6, 0.01, "auto")
    for p in range(3):
        np.testing.assert_array_equal(_exposures(engine, z[p:p + 1], 6, 0.01, "auto")[:, 0], x[:, p])
