"""The slicing arithmetic of the FP64 contraction (hjm_contract.cu), restated
in numpy: the slices of a normal are exact in FP16 and sum to it, those of a
response likewise, and the sums of the two exact levels over a 12-chunk group
stay within the FP32 accumulators' exact range."""
from __future__ import annotations

import numpy as np
import pytest

GRID, SHIFT, TOP, LEVELS = 2.0**-7, 2.0**10, 8, 5


def slice_normals(phi):
    """a0..a3 by the kernel's FP32 operations (each exact until the last rounding)."""
    g, out = np.float32(98304.0), []
    d = phi.astype(np.float32)
    for s in range(3):
        t = (d.astype(np.float64) * (SHIFT if s else 1.0) + float(g)).astype(np.float32)
        a = t - g
        d = (d.astype(np.float64) * (SHIFT if s else 1.0) - a).astype(np.float32)
        out.append(a)
    out.append((d * np.float32(SHIFT)).astype(np.float16).astype(np.float32))
    return out


def slice_responses(r):
    e = np.frexp(np.max(np.abs(r)))[1]
    x = np.ldexp(r, TOP - e)
    out = []
    for s in range(LEVELS):
        b = np.rint(x) if s < LEVELS - 1 else x.astype(np.float16).astype(np.float64)
        out.append(b)
        x = (x - b) * SHIFT
    return out


@pytest.mark.parametrize("scale", [1.0, 2.0**-9, 2.0**-20])
def test_normal_slices_are_exact(scale):
    phi = np.clip(np.random.default_rng(1).standard_normal(200_000) * scale, -5.77, 5.77).astype(np.float32)
    a = slice_normals(phi)
    for s in a:
        assert np.array_equal(s.astype(np.float16).astype(np.float32), s)
    for s in a[:3]:
        assert np.array_equal(np.rint(s / GRID) * GRID, s)
    total = sum(s.astype(np.float64) * SHIFT**-i for i, s in enumerate(a))
    big = np.abs(phi) >= 2.0**-14
    assert np.array_equal(total[big], phi[big].astype(np.float64))
    # below, the fourth slice rounds to 11 bits of at most half the third's grid
    assert np.max(np.abs(total - phi)) <= 2.0**-40


@pytest.mark.parametrize("shape", ["constant", "decaying", "oscillating"])
def test_level_sums_stay_exact(shape):
    rng = np.random.default_rng(7)
    n, m = 576, 4000  # one accumulator group: 12 chunks of 48 values
    t = np.arange(n)
    r = {"constant": np.full(n, 0.0064), "decaying": 0.01 * np.exp(-t / 90.0),
         "oscillating": 0.004 * np.cos(t / 17.0) + 1e-4 * rng.standard_normal(n)}[shape]
    b = slice_responses(r)
    for s in b:
        assert np.array_equal(s.astype(np.float16).astype(np.float64), s)
    phi = np.clip(rng.standard_normal((m, n)), -5.77, 5.77).astype(np.float32)
    a = slice_normals(phi)
    for lev in range(2):
        acc = sum(a[i].astype(np.float64) @ b[lev - i] for i in range(lev + 1))
        assert np.max(np.abs(acc)) / GRID < 2.0**24  # in grid units: the accumulators' exact range
