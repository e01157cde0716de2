"""The arithmetic of the FP64 contraction (hjm_contract.cu), restated in numpy:
the slices of a normal are exact in FP16 and sum to it, those of a response
likewise, the sums of the two exact levels over a 12-chunk group stay within the
FP32 accumulators' exact range, and the closed (random-walk) form of the step's
responses equals the recursion over the lags."""
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


def _advance(v, c, pc):
    d = np.append(v[1:] - v[:-1], v[-1] - v[-2])
    e = v + c * d
    return v + 0.5 * c * (d + np.append(e[1:] - e[:-1], e[-1] - e[-2])) if pc else e


def _fma(a, b, c):
    """a b + c rounded once (the product's tail beyond extended precision aside)."""
    return (a.astype(np.longdouble) * b + c).astype(float)


def _walk(S, c, M, pc):
    """The kernels' closed form of the step's responses and their running sums."""
    L, m = len(S) - 1, np.arange(M)
    a0, a1, a2 = (1 - c + c * c / 2, c - c * c, c * c / 2) if pc else (1 - c, c, 0.0)
    la = np.log1p(np.longdouble(-c) + (np.longdouble(c) ** 2 / 2 if pc else 0))
    d = S[L] - S[L - 1]
    dev = np.array([S[t] - (S[L] + (t - L) * d) if t < L - 1 else 0.0 for t in range(L + 1)])
    f, h = np.exp(m * la).astype(float), np.exp((m + 1) * la).astype(float)
    f1, h1, g, tail = np.zeros(M), np.zeros(M), np.zeros(M), np.ones(M)
    F, G = [], []
    for i in range(L - 2):
        tail = tail - h
        g = _fma(tail, np.float64(1.0 / (a1 + a2)), -(a2 / (a1 + a2)) * g)
        F.append(f)
        G.append(g)
        f, f1 = _fma((m - i) * (a1 / a0), f, (2 * m - i + 1) * (a2 / a0) * f1) * (1.0 / (i + 1)), f
        h, h1 = _fma((m + 1 - i) * (a1 / a0), h, (2 * m - i + 3) * (a2 / a0) * h1) * (1.0 / (i + 1)), h
    R, C = np.zeros((M, L + 1)), np.zeros((M, L + 1))
    for j in range(2, L + 1):
        at = S[L] + (j - L) * d
        R[:, j] = at + m * c * d
        C[:, j] = (m + 1) * (at + 0.5 * m * c * d)
        for i in range(L - 1 - j):
            R[:, j] = _fma(F[i], dev[j + i], R[:, j])
            C[:, j] = _fma(G[i], dev[j + i], C[:, j])
    return R, C


@pytest.mark.parametrize("pc", [False, True], ids=["euler", "predictor-corrector"])
@pytest.mark.parametrize("c,M", [(0.02, 2450), (0.5, 98), (0.1, 290)])
def test_walk_form_of_the_responses(pc, c, M):
    """The responses against the recursion over the lags in extended precision:
    48 recurrence steps of a few roundings, relative to each date's largest.
    (Their sums enter every date's discount: the GPU tests hold them.)"""
    T = 0.5 * np.arange(51)
    for S in (0.002 - 0.0006 * T + 2e-5 * T**2, 0.004 * np.cos(np.arange(51) / 7.0)):
        R, _ = _walk(S, c, M, pc)
        v, want = S.astype(np.longdouble), np.zeros((M, 51), dtype=np.longdouble)
        for m in range(M):
            want[m] = v
            v = _advance(v, np.longdouble(c), pc)
        for j in range(2, 51):
            assert np.max(np.abs(R[:, j] - want[:, j])) <= 48 * 4 * 2.0**-53 * np.max(np.abs(want[:, j]))


def _ramp_responses(nt, c, m, j, pc):
    """mresp_table_kernel's tail sums: G2, CG2 (responses to e_L), G1, CG1 (to
    e_{L-1}) and G2 a lag on, of date j at lag m."""
    a0, a1, a2 = (1 - c + 0.5 * c * c, c - c * c, 0.5 * c * c) if pc else (1 - c, c, 0.0)
    r1, r2, inv, b2 = a1 / a0, a2 / a0, 1 / (a1 + a2), a2 / (a1 + a2)
    mean = c * (m + 1.0)
    n = min(128, int(mean + 10.0 * np.sqrt(mean)) + 12)
    f, h = np.zeros(n), np.zeros(n)
    f[0], h[0] = np.exp(m * np.log1p(a0 - 1)), np.exp((m + 1) * np.log1p(a0 - 1))
    for i in range(n - 1):
        f[i + 1] = ((m - i) * r1 * f[i] + (2 * m - i + 1) * r2 * (f[i - 1] if i else 0.0)) / (i + 1)
        h[i + 1] = ((m + 1 - i) * r1 * h[i] + (2 * m - i + 3) * r2 * (h[i - 1] if i else 0.0)) / (i + 1)
    q = nt - 1 - j
    i = np.arange(n)
    up = np.maximum(i - q + 1, 0)
    tail = np.append(np.cumsum(h[::-1])[::-1][1:], 0.0)
    g = np.zeros(n)
    for k in range(n):
        g[k] = tail[k] * inv - (b2 * g[k - 1] if k else 0.0)
    down = np.where(i >= q - 1, q - i, 0)
    return (up * f)[::-1].sum(), (up * g).sum(), (down * f)[::-1].sum(), (down * g).sum(), (up * h)[::-1].sum()


@pytest.mark.parametrize("nt,c,stride,B,pc", [(51, 0.02, 50, 20, False), (51, 0.02, 50, 24, True), (61, 0.04, 25, 30, True),
                                              (51, 0.5, 2, 28, False), (35, 0.1, 10, 34, False), (35, 0.5, 2, 33, True)])
def test_walk_tails_equal_the_recursion_over_the_lags(nt, c, stride, B, pc):
    """The mixed response table's closed form against the step's recursion in
    extended precision: entries that count (2^-30 and more) to FP32's rounding,
    smaller ones to 2^-54, half of that rounding at 2^-30."""
    L = nt - 1
    a0, a1, a2 = 1 - c + 0.5 * c * c, c - c * c, 0.5 * c * c
    M = (B - 1) * stride
    hist = np.zeros((2, M + 1, nt), dtype=np.longdouble)
    v = np.zeros((2, nt), dtype=np.longdouble)
    v[0, L] = v[1, L - 1] = 1
    for m in range(M + 1):
        hist[:, m] = v
        w = v.copy()
        w[:, :L] += c * (v[:, 1:] - v[:, :L])
        if pc:
            w[:, : L - 1] = a0 * v[:, : L - 1] + a1 * v[:, 1:L] + a2 * v[:, 2:]
        w[:, L] = v[:, L] + c * (v[:, L] - v[:, L - 1])
        v = w
    cum = np.cumsum(hist, axis=1)
    for j in sorted({2, B // 2, B - 1, B}):
        for m in sorted({0, 1, stride, (j - 1) * stride // 2, (j - 1) * stride - 1}):
            got = _ramp_responses(nt, c, m, j, pc)
            want = [hist[0, m, j], cum[0, m, j], hist[1, m, j], cum[1, m, j], hist[0, m + 1, j]]
            for x, y in list(zip(got, want))[: 5 if pc else 2]:
                assert abs(x - float(y)) <= max(2.0 ** -24 * abs(float(y)), 2.0 ** -54), (j, m, x, y)


@pytest.mark.parametrize("pc", [False, True], ids=["euler", "predictor-corrector"])
@pytest.mark.parametrize("c,M", [(0.02, 2450), (0.5, 98), (0.1, 290)])
def test_walk_form_of_the_running_sums(pc, c, M):
    """The responses' running sums against the cumulated recursion in extended
    precision: the responses' bound, and 48 roundings of the walk's upper tail
    (2^-53 each) that every sum's weight carries, 1 / (a1 + a2) <= 1 / (c - c^2 / 2) times."""
    T = 0.5 * np.arange(51)
    for S in (0.002 - 0.0006 * T + 2e-5 * T**2, 0.004 * np.cos(np.arange(51) / 7.0)):
        _, C = _walk(S, c, M, pc)
        v, total = S.astype(np.longdouble), np.zeros(51, dtype=np.longdouble)
        want = np.zeros((M, 51), dtype=np.longdouble)
        for m in range(M):
            total = total + v
            want[m] = total
            v = _advance(v, np.longdouble(c), pc)
        line = S[50] + (np.arange(51) - 50) * (S[50] - S[49])
        dev = np.cumsum(np.abs(S - line)[::-1])[::-1]
        for j in range(2, 51):
            bound = 48 * 4 * 2.0**-53 * np.max(np.abs(want[:, j])) + 48 * 2.0**-53 / (c - 0.5 * c * c) * dev[j]
            assert np.max(np.abs(C[:, j] - want[:, j])) <= bound
