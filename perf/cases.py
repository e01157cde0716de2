"""The work that users of this engine have it do, as measurable cases.

A case names the call (a valuation, the reference's drop-in call, the adjoint),
the market, the product, the precision, the time scheme and the sizes.  The
sizes are those of this repository's configurations, tests and benchmark: the
reference driver's own 25y call at its published 5,000 scenarios and at 1M
paths, the 10y swap from the default 5,000 paths to 4M, the 30y swap and
netting set on 61 tenors, and odd path counts between.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from cva_hjm_cuda_gb300.engine import HJMEngine, calculate_exposure_gpu, calculate_exposure_gpu_fp32
from cva_hjm_cuda_gb300.market import Market, NettingSet, RunConfig, Swap

DTAU = 0.5
# Polynomials whose values, printed to nine decimals, make the kind of PCA
# volatility table the reference's driver carries (powers of T per factor).
PCA_COEFFS = ((6.430655e-3, 0.0, 0.0, 0.0),
              (-3.55654284e-3, -5.68399973e-4, 1.18191505e-4, -3.59390010e-6),
              (-4.75067182e-3, 1.75417844e-3, -1.41524913e-4, 3.12740033e-6))
POLY_COEFFS = ((0.0064, 0.0, 0.0), (-0.0036, 0.0004, 0.0), (0.0020, -0.0006, 0.00002))


def _case(name, entry, market, precision, n_tenor, years, paths, *, dt=0.01, scheme="euler", swaps=1, pfe=False,
          checkpoint=0):
    c = {"entry": entry, "market": market, "precision": precision, "n_tenor": n_tenor, "years": years, "paths": paths,
         "dt": dt, "scheme": scheme, "swaps": swaps, "pfe": pfe, "checkpoint": checkpoint}
    return {"name": name, **c} if name else c


def listed():
    return [
        # the reference's own published measurement: its driver's 25y swap on its
        # PCA table, 5,000 scenarios, the double overload of its entry point
        _case("driver-25y-fp64-5k", "dropin", "pca", "fp64", 51, 25.0, 5000),
        # the same call at a production path count
        _case("driver-25y-fp64-1m", "dropin", "pca", "fp64", 51, 25.0, 1048576),
        # the float overload of the same call
        _case("driver-25y-fp32-1m", "dropin", "pca", "mixed", 51, 25.0, 1048576),
        # one interactive valuation at the default run size, EE + PFE + CVA
        _case("swap-10y-fp64-5k", "run", "poly", "fp64", 51, 10.0, 5000, pfe=True),
        # the benchmark's headline valuation
        _case("swap-10y-fp64-1m", "run", "poly", "fp64", 51, 10.0, 1048576, pfe=True),
        # the benchmark's mixed-precision valuation, the largest path count used in earnest
        _case("swap-10y-mixed-4m", "run", "poly", "mixed", 51, 10.0, 4194304, pfe=True),
        # a calibration's raw factors: a volatility table of no polynomial shape, an odd path count
        _case("table-10y-fp64-300k", "run", "table", "fp64", 51, 10.0, 300007, pfe=True),
        # the 64-swap netting set on the 30y grid
        _case("netting-30y-mixed-512k", "run", "poly", "mixed", 61, 30.0, 524288, swaps=64),
        # a 30y swap in FP64, an odd path count
        _case("swap-30y-fp64-100k", "run", "poly", "fp64", 61, 30.0, 100003),
        # the predictor-corrector scheme at half the default step's accuracy
        _case("pc-10y-fp64-200k", "run", "poly", "fp64", 51, 10.0, 200000, dt=0.02, scheme="predictor_corrector"),
        # CVA with its 112 sensitivities, the sampled states kept
        _case("adjoint-10y-1m", "adjoint", "poly", "mixed", 51, 10.0, 1048576),
        # the adjoint with its default curve checkpoints
        _case("adjoint-10y-ckpt32-256k", "adjoint", "poly", "mixed", 51, 10.0, 262144, checkpoint=32),
    ]


def draw(rng):
    entry = rng.choice(("run", "run", "run", "run", "dropin", "adjoint"))
    paths = int(round(math.exp(rng.uniform(math.log(200.0), math.log(1048576.0)))))
    if entry == "dropin":
        precision = rng.choice(("fp64", "mixed"))
        years = rng.choice((5, 10, 12, 15, 20, 25))
        return _case("", entry, rng.choice(("pca", "poly")), precision, 51, float(years), paths)
    n_tenor = rng.choice((51, 51, 61))
    years = rng.randint(2, 2 * (25 if n_tenor == 51 else 30)) / 2.0
    dt = rng.choice((0.005, 0.01, 0.01, 0.02))
    if entry == "adjoint":
        years = min(years, 15.0)
        return _case("", entry, "poly", "mixed", n_tenor, years, min(paths, 524288), dt=max(dt, 0.01),
                     checkpoint=rng.choice((0, 0, 16)))
    precision = rng.choice(("fp64", "fp64", "mixed"))
    scheme = rng.choice(("euler", "euler", "euler", "predictor_corrector"))
    market = rng.choice(("poly", "poly", "pca", "table"))
    cost = 1048576 * 2500  # path-steps of the largest FP64 case
    paths = min(paths, int(cost * (0.25 if market == "table" else 0.5) / (years / dt)))
    return _case("", entry, market, precision, n_tenor, years, paths, dt=dt, scheme=scheme,
                 swaps=rng.choice((1, 1, 1, rng.randint(2, 200))), pfe=rng.random() < 0.6)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _steps(case):
    stride = int(round(DTAU / case["dt"]))
    dates = int(round(case["years"] / DTAU))
    return stride, dates


def _inputs(case, seed):
    """The market, product and run numbers of a call, from the seed alone."""
    rng = np.random.default_rng([seed, 20261205])
    nt = case["n_tenor"]
    T = DTAU * np.arange(nt)
    _, dates = _steps(case)
    level, slope = 0.03 * rng.uniform(0.8, 1.3), 0.01 * rng.uniform(0.5, 1.5)
    e = np.exp(-T / 2.0)
    spot = level - slope * e + slope * (T / 2.0) * e
    scale = rng.uniform(0.85, 1.15, 3)
    coef = np.array(POLY_COEFFS) * scale[:, None]
    if case["market"] == "pca":
        p = np.array(PCA_COEFFS) * scale[:, None]
        vol = np.round(p @ np.stack([(T * 25.0 / T[-1]) ** d for d in range(4)]), 9)
    else:
        vol = coef @ np.stack([T**d for d in range(3)])
    if case["market"] == "table":
        vol = vol * (1.0 + 0.1 * np.cos(np.arange(nt) / 7.0 + rng.uniform(0.0, 1.0))[None, :])
    seg = 0.5 * (vol[:, 1:] + vol[:, :-1]) * DTAU
    drift = np.sum(vol * np.concatenate([np.zeros((3, 1)), np.cumsum(seg, axis=1)], axis=1), axis=0)
    if case["swaps"] > 1:
        n = case["swaps"]
        rate = rng.uniform(0.01, 0.04, n)
        book = {"notional": np.exp(rng.uniform(np.log(1e5), np.log(1e7), n)), "fixed_rate": rate,
                "n_periods": np.clip(np.rint(rng.uniform(1.0, case["years"], n) / DTAU), 1, dates).astype(np.int32),
                "payer": (rng.uniform(size=n) < 0.5).astype(np.int32)}
        accrual = None
    else:
        book = None
        accrual = np.zeros(nt)
        accrual[1:dates + 1] = DTAU
        if case["entry"] == "dropin":  # day-count fractions, as the reference's driver has them
            accrual[1:dates + 1] = np.round(DTAU + rng.choice((0.002778, 0.005556, 0.011111, 0.016667), dates), 6)
    return {"spot": spot, "vol": vol, "drift": drift, "coef": coef, "book": book, "accrual": accrual,
            "notional": 1.0e6 * rng.uniform(0.5, 2.0), "strike": float(spot[1:dates + 1].mean()) * rng.uniform(0.85, 1.0),
            "hazard": rng.uniform(0.01, 0.03), "recovery": 0.4, "quantile": 0.975,
            "seed": 1234 if case["entry"] == "dropin" else int(rng.integers(1, 2**40))}


def prepare(case, seed):
    x = _inputs(case, seed)
    stride, dates = _steps(case)
    if case["entry"] == "dropin":
        real = np.float64 if case["precision"] == "fp64" else np.float32
        arrays = [np.ascontiguousarray(x[k], dtype=real) for k in ("accrual", "spot", "drift")]
        return {"case": case, "call": [x["notional"], x["strike"], case["years"], DTAU, *arrays,
                                       np.ascontiguousarray(x["vol"].ravel(), dtype=real), 0.0, 1, case["paths"],
                                       case["dt"]], "real": real}
    nt = case["n_tenor"]
    eng = HJMEngine(0)
    eng.set_scheme(case["scheme"])
    cfg = RunConfig(n_paths=case["paths"], n_steps=stride * dates, dt=case["dt"], seed=x["seed"], hazard=x["hazard"],
                    recovery=x["recovery"], pfe_quantile=x["quantile"])
    product = (NettingSet(**x["book"]) if x["book"] else
               Swap(notional=x["notional"], strike=x["strike"], n_periods=dates, n_tenor=nt, accrual=x["accrual"]))
    market = Market(n_tenor=nt, dtau=DTAU, spot=x["spot"], vol=x["vol"], drift=x["drift"])
    return {"case": case, "engine": eng, "cfg": cfg, "product": product, "market": market, "spot": x["spot"],
            "coef": x["coef"]}


def run(state):
    """One call as a user makes it, host data in and results on the host: the
    market and the product are set, then the valuation or the adjoint runs.
    Mixed precision prices in FP32 (the drop-in's float overload returns
    floats), so its results are kept as FP32 arrays."""
    case = state["case"]
    if case["entry"] == "dropin":
        ee = np.zeros(51, dtype=state["real"])
        call = calculate_exposure_gpu if state["real"] is np.float64 else calculate_exposure_gpu_fp32
        call(ee, *state["call"])
        return {"ee": ee}
    eng, cfg = state["engine"], state["cfg"]
    real = np.float64 if case["precision"] == "fp64" else np.float32
    if case["entry"] == "adjoint":
        eng.set_market_poly(case["n_tenor"], DTAU, state["spot"], state["coef"])
        eng.set_swap(state["product"])
        s = eng.run_adjoint(cfg, checkpoint_every=case["checkpoint"])
        return {"cva": np.array([s.cva, s.cva_stderr, s.dcva_dhazard]).astype(real),
                "dspot": s.dcva_dspot.astype(real), "ddrift": s.dcva_ddrift.astype(real),
                "dcoef": s.dcva_dvolcoef.astype(real)}
    eng.set_market(state["market"])
    if case["swaps"] > 1:
        eng.set_netting_set(state["product"])
    else:
        eng.set_swap(state["product"])
    v = eng.run(cfg, case["precision"], pfe=case["pfe"])
    out = {"ee": v.ee.astype(real), "cva": np.array([v.cva, v.cva_stderr, v.dcva_dhazard]).astype(real)}
    if case["pfe"]:
        out["pfe"] = v.pfe.astype(real)
    return out


def work(case):
    """Host arrays in and results out; per path-step three normals (two radii,
    two angles and their products, ~30 flops) and three scalar states with
    their sums (~20), per sampled date two exponentials and the cash flow
    (~60); the adjoint as much again for its 12 gathered sums."""
    stride, dates = _steps(case)
    nt = case["n_tenor"]
    steps = stride * (dates - 1)
    flops = case["paths"] * (50.0 * steps + 60.0 * dates)
    if case["entry"] == "adjoint":
        flops += case["paths"] * 24.0 * steps
    values = 8 if case["precision"] == "fp64" else 4
    return {"bytes": float(values * (6 * nt + 2 * nt + 3)), "flops": float(flops)}


# ---------------------------------------------------------------------------
# the same results in 64 bits, in plain torch
# ---------------------------------------------------------------------------
_M32 = 0xFFFFFFFF


def _mul_hi_lo(m, x):
    """High and low words of the 32 x 32 bit product (int64 tensors)."""
    lo16 = (x & 0xFFFF) * m
    hi16 = (x >> 16) * m
    t = hi16 + (lo16 >> 16)
    return t >> 16, ((t & 0xFFFF) << 16) | (lo16 & 0xFFFF)


def _normals(p0, n, first, last, seed, dev):
    """[n][last - first][3] draws of paths p0.. and steps first..last - 1: Philox4x32-10
    with counter (step, 0, path lo, path hi) and the seed as key, Box-Muller on 24-bit uniforms."""
    path = torch.arange(p0, p0 + n, device=dev, dtype=torch.int64)[:, None]
    step = torch.arange(first, last, device=dev, dtype=torch.int64)[None, :]
    c0, c1 = step.expand(n, -1), torch.zeros((), device=dev, dtype=torch.int64)
    c2, c3 = (path & _M32).expand(-1, last - first), path >> 32
    k0, k1 = seed & _M32, seed >> 32
    for _ in range(10):
        h0, l0 = _mul_hi_lo(0xD2511F53, c0)
        h1, l1 = _mul_hi_lo(0xCD9E8D57, c2)
        c0, c1, c2, c3 = h1 ^ c1 ^ k0, l1, h0 ^ c3 ^ k1, l0
        k0, k1 = (k0 + 0x9E3779B9) & _M32, (k1 + 0xBB67AE85) & _M32
    u = [(c >> 8).double() * 2.0**-24 for c in (c0, c1, c2, c3)]
    r0, r1 = torch.sqrt(-2.0 * torch.log1p(-u[0])), torch.sqrt(-2.0 * torch.log1p(-u[2]))
    a0, a1 = math.pi * (2.0 * u[1] - 1.0), math.pi * (2.0 * u[3] - 1.0)
    return torch.stack([r0 * torch.cos(a0), r0 * torch.sin(a0), r1 * torch.cos(a1)], dim=2)


def _slope(f):
    d = f[..., 1:] - f[..., :-1]
    return torch.cat([d, d[..., -1:]], dim=-1)


def _advance(f, c, scheme):
    """One noise-free, drift-free step of the curve f[..., tenor]."""
    e = f + c * _slope(f)
    return e if scheme == "euler" else f + 0.5 * c * (_slope(f) + _slope(e))


def _curve(spot, drift, stride, dates, dt, scheme):
    """The deterministic curve's samples and its sums up to each date's sampling."""
    c = dt / DTAU
    f, total = spot, spot * stride
    samp, sums = [spot[1]], [total[1]]
    for b in range(1, dates):
        for _ in range(stride):
            a = drift * dt + c * _slope(f)
            if scheme == "euler":
                f = f + a
            else:
                f = f + 0.5 * (a + drift * dt + c * _slope(f + a))
            total = total + f
        samp.append(f[b + 1])
        sums.append(total[b + 1])
    return torch.stack(samp), torch.stack(sums)


def _responses(rows, stride, dates, c, scheme):
    """[evolved step][row][2 (dates - 1)]: what one unit of each loading row, injected at a step,
    adds to the sample of dates 2.. and to its running sum."""
    n = stride * (dates - 1)
    h = rows + 0.5 * c * _slope(rows) if scheme != "euler" else rows
    lag, acc = [], []
    total = torch.zeros_like(h)
    for _ in range(max(n, 1)):
        total = total + h
        lag.append(h)
        acc.append(total)
        h = _advance(h, c, scheme)
    lag, acc = torch.stack(lag), torch.stack(acc)
    out = torch.zeros((n, rows.shape[0], 2 * (dates - 1)), dtype=torch.float64, device=rows.device)
    for j in range(2, dates + 1):
        last = stride * (j - 1)  # steps that date j sees
        out[:last, :, 2 * (j - 2)] = lag[:last, :, j].flip(0)
        out[:last, :, 2 * (j - 2) + 1] = acc[:last, :, j].flip(0)
    return out


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x = _inputs(case, seed)
    stride, dates = _steps(case)
    nt, dt, scheme = case["n_tenor"], case["dt"], case["scheme"]
    real32 = case["entry"] == "dropin" and case["precision"] != "fp64"
    cast = (lambda a: np.asarray(a, dtype=np.float32).astype(np.float64)) if real32 else (lambda a: np.asarray(a))
    t64 = lambda a: torch.tensor(cast(a), dtype=torch.float64, device=dev)  # noqa: E731
    adjoint = case["entry"] == "adjoint"
    spot, vol, drift = t64(x["spot"]), t64(x["vol"]), t64(x["drift"])
    if x["book"]:
        pay_a, pay_b = torch.zeros(nt, dtype=torch.float64, device=dev), torch.zeros(nt, dtype=torch.float64, device=dev)
        for n, r, m, p in zip(*(x["book"][k] for k in ("notional", "fixed_rate", "n_periods", "payer"))):
            pay_a[1:m + 1] += (1.0 if p else -1.0) * n * DTAU
            pay_b[1:m + 1] += (1.0 if p else -1.0) * n * DTAU * r
    else:
        pay_a = t64(x["accrual"]) * float(cast(x["notional"]))
        pay_b = pay_a * float(cast(x["strike"]))
    pay_a, pay_b = pay_a[1:dates + 1], pay_b[1:dates + 1]
    haz, rec = (0.0, 0.0) if case["entry"] == "dropin" else (x["hazard"], x["recovery"])
    time = DTAU * torch.arange(dates + 1, dtype=torch.float64, device=dev)
    surv = torch.exp(-haz * time)
    w = torch.zeros(dates + 1, dtype=torch.float64, device=dev)
    w[1:] = (1.0 - rec) * (surv[:-1] - surv[1:])
    dw = torch.zeros_like(w)
    dw[1:] = (1.0 - rec) * (-time[:-1] * surv[:-1] + time[1:] * surv[1:])

    if adjoint:
        coef = t64(x["coef"]).requires_grad_(True)
        powers = torch.stack([(DTAU * torch.arange(nt, dtype=torch.float64, device=dev)) ** d for d in range(3)])
        sig = coef @ powers
        seg = 0.5 * (sig[:, 1:] + sig[:, :-1]) * DTAU
        mu = torch.sum(sig * torch.cat([torch.zeros_like(sig[:, :1]), torch.cumsum(seg, 1)], 1), 0)
        spot_g, mu_g = spot.clone().requires_grad_(True), mu.detach().clone().requires_grad_(True)
        samp, sums = _curve(spot_g, mu_g, stride, dates, dt, scheme)
        vol = sig.detach()
        unit = _responses(powers, stride, dates, dt / DTAU, scheme)
        grad = torch.zeros(3, 3, dtype=torch.float64, device=dev)
        xb, ab = torch.zeros(dates, dtype=torch.float64, device=dev), torch.zeros(dates, dtype=torch.float64, device=dev)
    else:
        samp, sums = _curve(spot, drift, stride, dates, dt, scheme)
    mean_s, mean_a = samp.detach(), sums.detach()
    load = _responses(math.sqrt(dt) * vol, stride, dates, dt / DTAU, scheme)
    steps = load.shape[0]
    load = load.reshape(steps * 3, -1)

    n_all = case["paths"]
    rows = max(1, min(n_all, int(4.0e7 / max(steps, 1))))
    ee = torch.zeros(dates + 1, dtype=torch.float64, device=dev)
    c1 = c2 = 0.0
    store = []
    for p0 in range(0, n_all, rows):
        n = min(rows, n_all - p0)
        xs, am = mean_s.expand(n, -1).clone(), mean_a.expand(n, -1).clone()
        if steps:
            phi = _normals(p0, n, stride, stride * dates, x["seed"], dev)
            h = phi.reshape(n, -1) @ load
            xs[:, 1:] += h[:, 0::2]
            am[:, 1:] += h[:, 1::2]
        D = torch.exp(-am * dt)
        lib = (torch.exp(xs * DTAU) - 1.0) / DTAU
        cf = D * (pay_a * lib - pay_b)
        E = torch.zeros(n, dates + 1, dtype=torch.float64, device=dev)
        v = torch.flip(torch.cumsum(torch.flip(cf, (1,)), 1), (1,))
        E[:, :dates] = torch.clamp(v, min=0.0)
        ee += E.sum(0)
        cva = E @ w
        c1, c2 = c1 + float(cva.sum()), c2 + float((cva * cva).sum())
        if case["pfe"]:
            store.append(E)
        if adjoint:
            bar = torch.cumsum((v > 0.0).double() * w[:dates], 1)  # d cva / d cash flow of date i: dates j < i
            xbar, abar = bar * D * pay_a * torch.exp(xs * DTAU), -dt * bar * cf
            xb += xbar.sum(0)
            ab += abar.sum(0)
            if steps:
                seeds = torch.stack([xbar[:, 1:], abar[:, 1:]], 2).reshape(n, -1)
                for k in range(3):
                    for d in range(3):
                        grad[k, d] += torch.sum((phi[:, :, k] @ unit[:, d, :]) * seeds)
    ee = ee / n_all
    full = np.zeros(nt)
    full[:dates + 1] = ee.cpu().numpy()
    if case["entry"] == "dropin":
        return {"ee": np.concatenate([full, np.zeros(51 - nt)]) if nt < 51 else full}
    mean = c1 / n_all
    var = max(c2 / n_all - mean * mean, 0.0) * n_all / max(n_all - 1, 1)
    head = np.array([float(ee @ w), math.sqrt(var / n_all), float(ee @ dw)])
    if adjoint:
        total = torch.sum(samp * xb / n_all) + torch.sum(sums * ab / n_all)
        total.backward()
        torch.sum(mu * mu_g.grad).backward()
        dcoef = coef.grad + math.sqrt(dt) * grad / n_all
        return {"cva": head, "dspot": spot_g.grad.cpu().numpy(), "ddrift": mu_g.grad.cpu().numpy(),
                "dcoef": dcoef.cpu().numpy()}
    out = {"ee": full, "cva": head}
    if case["pfe"]:
        rank = min(max(math.ceil(x["quantile"] * n_all - 1e-7), 1), n_all)
        pfe = np.zeros(nt)
        for j in range(dates + 1):
            col = torch.cat([e[:, j] for e in store])
            pfe[j] = float(torch.kthvalue(col, rank).values)
        out["pfe"] = pfe
    return out
