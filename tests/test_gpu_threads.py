"""Distinct contexts driven from different threads at the same time (the
header's promise), with runs of different sizes on the same kernels."""
from __future__ import annotations

import threading

import numpy as np
import pytest

from cva_hjm_cuda_gb300.market import DEFAULT_VOL_COEFFS, Market, RunConfig, Swap

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["fp64", "fp64-convected", "mixed", "adjoint"])
def test_contexts_on_threads_with_different_date_counts(mode):
    """Each thread's results equal its own single-threaded run, bit for bit, and no
    call fails: a kernel's shared-memory limit is not another run's size."""
    from cva_hjm_cuda_gb300.engine import HJMEngine

    dates = (50, 20, 4, 33)
    reps = 60 if mode == "fp64-convected" else 300
    gate = threading.Barrier(len(dates))
    wrong = []

    def drive(nd):
        try:
            with HJMEngine(0) as eng:
                mk = Market()
                eng.set_market_poly(51, 0.5, mk.spot, DEFAULT_VOL_COEFFS)
                eng.set_swap(Swap(n_periods=nd))
                eng.set_remainder_form("convect" if mode == "fp64-convected" else "auto")
                cfg = RunConfig(n_paths=200, n_steps=10 * nd, dt=0.05, seed=nd)

                def value():
                    if mode == "adjoint":
                        return eng.run_adjoint(cfg, checkpoint_every=0).dcva_dspot
                    return eng.run(cfg, mode.split("-")[0], pfe=False).ee

                with lock:
                    want = value()
                gate.wait(timeout=60)
                for _ in range(reps):
                    if not np.array_equal(value(), want):
                        wrong.append((nd, "differs"))
        except Exception as e:  # noqa: BLE001
            wrong.append((nd, str(e)[-120:]))
            gate.abort()

    lock = threading.Lock()
    threads = [threading.Thread(target=drive, args=(nd,)) for nd in dates]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert wrong == []
