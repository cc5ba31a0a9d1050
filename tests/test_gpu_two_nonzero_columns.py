"""The primal steps of operators with two nonzeros a column: numbers of columns around a thread's 2
(FP64) or 4 (FP32) and a CTA's 512 or 1,024, with shared and with own column bounds, classic and
Halpern, against the oracle. Tolerances and rounding of the inputs as in tests/test_gpu_steps.py
(1e-12 and 1e-5 after 8 steps)."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_steps import _check32, _check64, _device, _equilibrated, _f32, _start, _steps

pytestmark = pytest.mark.gpu


def _lp(n, shared):
    from samaya_gb300.model import LpProblem
    rng = np.random.default_rng(n)
    m = max(2, min(40, n // 3))
    rows = np.array([np.sort(rng.permutation(m)[:2]) for _ in range(n)])
    lower = np.concatenate([np.zeros(n), rng.uniform(-1.0, 0.0, m)])
    upper = np.concatenate([np.full(n, np.inf), rng.uniform(0.0, 1.0, m)])
    if not shared:
        lower[:n] = rng.uniform(-1.0, 0.0, n)
        upper[:n] = rng.uniform(0.0, 1.0, n)
    return LpProblem(m, n, 2 * np.arange(n + 1), rows.ravel(), rng.uniform(0.5, 2.0, 2 * n),
                     rng.uniform(-1.0, 1.0, n + m), lower, upper)


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 7, 511, 512, 513, 1023, 1025, 4099])
@pytest.mark.parametrize("shared", [True, False])
def test_two_nonzero_columns(engine, oracle, n, shared):
    rng = np.random.default_rng(17)
    lp = _lp(n, shared)
    e = _equilibrated(lp, rng)
    start = _start(rng, e)
    steps = _steps(e)
    for precision in (0, 2):
        check = _check64 if precision == 0 else _check32
        round_ = (lambda a: a) if precision == 0 else _f32
        v, y, v0, y0 = (round_(a) for a in start)
        tau, sigma = (float(round_(np.float64(a))) for a in steps)
        args = (e["m"], e["n"], e["colptr"], e["rowidx"]) + tuple(
            round_(e[k]) for k in ("vals", "cost", "lower", "upper"))
        dev = _device(engine, e, precision)
        dev.set_original(e["cs"], e["rs"], lp.cost, lp.lower, lp.upper)
        dev.set_state(*start, precision=min(precision, 1))
        for k in range(8):
            dev.halpern_step(*steps, 3 + k)
            dev.advance()
        got = dev.download()
        want = oracle.halpern_steps(*args, tau, sigma, 8, 3, v, y, v0, y0)
        for a, b in (("v", "v"), ("y", "y"), ("v_erg", "v_hat"), ("y_erg", "y_hat")):
            check(got[a], want[b])
        dev.set_state(start[0], start[1], start[0], start[1], precision=min(precision, 1))
        for k in range(8):
            dev.step(*steps, 1.0, k)
            dev.advance()
        got = dev.download()
        dev.close()
        state = dict(v=v.copy(), v_prev=v.copy(), y=y.copy(), v_erg=np.zeros_like(v),
                     y_erg=np.zeros_like(y))
        want = oracle.pdhg_steps(*args, tau, sigma, 8, 0, state)
        for a in ("v", "y", "v_erg", "y_erg"):
            check(got[a], want[a])
