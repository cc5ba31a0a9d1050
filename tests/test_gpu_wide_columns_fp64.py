"""The primal steps of two nonzeros a column in FP64, which take 16 bytes of every vector a thread from
80,000 columns on: numbers of columns around that and around a CTA's 512, about 20 nonzeros a row,
shared and own column bounds, classic and Halpern, against the oracle. Tolerance and rounding of the
inputs as in tests/test_gpu_steps.py (1e-12 after 8 steps)."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_steps import _check64, _device, _equilibrated, _start, _steps

pytestmark = pytest.mark.gpu


def _lp(n, shared):
    from samaya_gb300.model import LpProblem
    rng = np.random.default_rng(n)
    m = n // 10
    first = rng.integers(0, m, n)
    second = (first + rng.integers(1, m, n)) % m
    rows = np.sort(np.stack([first, second], axis=1), axis=1)
    lower = np.concatenate([np.zeros(n), rng.uniform(-1.0, 0.0, m)])
    upper = np.concatenate([np.full(n, np.inf), rng.uniform(0.0, 1.0, m)])
    if not shared:
        lower[:n] = rng.uniform(-1.0, 0.0, n)
        upper[:n] = rng.uniform(0.0, 1.0, n)
    return LpProblem(m, n, 2 * np.arange(n + 1), rows.ravel(), rng.uniform(0.5, 2.0, 2 * n),
                     rng.uniform(-1.0, 1.0, n + m), lower, upper)


@pytest.mark.parametrize("n", [79999, 80000, 80001, 80383, 80384, 80385])
@pytest.mark.parametrize("shared", [True, False])
def test_wide_columns(engine, oracle, n, shared):
    rng = np.random.default_rng(17)
    lp = _lp(n, shared)
    e = _equilibrated(lp, rng)
    v, y, v0, y0 = start = _start(rng, e)
    steps = _steps(e)
    args = (e["m"], e["n"], e["colptr"], e["rowidx"]) + tuple(
        e[k] for k in ("vals", "cost", "lower", "upper"))
    dev = _device(engine, e, 0)
    dev.set_original(e["cs"], e["rs"], lp.cost, lp.lower, lp.upper)
    dev.set_state(*start, precision=0)
    for k in range(8):
        dev.halpern_step(*steps, 3 + k)
        dev.advance()
    got = dev.download()
    want = oracle.halpern_steps(*args, *map(float, steps), 8, 3, v, y, v0, y0)
    for a, b in (("v", "v"), ("y", "y"), ("v_erg", "v_hat"), ("y_erg", "y_hat")):
        _check64(got[a], want[b])
    dev.set_state(v, y, v, y, precision=0)
    for k in range(8):
        dev.step(*steps, 1.0, k)
        dev.advance()
    got = dev.download()
    dev.close()
    state = dict(v=v.copy(), v_prev=v.copy(), y=y.copy(), v_erg=np.zeros_like(v),
                 y_erg=np.zeros_like(y))
    want = oracle.pdhg_steps(*args, *map(float, steps), 8, 0, state)
    for a in ("v", "y", "v_erg", "y_erg"):
        _check64(got[a], want[a])
