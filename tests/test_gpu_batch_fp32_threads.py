"""Batches with FP32 storage on both sides of the rule for a CTA's threads: rows and columns of the
largest LP a CTA up to 1,600 (256 threads), above (384), and for the Halpern iteration from 3,000 on
(512), a CTA per LP, alone and together with a small one; slices partly filled.

The averaging iteration against the oracle, the Halpern iteration before its first evaluation against
the oracle's steps on the problem equilibrated by the device's factors, with the tolerance (and its
reason) of tests/test_gpu_batch_clusters.py for FP32: 1e-3 of (1 + max |reference|)."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_batch_clusters import _differs, _lengths, _lp

pytestmark = pytest.mark.gpu

SIZES = [(1, 3), (33, 97), (500, 1099), (500, 1101), (1000, 1999), (1000, 2001)]


@pytest.fixture(autouse=True)
def cta_per_lp(monkeypatch):
    monkeypatch.setenv("SG_MAX_CLUSTER", "1")


def _problems(m, n):
    return [_lp(n, _lengths(m, 1, min(n, 14), m + n), m + n),
            _lp(70, _lengths(31, 1, 9, m + n + 1), m + n + 1)]


def _solve(engine, probs, iterations, algorithm):
    from samaya_gb300.batch import BatchSolver
    s = BatchSolver.from_problems(probs, engine.PdlpOptions(
        tol=1e-30, max_iterations=iterations, precision=engine.FP32_REFINED,
        algorithm=algorithm))
    res, again = s.solve(), s.solve()
    s.close()
    for a, b in zip(res, again):
        assert np.array_equal(a.x, b.x) and np.array_equal(a.y, b.y)
    return res


@pytest.mark.parametrize("m,n", SIZES)
def test_averaging(engine, oracle, m, n):
    probs = _problems(m, n)
    for iterations in (1, 100):
        for lp, r in zip(probs, _solve(engine, probs, iterations, engine.REFERENCE)):
            ref = oracle.pdlp_solve(*lp.arrays(), tol=1e-30, max_iter=iterations)
            assert _differs(r.x, ref.x) <= 1e-3 and _differs(r.y, ref.y) <= 1e-3, iterations


@pytest.mark.parametrize("m,n", SIZES)
def test_halpern(engine, oracle, m, n):
    probs = _problems(m, n)
    for lp, r in zip(probs, _solve(engine, probs, 37, engine.HALPERN)):
        with engine.PdlpSolver(lp, engine.PdlpOptions(algorithm=engine.HALPERN,
                                                      autotune=False)) as s:
            cs, rs, _, eta = s.equilibration()
        nv = lp.n
        cols = np.repeat(np.arange(nv), np.diff(lp.colptr))
        scale = np.concatenate([cs, 1.0 / rs])
        cost, lower, upper = lp.cost * scale, lp.lower / scale, lp.upper / scale
        bound = np.maximum(*[np.where(np.isfinite(b[nv:]), np.abs(b[nv:]), 0.0)
                             for b in (lower, upper)])
        cn, bn = np.linalg.norm(cost[:nv]), np.linalg.norm(bound)
        omega = cn / bn if cn > 1e-10 and bn > 1e-10 else 1.0
        zv, zy = np.zeros(nv + lp.m), np.zeros(lp.m)
        ref = oracle.halpern_steps(lp.m, nv, lp.colptr, lp.rowidx,
                                   rs[lp.rowidx] * lp.vals * cs[cols], cost, lower, upper,
                                   eta / omega, eta * omega, 37, 0, zv, zy, zv, zy)
        assert _differs(r.x, ref["v_hat"] * scale) <= 1e-3
        assert _differs(r.y, ref["y_hat"] * rs) <= 1e-3
