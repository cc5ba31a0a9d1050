"""The setup's passes where their split over CTAs and warps can go wrong: rows cut into several
tiles, empty rows and columns, 255 to 257 and 513 nonzeros (a warp scales 256 at a time), one
nonzero, bounds that are 0, infinite (not divided) and others.

Scales and the operator norm against the oracle (the reference's Ruiz passes) and against numpy
(the enhanced passes): a statistic sums at most 30,000 products, 30,000 * 2^-53 = 3e-12, eleven
passes halve (square root) and add such errors: 1e-11. One iteration then covers the scaled
matrix, cost and bounds: 1e-9 of (1 + max |reference|)."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_batch_clusters import _differs, _lp

pytestmark = pytest.mark.gpu

LPS = {
    "one nonzero": (2, [1]),
    "255 nonzeros": (90, [85, 0, 85, 85]),
    "257 nonzeros": (90, [85, 0, 85, 0, 87]),
    "513 nonzeros": (600, [0] * 40 + [513] + [0] * 40),
    # More work than the cluster's power iteration takes: the tile kernels.
    "large split rows": (40000, [30000, 4100, 33, 129] + [0, 1, 2, 7] * 700),
    "split rows": (9100, [9000, 1, 0, 4100, 33, 129] + [0, 1, 2, 7] * 700),
}


@pytest.mark.parametrize("name", list(LPS))
def test_setup_passes(engine, oracle, name):
    n, lengths = LPS[name]
    lp = _lp(n, lengths, 5)
    rng = np.random.default_rng(6)
    lp.lower[:n] = rng.choice([-np.inf, 0.0, -1.25, -0.0], n)
    lp.upper[:n] = rng.choice([np.inf, 4.0, 0.0], n)
    cols = np.repeat(np.arange(n), np.diff(lp.colptr))
    rows, a = lp.rowidx, np.abs(lp.vals)
    cs, rs = np.ones(n), np.ones(lp.m)
    for k in range(11):
        cn, rn = np.zeros(n), np.zeros(lp.m)
        (np.maximum if k < 10 else np.add).at(cn, cols, a * rs[rows])
        (np.maximum if k < 10 else np.add).at(rn, rows, a * cs[cols])
        cn, rn = cn * cs, rn * rs
        cs = np.where(cn > 0, cs / np.sqrt(np.where(cn > 0, cn, 1.0)), cs)
        rs = np.where(rn > 0, rs / np.sqrt(np.where(rn > 0, rn, 1.0)), rs)
    scaled = rs[rows] * lp.vals * cs[cols]
    u, sigma = np.asarray(oracle.power_start(lp.m))[:lp.m], 0.0
    for _ in range(20):
        v, w = np.zeros(n), np.zeros(lp.m)
        np.add.at(v, cols, scaled * (u / np.linalg.norm(u))[rows])
        np.add.at(w, rows, scaled * v[cols])
        u, sigma = w, np.linalg.norm(w) / np.linalg.norm(v)
    enhanced = (cs, rs, np.sqrt((1.01 * sigma) ** 2 + 1.0))
    ref = oracle.setup(lp.m, n, lp.colptr, lp.rowidx, lp.vals)
    reference = (ref[1], ref[0], ref[4])
    for algorithm, expect in ((engine.REFERENCE, reference), (engine.ENHANCED, enhanced)):
        s = engine.PdlpSolver(lp, engine.PdlpOptions(
            tol=1e-30, max_iterations=1, algorithm=algorithm, autotune=False))
        got = s.equilibration()
        for g, e in zip(got, expect):
            assert np.all(np.abs(g - e) <= 1e-11 * np.abs(e)), (name, algorithm)
        if algorithm == engine.REFERENCE:
            r = s.solve()
            one = oracle.pdlp_solve(*lp.arrays(), tol=1e-30, max_iter=1)
            assert _differs(r.x, one.x) <= 1e-9 and _differs(r.y, one.y) <= 1e-9


@pytest.mark.parametrize("supplies, demands", [(7, 9), (60, 81), (200, 301)])
def test_enhanced_scales_of_a_transportation_lp_to_the_bit(engine, supplies, demands):
    """One cluster's passes and the tile kernels'. Every nonzero is 1 and a column holds two, so
    the ten maximum passes are the same IEEE products, roots and quotients in any order; the rows'
    sums of the last pass take up to `demands` terms in another order: with the three operations
    after them (demands + 3) * 2^-53."""
    n, m = supplies * demands, supplies + demands
    rowidx = np.empty((n, 2), dtype=np.int32)
    rowidx[:, 0] = np.repeat(np.arange(supplies), demands)
    rowidx[:, 1] = supplies + np.tile(np.arange(demands), supplies)
    lp = engine.LpProblem(
        m=m, n=n, colptr=np.arange(0, 2 * n + 1, 2, dtype=np.int64), rowidx=rowidx.reshape(-1),
        vals=np.ones(2 * n), cost=np.concatenate([np.arange(n) % 7 + 1.0, np.zeros(m)]),
        lower=np.concatenate([np.zeros(n), np.ones(m)]),
        upper=np.concatenate([np.full(n, np.inf), np.ones(m)]))
    s = engine.PdlpSolver(lp, engine.PdlpOptions(
        tol=1e-30, max_iterations=1, algorithm=engine.ENHANCED, autotune=False))
    got = s.equilibration()
    cs, rs = np.ones(lp.n), np.ones(lp.m)
    cols, rows = np.repeat(np.arange(lp.n), np.diff(lp.colptr)), lp.rowidx
    for k in range(11):
        cn, rn = np.zeros(lp.n), np.zeros(lp.m)
        (np.maximum if k < 10 else np.add).at(cn, cols, rs[rows])
        (np.maximum if k < 10 else np.add).at(rn, rows, cs[cols])
        cs, rs = cs / np.sqrt(cn * cs), rs / np.sqrt(rn * rs)
    assert np.array_equal(got[0], cs)
    assert np.all(np.abs(got[1] - rs) <= (demands + 3) * 2.0 ** -53 * rs)
