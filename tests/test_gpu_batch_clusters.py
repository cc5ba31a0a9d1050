"""The batch's cluster kernels at the edges of their layout: rows of 0 to 129 nonzeros (slices of
32 rows and of 8, partly filled ones, rows of more than 32 on warps), clusters of 1 to 16 CTAs,
and state and gathered vectors in shared or in device memory, also in one batch.

Every LP runs a fixed number of iterations, past one evaluation and restart. Tolerances, of
(1 + max |reference|): the PDHG map is nonexpansive, so an iteration's rounding errors (at most
about 130 products and 10 operations a row) add up over 100 iterations and the scales' quotients
(up to 1e2) to 100 * 140 * 1e2 * 2^-53 = 2e-10 in FP64: 1e-9. In FP32 the same count with the
errors' random signs, sqrt(100 * 140) * 1e1 * 2^-24 = 7e-5, once more for the rounded data and the
step sizes that follow from them: 1e-3. The Halpern iteration is compared with the single-LP engine
(other kernels), FP64."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ITERATIONS = 100
EDGES = [0, 1, 2, 3, 4, 5, 8, 31, 32, 33, 63, 64, 65, 128, 129]


def _lp(n, lengths, seed):
    """A feasible LP with rows of the given numbers of nonzeros: equality, one-sided and free
    rows around the product with a point inside the columns' bounds."""
    from samaya_gb300.model import LpProblem
    rng = np.random.default_rng(seed)
    m = len(lengths)
    cols = np.concatenate([np.sort(rng.permutation(n)[:k]) for k in lengths] +
                          [np.zeros(0)]).astype(np.int64)
    rows = np.repeat(np.arange(m), lengths)
    vals = rng.uniform(0.5, 2.0, cols.size) * rng.choice([-1.0, 1.0], cols.size)
    by_col = np.lexsort((rows, cols))
    colptr = np.concatenate([[0], np.cumsum(np.bincount(cols, minlength=n))])
    x = rng.uniform(0.0, 3.0, n)
    ax = np.zeros(m)
    np.add.at(ax, rows, vals * x[cols])
    kind = rng.integers(0, 4, m)
    lower = np.concatenate([np.zeros(n), np.where(kind <= 1, ax, -np.inf)])
    upper = np.concatenate([np.full(n, 4.0), np.where((kind == 0) | (kind == 2), ax, np.inf)])
    cost = np.concatenate([rng.uniform(-1.0, 1.0, n), np.zeros(m)])
    return LpProblem(m, n, colptr, rows[by_col], vals[by_col], cost, lower, upper)


def _lengths(m, least, most, seed):
    return np.random.default_rng(seed).integers(least, most + 1, m)


# 16 CTAs and 8 for a single LP and few, 1 for many; 15,000 + 9,000 vector entries in shared memory
# without the state in FP64; 40,000 + 17,000 in device memory in both types.
BATCHES = {
    "one row": lambda: [_lp(1, [1], 1)],
    "no rows": lambda: [_lp(5, [], 2), _lp(40, _lengths(9, 0, 5, 2), 2)],
    "long rows": lambda: [_lp(150, EDGES, 3), _lp(150, EDGES * 7, 4)],
    "partial slices": lambda: [_lp(97, _lengths(33, 0, 6, 5), 5), _lp(31, _lengths(65, 0, 6, 6), 6)],
    "many": lambda: [_lp(60 + k, _lengths(20 + k % 50, 0, 5, k), k) for k in range(400)],
    "one large": lambda: [_lp(3000, _lengths(1500, 4, 20, 7), 7)],
    "some": lambda: [_lp(1200, _lengths(500, 10, 20, k), k) for k in range(40)],
    "every memory": lambda: [_lp(97, _lengths(33, 0, 6, 8), 8),
                             _lp(15000, _lengths(9000, 3, 7, 9), 9),
                             _lp(40000, _lengths(17000, 3, 7, 10), 10)],
}


def _differs(a, b):
    return np.max(np.abs(a - b), initial=0.0) / (1.0 + np.max(np.abs(b), initial=0.0))


@pytest.mark.parametrize("name", list(BATCHES))
def test_cluster_kernels_at_their_edges(engine, oracle, name):
    from oracle.unroll_oracle import UnrolledPdhg as UnrollOracle
    from samaya_gb300.batch import BatchSolver
    from samaya_gb300.diff import UnrolledPdhg
    probs = BATCHES[name]()

    def solve(**options):
        s = BatchSolver.from_problems(probs, engine.PdlpOptions(
            tol=1e-30, max_iterations=ITERATIONS, **options))
        res, again = s.solve(), s.solve()
        s.close()
        for a, b in zip(res, again):
            assert np.array_equal(a.x, b.x) and np.array_equal(a.y, b.y)
        return res

    refs = [oracle.pdlp_solve(*lp.arrays(), tol=1e-30, max_iter=ITERATIONS) for lp in probs]
    for precision, bar in ((engine.FP64, 1e-9), (engine.FP32_REFINED, 1e-3)):
        for k, (r, ref) in enumerate(zip(
                solve(algorithm=engine.REFERENCE, precision=precision), refs)):
            assert _differs(r.x, ref.x) <= bar and _differs(r.y, ref.y) <= bar, (k, precision)
    few = probs[:3]
    for k, (lp, r) in enumerate(zip(few, solve(algorithm=engine.HALPERN))):
        ref = engine.solve_pdlp(lp, engine.PdlpOptions(
            tol=1e-30, max_iterations=ITERATIONS, algorithm=engine.HALPERN, autotune=False))
        assert _differs(r.x, ref.x) <= 1e-9 and _differs(r.y, ref.y) <= 1e-9, k
    # (A converged LP's projections meet their bounds within rounding errors, and then either
    # bound's gradient is right.)
    if min(lp.m for lp in probs) <= 1:
        return
    b = BatchSolver.from_problems(few)
    un = UnrolledPdhg(b, iterations=ITERATIONS, checkpoint_every=48)
    v = un.forward()
    w = np.random.default_rng(11).standard_normal(v.size)
    grads = un.adjoint(w)
    b.close()
    off = 0
    for k, lp in enumerate(few):
        part = slice(off, off + lp.n + lp.m)
        o = UnrollOracle(lp.m, lp.n, lp.colptr, lp.rowidx, lp.vals)
        assert _differs(v[part], o.forward(lp.cost, lp.lower, lp.upper, ITERATIONS)) <= 1e-9, k
        for got, ref in zip(grads, o.adjoint(lp.cost, lp.lower, lp.upper, ITERATIONS, w[part])):
            assert _differs(got[part], ref) <= 1e-9, k
        off += lp.n + lp.m


@pytest.mark.parametrize("count", [1, 152, 153])
def test_adjoint_with_an_sm_to_a_cta_and_with_two_ctas_to_one(engine, count):
    """Up to one small LP per SM, and one more: the adjoint has a kernel for each. Every copy's
    gradients against the oracle's, to 1e-9 as above."""
    from oracle.unroll_oracle import UnrolledPdhg as UnrollOracle
    from samaya_gb300.batch import BatchSolver
    from samaya_gb300.diff import UnrolledPdhg
    lp = _lp(40, [5, 1, 7, 40, 3] * 4, 9)
    b = BatchSolver.from_problems([lp] * count)
    un = UnrolledPdhg(b, iterations=30, checkpoint_every=16)
    un.forward()
    w = np.random.default_rng(12).standard_normal(lp.n + lp.m)
    grads = un.adjoint(np.tile(w, count))
    b.close()
    o = UnrollOracle(lp.m, lp.n, lp.colptr, lp.rowidx, lp.vals)
    for got, ref in zip(grads, o.adjoint(lp.cost, lp.lower, lp.upper, 30, w)):
        for part in np.split(got, count):
            assert _differs(part, ref) <= 1e-9
