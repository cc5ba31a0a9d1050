"""FP64 batches of LPs whose vectors leave no room for a second CTA on an SM (512 threads): on both sides
of that size, with the vectors in shared and in device memory, alone and together with small LPs,
solves (the oracle's iterates) and the unrolled layer, with the tolerances (and their reasons) of
tests/test_gpu_batch_clusters.py: 1e-9 of (1 + max |reference|)."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_batch_clusters import _differs, _lengths, _lp

pytestmark = pytest.mark.gpu

ITERATIONS = 70
# (n + m + 2) doubles against 105 KB (13,440) and 219 KB (28,032) of shared memory.
BATCHES = {
    "below": lambda: [_lp(9000, _lengths(4438, 3, 7, 1), 1)],
    "above": lambda: [_lp(9002, _lengths(4438, 3, 7, 2), 2)],
    "in shared memory": lambda: [_lp(14001, _lengths(9001, 3, 7, 3), 3), _lp(97, [5] * 33, 3)],
    "in device memory": lambda: [_lp(20011, _lengths(9001, 3, 7, 4), 4), _lp(97, [5] * 33, 4),
                                 _lp(9000, _lengths(4000, 3, 7, 5), 5)],
}


@pytest.mark.parametrize("name", list(BATCHES))
def test_large_batches(engine, oracle, name):
    from oracle.unroll_oracle import UnrolledPdhg as UnrollOracle
    from samaya_gb300.batch import BatchSolver
    from samaya_gb300.diff import UnrolledPdhg
    probs = BATCHES[name]()
    for algorithm in (engine.REFERENCE, engine.HALPERN):
        s = BatchSolver.from_problems(probs, engine.PdlpOptions(
            tol=1e-30, max_iterations=ITERATIONS, algorithm=algorithm))
        res, again = s.solve(), s.solve()
        s.close()
        for lp, a, b in zip(probs, res, again):
            assert np.array_equal(a.x, b.x) and np.array_equal(a.y, b.y)
            if algorithm == engine.REFERENCE:
                ref = oracle.pdlp_solve(*lp.arrays(), tol=1e-30, max_iter=ITERATIONS)
            else:  # the step launches
                ref = engine.solve_pdlp(lp, engine.PdlpOptions(
                    tol=1e-30, max_iterations=ITERATIONS, algorithm=algorithm, autotune=False,
                    tile_nnz=512))
            assert _differs(a.x, ref.x) <= 1e-9 and _differs(a.y, ref.y) <= 1e-9
    b = BatchSolver.from_problems(probs)
    un = UnrolledPdhg(b, iterations=30, checkpoint_every=16)
    v = un.forward()
    w = np.random.default_rng(11).standard_normal(v.size)
    grads = un.adjoint(w)
    b.close()
    off = 0
    for lp in probs:
        part = slice(off, off + lp.n + lp.m)
        o = UnrollOracle(lp.m, lp.n, lp.colptr, lp.rowidx, lp.vals)
        assert _differs(v[part], o.forward(lp.cost, lp.lower, lp.upper, 30)) <= 1e-9
        for got, ref in zip(grads, o.adjoint(lp.cost, lp.lower, lp.upper, 30, w[part])):
            assert _differs(got[part], ref) <= 1e-9
        off += lp.n + lp.m
