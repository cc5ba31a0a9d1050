"""Batches of small LPs (at most 512 rows and columns each), whose rows take several lanes: operators of
64, 65, 128 and 129 rows, rows of 0 to 40 nonzeros (32 and 33 on both sides of the warp's rows), the
largest small LP and one past it, alone and many. Solves in both storages and the unrolled layer
against the oracles, with the tolerances (and their reasons) of tests/test_gpu_batch_clusters.py: 1e-9
in FP64 and 1e-3 in FP32, of (1 + max |reference|), after 100 iterations."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_batch_clusters import ITERATIONS, _differs, _lp

pytestmark = pytest.mark.gpu


def _mixed(m, n, seed):
    """Rows of 0 to 40 nonzeros, 31 to 34 among them."""
    rng = np.random.default_rng(seed)
    lengths = rng.integers(0, min(n, 12) + 1, m)
    some = [k for k in (0, 1, 3, 4, 5, 31, 32, 33, 34, 40) if k <= n]
    at = rng.permutation(m)[:len(some)]
    lengths[at] = some[:at.size]
    return _lp(n, lengths, seed)


BATCHES = {
    "64 and 65 rows": lambda: [_mixed(64, 129, 1), _mixed(65, 128, 2)],
    "128 and 129 rows": lambda: [_mixed(128, 64, 3), _mixed(129, 65, 4)],
    "one to nine rows": lambda: [_mixed(m, 40, 10 + m) for m in range(1, 10)],
    "long rows": lambda: [_lp(90, [40] * 30, 5), _lp(90, [33, 32] * 9, 6)],
    "no nonzeros": lambda: [_lp(7, [0, 0, 0], 7), _mixed(20, 30, 8)],
    "512": lambda: [_mixed(180, 332, 9)],
    "513": lambda: [_mixed(181, 332, 9), _mixed(40, 60, 10)],
    "many": lambda: [_mixed(20 + k % 60, 50 + k % 90, 100 + k) for k in range(330)],
}


@pytest.mark.parametrize("name", list(BATCHES))
def test_small_batches(engine, oracle, name):
    from samaya_gb300.batch import BatchSolver
    probs = BATCHES[name]()
    refs = [oracle.pdlp_solve(*lp.arrays(), tol=1e-30, max_iter=ITERATIONS) for lp in probs]
    for precision, bar in ((engine.FP64, 1e-9), (engine.FP32_REFINED, 1e-3)):
        for algorithm in (engine.REFERENCE, engine.HALPERN):
            s = BatchSolver.from_problems(probs, engine.PdlpOptions(
                tol=1e-30, max_iterations=ITERATIONS, precision=precision, algorithm=algorithm))
            res, again = s.solve(), s.solve()
            s.close()
            for k, (a, b) in enumerate(zip(res, again)):
                assert np.array_equal(a.x, b.x) and np.array_equal(a.y, b.y)
                if algorithm == engine.REFERENCE:
                    assert _differs(a.x, refs[k].x) <= bar, (k, precision)
                    assert _differs(a.y, refs[k].y) <= bar, (k, precision)
            if algorithm == engine.HALPERN and precision == engine.FP64:
                # The step launches (tile_nnz): no code of the clusters'.
                for lp, a in list(zip(probs, res))[:4]:
                    ref = engine.solve_pdlp(lp, engine.PdlpOptions(
                        tol=1e-30, max_iterations=ITERATIONS, algorithm=engine.HALPERN,
                        autotune=False, tile_nnz=256))
                    assert _differs(a.x, ref.x) <= bar and _differs(a.y, ref.y) <= bar


@pytest.mark.parametrize("name", [k for k in BATCHES if k != "many"])
@pytest.mark.parametrize("copies", [1, 160])
def test_small_unrolled(engine, name, copies):
    """Also with more CTAs than SMs, where the adjoint has a kernel of its own: the iterate and the
    gradients."""
    from oracle.unroll_oracle import UnrolledPdhg as UnrollOracle
    from samaya_gb300.batch import BatchSolver
    from samaya_gb300.diff import UnrolledPdhg
    probs = [lp for lp in BATCHES[name]() if lp.m > 9] or BATCHES[name]()[-1:]
    if copies > 1:
        probs = probs[:1]
    iterations = 40
    b = BatchSolver.from_problems(probs * copies)
    un = UnrolledPdhg(b, iterations=iterations, checkpoint_every=16)
    v = un.forward()
    total = sum(lp.n + lp.m for lp in probs)
    w = np.random.default_rng(11).standard_normal(total)
    grads = un.adjoint(np.tile(w, copies))
    b.close()
    off = 0
    for lp in probs:
        part = slice(off, off + lp.n + lp.m)
        o = UnrollOracle(lp.m, lp.n, lp.colptr, lp.rowidx, lp.vals)
        ref_v = o.forward(lp.cost, lp.lower, lp.upper, iterations)
        refs = o.adjoint(lp.cost, lp.lower, lp.upper, iterations, w[part])
        for copy in range(copies):
            at = slice(copy * total + part.start, copy * total + part.stop)
            assert _differs(v[at], ref_v) <= 1e-9
            for got, ref in zip(grads, refs):
                assert _differs(got[at], ref) <= 1e-9
        off += lp.n + lp.m
