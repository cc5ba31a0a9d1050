"""Small LPs on the two sides of the choice between one cluster (chunk_kernel) and the step launches,
which share no step code: a caller who asks for a shape of the step launches (here tile_nnz) gets
them. The cluster's iterations, the batch's (the cluster's steps, one LP to a cluster) and the step
launches end at the same points past restarts; the rows that a solve leaves out of the step launches
change no bit of them; and an LP with one long row takes them by itself.

Tolerances, of (1 + max |value|): test_gpu_batch_clusters.py's 2e-10 for 100 iterations in FP64, times
4 for 400 and times 10 for primal weights that restarts move (they come from the iterates), 8e-9: 1e-8.
FP32, whose sums keep the step launches' order, 100 iterations without a restart's weight: 1e-3."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_batch_clusters import EDGES, _differs, _lengths, _lp
from test_gpu_inert_rows import _inert, _with_empty_rows

pytestmark = pytest.mark.gpu

LPS = {
    "edges": lambda: _lp(150, EDGES * 2, 3),
    "random": lambda: _lp(700, _lengths(300, 5, 20, 3), 3),
    "few columns": lambda: _lp(40, _lengths(400, 0, 9, 11), 11),
}


def _solve(engine, lp, iterations, **options):
    r = engine.solve_pdlp(lp, engine.PdlpOptions(tol=1e-30, inner_tol=1e-30, autotune=False,
                                                 max_iterations=iterations, **options))
    assert r.iterations == iterations
    return r


def _on_steps(r):
    return r.kernel_launches >= 2 * r.iterations


@pytest.mark.parametrize("name", list(LPS))
@pytest.mark.parametrize("algorithm", ["REFERENCE", "ENHANCED", "HALPERN"])
def test_cluster_batch_and_step_launches_agree_past_restarts(engine, name, algorithm):
    from samaya_gb300.batch import BatchSolver
    lp = LPS[name]()
    algorithm = getattr(engine, algorithm)
    # (The batch restarts the enhanced PDHG at 0.36, a single LP's solve at 0.1.)
    forced = 0.36 if algorithm == engine.ENHANCED else 0.0
    on_cluster = _solve(engine, lp, 400, algorithm=algorithm, artificial_restart=forced)
    on_steps = _solve(engine, lp, 400, algorithm=algorithm, artificial_restart=forced,
                      tile_nnz=512)
    assert not _on_steps(on_cluster) and _on_steps(on_steps)
    assert on_cluster.restarts == on_steps.restarts > 0
    s = BatchSolver.from_problems([lp], engine.PdlpOptions(tol=1e-30, max_iterations=400,
                                                           algorithm=algorithm))
    in_batch = s.solve()[0]
    s.close()
    for r in (on_cluster, in_batch):
        assert _differs(r.x, on_steps.x) <= 1e-8 and _differs(r.y, on_steps.y) <= 1e-8


@pytest.mark.parametrize("option", ["tile_nnz", "tile_split", "row_groups", "segment_staging"])
def test_asked_shapes_run(engine, option):
    lp = LPS["random"]()
    value = {"tile_nnz": 1024, "tile_split": 64}.get(option, 1)
    for precision, bar in (("FP64", 1e-8), ("FP32_THEN_FP64", 1e-3)):
        options = dict(precision=getattr(engine, precision), algorithm=engine.HALPERN)
        r = _solve(engine, lp, 100, **{option: value}, **options)
        assert _on_steps(r), precision
        ref = _solve(engine, lp, 100, **options)
        assert not _on_steps(ref), precision
        assert _differs(r.x, ref.x) <= bar and _differs(r.y, ref.y) <= bar, precision


@pytest.mark.parametrize("algorithm,precision", [("REFERENCE", "FP64"), ("HALPERN", "FP64"),
                                                 ("HALPERN", "FP32_THEN_FP64")])
def test_inert_rows_left_out_of_the_step_launches(engine, algorithm, precision):
    from samaya_gb300 import generators as g
    from samaya_gb300.problem import make_problem
    for base in (g.random_sparse_lp(300, 800, seed=5), g.transportation_lp(30, 60, seed=2)):
        model = _with_empty_rows(base, seed=1)
        lp, _ = make_problem(model)
        out = []
        for keep in (False, True):
            options = engine.PdlpOptions(
                tol=1e-30, inner_tol=1e-30, max_iterations=300, autotune=False, tile_nnz=256,
                keep_inert_rows=keep, algorithm=getattr(engine, algorithm),
                precision=getattr(engine, precision))
            with engine.PdlpSolver(lp, options) as s:
                rows, _, _, _ = s.step_rows()
                assert rows == lp.m - (0 if keep else _inert(model))
                out.append(s.solve())
            assert _on_steps(out[-1])
        a, b = out
        assert np.array_equal(a.x, b.x) and np.array_equal(a.y, b.y)


@pytest.mark.parametrize("longest,on_steps", [(4141, False), (4142, True), (5000, True)])
def test_one_long_row(engine, oracle, longest, on_steps):
    """A row is a warp's chain on the cluster; step launches split it."""
    lp = _lp(5000, [longest] + [6] * 200, longest)
    assert (2 * lp.nnz + 5 * (lp.n + lp.m) + 66 * longest > 310000) == on_steps
    r = _solve(engine, lp, 100, algorithm=engine.REFERENCE)
    assert _on_steps(r) == on_steps
    ref = oracle.pdlp_solve(*lp.arrays(), tol=1e-30, max_iter=100)
    assert _differs(r.x, ref.x) <= 1e-8 and _differs(r.y, ref.y) <= 1e-8


@pytest.mark.parametrize("m,n,on_steps", [(5400, 12000, False), (5900, 13400, True)])
def test_fp32_limit(engine, m, n, on_steps):
    """2 nnz + 8 (n + m) below and above 300,000: the same iterations on both sides."""
    rng = np.random.default_rng(m)
    lp = _lp(n, rng.multinomial(6 * n, np.full(m, 1.0 / m)), m)
    assert (2 * lp.nnz + 8 * (lp.n + lp.m) > 300000) == on_steps
    options = dict(precision=engine.FP32_THEN_FP64, algorithm=engine.HALPERN)
    r = _solve(engine, lp, 100, **options)
    assert _on_steps(r) == on_steps
    ref = _solve(engine, lp, 100, tile_nnz=512, **options)
    assert _differs(r.x, ref.x) <= 1e-3 and _differs(r.y, ref.y) <= 1e-3
