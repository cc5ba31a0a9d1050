"""Where the device cannot hold a cluster (a process that owns a slice of the GPU; here
SG_MAX_CLUSTER, which caps the size the device is asked for), small LPs take the step launches and
batches smaller clusters, down to a CTA per LP, with the answers of the clusters.

Tolerances (and their reasons) of tests/test_gpu_batch_clusters.py: the same iterations with sums in
another order, 1e-9 in FP64 and 1e-3 in FP32, of (1 + max |value|)."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_batch_clusters import _differs, _lengths, _lp

pytestmark = pytest.mark.gpu

ITERATIONS = 100


@pytest.mark.parametrize("precision,bar", [("FP64", 1e-9), ("FP32_THEN_FP64", 1e-3)])
@pytest.mark.parametrize("algorithm", ["REFERENCE", "HALPERN"])
def test_small_lp_without_a_cluster_takes_the_step_launches(engine, monkeypatch, precision, bar,
                                                            algorithm):
    lp = _lp(700, _lengths(300, 5, 20, 3), 3)

    def solve():
        return engine.solve_pdlp(lp, engine.PdlpOptions(
            tol=1e-30, inner_tol=1e-30, max_iterations=ITERATIONS, autotune=False,
            precision=getattr(engine, precision), algorithm=getattr(engine, algorithm)))

    on_cluster = solve()
    assert on_cluster.kernel_launches < ITERATIONS
    for most in ("1", "2"):
        monkeypatch.setenv("SG_MAX_CLUSTER", most)
        r = solve()
        assert r.kernel_launches >= 2 * ITERATIONS, most
        assert r.iterations == on_cluster.iterations == ITERATIONS
        assert _differs(r.x, on_cluster.x) <= bar and _differs(r.y, on_cluster.y) <= bar, most


@pytest.mark.parametrize("most", ["1", "2", "4"])
def test_batches_take_smaller_clusters(engine, monkeypatch, most):
    from samaya_gb300.batch import BatchSolver
    from samaya_gb300.diff import UnrolledPdhg
    probs = [_lp(1200, _lengths(500, 10, 20, k), k) for k in range(3)]

    def outputs():
        out = []
        for precision in (engine.FP64, engine.FP32_REFINED):
            s = BatchSolver.from_problems(probs, engine.PdlpOptions(
                tol=1e-30, max_iterations=ITERATIONS, precision=precision))
            out.append(np.concatenate([np.concatenate([r.x, r.y]) for r in s.solve()]))
            s.close()
        b = BatchSolver.from_problems(probs)
        un = UnrolledPdhg(b, iterations=ITERATIONS, checkpoint_every=48)
        v = un.forward()
        out += [v, *un.adjoint(np.random.default_rng(5).standard_normal(v.size))]
        b.close()
        return out

    refs = outputs()
    monkeypatch.setenv("SG_MAX_CLUSTER", most)
    for k, (got, ref) in enumerate(zip(outputs(), refs)):
        assert _differs(got, ref) <= (1e-3 if k == 1 else 1e-9), k
