"""Small LPs whose iterations run on one cluster, at the edges of that rule and of the kernel:
work 2 nnz + 5 (n + m) on both sides of 6,000, 12,000, 25,000 and 50,000 (4, 8, 16 CTAs), 24,000,
48,000 and 112,000 (lanes a row takes) and 220,000 (step launches), rows of 0 to 129 nonzeros (in
FP32 a row of 129 takes the step launches), one row, and iteration limits inside a chunk, at its end
and after a restart.

Against the oracle after a fixed number of iterations, with the tolerances (and their reasons) of
tests/test_gpu_batch_clusters.py: 1e-9 in FP64, 1e-3 for the FP32 phase of the precision switch,
of (1 + max |reference|). The Halpern iteration is checked before its first evaluation, T(z) from
zero on the problem equilibrated by the device's factors."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_batch_clusters import EDGES, _differs, _lengths, _lp

pytestmark = pytest.mark.gpu


def _near(work, side, seed):
    """A random LP of about 12 nonzeros a row with 2 nnz + 5 (n + m) just below or above work."""
    m = work // 39 + side * 10
    lp = _lp(2 * m, np.full(m, 12), seed)
    assert (2 * lp.nnz + 5 * (lp.n + lp.m) > work) == (side > 0)
    return lp


LPS = {
    "one row": lambda: _lp(3, [2], 1),
    "edges": lambda: _lp(150, EDGES, 3),
    "up to 128": lambda: _lp(150, EDGES[:-1] * 5, 4),
    "step launches": lambda: _near(220000, 1, 10),
    "few columns": lambda: _lp(40, _lengths(900, 0, 9, 11), 11),
}


for _k, _work in enumerate((6000, 12000, 24000, 25000, 48000, 50000, 112000, 220000)):
    LPS[f"below {_work}"] = lambda w=_work, k=_k: _near(w, -1, 20 + k)
    LPS[f"above {_work}"] = lambda w=_work, k=_k: _near(w, 1, 40 + k)


@pytest.mark.parametrize("name", list(LPS))
def test_chunk_matches_the_oracle(engine, oracle, name):
    lp = LPS[name]()

    def solve(iterations, **options):
        s = engine.PdlpSolver(lp, engine.PdlpOptions(
            tol=1e-30, max_iterations=iterations, autotune=False, **options))
        factors = s.equilibration()
        r, again = s.solve(), s.solve()
        assert np.array_equal(r.x, again.x) and np.array_equal(r.y, again.y)
        return r, factors

    for iterations in (1, 64, 130):
        r, _ = solve(iterations, algorithm=engine.REFERENCE)
        ref = oracle.pdlp_solve(*lp.arrays(), tol=1e-30, max_iter=iterations)
        assert _differs(r.x, ref.x) <= 1e-9 and _differs(r.y, ref.y) <= 1e-9, iterations
    for precision, bar in ((engine.FP64, 1e-9), (engine.FP32_THEN_FP64, 1e-3)):
        r, (cs, rs, _, eta) = solve(37, algorithm=engine.HALPERN, precision=precision)
        n = lp.n
        cols = np.repeat(np.arange(n), np.diff(lp.colptr))
        scale = np.concatenate([cs, 1.0 / rs])
        cost, lower, upper = lp.cost * scale, lp.lower / scale, lp.upper / scale
        bound = np.maximum(*[np.where(np.isfinite(b[n:]), np.abs(b[n:]), 0.0)
                             for b in (lower, upper)])
        cn, bn = np.linalg.norm(cost[:n]), np.linalg.norm(bound)
        omega = cn / bn if cn > 1e-10 and bn > 1e-10 else 1.0
        zv, zy = np.zeros(n + lp.m), np.zeros(lp.m)
        ref = oracle.halpern_steps(lp.m, n, lp.colptr, lp.rowidx,
                                   rs[lp.rowidx] * lp.vals * cs[cols], cost, lower, upper,
                                   eta / omega, eta * omega, 37, 0, zv, zy, zv, zy)
        assert _differs(r.x, ref["v_hat"] * scale) <= bar, precision
        assert _differs(r.y, ref["y_hat"] * rs) <= bar, precision
