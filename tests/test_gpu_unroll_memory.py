"""The unrolled layer when its checkpoints do not fit the device: the call says so, the adjoint finds no
forward pass to go back through, and the batch works on with a smaller one."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_batch_clusters import _lengths, _lp

pytestmark = pytest.mark.gpu

OUT_OF_MEMORY, NOT_READY = "out of memory", "must run before its adjoint"


def test_checkpoints_past_the_memory(engine):
    from samaya_gb300.batch import BatchSolver
    from samaya_gb300.diff import UnrolledPdhg
    lp = _lp(40, _lengths(20, 1, 6, 1), 1)
    b = BatchSolver.from_problems([lp])
    small = UnrolledPdhg(b, iterations=20, checkpoint_every=8)
    v = small.forward()
    w = np.random.default_rng(2).standard_normal(v.size)
    grads = small.adjoint(w)
    # 2^31 - 1 checkpoints of 140 doubles: 2.4 TB.
    for _ in range(2):
        with pytest.raises(Exception, match=OUT_OF_MEMORY):
            UnrolledPdhg(b, iterations=2**31 - 1, checkpoint_every=1).forward()
        with pytest.raises(Exception, match=NOT_READY):
            small.adjoint(w)
        assert np.array_equal(small.forward(), v)
        for got, ref in zip(small.adjoint(w), grads):
            assert np.array_equal(got, ref)
    b.close()
