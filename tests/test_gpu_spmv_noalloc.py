"""sg_spmv_noalloc at the edges of its split: empty and single rows, rows of 64 / 65 (a warp's) and
1,024 / 1,025 (the CTA's) nonzeros, rows over the ends of chunks, 16,384 and 16,385 nonzeros (one
launch and two), and average lengths from 0 to 40 (1 to 32 lanes a row).

Against numpy. A row's sum is at most 80 additions deep over terms of |a x| <= 1, at most 16,385 of
them: 80 * 2^-53 * 16,385 = 1.5e-10 at worst, a hundredth of that by its random signs and the
absolute 1e-10 allowed here."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROWS = {
    "no nonzeros": [0] * 70,
    "one": [1],
    "empty ends": [0, 0, 3, 0, 0],
    "64 and 65": [64, 65, 0, 65, 64] * 9,
    "1024 and 1025": [1024, 1, 1025, 0, 1024, 1025],
    "one row, one launch": [16384],
    "one row, two launches": [16385],
    "one launch at most": [3] * 4096 + [4096],
    "two launches at least": [3] * 4096 + [4097],
    "a row over many chunks": [1] * 300 + [9000] + [2] * 300 + [9000, 0, 0],
    "average 15": [11, 15, 19, 0, 30] * 400,
    "average 40": [40, 39, 41] * 500,
    "mixed": [0, 1, 2, 31, 32, 33, 255, 256, 257] * 30,
}


@pytest.mark.parametrize("name", list(ROWS))
def test_noalloc_spmv_splits(engine, name):
    torch = pytest.importorskip("torch")
    from samaya_gb300 import _native
    lib = _native.load()
    f = lib.sg_spmv_noalloc
    f.restype = ctypes.c_int
    f.argtypes = [ctypes.c_int, ctypes.c_longlong] + [ctypes.c_void_p] * 6
    lens = np.array(ROWS[name])
    m, n, nnz = lens.size, 17000, int(lens.sum())
    rng = np.random.default_rng(3)
    ptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    idx = rng.integers(0, n, max(nnz, 1)).astype(np.int32)
    val = rng.uniform(-1.0, 1.0, max(nnz, 1))
    x = rng.uniform(-1.0, 1.0, n)
    want = np.bincount(np.repeat(np.arange(m), lens), weights=val[:nnz] * x[idx[:nnz]],
                       minlength=m)
    d = [torch.from_numpy(a).cuda() for a in (ptr, idx, val, x)]
    got = []
    for _ in range(2):
        y = torch.full((m,), float("nan"), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        assert f(m, nnz, *[a.data_ptr() for a in d], y.data_ptr(), None) == 0
        torch.cuda.synchronize()
        got.append(y.cpu().numpy())
    assert np.max(np.abs(got[0] - want)) <= 1e-10
    assert np.array_equal(got[0], got[1])
