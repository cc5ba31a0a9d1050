"""The tuner's cache: its choice for an operator holds for the iteration it was timed in, both
operators' rows and the algorithm's step kernels, and lines of the file's earlier format (shapes timed
for one step alone) are not taken."""
from __future__ import annotations

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SCRIPT = """
import sys
sys.path.insert(0, {root!r})
import numpy as np
import samaya_gb300 as sg
from samaya_gb300.model import LpProblem
m, n = 4000, 40000


def lp(columns):
    # Rows of 70 nonzeros, the same for every call; the columns' lengths differ.
    cols = columns.reshape(m, 70)
    rows = np.repeat(np.arange(m), 70)
    order = np.lexsort((rows, cols.ravel()))
    colptr = np.concatenate([[0], np.cumsum(np.bincount(cols.ravel(), minlength=n))])
    return LpProblem(m, n, colptr, rows[order], np.ones(rows.size), np.ones(n + m),
                     np.zeros(n + m), np.concatenate([np.ones(n), np.full(m, 70.0)]))


even = lp((np.arange(m * 70) * 7) % n)
uneven = lp(np.concatenate([np.arange(70 * m - n) % (n // 5), np.arange(n)])[:70 * m])
for p, algorithm in ((even, sg.HALPERN), (even, sg.ENHANCED), (uneven, sg.HALPERN)):
    with sg.PdlpSolver(p, sg.PdlpOptions(algorithm=algorithm)) as s:
        print(s.tile_shapes())
"""


def _run(path):
    r = subprocess.run([sys.executable, "-c", SCRIPT.format(root=ROOT)],
                       env=dict(os.environ, SG_TILE_CACHE=str(path)), capture_output=True,
                       text=True, timeout=600)
    assert r.returncode == 0, r.stderr
    return r.stdout


def test_choices_are_kept_by_iteration(tmp_path):
    path = tmp_path / "tiles.txt"
    # A line of the earlier format for the rows of both LPs: a capacity that no candidate has.
    old = "4000 280000 70 4000 0 0 0 0 0 16384 256 128 0 0 0 0"
    path.write_text(old + "\n")
    out = _run(path)
    lines = path.read_text().splitlines()
    assert lines[0] == old and len(lines) == 7
    assert len({tuple(x.split()[:9]) for x in lines[1:]}) == 6
    assert _run(path) == out
    assert path.read_text().splitlines() == lines
