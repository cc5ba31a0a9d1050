"""The cluster kernels' operator layout on the CPU (tests/c/cluster_layout_driver.cpp)."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_every_nonzero_has_its_place(tmp_path):
    exe = str(tmp_path / "layout")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I",
                    os.path.join(os.path.dirname(HERE), "samaya_gb300", "csrc"),
                    os.path.join(HERE, "c", "cluster_layout_driver.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
