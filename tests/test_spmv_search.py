"""sg_spmv_noalloc's search of the row starts up to 2^31 - 1 rows, its source on the CPU
(tests/c/spmv_search_driver.cpp)."""
from __future__ import annotations

import os
import re
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_search_of_many_rows(tmp_path):
    with open(os.path.join(os.path.dirname(HERE), "samaya_gb300", "csrc", "sg_noalloc.cu")) as f:
        search = re.search(r"__device__ __forceinline__ int lower_bound_ptr\(.*?\n}\n", f.read(),
                           re.S).group(0)
    with open(os.path.join(HERE, "c", "spmv_search_driver.cpp")) as f:
        (tmp_path / "driver.cpp").write_text(f.read().replace("// SEARCH", search))
    exe = str(tmp_path / "driver")
    subprocess.run(["g++", "-std=c++20", "-O1", "-fwrapv", "-pthread", str(tmp_path / "driver.cpp"),
                    "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    if r.returncode == 2:
        pytest.skip("no address space for 2^31 row starts")
    assert r.returncode == 0, (r.returncode, r.stdout)
