"""A bounded wait that gives up in one CTA of a cluster, in the batched kernels' own sources on the
CPU: their control flow runs with a host thread per CTA (tests/c/cluster_failure_driver.cpp), and in
every case all CTAs must pass the same cluster barriers, none may store into the shared memory of
one that has ended, and the failure must be reported. (Nothing makes a wait fail on a GPU.)"""
from __future__ import annotations

import os
import re
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "samaya_gb300", "csrc")


def _text(name):
    with open(os.path.join(CSRC, name)) as f:
        return f.read()


def _cut(text, marker):
    """The text before the marker (the launches), its namespaces closed."""
    assert text.count(marker) == 1, marker
    return text[:text.index(marker)]


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_every_cta_leaves_together(tmp_path):
    files = {
        "sg_cluster_steps.cuh": _text("sg_cluster_steps.cuh"),
        "sg_batch.cuh": re.sub(r"#include [<\"](cuda_runtime|sg_common).*", "",
                               _text("sg_batch.cuh")),
        "sg_batch_device.cuh": _cut(_text("sg_batch_device.cuh"),
                                    "// The configuration of a launch") + "}\n}\n",
        "sg_batch.cu": _cut(_text("sg_batch.cu"),
                            "__global__ void batch_deadline_kernel") + "}\n",
        "sg_batch_solve.cuh": _cut(_text("sg_batch_solve.cuh"),
                                   "// go() with the kernel of a mode and") + "}\n",
        "sg_batch_unroll.cu": _cut(_text("sg_batch_unroll.cu"),
                                   "namespace {\n\n// go() with the kernel of a mode") + "}\n",
    }
    # The barrier that carries a failure is the kernels' own.
    stopped = re.search(r"__device__ __forceinline__ bool cluster_stopped\(.*?\n}\n",
                        _text("sg_cluster.cuh"), re.S)
    with open(os.path.join(HERE, "c", "emulated_cluster.cuh")) as f:
        files["sg_cluster.cuh"] = f.read().replace("// CLUSTER_STOPPED",
                                                   stopped.group(0) if stopped else "")
    for name, text in files.items():
        # A thread is a CTA: the thread that stores to CTA q stores to all.
        text = text.replace("if (threadIdx.x < size && sh.fail != 0) {\n"
                            "    st_cluster(map_rank(shared_addr(&sh.stop), threadIdx.x), 1u);",
                            "for (unsigned q = 0; q < size && sh.fail != 0; ++q) {\n"
                            "    st_cluster(map_rank(shared_addr(&sh.stop), q), 1u);")
        (tmp_path / name).write_text(text)
    for name in ("cluster_failure_driver.cpp", "emulated_device.h"):
        shutil.copy(os.path.join(HERE, "c", name), tmp_path)
    exe = str(tmp_path / "driver")
    subprocess.run(["g++", "-std=c++20", "-O1", "-w", "-pthread", "-I", str(tmp_path),
                    str(tmp_path / "cluster_failure_driver.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
