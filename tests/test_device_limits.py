"""Limits that the CUDA runtime keeps per device are kept per device by the
engine too: a process may use several."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "rwig_b200", "csrc")


def test_shared_memory_limit_is_raised_on_each_device(tmp_path):
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    if not shutil.which("g++") or not os.path.isdir(cuda):
        pytest.skip("g++ or the CUDA headers are not available")
    exe = str(tmp_path / "context_main")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", cuda, "-o", exe,
                    os.path.join(ROOT, "tests", "cudart_stub", "context_main.cpp"),
                    "-x", "c++", os.path.join(CSRC, "context.cu")], check=True)
    run = subprocess.run([exe], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout


@pytest.mark.parametrize("name", ["sinkhorn_resident.cu", "dgemm.cuh", "ozaki.cu", "ozaki.cuh", "batch.cu"])
def test_no_process_wide_guard(name):
    """No static variable guards a cudaFuncSetAttribute call."""
    src = open(os.path.join(CSRC, name)).read()
    assert not re.search(r"\bstatic (bool|int|size_t) (attr|cache|tried)", src)
    assert "raise_smem(" in src
