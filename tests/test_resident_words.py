"""A resident Sinkhorn solve in which any CTA's bounded wait ran out is an error
for the host, whichever CTA left first."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_outcome_of_the_words(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("g++ is not available")
    exe = str(tmp_path / "words_main")
    src = os.path.join(ROOT, "tests", "cudart_stub", "words_main.cpp")
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-o", exe, src], check=True)
    run = subprocess.run([exe], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout


def test_every_cta_reports():
    """The kernel's end goes through words_leave in every CTA, not in CTA 0 alone."""
    src = open(os.path.join(ROOT, "rwig_b200", "csrc", "sinkhorn_resident.cu")).read()
    assert "kResKerr" not in src
    assert "  if (tid == 0) {\n    if (GRAD && done && cta == 0)" in src and "words_leave(p.res, cta," in src
