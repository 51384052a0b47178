"""A wait between the CTAs of a two-sided Jacobi that runs out makes the solve an error,
in whichever CTA it is: in the last round of a sweep only that one knows. The rule
(tree-embedding_gb300/csrc/jacobi_sched.h) is host/device code; this compiles it for the
host and goes through every set of CTAs."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "tree-embedding_gb300", "csrc")


def test_a_wait_that_ran_out_is_reported(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    exe = str(tmp_path / "jacobi_report_check")
    subprocess.run([cxx, "-O1", "-std=c++17", "-I", CSRC,
                    os.path.join(HERE, "native", "jacobi_report_check.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout + out.stderr
    assert "mismatches 0" in out.stdout
