"""The quotient that dependencies are divided by is the IEEE division's, bit for bit (host
code, compiled here)."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="nvcc absent")
def test_quotients_are_the_divisions(tmp_path):
    csrc = os.path.join(ROOT, "graph-utils_gb300", "csrc")
    exe = tmp_path / "quotient_check"
    r = subprocess.run(["nvcc", "-std=c++17", "-O2", "-I" + csrc, "-I" + os.path.join(ROOT, "include"), "-gencode",
                        "arch=compute_103a,code=sm_103a", os.path.join(ROOT, "tests", "cpp", "quotient_check.cu"), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
