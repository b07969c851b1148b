"""The list scan's plan (mestrado_gb300/csrc/list_plan.cuh) on list lengths up to 2^31 - 1, against a restatement in
64 bits (host build, CPU): a query over more than 2^30 rows must not take more rows of a list in its first pass than
the record between the passes holds."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_plan(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    exe = str(tmp_path / "lp_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-Wall", "-I", os.path.join(ROOT, "mestrado_gb300", "csrc"), "-o", exe,
                    os.path.join(ROOT, "tests", "native", "lp_check.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    print(r.stdout)
    assert r.returncode == 0, r.stdout
