"""The bit-level rounding of a double to a float (csrc/df64.cuh, d2f) against the
conversion, on the host.  No GPU."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "fel-multi-phase-flow_gb300", "csrc")


def test_d2f_rounds_as_the_conversion(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    exe = tmp_path / "d2f_check"
    subprocess.run([cxx, "-std=c++17", "-O2", "-ffp-contract=off", "-I", CSRC, os.path.join(HERE, "d2f_check.cpp"),
                    "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.strip() == "0"
