"""The thresholds of the snap outside the interface band (csrc/snap.cuh) against the
comparisons they stand for, on the host, for every steepness that is accepted (a reversed
profile, beta < 0, too): found at once and exact.  No GPU."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "fel-multi-phase-flow_gb300", "csrc")


def test_snap_thresholds(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    exe = tmp_path / "snap_check"
    subprocess.run([cxx, "-std=c++17", "-O2", "-ffp-contract=off", "-I", CSRC, os.path.join(HERE, "snap_check.cpp"),
                    "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=60).stdout
    assert out.strip() == "0"
