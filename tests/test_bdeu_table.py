"""The library's fixed-point lgamma table, sums of logarithms in pairs of
doubles (bdeu_table_into, eddy_host.cpp), against lgammal: every entry is
the nearest step, or within a hundredth of a step of being so.  That is
looser than its own error (n 2^-58 against a step of 2^-44 to 2^-31) and
covers lgammal's of an 80-bit long double (a few 2^-64 of values up to 2^20).
CPU only."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(ROOT, "eddy-gpu_gb300", "csrc")


def test_table_entries_are_the_nearest_steps(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "bdeu_table")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(ROOT, "include"),
                    "-I", CSRC, os.path.join(HERE, "bdeu_table_main.cpp"),
                    os.path.join(CSRC, "eddy_host.cpp"), "-o", exe], check=True)
    counts = [1, 2, 3, 17, 60, 301, 1000, 4096, 20000]
    r = subprocess.run([exe] + [str(n) for n in counts], capture_output=True, text=True, check=True)
    worst = [float(x) for x in r.stdout.split()]
    assert len(worst) == len(counts)
    assert max(worst) <= 0.51, dict(zip(counts, worst))
