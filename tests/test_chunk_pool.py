"""The pool that holds the sets' kept outputs (eddy_pool.h): page-locked up to
a bound, ordinary memory past it, what a call takes for itself given back.
CPU only, over a counting allocator."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "eddy-gpu_gb300", "csrc")


def test_pool_of_kept_outputs(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "chunk_pool")
    subprocess.run(["g++", "-O1", "-g", "-std=c++17", "-Wall", "-Werror", "-I", CSRC,
                    os.path.join(HERE, "chunk_pool_main.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, check=True).stdout.splitlines()
    assert len(out) == 12 and all(line.startswith("ok ") for line in out), out
