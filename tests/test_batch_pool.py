"""The pool of device buffers of the batch calls (batch_pool.cpp), on the CPU over a device that the
check plays: reuse, bounds, contexts, a reset after which addresses are given out again, and
a full device."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "adb_gb300", "csrc")
CUDA = "/usr/local/cuda/include"


def test_pool(tmp_path):
    if not shutil.which("g++") or not os.path.isdir(CUDA):
        pytest.skip("needs g++ and the CUDA headers")
    exe = str(tmp_path / "check")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-I", CUDA, "-o", exe, os.path.join(HERE, "batch_pool_check.cpp"),
                           os.path.join(CSRC, "batch_pool.cpp")])
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
