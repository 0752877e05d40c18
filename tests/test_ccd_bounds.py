"""Error bounds of the FP32 vectors that the trajectory certificates and the FP32 root
verification are proved from, on the CPU: compiled from the header the kernels use, at the
values where the roundings are largest. A bound has no tolerance."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA = "/usr/local/cuda/include"


@pytest.mark.parametrize("seed", [1, 2])
def test_bounds_hold(tmp_path, seed):
    if not shutil.which("g++") or not os.path.isdir(CUDA):
        pytest.skip("needs g++ and the CUDA headers")
    exe = str(tmp_path / "check")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", CUDA, "-o", exe,
                           os.path.join(HERE, "ccd_bounds_check.cpp")])
    r = subprocess.run([exe, str(seed)], capture_output=True, text=True)
    print(r.stdout)
    assert r.returncode == 0
