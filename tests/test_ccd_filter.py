"""The FP32 certificates that a trajectory has no time of impact, on the CPU: compiled from
the header the kernels use and compared with the FP64 test over sizes, distances, motions
and offsets, with lattice, planar and sliver configurations among them. A certified candidate
must have a time of impact of exactly 1; there is no tolerance."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA = "/usr/local/cuda/include"


@pytest.mark.parametrize("seed", [1, 2])
def test_certificates_hold(tmp_path, seed):
    if not shutil.which("g++") or not os.path.isdir(CUDA):
        pytest.skip("needs g++ and the CUDA headers")
    exe = str(tmp_path / "check")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", CUDA, "-o", exe,
                           os.path.join(HERE, "ccd_filter_check.cpp")])
    r = subprocess.run([exe, str(seed)], capture_output=True, text=True)
    print(r.stdout)
    assert r.returncode == 0 and "contradictions 0" in r.stdout
