"""Batch calls after a cudaDeviceReset, as a program that ends its context between two uses makes
them: in a process of their own, the same results before and after."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CODE = """
import numpy as np
from adb_gb300 import _lib, abdtk
x = np.random.default_rng(0).normal(size=(300, 4, 3)) * 0.02
def calls():
    t, d = abdtk.ee_distance_batch(x)
    return [t, d] + [np.asarray(a) for a in abdtk.ipc_hess_ee_batch(x)]
want = calls()
for _ in range(3):
    calls()
    assert _lib.lib().cudaDeviceReset() == 0
    for n in (1, 300):
        abdtk.ipc_hess_pt_batch(x[:n])
    assert all(np.array_equal(a, b) for a, b in zip(calls(), want))
print("equal")
"""


def test_after_a_reset(gpu_lib):
    r = subprocess.run([sys.executable, "-c", CODE], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "equal" in r.stdout, r.stderr
