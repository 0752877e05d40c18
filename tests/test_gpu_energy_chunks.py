"""Energy totals of scenes whose number of terms lies around a half chunk (256), a chunk (512) and two:
the line-search total against the sum of the bodies' totals alone. The bodies float apart, so a
body is one term of the same sign; summing n of them rounds by at most n 2^-53 of the total."""
import numpy as np
import pytest

from adb_gb300 import scene as S

pytestmark = pytest.mark.gpu


def total(lo, hi):
    from adb_gb300.abd import ABD
    rng = np.random.default_rng(7)
    sb = S.SceneBuilder()
    for k in range(lo, hi):
        sb.add(S.cube_mesh(), (3.0 * (k % 33), 5.0, 3.0 * (k // 33)))
    sc = sb.build()
    dq = (1e-2 * rng.uniform(-1, 1, (1100, 12)))[lo:hi]
    e = ABD(sc, S.workload_config("cubes")).energy(sc.q0, dq)
    assert e["counts"].sum() == 0
    return float(e["terms"][0, 5])


@pytest.mark.parametrize("n", [1, 2, 255, 256, 257, 511, 512, 513, 768, 1024, 1025])
def test_total(gpu_lib, n):
    parts = [total(k, min(k + 100, n)) for k in range(0, n, 100)]
    assert abs(total(0, n) - sum(parts)) <= 2 * n * 2.0 ** -53 * sum(np.abs(parts))
