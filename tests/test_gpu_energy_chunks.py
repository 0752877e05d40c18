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


@pytest.mark.parametrize("n", [1, 2, 127, 128, 129])
def test_scenes(gpu_lib, n):
    """Totals of n scenes in one handle (their ranges found in one launch up to 128) against the same
    scenes alone, bit for bit; a scene's lists are empty, of one overlap or of several."""
    from adb_gb300.abd import ABD
    rng = np.random.default_rng(n)
    sb = S.SceneBuilder()
    for k in range(n):
        for j in range(1 + k % 3):
            sb.add(S.cube_mesh(), (4.0 * (k % 12), 0.5 + S.GROUND_SHIFT + 0.01 + 1.015 * j, 4.0 * (k // 12)), scene_id=k)
    sc, cfg = sb.build(), S.workload_config("cubes")
    dq = 1e-3 * rng.uniform(-1, 1, sc.q0.shape)
    e = ABD(sc, cfg).energy(sc.q0, dq)["terms"]
    for k in sorted({0, n // 2, n - 1}):
        b0, b1 = sc.scene_ranges()[k]
        alone = ABD(sc.body_range(b0, b1), cfg).energy(sc.q0[b0:b1], dq[b0:b1])["terms"]
        assert e[k, 5] != 0 and np.array_equal(alone[0], e[k])
