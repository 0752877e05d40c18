"""Newton systems of scenes in a large batch against the same scenes alone, bit for bit: more pairs
in the batch than any size from which the pair-term kernels launch differently, with mollified
edge pairs and friction."""
import numpy as np
import pytest

from adb_gb300 import scene as S

pytestmark = pytest.mark.gpu


def touching_pairs(n, lo, hi, seed):
    rng = np.random.default_rng(seed)
    sb, ico = S.SceneBuilder(), S.icosphere_mesh(2, 0.5)
    side = int(np.ceil(np.sqrt(n)))
    for k, d in enumerate(np.geomspace(lo, hi, n)):
        at = np.array([4.0 * (k % side), 3.0, 4.0 * (k // side)])
        for j in range(2):
            sb.add(ico, at + j * d * np.array([0.8, 0.5, -0.33]), S.rotation_zyx(*rng.uniform(-1e-3, 1e-3, 3)), scene_id=k)
    return sb.build()


@pytest.mark.parametrize("n,lo,hi", [(16, 0.01, 0.1), (90, 0.03, 0.12)])
def test_system_of_a_large_batch(gpu_lib, n, lo, hi):
    from adb_gb300.abd import ABD
    sc, cfg = touching_pairs(n, lo, hi, n), S.workload_config("batched")
    q = sc.q0 + np.random.default_rng(1).uniform(-1e-4, 1e-4, sc.q0.shape)  # moved: friction
    bat = ABD(sc, cfg)
    assert len(bat.cull(1, q)[2]) > (16384 if n == 16 else 65536)
    grad, diag, keys, off = bat.newton_system(q)
    for k in (0, n // 3, n - 1):
        b0, b1 = sc.scene_ranges()[k]
        g1, d1, k1, o1 = ABD(sc.body_range(b0, b1), cfg).newton_system(q[b0:b1])
        mine = [i for i, (a, b) in enumerate(np.asarray(keys).reshape(-1, 2)) if b0 <= a < b1]
        assert np.array_equal(g1, grad.reshape(-1, 12)[b0:b1].reshape(g1.shape))
        assert np.array_equal(d1, diag[b0:b1]) and np.array_equal(o1, off[mine])
        assert len(mine) == 1 and np.abs(o1).max() > 0
