"""Binning through clusters of 32 primitives (cull.cu): bodies of a few primitives, of more than the
64 from which the clusters are tested, and both mixed, so that clusters hold the ends of two
bodies. Pair sets and the step bound equal the oracle's."""
import numpy as np
import pytest

from adb_gb300 import scene as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kinds", [("cube",), ("ico1", "cube"), ("ico2", "cube", "ico1"), ("ico3", "cube"), ("torus", "cube", "ico2")])
def test_mixed_bodies(gpu_lib, oracle_lib, kinds):
    from adb_gb300.abd import ABD
    mesh = {"cube": S.cube_mesh(), "torus": S.torus_mesh(nu=17, nv=9), **{"ico%d" % k: S.icosphere_mesh(k, 0.5) for k in (1, 2, 3)}}
    rng = np.random.default_rng(len(kinds))
    sb = S.SceneBuilder()
    for k in range(18):
        sb.add(mesh[kinds[k % len(kinds)]], 0.93 * np.array([k % 3, k // 9, (k // 3) % 3]) + rng.uniform(-.03, .03, 3),
               S.random_rotation(rng))
    sc, cfg = sb.build(), S.workload_config("pile")
    gpu, orc = ABD(sc, cfg), oracle_lib.OracleSim(sc, cfg)
    o = orc.cull(1, sc.q0)
    assert len(o[0]) + len(o[2]) > 20
    for a, b in zip(gpu.cull(1, sc.q0), o):
        assert a.shape == b.shape and np.array_equal(a, b)
    dq = rng.normal(size=sc.q0.shape) * 0.02
    for a, b in zip(gpu.cull(2, sc.q0, dq), orc.cull(2, sc.q0, dq)):
        assert np.array_equal(a, b)
    assert gpu.cull(3, sc.q0, dq) == orc.cull(3, sc.q0, dq)
