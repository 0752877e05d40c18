"""Candidate lists of the pair cull (cull.cu): overlaps whose candidates for the FP64 test are none, a
few, around the shared-memory sort's 2048 and more, and so many of them that the staging buffer
grows and the cull repeats. Sets, order and distance types equal the oracle's."""
import numpy as np
import pytest

from adb_gb300 import scene as S


def touching(pairs, lo, hi):
    """2 * pairs spheres, pairs apart from each other; the two of a pair almost coincide, shifted
    by lo .. hi (geometrically)."""
    sc = S.sphere_pile(2 * pairs, 1, 1, subdiv=2, jitter=0.0, vel_sigma=0.0, seed=3)
    q = sc.q0.copy()
    q[1::2, :3] = q[::2, :3] + np.array([0.8, 0.5, -0.33]) * np.geomspace(lo, hi, pairs)[:, None]
    return sc, q


@pytest.mark.gpu
@pytest.mark.parametrize("pairs,lo,hi", [(1, 2.0, 2.0), (24, 0.005, 1.2), (100, 0.06, 0.12)])
def test_lists(gpu_lib, oracle_lib, pairs, lo, hi):
    from adb_gb300.abd import ABD
    sc, q = touching(pairs, lo, hi)
    cfg = S.workload_config("pile")
    gpu, orc = ABD(sc, cfg), oracle_lib.OracleSim(sc, cfg)
    o = orc.cull(1, q)
    for _ in range(2):  # the second cull starts with the staging the first one grew
        for a, b in zip(gpu.cull(1, q), o):
            assert a.shape == b.shape and np.array_equal(a, b)
    n = np.bincount(np.concatenate([o[0][:, 0], o[2][:, 0]]).astype(int) // 2, minlength=pairs)
    assert (pairs == 1) == (n.sum() == 0)
    if pairs == 24:
        assert n.max() > 2048 and n.min() < 200
    if pairs == 100:
        assert n[n < 1700].sum() > 65536


@pytest.mark.gpu
@pytest.mark.parametrize("subdiv,shift", [(0, 0.3), (1, 0.01), (1, 0.2), (1, 0.9)])
def test_short_lists(gpu_lib, oracle_lib, subdiv, shift):
    """Lists that are staged together: of few box hits, and of more than the queue of hits holds."""
    from adb_gb300.abd import ABD
    sb, rng = S.SceneBuilder(), np.random.default_rng(4)
    for k in range(12):
        sb.add(S.icosphere_mesh(subdiv, 0.5), np.array([3.0 * (k // 2), 2.0, 0.0]) + (k % 2) * shift * np.array([0.8, 0.5, -0.33]),
               S.rotation_zyx(*rng.uniform(-1e-2, 1e-2, 3)))
    sc, cfg = sb.build(), S.workload_config("pile")
    gpu, orc = ABD(sc, cfg), oracle_lib.OracleSim(sc, cfg)
    dq = rng.normal(size=sc.q0.shape) * 0.01
    for args in ((1, sc.q0), (2, sc.q0, dq)):
        for a, b in zip(gpu.cull(*args), orc.cull(*args)):
            assert a.shape == b.shape and np.array_equal(a, b)
    assert gpu.cull(3, sc.q0, dq) == orc.cull(3, sc.q0, dq)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 1023, 1024, 1025, 2047, 2048, 2049])
def test_counts_of_many_overlaps(gpu_lib, oracle_lib, n):
    """n overlaps of 2 n bodies: the scans of the counts by bodies and by overlaps around a tile."""
    from adb_gb300.abd import ABD
    sb, mesh = S.SceneBuilder(), S.cube_mesh()
    for k in range(n):
        at = np.array([3.0 * (k % 46), 2.0, 3.0 * (k // 46)])
        sb.add(mesh, at)
        sb.add(mesh, at + np.array([0.1 * (k % 7) / 7, 1.0 + 0.04 * (k % 3) / 3, 0.2]))
    sc, cfg = sb.build(), S.workload_config("pile")
    g, o = ABD(sc, cfg).cull(1, sc.q0), oracle_lib.OracleSim(sc, cfg).cull(1, sc.q0)
    assert len(o[0]) + len(o[2]) > n
    for a, b in zip(g, o):
        assert a.shape == b.shape and np.array_equal(a, b)
