"""Spatial-hash queries in FP32 with an FP64 second pass (shash.cu) against the oracle's
restatement of the bucket walk, over the forms the path accepts: pair sets, order, types and
step bounds bit for bit. Grids from one bucket per axis pair to thousands, cells smaller and
larger than the primitives, scaled thresholds, aligned scenes whose edges are parallel and
coplanar (where no FP32 certificate holds), several scenes in one handle, and more
candidates than the list holds at a time."""
import dataclasses

import numpy as np
import pytest

from adb_gb300 import scene as S

pytestmark = pytest.mark.gpu


def build(kind, n, seed):
    rng = np.random.default_rng(seed)
    sb = S.SceneBuilder()
    for k in range(n):
        if kind == "random":
            mesh = S.cube_mesh() if k % 2 else S.icosphere_mesh(1, 0.5)
            sb.add(mesh, rng.uniform(-1.5, 1.5, 3) + (0.0, 3.0, 0.0), S.random_rotation(rng))
        elif kind == "aligned":   # cubes on a lattice, faces 0.0625 apart
            sb.add(S.cube_mesh(), (1.0625 * (k % 3), 3.0 + 1.0625 * (k // 3), 0.25 * (k % 2)))
        else:                     # dense meshes inside one another's reach
            sb.add(S.icosphere_mesh(3, 0.5), (1.01 * k, 3.0, 0.0))
    return sb.build()


def assert_sets_equal(g, o):
    for name, a, b in zip(("pt", "pt_type", "ee", "ee_type", "vg"), g, o):
        assert a.shape == b.shape and np.array_equal(a, b), name


@pytest.mark.parametrize("kind", ["random", "aligned"])
@pytest.mark.parametrize("bits,dx,sf", [(1, 0.8, 1.0), (6, 0.8, 1.0), (6, 0.8, 2.5), (3, 0.2, 1.0), (8, 0.11, 0.5)])
def test_sets_and_bounds(gpu_lib, oracle_lib, kind, bits, dx, sf):
    from adb_gb300.abd import ABD
    sc = build(kind, 9, 3)
    cfg = S.Config(dhat=1e-2, iaabb=0, full_ccd=True, sh_bits=bits, sh_dx=dx, sh_min_xyz=-5.0, safe_factor=sf)
    gpu, orc = ABD(sc, cfg), oracle_lib.OracleSim(sc, cfg)
    assert_sets_equal(gpu.cull(1, sc.q0), orc.cull(1, sc.q0))
    rng = np.random.default_rng(2)
    hits = 0
    for k in range(4):
        dq = np.zeros_like(sc.q0)
        # rigid translations along an axis keep aligned edges parallel, then free motion
        dq[:, :3] = rng.choice((-0.5, 0.0, 0.5), dq[:, :3].shape) if k < 2 else rng.normal(size=dq[:, :3].shape)
        if k == 3:
            dq += rng.normal(size=dq.shape) * 0.1
        for fix in (False, True):
            c2 = dataclasses.replace(cfg, sh_fix_edge_trajectory=fix)
            g2, o2 = ABD(sc, c2), oracle_lib.OracleSim(sc, c2)
            tg, to = g2.cull(3, sc.q0, dq), o2.cull(3, sc.q0, dq)
            assert tg == to
            hits += to < 1.0
        assert_sets_equal(gpu.cull(2, sc.q0, 0.05 * dq), orc.cull(2, sc.q0, 0.05 * dq))
    assert hits >= 2


def test_more_candidates_than_the_list(gpu_lib, oracle_lib):
    """1920 x 1920 edge pairs within reach: the queries run in parts."""
    from adb_gb300.abd import ABD
    sc = build("dense", 2, 0)
    cfg = S.Config(dhat=4.0, iaabb=2, sh_dx=4.0, sh_bits=2, ground=False)
    gpu, orc = ABD(sc, cfg), oracle_lib.OracleSim(sc, cfg)
    g, o = gpu.cull(1, sc.q0), orc.cull(1, sc.q0)
    assert len(g[2]) > 1 << 21
    assert_sets_equal(g, o)


def test_scenes_stay_apart(gpu_lib):
    """Two scenes in one place: each gets the sets it has alone."""
    from adb_gb300.abd import ABD
    a = build("random", 5, 7)
    sc = S.concat_scenes(a, a)
    sc.scene_id = np.repeat(np.arange(2), 5).astype(np.int32)
    cfg = S.Config(dhat=1e-2, iaabb=2, sh_min_xyz=-5.0, ground=False)
    one, both = ABD(a, cfg).cull(1, a.q0), ABD(sc, cfg).cull(1, sc.q0)
    for k in (0, 2):
        shifted = one[k] + np.array([5, 0, 5, 0], np.int32)
        assert np.array_equal(both[k], np.concatenate([one[k], shifted]))
    for k in (1, 3):
        assert np.array_equal(both[k], np.concatenate([one[k], one[k]]))
