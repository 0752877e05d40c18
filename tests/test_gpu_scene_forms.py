"""The two forms of the pair terms (scenes below and from 512 bodies on; newton.cu): scenes around
that size against the oracle at the 1e-9 relative bar of every Newton system, one handle with
scenes on both sides (in which both forms run over the same pairs' buffers) against each
scene alone bit for bit, with mollified edge pairs and friction, and the large form's 9 x 9
projection off, and with stiffnesses outside the FP32 range."""
import dataclasses

import numpy as np
import pytest

from adb_gb300 import scene as S

pytestmark = pytest.mark.gpu
REL = 1e-9


def lattice(n, seed, tilt=1e-2):
    """Columns of cubes, a sphere in three, a little off alignment."""
    rng = np.random.default_rng(seed)
    sb, cube, ico = S.SceneBuilder(), S.cube_mesh(), S.icosphere_mesh(1, 0.5)
    for k in range(n):
        a, b, c = rng.uniform(-tilt, tilt, 3)
        p = (1.015 * (k % 3), 3.0 + 1.015 * (k // 9), 1.015 * ((k // 3) % 3))
        sb.add(ico if (k // 2) % 3 == 2 else cube, p, S.rotation_zyx(a, b, c))
    return sb.build()


def config(**kw):
    return dataclasses.replace(S.workload_config("cubes"), ground=False, mu=0.2, **kw)


def rel(a, b):
    return float(np.abs(a - b).max() / max(np.abs(b).max(), 1e-300))


def moved(sc, seed):
    return sc.q0 + np.random.default_rng(seed).uniform(-1e-4, 1e-4, sc.q0.shape)  # friction


def against_oracle(oracle_lib, sc, cfg, q):
    from adb_gb300.abd import ABD
    gpu, orc = ABD(sc, cfg), oracle_lib.OracleSim(sc, cfg)
    got, want = gpu.newton_system(q), orc.newton_system(q)
    assert len(want[2]) and np.array_equal(got[2], want[2])
    print("%d bodies: grad %.1e diag %.1e off %.1e" % (sc.n_bodies, *(rel(got[i], want[i]) for i in (0, 1, 3))))
    assert all(rel(got[i], want[i]) <= REL for i in (0, 1, 3))


@pytest.mark.parametrize("n", [511, 512, 513])
def test_sizes(gpu_lib, oracle_lib, n):
    sc = lattice(n, n)
    against_oracle(oracle_lib, sc, config(), moved(sc, n))


@pytest.mark.parametrize("kappa,psd", [(1e-4, False), (1e30, True), (1e-44, True)])
def test_large_form_options(gpu_lib, oracle_lib, kappa, psd):
    sc = lattice(520, 1)
    against_oracle(oracle_lib, sc, config(kappa=kappa, psd=psd), sc.q0)


@pytest.mark.parametrize("sizes", [(3, 512, 27, 511), (513, 2, 640)])
def test_both_forms_in_one_handle(gpu_lib, sizes):
    from adb_gb300.abd import ABD
    parts = [lattice(n, n) for n in sizes]
    sc = parts[0]
    for p in parts[1:]:
        sc = S.concat_scenes(sc, p)
    sc.scene_id = np.concatenate([np.full(p.n_bodies, k, np.int32) for k, p in enumerate(parts)])
    q = moved(sc, 0)
    cfg = config()
    grad, diag, keys, off = ABD(sc, cfg).newton_system(q)
    keys = np.asarray(keys).reshape(-1, 2)
    for k, (b0, b1) in enumerate(sc.scene_ranges()):
        assert b1 - b0 == sizes[k]
        g1, d1, k1, o1 = ABD(sc.body_range(b0, b1), cfg).newton_system(q[b0:b1])
        mine = (keys[:, 0] >= b0) & (keys[:, 0] < b1)
        assert np.array_equal(np.asarray(k1).reshape(-1, 2) + b0, keys[mine])
        assert np.array_equal(g1, grad.reshape(-1, 12)[b0:b1].reshape(g1.shape))
        assert np.array_equal(d1, diag[b0:b1]) and np.array_equal(o1, off[mine])
