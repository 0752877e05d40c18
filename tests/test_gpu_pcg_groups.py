"""The CG with one body group per CTA, whose CTAs exchange tagged words (k_pcg1), at its edges:
one group and a part of one, group counts around a warp of sums, bodies with more row blocks
than the registers hold, several scenes of different sizes that converge apart, and the
iteration caps. Newton steps against the oracle's direct solve at the 1e-9 relative bar of
every Newton step, and scenes in a batch bit for bit as alone."""
import dataclasses

import numpy as np
import pytest

from adb_gb300 import scene as S

pytestmark = pytest.mark.gpu
REL = 1e-9


def cluster(n, seed, spacing=1.012, subdiv=1):
    """n icospheres on a lattice, neighbours within the activation distance."""
    rng = np.random.default_rng(seed)
    sb = S.SceneBuilder()
    mesh = S.icosphere_mesh(subdiv, 0.5)
    side = int(np.ceil(n ** (1.0 / 3.0)))
    for k in range(n):
        p = spacing * np.array([k % side, (k // side) % side, k // side ** 2]) + (0.0, 3.0, 0.0)
        sb.add(mesh, p, S.random_rotation(rng), mass=1000.0 * mesh.volume)
    return sb.build()


def config(**kw):
    # the activation distance reaches the flat sides of the coarse spheres
    return dataclasses.replace(S.workload_config("pile"), dhat=2.5e-2, tri_direct=False, **kw)


@pytest.mark.parametrize("n", [1, 5, 8, 9, 64, 257])
def test_steps_match_oracle(gpu_lib, oracle_lib, n):
    from adb_gb300.abd import ABD
    sc, cfg = cluster(n, n), config()
    gpu, orc = ABD(sc, cfg), oracle_lib.OracleSim(sc, cfg)
    dq, its = gpu.newton_dq(sc.q0)
    ref = orc.newton_dq(sc.q0)
    assert its > 0
    assert float(np.abs(dq - ref).max() / np.abs(ref).max()) <= REL


def test_many_row_blocks(gpu_lib, oracle_lib):
    """A body in touch with 26 others: row blocks past the two that a part keeps in registers."""
    from adb_gb300.abd import ABD
    sc = cluster(27, 3, spacing=0.68)
    cfg = config()
    gpu, orc = ABD(sc, cfg), oracle_lib.OracleSim(sc, cfg)
    keys = gpu.newton_system(sc.q0)[2]
    assert np.bincount(keys.ravel()).max() > 8
    dq, _ = gpu.newton_dq(sc.q0)
    ref = orc.newton_dq(sc.q0)
    assert float(np.abs(dq - ref).max() / np.abs(ref).max()) <= REL


def test_scenes_converge_apart_bitwise(gpu_lib):
    from adb_gb300.abd import ABD
    parts = [cluster(n, 7 + n) for n in (3, 40, 8, 17)]
    sc = parts[0]
    for p in parts[1:]:
        sc = S.concat_scenes(sc, p)
    sc.scene_id = np.concatenate([np.full(p.n_bodies, k, np.int32) for k, p in enumerate(parts)])
    cfg = config()
    both, its = ABD(sc, cfg).newton_dq(sc.q0)
    alone = [ABD(p, cfg).newton_dq(p.q0) for p in parts]
    assert np.array_equal(both, np.concatenate([a[0] for a in alone]))
    assert its == max(a[1] for a in alone) and len({a[1] for a in alone}) > 1


@pytest.mark.parametrize("cap", [0, 1, 3])
def test_iteration_cap(gpu_lib, cap):
    from adb_gb300.abd import ABD
    sc = cluster(40, 2)
    dq, its = ABD(sc, config(pcg_max_iter=cap)).newton_dq(sc.q0)
    assert its == cap and np.all(np.isfinite(dq)) and (cap > 0 or not dq.any())
