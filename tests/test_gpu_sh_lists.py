"""The candidate list of the spatial-hash queries (shash.cu): sized by the scene, so that a handle of
few bodies stays small; grown when a run leaves more; sets and bounds of the oracle either
way, the first time and again."""
import dataclasses

import numpy as np
import pytest

from adb_gb300 import scene as S

pytestmark = pytest.mark.gpu


def test_memory_of_a_small_handle(gpu_lib):
    torch = pytest.importorskip("torch")
    from adb_gb300.abd import ABD
    sc = S.cube_stack(10, gap=0.01, seed=1)
    cfg = dataclasses.replace(S.workload_config("cubes"), iaabb=0, full_ccd=True)

    def used():
        torch.cuda.synchronize()
        return -torch.cuda.mem_get_info()[0]

    def handle():
        sim = ABD(sc, cfg)
        sim.cull(1, sc.q0)
        sim.cull(3, sc.q0, cfg.dt * sc.dqdt)
        return sim

    keep = [handle()]
    before = used()
    keep += [handle() for _ in range(16)]
    # the bucket table has 2 MB; the list alone was 16 MB
    assert (used() - before) / 16 < 9 << 20


def test_growth(gpu_lib, oracle_lib):
    """480 x 480 edge pairs within reach where the list starts with 30720 entries."""
    from adb_gb300.abd import ABD
    sb = S.SceneBuilder()
    for k in range(2):
        sb.add(S.icosphere_mesh(2, 0.5), (1.01 * k, 3.0, 0.0))
    sc = sb.build()
    cfg = S.Config(dhat=4.0, iaabb=0, full_ccd=True, sh_dx=4.0, sh_bits=2, ground=False)
    gpu, orc = ABD(sc, cfg), oracle_lib.OracleSim(sc, cfg)
    want = orc.cull(1, sc.q0)
    assert len(want[2]) > 1 << 17
    dq = np.zeros_like(sc.q0)
    dq[1, 0] = -0.5
    bound = orc.cull(3, sc.q0, dq)
    assert bound < 1.0
    for _ in range(2):
        assert all(np.array_equal(a, b) for a, b in zip(gpu.cull(1, sc.q0), want))
        assert gpu.cull(3, sc.q0, dq) == bound


def test_runs_grow_again(gpu_lib):
    """Two spheres whose 1920 x 1920 edge pairs are within reach, then many that reach nothing: only the
    former are taken in short runs."""
    from adb_gb300.abd import ABD
    mesh = S.icosphere_mesh(3, 0.5)
    cfg = S.Config(dhat=4.0, iaabb=2, sh_dx=4.0, sh_bits=3, ground=False)

    def cull(others):
        sb = S.SceneBuilder()
        for k in range(2):
            sb.add(mesh, (1.01 * k, 3.0, 0.0))
        for k in range(others):
            sb.add(mesh, (20.0 + 4.0 * k, 3.0, 0.0))
        sc = sb.build()
        sim = ABD(sc, cfg)
        sim.cull(1, sc.q0)
        sim.profile(True)
        sets = sim.cull(1, sc.q0)
        return sets, sum(v["launches"] for k, v in sim.kernel_times().items() if "hash" in k)

    alone, few = cull(0)
    sets, launches = cull(30)
    assert few > 0 and all(np.array_equal(a, b) for a, b in zip(alone, sets))
    # 57 600 edges past the pair: at most a doubling run each, of two launches, for log2(61440)
    assert launches <= few + 2 * 20


def test_memory_of_the_buckets(gpu_lib):
    """2^24 buckets (xyz_bits 8) of 8 bytes."""
    torch = pytest.importorskip("torch")
    from adb_gb300.abd import ABD
    sc = S.cube_stack(2, gap=0.01, seed=1)
    cfg = dataclasses.replace(S.workload_config("cubes"), iaabb=0, sh_bits=8)
    ABD(sc, cfg).cull(1, sc.q0)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    sim = ABD(sc, cfg)
    sim.cull(1, sc.q0)
    torch.cuda.synchronize()
    # two arrays, by the steps in which buffers grow 66 MB each (a third one would make 198)
    assert before - torch.cuda.mem_get_info()[0] < 160 << 20
