"""The list of trajectory candidates that the FP32 certificates leave (cull.cu): sized by the scene,
so that a handle of few bodies stays small, and a step with more candidates than it holds gives
the oracle's bound bit for bit, the first time and once the list has grown."""
import numpy as np
import pytest

from adb_gb300 import scene as S

pytestmark = pytest.mark.gpu


def test_memory_of_a_small_handle(gpu_lib):
    torch = pytest.importorskip("torch")
    from adb_gb300.abd import ABD
    sc, cfg = S.cube_stack(10, gap=0.01, seed=1), S.workload_config("cubes")

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
    # buffers of 1024 entries or a few thousand; the list alone was 16 MB
    assert (used() - before) / 16 < 6 << 20


def rod(sides, axis):
    """A closed prism of length 8 along an axis: edges as long as the body."""
    t = 2.0 * np.pi * np.arange(sides) / sides
    ring = np.stack([np.zeros(sides), 0.3 * np.cos(t), 0.3 * np.sin(t)], 1)
    v = np.concatenate([ring - (4.0, 0.0, 0.0), ring + (4.0, 0.0, 0.0), [(-4.0, 0.0, 0.0), (4.0, 0.0, 0.0)]])
    f = []
    for k in range(sides):
        n = (k + 1) % sides
        f += [(k, sides + k, n), (n, sides + k, sides + n), (k, n, 2 * sides), (sides + n, sides + k, 2 * sides + 1)]
    f = np.array(f, np.int32)[:, ::-1]
    v = v.astype(np.float32).astype(np.float64)
    return S.Mesh(np.roll(v, axis, 1), f, S.extract_edges(f))


def test_more_candidates_than_the_list(gpu_lib, oracle_lib):
    from adb_gb300 import abdtk
    from adb_gb300.abd import ABD
    mesh = [rod(64, 0), rod(64, 2)]
    sb = S.SceneBuilder()
    sb.add(mesh[0], (0.0, 3.0, 0.0))
    sb.add(mesh[1], (0.0, 3.7, 0.0), S.rotation_zyx(0.03, 0.02, 0.01))
    sc, cfg = sb.build(), S.workload_config("pile")
    dq = np.zeros_like(sc.q0)
    dq[1, 1] = -1.5
    # the long edges of one cross those of the other: more pairs that meet, by a sample of all,
    # than the 4096 candidates that so few primitives have room for
    rng = np.random.default_rng(0)
    v = [m.vertices @ q[3:].reshape(3, 3) + q[:3] for m, q in zip(mesh, sc.q0)]
    n = 20000
    a, b = (w[m.edges[rng.integers(len(m.edges), size=n)]] for w, m in zip(v, mesh))
    x = np.concatenate([a, b, a, b + dq[1, :3]], 1)
    assert (abdtk.ee_collision_time_batch(x) < 1.0).mean() * len(mesh[0].edges) * len(mesh[1].edges) > 2 * 4096
    gpu, want = ABD(sc, cfg), oracle_lib.OracleSim(sc, cfg).cull(3, sc.q0, dq)
    assert want < 1.0
    for _ in range(3):
        assert gpu.cull(3, sc.q0, dq) == want
