"""The bounded waits of the CG whose CTAs exchange tagged words (k_pcg1): with a limit of few polls a
solve gives up at any of its exchanges (groups of sums, neighbours' z, row blocks past the
registers) and the call reports it, or it ends as ever; the next solve on the handle with the
normal limit gives the bits of an undisturbed one."""
import numpy as np
import pytest

from adb_gb300 import scene as S
from test_gpu_pcg_groups import cluster, config

pytestmark = pytest.mark.gpu
NORMAL = 1 << 21


def scenes(kind):
    if kind == "batch":
        parts = [cluster(n, 7 + n) for n in (3, 40, 8, 17)]
        sc = parts[0]
        for p in parts[1:]:
            sc = S.concat_scenes(sc, p)
        sc.scene_id = np.concatenate([np.full(p.n_bodies, k, np.int32) for k, p in enumerate(parts)])
        return sc
    return cluster(27, 3, spacing=0.68) if kind == "blocks" else cluster(257, 257)


@pytest.mark.parametrize("kind", ["groups", "blocks", "batch"])
def test_giving_up(gpu_lib, kind):
    from adb_gb300._lib import AbdError
    from adb_gb300.abd import ABD
    sc, cfg = scenes(kind), config()
    want, its = ABD(sc, cfg).newton_dq(sc.q0)
    sim = ABD(sc, cfg)
    gave_up = 0
    for polls in (0, 1, 2, 3, 5, 8, 20, 50, 200):
        sim.set_poll_limit(polls)
        try:
            got = sim.newton_dq(sc.q0)[0]
            assert np.array_equal(got, want)
        except AbdError as e:
            assert "ABD_ERR_CUDA" in str(e) and "did not arrive" in str(e)
            gave_up += 1
        sim.set_poll_limit(NORMAL)
        got, k = sim.newton_dq(sc.q0)
        assert k == its and np.array_equal(got, want)
    assert gave_up > 0  # with no poll at all at least


def test_frame_after_giving_up(gpu_lib):
    from adb_gb300._lib import AbdError
    from adb_gb300.abd import ABD
    sc, cfg = cluster(64, 64), config(max_iter_frame=2)
    ref, sim = ABD(sc, cfg), ABD(sc, cfg)
    want = ref.step(1, raise_on_error=False).status
    sim.set_poll_limit(0)
    with pytest.raises(AbdError):
        sim.step(1)
    sim.set_poll_limit(NORMAL)
    sim.set_state(sc.q0, sc.dqdt)
    sim.iter = 0
    assert sim.step(1, raise_on_error=False).status == want
    assert all(np.array_equal(a, b) for a, b in zip(sim.state(), ref.state()))
