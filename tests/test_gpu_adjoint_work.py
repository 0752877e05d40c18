"""Algorithmic bytes that the profile of an adjoint states for its CG: every iteration of each of its
solves on one system reads at least the diagonal blocks and the vectors."""
import dataclasses

import numpy as np
import pytest

from adb_gb300 import scene as S

pytestmark = pytest.mark.gpu


def test_bytes_of_every_solve(gpu_lib):
    from adb_gb300.abd import ABD
    sc = S.diff_grid(seed=1, n=2, spacing=1.015, lift=0.515)
    sim = ABD(sc, dataclasses.replace(S.workload_config("diff"), mu=0.1, max_iter_frame=8))
    sim.step(1)
    q = sim.state()[0]
    sim.profile(True)
    sim.adjoint_frame(sc.q0, sc.dqdt, q, np.random.default_rng(0).normal(size=sc.q0.shape))
    pcg, inverse = (sim.kernel_times()[k] for k in ("pcg", "block_inverse"))
    assert sim.adjoint_stats()[0] > 1 and pcg["units"] > 0
    assert pcg["bytes"] >= pcg["units"] * sc.n_bodies * (1152.0 + 6 * 96.0)
    assert inverse["units"] == 1  # formed once
