"""Mollified edge-edge pairs (near-parallel edges, the full 9 x 9 projection by one warp)
against the oracle: Newton systems of cube lattices a little off alignment, where most
edge pairs are mollified, with and without the projection and with stiffnesses outside the
FP32 range (the projection then starts from the identity). The bar is the 1e-9 relative of
every Newton system of this library."""
import dataclasses

import numpy as np
import pytest

from adb_gb300 import scene as S

pytestmark = pytest.mark.gpu
REL = 1e-9


def rel(a, b):
    return float(np.abs(a - b).max() / max(np.abs(b).max(), 1e-300))


@pytest.mark.parametrize("tilt,kappa,psd", [(1e-2, 1e-4, True), (1e-3, 1e-4, True), (1e-2, 1e-4, False),
                                            (1e-2, 1e30, True), (1e-2, 1e-44, True)])
@pytest.mark.parametrize("n", [2, 3, 27])
def test_newton_system_of_nearly_parallel_edges(gpu_lib, oracle_lib, n, tilt, kappa, psd):
    from adb_gb300.abd import ABD
    rng = np.random.default_rng(n)
    sb = S.SceneBuilder()
    for k in range(n):
        a, b, c = rng.uniform(-tilt, tilt, 3)
        sb.add(S.cube_mesh(), (1.015 * (k % 3), 3.0 + 1.015 * (k // 9), 1.015 * ((k // 3) % 3)), S.rotation_zyx(a, b, c))
    sc = sb.build()
    cfg = dataclasses.replace(S.workload_config("cubes"), kappa=kappa, psd=psd, ground=False)
    gpu, orc = ABD(sc, cfg), oracle_lib.OracleSim(sc, cfg)
    gg, gd, gk, gv = gpu.newton_system(sc.q0)
    og, od, ok, ov = orc.newton_system(sc.q0)
    assert len(ok) and np.array_equal(gk, ok)
    print("bodies %d: grad %.1e diag %.1e off %.1e" % (n, rel(gg, og), rel(gd, od), rel(gv, ov)))
    assert rel(gg, og) <= REL and rel(gd, od) <= REL and rel(gv, ov) <= REL
