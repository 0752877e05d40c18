"""Direct solve of block-tridiagonal scenes by elimination levels (tri.cu): chains whose
lengths lie around the level boundaries (powers of two and their neighbours), unbroken and
with a missing link, against the oracle's direct block Cholesky. Both solve the same SPD
system with backward-stable factorizations, so the steps meet the 1e-9 relative bar that
holds for every Newton step of this library."""
import numpy as np
import pytest

from adb_gb300 import scene as S

pytestmark = pytest.mark.gpu
REL = 1e-9


@pytest.mark.parametrize("n", [1, 2, 3, 4, 7, 8, 9, 17])
@pytest.mark.parametrize("broken", [False, True])
def test_chain_lengths_match_oracle(gpu_lib, oracle_lib, n, broken):
    from adb_gb300.abd import ABD
    # links 0.006 apart where they touch (activation distance 0.01), free to move
    sc = S.torus_chain(n=n, gap=0.006, seed=n)
    sc.mass[0] = sc.mass[-1] if n > 1 else 1000.0
    sc.Ic[0] = sc.mass[0] / 12.0
    if broken:
        sc.q0[n // 2:, 0] -= 0.05   # pushed together: one contact opens
    cfg = S.workload_config("chain")
    gpu, orc = ABD(sc, cfg), oracle_lib.OracleSim(sc, cfg)
    keys = gpu.newton_system(sc.q0)[2]
    assert len(keys) == n - 1 - (1 if broken and n > 1 else 0)
    dq, its = gpu.newton_dq(sc.q0)
    ref = orc.newton_dq(sc.q0)
    assert its == 0
    err = float(np.abs(dq - ref).max() / np.abs(ref).max())
    print("links %d broken %d: %.2e from the oracle" % (n, broken, err))
    assert err <= REL
