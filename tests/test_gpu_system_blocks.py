"""Off-diagonal blocks as abd_newton_system returns them (gathered on the device, copied at
once): overlaps without a contact among them, none at all, more and fewer places than
blocks. Values and keys bit for bit the same whatever the number of places, and the whole
system against the oracle."""
import ctypes as C

import numpy as np
import pytest

from adb_gb300 import scene as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,spacing", [(1, 1.0), (9, 1.3), (64, 1.012)])
def test_blocks(gpu_lib, oracle_lib, n, spacing):
    from adb_gb300 import _lib as L
    from adb_gb300.abd import ABD
    sb = S.SceneBuilder()
    mesh = S.icosphere_mesh(1, 0.5)
    rng = np.random.default_rng(n)
    for k in range(n):
        p = spacing * np.array([k % 4, k // 16, (k // 4) % 4]) + (0.0, 3.0, 0.0)
        sb.add(mesh, p, S.random_rotation(rng), mass=1000.0 * mesh.volume)
    sc = sb.build()
    cfg = S.workload_config("pile")
    cfg.dhat = 2.5e-2
    gpu = ABD(sc, cfg)
    grad, diag, keys, vals = gpu.newton_system(sc.q0)
    og, od, ok, ov = oracle_lib.OracleSim(sc, cfg).newton_system(sc.q0)
    assert np.array_equal(keys, ok)
    if len(ok):
        assert np.abs(vals - ov).max() <= 1e-9 * np.abs(ov).max()
    for room in sorted({1, max(1, len(keys) - 1), len(keys) + 3}):
        k2, v2, m = np.full((room, 2), -7, np.int32), np.full((room, 12, 12), -7.0), C.c_int()
        q = np.ascontiguousarray(sc.q0)
        assert gpu_lib.abd_newton_system(gpu._h, L.dptr(q), L.dptr(grad), L.dptr(diag), C.byref(m), L.iptr(k2),
                                         L.dptr(v2), room) == 0
        use = min(room, len(keys))
        assert m.value == len(keys)
        assert np.array_equal(k2[:use], keys[:use]) and np.array_equal(v2[:use], vals[:use])
        assert np.all(k2[use:] == -7) and np.all(v2[use:] == -7.0)
