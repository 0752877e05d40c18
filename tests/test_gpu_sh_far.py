"""Spatial-hash queries of bodies beyond the cells that an int counts (2^31 of them on an axis): all
their coordinates fall into the last cell. A body out there changes neither the sets nor the
step bounds of the others."""
import dataclasses

import numpy as np
import pytest

from adb_gb300 import scene as S

pytestmark = pytest.mark.gpu


def build(far):
    sb = S.SceneBuilder()
    for k in range(4):
        mesh = S.cube_mesh() if k % 2 else S.icosphere_mesh(1, 0.5)
        sb.add(mesh, (1.04 * k, 3.0, 0.0), S.rotation_zyx(0.0, 0.01 * k, 0.0))
    if far:
        sb.add(S.cube_mesh(), far)
    return sb.build()


@pytest.mark.parametrize("axes", [(1, 0, 0), (0, 1, 0), (1, 1, 1)])
def test_far_body(gpu_lib, axes):
    from adb_gb300.abd import ABD
    cfg = S.Config(dhat=1e-2, iaabb=0, full_ccd=True, sh_min_xyz=-5.0, ground=False)
    out = []
    for far in (None, tuple(4e9 * a + 10.0 for a in axes)):
        sc = build(far)
        sim = ABD(sc, cfg)
        dq = np.zeros_like(sc.q0)
        dq[:4, 0] = (0.6, 0.0, 0.3, -0.4)
        out.append((sim.cull(1, sc.q0), sim.cull(3, sc.q0, dq)))
    assert len(out[0][0][0]) and out[0][1] < 1.0
    assert all(np.array_equal(a, b) for a, b in zip(out[0][0], out[1][0])) and out[0][1] == out[1][1]


@pytest.mark.parametrize("cells", [(1 << 22, 1 << 21, 1 << 21), (1 << 11, 1 << 10, 1 << 10), (1 << 30, 1 << 30, 1)])
def test_too_many_cells(gpu_lib, cells):
    """Motions over more cells than a table can hold are refused, those whose number of cells is a
    multiple of 2^64 (the first) among them."""
    from adb_gb300._lib import AbdError
    from adb_gb300.abd import ABD
    sb = S.SceneBuilder()
    sb.add(S.cube_mesh(), (32.0, 32.0, 32.0))
    sb.add(S.cube_mesh(), (64.0 * 5 + 32.0, 32.0, 32.0))
    sc = sb.build()
    sim = ABD(sc, S.Config(iaabb=0, full_ccd=True, sh_min_xyz=0.0, sh_dx=64.0, ground=False))
    dq = np.zeros_like(sc.q0)
    dq[0, :3] = [64.0 * (n - 1) for n in cells]
    with pytest.raises(AbdError, match="too many cell registrations"):
        sim.cull(3, sc.q0, dq)
    assert sim.cull(3, sc.q0, np.zeros_like(dq)) == 1.0
