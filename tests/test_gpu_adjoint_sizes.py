"""Adjoint of scenes of few and many entries (the orthogonalisation's vectors: below and around
256, around 1024, 3072, and up to and past what one CTA holds): bodies that touch only the ground, so that a
body's gradients do not depend on how many others there are. GMRES stops at a residual of 1e-12 of
|b|, and an entry of the solution moves by at most the residual over the smallest mass (a
twelfth of the largest here): 1e-9 of the largest gradient has a margin of 80."""
import numpy as np
import pytest

from adb_gb300 import scene as S

pytestmark = pytest.mark.gpu
ALL = 1040


def resting(n):
    sb = S.SceneBuilder()
    for k in range(n):
        sb.add(S.cube_mesh(), (2.0 * (k % 33), 0.5 + S.GROUND_SHIFT + 0.01, 2.0 * (k // 33)))
    return sb.build()


def gradients(n):
    from adb_gb300.abd import ABD
    rng = np.random.default_rng(3)
    v, g, d = (rng.uniform(-1, 1, (ALL, 12))[:n] for _ in range(3))
    sc = resting(n)
    d[:, 3:] = 0.0  # a shear leaves the orthogonality energy's Hessian indefinite
    q1 = sc.q0 + 1e-3 * d
    sim = ABD(sc, S.workload_config("cubes"))
    return sim.cull(1, q1)[4], sim.adjoint_frame(sc.q0, 0.1 * v, q1, g)


@pytest.fixture(scope="module")
def whole(gpu_lib):
    return gradients(ALL)


@pytest.mark.parametrize("n", [1, 2, 21, 22, 86, 256, 257, 1024])
def test_part_of_the_bodies(whole, n):
    vg, part = gradients(n)
    assert len(vg) >= 2 * n
    for a, b in zip(part[:2], whole[1][:2]):
        assert np.abs(a - b[:n]).max() <= 1e-9 * np.abs(b).max()
