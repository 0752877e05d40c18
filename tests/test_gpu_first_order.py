"""Projections that end with the first-order correction (abd_ipc.cuh): Hessian blocks of pairs whose
reduced matrices have eigenvalues of both signs, from well separated to nearly equal and nearly
zero, against an eigen-decomposition by LAPACK of the unprojected Hessian. An eigen-decomposition of
n = 12 is backward stable to about n * 2^-53 of the norm and a projection onto the cone is
Lipschitz with constant 1, so 1e-13 of each block's norm covers both sides and the derivatives'
own rounding (some hundred operations on values within it)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def stencils(kind, n, seed):
    rng = np.random.default_rng(seed)
    X = rng.normal(size=(n, 4, 3))
    X[: n // 4, 0] = X[: n // 4, 1:].mean(1) + 1e-3 * rng.normal(size=(n // 4, 3))    # near the face
    X[n // 4: n // 2, 2:] = X[n // 4: n // 2, :2] + 0.3 * rng.normal(size=(n // 2 - n // 4, 2, 3))
    X[: n // 8, :] *= np.array([1.0, 1.0, 1e-3])                                       # nearly flat
    return X * 0.02


@pytest.mark.parametrize("kappa", [0.5, 1e-4, 1e12])
@pytest.mark.parametrize("kind", ["pt", "ee"])
def test_projection(gpu_lib, kind, kappa):
    from adb_gb300 import abdtk
    X = stencils(kind, 4000, 11)
    t, d = (abdtk.pt_distance_batch if kind == "pt" else abdtk.ee_distance_batch)(X)
    X, t, d = X[d > 1e-12], t[d > 1e-12], d[d > 1e-12]
    hess = abdtk.ipc_hess_pt_batch if kind == "pt" else abdtk.ipc_hess_ee_batch
    out = []
    try:
        for psd in (False, True):
            abdtk.set_params(dhat=2 * float(d.max()), kappa=kappa, eps_x=1e-3, psd=psd)
            out.append(np.asarray(hess(X, t, d)[0]).reshape(-1, 12, 12))
    finally:
        abdtk.set_params(dhat=1e-4, kappa=1e-3, psd=True)
    w, V = np.linalg.eigh(0.5 * (out[0] + out[0].transpose(0, 2, 1)))
    want = np.einsum("nik,nk,njk->nij", V, np.maximum(w, 0), V)
    err = np.abs(out[1] - want).max((1, 2)) / np.abs(w).max(1)
    print("%s kappa %g: %d stencils, worst %.1e" % (kind, kappa, len(X), err.max()))
    assert (w.min(1) < 0).any() and err.max() <= 1e-13
