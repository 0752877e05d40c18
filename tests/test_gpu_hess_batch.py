"""Batched pair Hessians (prims.cu), whose CTAs take the stencils by projection size and the
mollified ones by a warp each: counts around a warp, a CTA's share and past the size from
which the shares grow, mollified shares from none to all, types given and not, projected and
not, each against the oracle at the 1e-9 relative bar of the pair Hessians."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
REL = 1e-9


def rel(a, b):
    return float(np.abs(a - b).max() / max(np.abs(b).max(), 1e-300))


def stencils(n, parallel, seed):
    rng = np.random.default_rng(seed)
    X = rng.normal(size=(n, 4, 3)) * 0.02
    k = int(round(parallel * n))
    X[:k, 3] = X[:k, 2] + (X[:k, 1] - X[:k, 0]) * 1.3 + 1e-4 * rng.normal(size=(k, 3))
    return X[rng.permutation(n)]


@pytest.mark.parametrize("n,parallel", [(1, 0.0), (1, 1.0), (31, 0.3), (33, 1.0), (129, 0.1), (400, 0.0), (9800, 0.05)])
@pytest.mark.parametrize("given", [False, True])
@pytest.mark.parametrize("psd", [False, True])
def test_batches(gpu_lib, oracle_lib, n, parallel, given, psd):
    from adb_gb300 import abdtk
    O = oracle_lib
    X = stencils(n, parallel, n)
    keep = dict(abdtk.PARAMS)
    for kind in ("pt", "ee"):
        t, d = (abdtk.pt_distance_batch if kind == "pt" else abdtk.ee_distance_batch)(X)
        dhat = float(d.max()) * 2
        abdtk.set_params(dhat=dhat, kappa=0.5, eps_x=1e-3, psd=psd)
        try:
            args = (X, t, d) if given else (X,)
            out = abdtk.ipc_hess_pt_batch(*args) if kind == "pt" else abdtk.ipc_hess_ee_batch(*args)
        finally:
            abdtk.set_params(**keep)
        for i in range(0, n, max(1, n // 300)):
            if kind == "pt":
                Ho, go = O.ipc_hess_pt(X[i].ravel(), t[i], d[i], dhat, 0.5, psd=psd)
            else:
                Ho, go, mo = O.ipc_hess_ee(X[i].ravel(), t[i], d[i], dhat, 0.5, 1e-3, psd=psd)
                assert abs(out[2][i] - mo) <= 1e-12
            assert rel(out[0][i], Ho) <= REL and rel(out[1][i], go) <= REL
