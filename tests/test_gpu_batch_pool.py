"""Device buffers kept between batch calls (prims.cu): calls of sizes up and down, larger than a kept
buffer may be, and of several threads at once, against the same calls alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(1, 5000, 3, 40000, 7, 5000), (300, 300, 200000, 300)])
def test_sizes_and_threads(gpu_lib, sizes):
    from adb_gb300 import abdtk
    X = np.random.default_rng(0).normal(size=(max(sizes), 4, 3)) * 0.02
    t, d = abdtk.ee_distance_batch(X)
    abdtk.set_params(dhat=2 * float(d.max()), kappa=1e-3, eps_x=1e-3)
    try:
        few = 300
        want = [np.asarray(a) for a in abdtk.ipc_hess_ee_batch(X[:few], t[:few], d[:few])]
        out = {}

        def work(k):
            got = []
            for n in sizes:
                got.append([np.asarray(a)[:few].copy() for a in abdtk.ipc_hess_ee_batch(X[:n], t[:n], d[:n])])
                t2, d2 = abdtk.ee_distance_batch(X[:n])
                got[-1] += [np.array_equal(t2, t[:n]) and np.array_equal(d2, d[:n])]
            out[k] = got

        threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
        for th in threads:
            th.start()
        for th in threads:
            th.join()
    finally:
        abdtk.set_params(dhat=1e-4, kappa=1e-3)
    assert len(out) == 4
    for got in out.values():
        for n, g in zip(sizes, got):
            assert g[-1]
            for a, b in zip(g[:-1], want):
                assert np.array_equal(a, b[:min(n, few)])
