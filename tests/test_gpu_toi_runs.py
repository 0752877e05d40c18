"""Batched times of impact whose warps stream over the trajectories (prims.cu, noalloc.cu): sizes
around a warp and a block and past the size from which a warp takes several rounds, bit for bit against the
oracle (a sample) and against the same trajectories in small batches; the minimum too."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def trajectories(n, seed):
    rng = np.random.default_rng(seed)
    x = rng.random((n, 8, 3))
    x[:, 5:] = x[:, 1:4] + 0.3 * (x[:, 5:] - 0.5)
    hit = rng.random(n) < 0.4
    t = rng.uniform(0.05, 1.0, (n, 1))
    b = rng.dirichlet((1, 1, 1), n)[:, :, None]
    foot = (b * (x[:, 1:4] + t[:, :, None] * (x[:, 5:] - x[:, 1:4]))).sum(1)
    x[:, 4] = np.where(hit[:, None], x[:, 0] + (foot - x[:, 0]) / t, x[:, 4])
    return x


@pytest.mark.parametrize("n", [1, 31, 127, 128, 129, 3000, 2 * 152 * 4 * 128 + 77])
def test_runs(gpu_lib, oracle_lib, n):
    from adb_gb300 import abdtk
    x = trajectories(n, n)
    pt, ee = abdtk.pt_collision_time_batch(x), abdtk.ee_collision_time_batch(x)
    m = min(n, 3000)
    assert np.array_equal(pt[:m], [oracle_lib.pt_collision_time(v) for v in x[:m]])
    assert np.array_equal(ee[:m], [oracle_lib.ee_collision_time(v) for v in x[:m]])
    if n > 3000:
        assert np.array_equal(pt, np.concatenate([abdtk.pt_collision_time_batch(x[k:k + 50000])
                                                  for k in range(0, n, 50000)]))
    dx = torch.from_numpy(np.ascontiguousarray(x.reshape(n, 24))).cuda()
    toi, mn = torch.full((n,), -1.0, dtype=torch.float64, device="cuda"), torch.zeros(1, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert gpu_lib.abd_pt_min_toi_noalloc(n, C.c_void_p(dx.data_ptr()), C.c_void_p(toi.data_ptr()),
                                          C.c_void_p(mn.data_ptr()), None) == 0
    torch.cuda.synchronize()
    assert np.array_equal(toi.cpu().numpy(), pt) and mn.item() == pt.min()
