"""Failure detection in the FP64 form's tensor-core kernels without a GPU fault:
a tile whose products are withheld by the wait-limit hook makes the waits on it
run out, in a level, the leaf stage and the weights of the breadth-first draws
and in the design Gram.  The kernels return, the session reports
EXAFAC_ERR_TIMEOUT, every sample it leaves is in range with a finite weight,
and the context stays usable."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

DIMS = (2001, 97, 611)


def optimizer(R, J):
    from rdist_tensor_gb300 import synthetic
    from rdist_tensor_gb300.api import AccumulatorStationary, Grid, LowRankTensor, STS_CP, SparseTensor, TensorGrid

    dims, idx, vals = synthetic.random_sparse(DIMS, 20000, seed=2)
    tg = TensorGrid(dims, Grid(np.ones(3, dtype=np.int32)))
    lr = LowRankTensor(R, tg)
    lr.set_factors(synthetic.gaussian_factors(dims, R, seed=R))
    opt = AccumulatorStationary(SparseTensor(tg, idx, vals, "none"), lr, STS_CP(lr), max_samples=J)
    opt.initialize_ground_truth_for_als()
    return opt


def status(opt):
    from rdist_tensor_gb300 import _lib

    out = _lib.StepInfo()
    _lib.call("exafac_als_step_info", opt._h, ctypes.byref(out), ctypes.c_void_p(0))
    return out.device_status


# one node chunk expanded per run, two chunks brought by bulk copies, and the
# 512-thread blocks with two node buffers (R = 70) and one (R = 128)
@pytest.mark.parametrize("R,J", [(25, 16385), (40, 8192), (70, 4096), (128, 2048)])
@pytest.mark.parametrize("site", [23, 24, 25, 26])
def test_withheld_products_report_timeout(R, J, site):
    from rdist_tensor_gb300 import _lib

    if site == 26 and R <= 32:
        pytest.skip("the digit Gram is for R > 32")
    assert J * R * (R + 1) // 2 >= 1 << 22
    opt = optimizer(R, J)
    opt.execute_ALS_step(0, J)
    assert status(opt) == 0
    _lib.call("exafac_als_set_wait_limit", opt._h, 256, (site << 32) | 3)
    opt.execute_ALS_step(1, J)
    torch.cuda.synchronize()
    assert status(opt) == 4  # EXAFAC_ERR_TIMEOUT
    with pytest.raises(_lib.ExafacError, match="wait ran out"):
        opt.step_info()
    s, w = opt.draw(0, J)
    s, w = s.cpu().numpy().view(np.uint32).astype(np.int64), w.cpu().numpy()
    for k in (1, 2):
        assert np.all((s[:, k] >= 0) & (s[:, k] < DIMS[k]))
    assert np.all(np.isfinite(w)) and np.all(w >= 0)
    if site != 26:  # the withheld tile's samples were not weighed
        assert np.any(w == 0)
    opt.deinitialize()
    opt2 = optimizer(R, J)
    for n in range(3):
        opt2.execute_ALS_step(n, J)
    assert status(opt2) == 0
    opt2.deinitialize()
