"""The session's pseudo-inverse over many blocks (32 < R <= 128) against the
oracle, at the ranks where its kernels change (elements per thread at 64 / 65
and 96 / 97, the Newton step at 92 / 93) and on singular Grams, which its
acceptance test sends to the Jacobi kernel.

The tolerance is that of the other FP64 step comparisons: with Gaussian
factors the design Gram's condition stays below 1e5, so FP64 rounding in
either implementation moves the factor by less than 1e5 x R x 1.1e-16 = 1.4e-9
of its size."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R,rank", [(33, 33), (64, 64), (65, 65), (92, 92), (93, 93), (96, 96), (97, 97), (128, 128),
                                    (40, 20), (100, 50)])
def test_step_inverse_matches_oracle(oracle_mod, R, rank):
    from rdist_tensor_gb300 import synthetic
    from rdist_tensor_gb300.api import AccumulatorStationary, CP_ARLS_LEV, Grid, LowRankTensor, SparseTensor, TensorGrid

    dims, idx, vals = synthetic.random_sparse((150, 140, 130), 30000, seed=9)
    f = synthetic.gaussian_factors(dims, R, seed=R)
    if rank < R:  # both other factors of rank `rank`, columns repeated: the Gram is singular
        for k in (1, 2):
            f[k] = np.ascontiguousarray(np.concatenate([f[k][:, :rank], f[k][:, :R - rank]], axis=1))
    tg = TensorGrid(dims, Grid(np.ones(3, dtype=np.int32)))
    lr = LowRankTensor(R, tg)
    lr.set_factors(f)
    J = 4096
    opt = AccumulatorStationary(SparseTensor(tg, idx, vals, "none"), lr, CP_ARLS_LEV(lr), max_samples=J)
    opt.initialize_ground_truth_for_als()
    ora = oracle_mod.OracleALS(dims, idx, vals, f, "cp_arls_lev")
    uni = np.random.default_rng(R).random((3, J))
    opt.execute_ALS_step(0, J, torch.as_tensor(uni, device="cuda"))
    out = ora.step(0, J, uni)
    got = lr.factors[0].data.cpu().numpy()
    assert np.all(np.isfinite(got))
    assert np.max(np.abs(got - out["factor"])) / np.max(np.abs(out["factor"])) < 1e-8
    opt.deinitialize()
