"""The FP64 form's Grams from exact digit products (design rows and factor
rows) against the oracle's step, at the ranks where the kernel's passes change
(one of 17 .. 64 columns, two of 65 .. 128), ragged row counts and heavy-tailed
rows.

Tolerance as in the other FP64 step comparisons: the digit products are within
FP64's own rounding of the sums, and with condition numbers below 1e5 that
moves the factor by less than 1e5 x R x 1.1e-16 = 1.4e-9 of its size."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R,J,kind", [(17, 30011, "gaussian"), (33, 8193, "heavy"), (48, 4001, "gaussian"),
                                      (64, 4096, "gaussian"), (65, 2049, "heavy"), (100, 1023, "gaussian"),
                                      (128, 4097, "gaussian")])
def test_step_matches_oracle(oracle_mod, R, J, kind):
    from rdist_tensor_gb300 import synthetic
    from rdist_tensor_gb300.api import AccumulatorStationary, CP_ARLS_LEV, Grid, LowRankTensor, SparseTensor, TensorGrid

    dims, idx, vals = synthetic.random_sparse((2600, 140, 530), 30000, seed=9)
    f = synthetic.gaussian_factors(dims, R, seed=R)
    if kind == "heavy":
        rng = np.random.default_rng(3)
        f = [np.ascontiguousarray(U * np.exp(rng.standard_normal((U.shape[0], 1)))) for U in f]
    tg = TensorGrid(dims, Grid(np.ones(3, dtype=np.int32)))
    lr = LowRankTensor(R, tg)
    lr.set_factors(f)
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
