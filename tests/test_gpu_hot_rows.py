"""Rows of tens of thousands of nonzeros (or hits) in the FP64 segmented
reductions: a row whose carries span more than 256 chunks is summed by a whole
block.  The exact step, the exact fit and sampled steps against the oracle, at
both forms of the reduction (R <= 32, above), and rows that span exactly 256 and
257 chunks of 128.  The sums are reproducible bit for bit.

Tolerances as in the other comparisons of exact and sampled FP64 steps with the
oracle (1e-9, 1e-8 of the factor)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def hot_tensor(counts, dims, seed):
    """counts[i] distinct nonzeros in row i of mode 0."""
    rng = np.random.default_rng(seed)
    rows, rest = [], []
    for i, c in enumerate(counts):
        rows.append(np.full(c, i, dtype=np.int64))
        rest.append(rng.choice(dims[1] * dims[2], size=c, replace=False))
    rows, rest = np.concatenate(rows), np.concatenate(rest)
    idx = np.stack([rows, rest // dims[2], rest % dims[2]], axis=1).astype(np.uint32)
    p = rng.permutation(len(idx))
    return idx[p], rng.standard_normal(len(idx))


def optimizer(dims, idx, vals, factors, J):
    from rdist_tensor_gb300.api import AccumulatorStationary, CP_ARLS_LEV, Grid, LowRankTensor, SparseTensor, TensorGrid

    tg = TensorGrid(np.array(dims), Grid(np.ones(3, dtype=np.int32)))
    lr = LowRankTensor(factors[0].shape[1], tg)
    lr.set_factors(factors)
    opt = AccumulatorStationary(SparseTensor(tg, idx, vals, "none"), lr, CP_ARLS_LEV(lr), max_samples=J)
    opt.initialize_ground_truth_for_als()
    return opt, lr


def rel_err(a, b):
    return np.max(np.abs(a - b)) / np.max(np.abs(b))


# row 1 begins at nonzero 64: 32800 nonzeros end in chunk 256, 32928 in chunk 257
@pytest.mark.parametrize("counts", [[64, 32800, 500], [64, 32928, 500], [45000, 3, 40000, 128, 1, 38000],
                                    [10, 58000]])
@pytest.mark.parametrize("R", [8, 32, 33, 100])
def test_exact_step_and_fit(oracle_mod, counts, R):
    from rdist_tensor_gb300 import synthetic

    dims = (len(counts), 300, 200)
    idx, vals = hot_tensor(counts, dims, seed=R)
    factors = synthetic.gaussian_factors(dims, R, seed=5)
    opt, lr = optimizer(dims, idx, vals, factors, 64)
    ora = oracle_mod.OracleALS(dims, idx, vals, factors, "cp_arls_lev")
    assert abs(opt.compute_exact_fit() - ora.fit()) < 1e-9
    ref = exact_mttkrp(dims, idx, vals, factors)
    G = (factors[1].T @ factors[1]) * (factors[2].T @ factors[2])
    opt.exact_step(0)
    got = lr.factors[0].data.cpu().numpy() * lr.sigma.cpu().numpy()
    want = ref @ np.linalg.pinv(G, rcond=1e-13, hermitian=True)
    assert rel_err(got, want) < 1e-9
    first = lr.factors[0].data.clone()
    lr2_opt, lr2 = optimizer(dims, idx, vals, factors, 64)
    lr2_opt.exact_step(0)
    assert torch.equal(first, lr2.factors[0].data)
    opt.deinitialize()
    lr2_opt.deinitialize()


def exact_mttkrp(dims, idx, vals, factors):
    M = np.zeros((dims[0], factors[0].shape[1]))
    np.add.at(M, idx[:, 0], vals[:, None] * factors[1][idx[:, 1]] * factors[2][idx[:, 2]])
    return M


@pytest.mark.parametrize("R", [8, 40])
def test_sampled_step(oracle_mod, R):
    from rdist_tensor_gb300 import synthetic

    dims, J = (5, 300, 200), 1 << 17
    idx, vals = hot_tensor([58000, 100, 55000, 7, 300], dims, seed=3)
    factors = synthetic.gaussian_factors(dims, R, seed=5)
    opt, lr = optimizer(dims, idx, vals, factors, J)
    ora = oracle_mod.OracleALS(dims, idx, vals, factors, "cp_arls_lev")
    uni = np.random.default_rng(R).random((3, J))
    opt.execute_ALS_step(0, J, torch.as_tensor(uni, device="cuda"))
    out = ora.step(0, J, uni)
    info = opt.step_info()
    assert info.hits == out["hits"]
    assert info.unique_samples > 40000  # nearly all of them hit rows 0 and 2: over 256 chunks each
    assert rel_err(lr.factors[0].data.cpu().numpy(), out["factor"]) < 1e-8
    opt.deinitialize()
