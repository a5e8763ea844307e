"""The mixed forms' pseudo-inverse over many blocks with its Newton step (R >
32: the session's factor, column, product and Newton kernels, with the step's two
forms at 92 / 93) on the session's own design Gram, and a singular Gram, which
the acceptance test sends to the Jacobi kernel before the Newton step.

Tolerance: X from the Newton step has a residual I - G X of the square of the
Cholesky inverse's (below 1e-16 for condition numbers below 1e5) plus the
rounding of its own two products of R terms and of X, each below R u (|G| |X|)
entry by entry: 8 R u (|G| |X| + 1).  A pseudo-inverse X of G satisfies X G X = X
to 1e-8 of its size when the kept eigenvalues' condition is below 1e6."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def gram_and_inverse(precision, R, rank):
    from rdist_tensor_gb300 import synthetic
    from rdist_tensor_gb300.api import AccumulatorStationary, CP_ARLS_LEV, Grid, LowRankTensor, SparseTensor, TensorGrid

    dims, idx, vals = synthetic.random_sparse((150, 140, 130), 30000, seed=9)
    f = synthetic.gaussian_factors(dims, R, seed=R)
    if rank < R:
        for k in (1, 2):
            f[k] = np.ascontiguousarray(np.concatenate([f[k][:, :rank], f[k][:, :R - rank]], axis=1))
    tg = TensorGrid(dims, Grid(np.ones(3, dtype=np.int32)))
    lr = LowRankTensor(R, tg)
    lr.set_factors(f)
    J = 4096
    opt = AccumulatorStationary(SparseTensor(tg, idx, vals, "none"), lr, CP_ARLS_LEV(lr), max_samples=J,
                                precision=precision)
    opt.initialize_ground_truth_for_als()
    opt.execute_ALS_step(0, J)
    _, _, G, X = opt.last_dedup()
    G, X = G.cpu().numpy(), X.cpu().numpy()
    opt.deinitialize()
    return G, X


@pytest.mark.parametrize("precision", ["tf32", "bf16"])
@pytest.mark.parametrize("R", [33, 64, 65, 91, 92, 93, 96, 97, 128])
def test_inverse(precision, R):
    G, X = gram_and_inverse(precision, R, R)
    G = np.triu(G) + np.triu(G, 1).T
    assert np.linalg.cond(G) < 1e5
    wide = np.eye(R) - G.astype(np.longdouble) @ X.astype(np.longdouble)
    assert np.all(np.abs(wide) <= 8 * R * U * (np.abs(G) @ np.abs(X) + 1.0))


@pytest.mark.parametrize("precision", ["tf32", "bf16"])
@pytest.mark.parametrize("R,rank", [(40, 20), (100, 50)])
def test_pseudo_inverse_of_singular_gram(precision, R, rank):
    G, X = gram_and_inverse(precision, R, rank)
    G = np.triu(G) + np.triu(G, 1).T
    assert np.all(np.isfinite(X))
    lam = np.linalg.eigvalsh(G)
    # the repeated columns' rows are equal numbers, so the null eigenvalues are roundings
    assert np.sum(lam > 1e-6 * lam[-1]) == rank
    assert np.max(np.abs(X @ G @ X - X)) <= 1e-8 * np.max(np.abs(X))
