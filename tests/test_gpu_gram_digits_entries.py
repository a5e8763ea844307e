"""The FP64 form's design Gram from digit products, entry by entry against the
same rows summed in extended precision: ordinary rows, columns whose rows differ
by many decades within a tile of 64, zero and subnormal columns, and rows with
values that overflow FP64's products.

Bound: a tile and entry lose at most 2^-50.6 of the product of the two columns'
largest values in the tile (cut of the rows to 2^-62 of them, the dropped digit
weights, the cut of the sum); the tiles' sums are FP64 sums of at most ntiles +
152 terms, each a rounding of 2^-53 of the sum of the terms' sizes.  The rows
are formed here by the same FP64 operations."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def design(R, J, kind):
    from rdist_tensor_gb300 import synthetic
    from rdist_tensor_gb300.api import AccumulatorStationary, CP_ARLS_LEV, Grid, LowRankTensor, SparseTensor, TensorGrid

    dims, idx, vals = synthetic.random_sparse((90, 140, 530, 61), 20000, seed=9)
    f = synthetic.gaussian_factors(dims, R, seed=R)
    rng = np.random.default_rng(R)
    if kind == "decades":  # within a column, different in each
        f = [np.ascontiguousarray(U * np.exp(8.0 * rng.standard_normal(U.shape))) for U in f]
    if kind == "columns":  # zero, and subnormal beside one of 1e80
        f[1][:, 3] = 0.0
        f[1][:, 4] *= 1e-300
        f[2][:, 4] *= 1e-15
        f[1][:, 5] *= 1e80
    if kind == "overflow":
        for k in (1, 2, 3):
            f[k][::7, 6] *= 1e120
            f[k][::5, 9] *= 1e100
    tg = TensorGrid(dims, Grid(np.ones(4, dtype=np.int32)))
    lr = LowRankTensor(R, tg)
    lr.set_factors(f)
    opt = AccumulatorStationary(SparseTensor(tg, idx, vals, "none"), lr, CP_ARLS_LEV(lr), max_samples=J)
    opt.initialize_ground_truth_for_als()
    kept = [u.data.cpu().numpy().copy() for u in lr.factors]
    opt.execute_ALS_step(0, J)
    s, w, G, _ = opt.last_dedup()
    s, w, G = s.cpu().numpy().view(np.uint32).astype(np.int64), w.cpu().numpy(), G.cpu().numpy()
    opt.deinitialize()
    with np.errstate(over="ignore"):
        X = kept[1][s[:, 1]] * kept[2][s[:, 2]]
        X = X * kept[3][s[:, 3]]
        X = X * np.sqrt(w)[:, None]
    return X, G


@pytest.mark.parametrize("R,J", [(33, 8193), (48, 4001), (64, 4096), (65, 2049), (100, 1023), (128, 4097)])
@pytest.mark.parametrize("kind", ["gaussian", "decades", "columns"])
def test_entries(R, J, kind):
    assert J * R * (R + 1) // 2 >= 1 << 22
    X, G = design(R, J, kind)
    assert np.all(np.isfinite(X))
    wide = X.astype(np.longdouble)
    ref = wide.T @ wide
    size = np.abs(wide).T @ np.abs(wide)
    ntiles = (X.shape[0] + 63) // 64
    lost = np.zeros_like(size)
    for t in range(ntiles):
        m = np.max(np.abs(wide[64 * t:64 * t + 64]), axis=0)
        lost += np.longdouble(2.0) ** -50.6 * m[:, None] * m
    bound = lost + (ntiles + 152) * np.longdouble(2.0) ** -53 * (size + lost) + np.longdouble(2.0) ** -1074 * ntiles
    assert np.array_equal(G, G.T)
    assert np.all(np.abs(G - ref) <= bound)
    if kind == "columns":
        assert np.all(G[3] == 0) and np.all(np.abs(X[:, 4]) < 2.0 ** -1022) and np.any(G[4, 5] != 0)


@pytest.mark.parametrize("R,J", [(40, 6001), (100, 1023)])
def test_overflowing_rows(R, J):
    """Infinities stay infinities, and what is finite in FP64 stays finite."""
    X, G = design(R, J, "overflow")
    assert np.any(np.isinf(X[:, 6])) and np.all(np.isfinite(np.delete(X, 6, axis=1)))
    assert np.max(np.abs(X[:, 9])) > 2.0 ** 877
    assert np.isposinf(G[6, 6])
    hit = np.isinf(X[:, 6])
    for b in range(R):
        if b == 6:
            continue
        t = np.sign(X[hit, 6]) * np.sign(X[hit, b])
        assert np.all(t != 0)  # Gaussian entries
        want = np.nan if (np.any(t > 0) and np.any(t < 0)) else t[0] * np.inf
        assert np.array_equal(G[6, b], want, equal_nan=True), b
    small = [b for b in range(R) if b not in (6, 9)]
    assert np.all(np.isfinite(G[np.ix_(small, small)]))
