"""The FP64 form's breadth-first STS-CP draws (digit products on the tensor
cores, marked samples drawn again depth first) against the CPU oracle's
depth-first draws: samples equal, weights to 1e-12 (the bound of the other
draw tests), at the edges of the tiles and ranks: odd ranks, ranks below and
above a 32-column chunk and the 64-column switch, one-leaf trees, partial
leaves, a last tile of one sample, heavy-tailed and skewed rows, and zero columns."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

CASES = [
    ((300, 120, 77), 17, 32769, "gaussian"),
    ((200, 31, 64), 32, 8192, "gaussian"),
    ((150, 33, 34), 33, 16385, "heavy"),
    ((500, 64, 65), 64, 4096, "gaussian"),
    ((140, 70, 300), 65, 4097, "sparse"),
    ((400, 99, 201), 100, 2048, "heavy"),
    ((300, 128, 129), 128, 2049, "gaussian"),
    ((17811, 97, 611), 58, 20001, "skewed"),
]


@pytest.mark.parametrize("dims,R,J,kind", CASES)
def test_draws_match_oracle(oracle_mod, dims, R, J, kind):
    from rdist_tensor_gb300.api import AccumulatorStationary, Grid, LowRankTensor, STS_CP, SparseTensor, TensorGrid

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(R)
    factors = []
    for d in dims:
        U = rng.standard_normal((d, R))
        if kind == "heavy":
            U *= np.exp(2.0 * rng.standard_normal((d, 1)))
        if kind == "skewed":  # the rare rows' tiles of the tail level: long sequences of leaves that stay
            U *= (1.0 + np.arange(d))[:, None] ** -0.55
        if kind == "sparse":
            U *= rng.random((d, R)) < 0.3
        factors.append(np.ascontiguousarray(U / np.sqrt((U * U).sum(axis=0))))
    idx = np.stack([rng.integers(0, d, size=2000) for d in dims], axis=1).astype(np.uint32)
    vals = rng.random(2000)
    tg = TensorGrid(np.array(dims), Grid(np.ones(len(dims), dtype=np.int32)))
    st = SparseTensor(tg, idx, vals, "none")
    lr = LowRankTensor(R, tg)
    lr.set_factors(factors)
    opt = AccumulatorStationary(st, lr, STS_CP(lr), max_samples=J)
    opt.initialize_ground_truth_for_als()
    ora = oracle_mod.OracleALS(dims, idx, vals, factors, "sts_cp")
    for n in range(len(dims)):
        uni = rng.random((len(dims), 2, J))
        s, w = opt.draw(n, J, torch.as_tensor(uni, device="cuda"))
        opt.step_info()  # raises on a device-side error
        ref = ora.draw(n, J, uni)
        got = s.cpu().numpy().astype(np.uint32)
        cols = [k for k in range(len(dims)) if k != n]
        assert np.array_equal(got[:, cols], ref[0][:, cols])
        np.testing.assert_allclose(w.cpu().numpy(), ref[1], rtol=1e-12)
    opt.deinitialize()
