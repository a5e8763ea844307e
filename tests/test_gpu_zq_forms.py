"""The FP64 form's breadth-first STS-CP draws in the forms the other draw tests
leave out, against the CPU oracle (samples equal, weights to 1e-12, the bound of
the other draw tests): two, four and five modes, fewer samples than the session
was opened for, and more tiles of samples than a block's shared memory holds
(the partition's prefix in global memory).  The number of kernels tells which
route a draw took."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


# (dims, R, J, the session's J, modes drawn)
CASES = [((3001, 700), 64, 4096, 4096, (0, 1)),
         ((901, 120, 77, 300), 48, 6001, 6001, (0, 1, 2, 3)),
         ((5003, 120, 77, 300, 64), 33, 9001, 9001, (0, 2, 4)),
         ((901, 120, 77), 58, 4097, 50000, (0, 1)),
         ((900, 120, 300), 100, 1000, 4097, (2,)),
         ((4001, 120, 90), 3, (1 << 21) + 77, (1 << 21) + 77, (1,)),
         ((301, 1, 70), 2, 1500000, 1500000, (0, 2)),
         ((130, 77), 1, (1 << 22) + 5, (1 << 22) + 5, (1,))]


@pytest.mark.parametrize("dims,R,J,Jmax,modes", CASES)
def test_draws_match_oracle(oracle_mod, dims, R, J, Jmax, modes):
    from rdist_tensor_gb300 import _lib
    from rdist_tensor_gb300.api import AccumulatorStationary, Grid, LowRankTensor, STS_CP, SparseTensor, TensorGrid

    rng = np.random.default_rng(R + len(dims))
    factors = []
    for d in dims:
        U = rng.standard_normal((d, R)) * (1.0 + np.arange(d))[:, None] ** -0.3
        factors.append(np.ascontiguousarray(U / np.sqrt((U * U).sum(axis=0))))
    idx = np.stack([rng.integers(0, d, size=2000) for d in dims], axis=1).astype(np.uint32)
    vals = rng.random(2000)
    tg = TensorGrid(np.array(dims), Grid(np.ones(len(dims), dtype=np.int32)))
    lr = LowRankTensor(R, tg)
    lr.set_factors(factors)
    opt = AccumulatorStationary(SparseTensor(tg, idx, vals, "none"), lr, STS_CP(lr), max_samples=Jmax)
    opt.initialize_ground_truth_for_als()
    ora = oracle_mod.OracleALS(dims, idx, vals, factors, "sts_cp")

    def launches(n, J, uni):
        before = _lib.load().exafac_kernel_launches()
        out = opt.draw(n, J, uni)
        return _lib.load().exafac_kernel_launches() - before, out

    for n in modes:
        uni = rng.random((len(dims), 2, J))
        few, _ = launches(n, 16, torch.as_tensor(uni[:, :, :16].copy(), device="cuda"))  # depth first
        taken, (s, w) = launches(n, J, torch.as_tensor(uni, device="cuda"))
        assert taken > few + 8 * (len(dims) - 1)  # two trees a mode, four kernels each at least
        opt.step_info()  # raises on a device-side error
        ref = ora.draw(n, J, uni)
        cols = [k for k in range(len(dims)) if k != n]
        assert np.array_equal(s.cpu().numpy().astype(np.uint32)[:, cols], ref[0][:, cols])
        np.testing.assert_allclose(w.cpu().numpy(), ref[1], rtol=1e-12)
    opt.deinitialize()
