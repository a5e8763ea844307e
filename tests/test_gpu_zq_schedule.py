"""The FP64 form's breadth-first STS-CP draws do not depend on how a level's
runs are spread over blocks, nor on the order the blocks run in: a tile of 128
slots is shared by several blocks, and with many times more blocks than fit on
the chip at once they run one wave after the other.  Samples are equal to the
CPU oracle's for every grid, weights to 1e-12 (the bound of the other draw
tests)."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

# (dims, R, J): both block sizes (R <= 64, above), one and several node chunks,
# trees with a tail level; the long mode's rows are skewed, so that a tile holds
# up to 128 runs
CASES = [((17811, 97, 611), 58, 20001), ((9001, 70, 300), 25, 16385), ((5003, 64, 129), 65, 4097)]


@pytest.mark.parametrize("dims,R,J", CASES)
def test_draws_do_not_depend_on_the_grid(oracle_mod, dims, R, J):
    from rdist_tensor_gb300 import _lib
    from rdist_tensor_gb300.api import AccumulatorStationary, Grid, LowRankTensor, STS_CP, SparseTensor, TensorGrid

    assert J * R * (R + 1) // 2 >= 1 << 22  # the breadth-first form
    rng = np.random.default_rng(R)
    factors = []
    for d in dims:
        U = rng.standard_normal((d, R)) * (1.0 + np.arange(d))[:, None] ** -0.55
        factors.append(np.ascontiguousarray(U / np.sqrt((U * U).sum(axis=0))))
    idx = np.stack([rng.integers(0, d, size=2000) for d in dims], axis=1).astype(np.uint32)
    tg = TensorGrid(np.array(dims), Grid(np.ones(len(dims), dtype=np.int32)))
    lr = LowRankTensor(R, tg)
    lr.set_factors(factors)
    vals = rng.random(2000)
    opt = AccumulatorStationary(SparseTensor(tg, idx, vals, "none"), lr, STS_CP(lr), max_samples=J)
    opt.initialize_ground_truth_for_als()
    ora = oracle_mod.OracleALS(dims, idx, vals, factors, "sts_cp")
    n = 1
    uni = rng.random((len(dims), 2, J))
    ref = ora.draw(n, J, uni)
    cols = [k for k in range(len(dims)) if k != n]
    dev = torch.as_tensor(uni, device="cuda")
    for blocks in (0, 1, 37, 152, 608, 4999):
        _lib.call("exafac_als_set_draw_blocks", opt._h, ctypes.c_int32(blocks))
        s, w = opt.draw(n, J, dev)
        opt.step_info()  # raises on a device-side error
        assert np.array_equal(s.cpu().numpy().astype(np.uint32)[:, cols], ref[0][:, cols]), blocks
        np.testing.assert_allclose(w.cpu().numpy(), ref[1], rtol=1e-12)
    opt.deinitialize()
