"""Sessions of different ranks in threads, each on its own stream: the same
factors, bit for bit, as one after the other.  (A kernel's limit of dynamic
shared memory is state of the process: set to one launch's size, it fell below
what another thread's launch of the same kernel needed, which was then refused.)
FP64 STS-CP sessions at three ranks and a mixed one, eager and replayed sweeps."""
import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

SESSIONS = [((2011, 97, 311), 58, 4001, "fp64"), ((1203, 400, 129), 66, 4097, "fp64"),
            ((901, 70, 300), 25, 16385, "fp64"), ((301, 120, 90), 100, 1000, "fp64"),
            ((901, 97, 300), 64, 4096, "tf32")]


def session(dims, R, J, precision):
    from rdist_tensor_gb300.api import AccumulatorStationary, Grid, LowRankTensor, STS_CP, SparseTensor, TensorGrid

    rng = np.random.default_rng(R)
    factors = []
    for d in dims:
        F = rng.standard_normal((d, R)) * (1.0 + np.arange(d))[:, None] ** -0.4
        factors.append(np.ascontiguousarray(F / np.sqrt((F * F).sum(axis=0))))
    idx = np.unique(np.stack([rng.integers(0, d, size=60000) for d in dims], axis=1), axis=0).astype(np.uint32)
    vals = rng.random(len(idx))
    tg = TensorGrid(np.array(dims), Grid(np.ones(len(dims), dtype=np.int32)))
    lr = LowRankTensor(R, tg)
    lr.set_factors(factors)
    opt = AccumulatorStationary(SparseTensor(tg, idx, vals, "none"), lr, STS_CP(lr), max_samples=J,
                                precision=precision)
    opt.initialize_ground_truth_for_als()
    uni = torch.as_tensor(rng.random((len(dims), len(dims), 2, J)), device="cuda")
    return opt, lr, uni, J


def sweeps(s):
    opt, _, uni, J = s
    for _ in range(5):
        opt.execute_sweeps(1, J, uni)


def test_threads_give_the_same_factors():
    ref = []
    for c in SESSIONS:
        s = session(*c)
        sweeps(s)
        torch.cuda.synchronize()
        s[0].step_info()
        ref.append([f.data.clone() for f in s[1].factors])
        s[0].deinitialize()
    for _ in range(3):
        live = [session(*c) for c in SESSIONS]
        torch.cuda.synchronize()
        errors = []

        def work(s):
            try:
                with torch.cuda.stream(torch.cuda.Stream()):
                    sweeps(s)
            except Exception as e:  # noqa: BLE001 (reported below)
                errors.append(e)

        threads = [threading.Thread(target=work, args=(s,)) for s in live]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        torch.cuda.synchronize()
        assert not errors, errors
        for s, r in zip(live, ref):
            s[0].step_info()
            for f, g in zip(s[1].factors, r):
                assert torch.equal(f.data, g)
            s[0].deinitialize()
