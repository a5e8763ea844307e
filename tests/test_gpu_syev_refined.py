"""The refined eigendecomposition of the FP64 form's sampling matrices
(exafac_syev_refined) on the spectra it has to face: separated, clustered at
one and at many scales, repeated, rank-deficient, spread over 16 decades,
diagonal.  Checked: the residual and orthonormality, the eigenvalues against
LAPACK's, and that a clustered spectrum costs no more than the plain FP64
Jacobi (exafac_syev): X that loses its orthonormality there would make the call
start over from A.

Tolerances: A^T A-type products of R terms in FP64 leave |A v - lambda v| and
|V^T V - I| below c R u with u = 2^-53 (c = 8 covers the Jacobi criterion R eps
= 2 R u applied over the sweeps), and Weyl's inequality bounds the eigenvalues'
error by the residual; LAPACK's own is within R u |A|."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def spectrum(kind, R, rng):
    if kind == "separated":
        return np.arange(1.0, R + 1.0)
    if kind == "cluster_1e-9":
        return 1.0 + 1e-9 * rng.standard_normal(R)
    if kind == "two_clusters":
        return np.where(np.arange(R) < R // 2, 1.0, 5.0) * (1.0 + 1e-8 * rng.standard_normal(R))
    if kind == "all_scales":
        return 1.0 + 10.0 ** (-8.0 * rng.random(R) - 1.0)
    if kind == "repeated":
        return np.repeat(np.arange(1.0, R // 4 + 2.0), 4)[:R]
    if kind == "null_half":
        return np.where(np.arange(R) < R // 2, 0.0, 1.0 + rng.random(R))
    if kind == "decades":
        return 10.0 ** (-16.0 * rng.random(R))
    return None


def matrix(kind, R, seed=0):
    rng = np.random.default_rng(R + seed)
    if kind == "diagonal":
        return np.diag(1.0 + rng.random(R))
    Q, _ = np.linalg.qr(rng.standard_normal((R, R)))
    A = (Q * spectrum(kind, R, rng)) @ Q.T
    return (A + A.T) / 2


def run(entry, A, V, lam, ws, nbytes):
    from rdist_tensor_gb300 import _lib

    p = lambda t: ctypes.c_void_p(t.data_ptr())
    _lib.call(entry, A.shape[0], p(A), p(V), p(lam), p(ws), ctypes.c_size_t(nbytes),
              ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))


def buffers(A):
    from rdist_tensor_gb300 import _lib

    R = A.shape[0]
    nbytes = _lib.load().exafac_syev_refined_workspace_bytes(R)
    ws = torch.empty(nbytes // 8 + 1, dtype=torch.float64, device="cuda")
    return (torch.as_tensor(A, device="cuda"), torch.empty((R, R), dtype=torch.float64, device="cuda"),
            torch.empty(R, dtype=torch.float64, device="cuda"), ws, nbytes)


@pytest.mark.parametrize("R", [1, 2, 4, 5, 6, 25, 32, 33, 64, 65, 100, 128])
@pytest.mark.parametrize("kind", ["separated", "cluster_1e-9", "two_clusters", "all_scales", "repeated", "null_half",
                                  "decades", "diagonal"])
def test_decomposition(R, kind):
    A = matrix(kind, R)
    b = buffers(A)
    run("exafac_syev_refined", *b)
    V, lam = b[1].cpu().numpy(), b[2].cpu().numpy()
    size = np.max(np.abs(lam))
    tol = 8 * max(R, 4) * U
    assert np.all(np.diff(lam) >= 0)
    assert np.max(np.abs(A @ V - V * lam)) <= tol * size
    assert np.max(np.abs(V.T @ V - np.eye(R))) <= tol
    assert np.max(np.abs(lam - np.linalg.eigvalsh(A))) <= 2 * tol * size * np.sqrt(R)


@pytest.mark.parametrize("R", [25, 58, 100])
@pytest.mark.parametrize("kind", ["cluster_1e-9", "two_clusters", "all_scales"])
def test_clusters_cost_no_more_than_the_plain_sweeps(R, kind):
    A = matrix(kind, R, seed=1)
    b = buffers(A)
    times = {}
    for entry in ("exafac_syev", "exafac_syev_refined"):
        best = float("inf")
        for _ in range(6):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            run(entry, *b)
            e1.record()
            e1.synchronize()
            best = min(best, e0.elapsed_time(e1))
        times[entry] = best
    assert times["exafac_syev_refined"] < times["exafac_syev"], times
