"""The weights of the FP64 form's breadth-first draws (digit products) against
exact rational arithmetic on the session's own Phi and factors: no larger an
error than the depth-first kernel's FP64 sum over the same samples, which the
same session takes when it draws fewer at a time.  Factors: Gaussian, nearly
collinear columns (large Phi with cancelling forms), and columns with one large
row in common (small entries of h where Phi is large, the case that a fixed
point shared by all of h serves worst).

Tolerance: the errors of the two kernels' forms are compared through the
weights R / (J q), whose product and quotient add two roundings each (2^-53): 4
x 2^-53 in all.  J is a power of two in both draws, so that R / J and J q cost
nothing more."""
import ctypes
from fractions import Fraction

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def make_factors(kind, dims, R):
    rng = np.random.default_rng(R)
    out = []
    for d in dims:
        F = rng.standard_normal((d, R))
        if kind == "collinear":
            eps = 10.0 ** (-3.0 * rng.random(R // 2))
            F[:, 1::2][:, :R // 2] = F[:, 0::2][:, :R // 2] + np.sqrt(2 * eps) * F[:, 1::2][:, :R // 2]
        if kind == "spiky":
            for c in range(R // 2, R):
                F[:, c] *= np.sqrt(10.0 ** (-3.0 * rng.random()) / d)
                F[0, c] = 1.0
        out.append(np.ascontiguousarray(F / np.sqrt((F * F).sum(axis=0))))
    return out


def exact_forms(h, phi):
    """h^T Phi h of each row of h, as Fractions."""
    R = h.shape[1]
    full = [[Fraction(0)] * R for _ in range(R)]
    k = 0
    for a in range(R):
        for b in range(a, R):
            full[a][b] = Fraction(float(phi[k]))
            k += 1
    scale = 1
    for row in full:
        for v in row:
            scale = max(scale, v.denominator)
    ints = [[int(v * scale) for v in row] for row in full]
    out = []
    for x in h:
        xs = [Fraction(float(v)) for v in x]
        s = max(v.denominator for v in xs)
        xi = [int(v * s) for v in xs]
        q = 0
        for a in range(R):
            row = ints[a]
            q += xi[a] * (row[a] * xi[a] + 2 * sum(row[b] * xi[b] for b in range(a + 1, R)))
        out.append(Fraction(q, scale * s * s))
    return out


@pytest.mark.parametrize("R,J", [(33, 16384), (64, 4096), (100, 2048)])
@pytest.mark.parametrize("kind", ["gaussian", "collinear", "spiky"])
def test_error_no_larger_than_the_depth_first_sum(kind, R, J):
    from rdist_tensor_gb300 import _lib
    from rdist_tensor_gb300.api import (AccumulatorStationary, Grid, LowRankTensor, STS_CP, SparseTensor, TensorGrid,
                                        _device_array)

    P = R * (R + 1) // 2
    assert J * P >= 1 << 22
    few = 256
    assert few * P < 1 << 22  # depth first
    dims = (60, 300, 200)
    f = make_factors(kind, dims, R)
    rng = np.random.default_rng(1)
    idx = np.stack([rng.integers(0, d, size=2000) for d in dims], axis=1).astype(np.uint32)
    vals = rng.random(2000)
    tg = TensorGrid(np.array(dims), Grid(np.ones(3, dtype=np.int32)))
    lr = LowRankTensor(R, tg)
    lr.set_factors(f)
    opt = AccumulatorStationary(SparseTensor(tg, idx, vals, "none"), lr, STS_CP(lr), max_samples=J)
    opt.initialize_ground_truth_for_als()
    uni = torch.rand((3, 2, J), generator=torch.Generator().manual_seed(R), dtype=torch.float64).cuda()
    s, w = opt.draw(0, J, uni)
    opt.step_info()
    p = ctypes.c_void_p()
    _lib.call("exafac_als_last_phi", opt._h, ctypes.byref(p))
    phi = _device_array(p.value, (P,), torch.float64).cpu().numpy()
    s1, w1 = opt.draw(0, few, uni[:, :, :few].contiguous())
    opt.step_info()
    assert torch.equal(s[:few, 1:], s1[:, 1:])
    U1, U2 = lr.factors[1].data.cpu().numpy(), lr.factors[2].data.cpu().numpy()
    s = s.cpu().numpy()
    h = U1[s[:few, 1]] * U2[s[:few, 2]]  # the kernels' own product, in FP64
    q = exact_forms(h, phi)
    err, ref = 0.0, 0.0
    for i in range(few):
        err = max(err, abs(float(Fraction(float(w[i])) * J * q[i] / R - 1)))
        ref = max(ref, abs(float(Fraction(float(w1[i])) * few * q[i] / R - 1)))
    assert err <= ref + 4 * U, (err, ref)
    opt.deinitialize()
