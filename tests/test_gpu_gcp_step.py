"""The fused loss of a GCP step (model, loss and derivative in one kernel, and
the gradient that zeroes its outputs) against the torch expression in FP64, at
the ranks where the lanes per entry and the access width change, on factors
that do and do not start on a 16-byte boundary; and the steps that keep to the
expression.

Tolerances: every term is a product of at most N positive factors summed over
R, then a logarithm or quotient of a value in [1e-2, 1e2], so the relative
rounding error of a sum of like-signed terms is below (N + R + 8) u; the
Poisson and Bernoulli losses and derivatives cancel, which is measured against
the sum of their terms' sizes.  100 u covers R <= 100 at u = 2^-24 / 2^-53."""
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _factors(dims, R, dt, aligned, g):
    out = []
    for d in dims:
        flat = torch.rand(d * R + 1, generator=g, device="cuda", dtype=dt) * 0.8 + 0.2
        U = flat[0 if aligned else 1:][:d * R].view(d, R)
        assert U.is_contiguous()
        out.append(U.requires_grad_())
    return out


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("kind", ["poisson", "bernoulli", "gaussian"])
@pytest.mark.parametrize("dims,R,J,aligned", [((5,), 1, 1, True), ((9, 8), 3, 31, True), ((7, 6, 5), 4, 33, False),
                                              ((30, 20, 10), 10, 1000, True), ((30, 20, 10), 32, 5000, True),
                                              ((30, 20, 10), 33, 777, True), ((40, 30, 20, 10), 100, 4099, True),
                                              ((3, 2, 2, 2, 2, 2, 2, 2), 6, 300, True)])
def test_fused_loss_matches_expression(kind, dtype, dims, R, J, aligned):
    from rdist_tensor_gb300 import gcp

    g = torch.Generator(device="cuda").manual_seed(R * 7 + J)
    U = _factors(dims, R, dtype, aligned, g)
    idx = torch.stack([torch.randint(0, d, (J,), generator=g, device="cuda") for d in dims], dim=1).to(torch.int32)
    x = torch.randint(0, 3, (J,), generator=g, device="cuda").to(dtype)
    w = torch.rand(J, generator=g, device="cuda", dtype=dtype) + 0.5
    f = gcp.SampledLoss.apply(kind, idx, x, w, *U)
    (3.0 * f).backward()

    u = 2.0 ** -24 if dtype == torch.float32 else 2.0 ** -53
    V = [q.detach().double() for q in U]
    rows = [V[k][idx[:, k].long()] for k in range(len(dims))]
    m = torch.ones_like(rows[0])
    for r in rows:
        m = m * r
    m, X, W = m.sum(dim=1), x.double(), w.double()
    ref = (W * gcp.loss_values(kind, X, m)).sum()
    if kind == "poisson":
        d, da, size = 1 - X / (m + gcp.EPS), 1 + X / m, (W * (m + X * (1 + torch.log(m).abs()))).sum()
    elif kind == "bernoulli":
        d, da = 1 / (m + 1) - X / (m + gcp.EPS), 1 / (m + 1) + X / m
        size = (W * (1 + torch.log(m + 1) + X * (1 + torch.log(m).abs()))).sum()
    else:
        d, da, size = 2 * (m - X), 2 * (m + X), (W * (m + X) ** 2).sum()
    assert f.shape == () and f.dtype == dtype
    assert abs(float(f.detach()) - float(ref)) <= 100 * u * float(size)
    for n in range(len(dims)):
        p, pa = 3 * (W * d)[:, None], 3 * (W * da)[:, None]
        for k in range(len(dims)):
            if k != n:
                p, pa = p * rows[k], pa * rows[k]
        G = torch.zeros_like(V[n]).index_add_(0, idx[:, n].long(), p.expand(J, R))
        A = torch.zeros_like(V[n]).index_add_(0, idx[:, n].long(), pa.expand(J, R))
        hits = float(torch.bincount(idx[:, n].long()).max())  # atomic sums of this many terms
        assert torch.all((U[n].grad.double() - G).abs() <= (100 + hits) * u * A)


def test_step_routes():
    """A step's fused objective equals the expression on the same sample; an
    overridden objective is the one that runs; a frozen factor gets no
    gradient."""
    from rdist_tensor_gb300 import gcp, synthetic

    dims, idx, vals = synthetic.random_sparse((20, 15, 10), 500, seed=1)
    seen = []

    class Own(gcp.GCP):
        def objective(self, *a):
            seen.append(1)
            return super().objective(*a)

    args = (idx.astype("int32"), vals, dims, 5)
    a, b = (cls(*args, loss="poisson", dtype=torch.float64, seed=4) for cls in (gcp.GCP, Own))
    fa, fb = a.step(300, 200), b.step(300, 200)
    assert seen == [1]
    assert abs(float(fa) - float(fb)) <= 1e-12 * abs(float(fb))
    for p, q in zip(a.factors, b.factors):
        assert torch.max((p.grad - q.grad).abs()) <= 1e-12 * torch.max(q.grad.abs())
    a.factors[1].requires_grad_(False)
    a.step(300, 200)
    assert a.factors[1].grad is None and a.factors[0].grad is not None
