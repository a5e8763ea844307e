"""A GCP step takes the module's own functions as they are at the time of the
step: a replaced ``loss_values`` or ``sampled_model`` is the one that runs, and
a replaced ``EPS`` counts.  Values are compared with the same step's own
expression in FP64 (1e-12: sums of some hundred like-sized terms)."""
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def model(loss):
    from rdist_tensor_gb300 import gcp, synthetic

    dims, idx, vals = synthetic.random_sparse((20, 15, 10), 500, seed=1)
    return gcp.GCP(idx.astype("int32"), abs(vals), dims, 5, loss=loss, dtype=torch.float64, seed=4)


@pytest.mark.parametrize("loss", ["poisson", "bernoulli", "gaussian"])
def test_replaced_loss_values_run(monkeypatch, loss):
    from rdist_tensor_gb300 import gcp

    plain = model(loss)
    f0 = float(plain.step(300, 200))
    g0 = [U.grad.clone() for U in plain.factors]
    own = gcp.loss_values
    monkeypatch.setattr(gcp, "loss_values", lambda kind, x, m: 3.0 * own(kind, x, m))
    other = model(loss)
    f1 = float(other.step(300, 200))
    assert abs(f1 - 3.0 * f0) <= 1e-12 * abs(f0)
    for a, U in zip(g0, other.factors):
        assert torch.max((U.grad - 3.0 * a).abs()) <= 1e-12 * torch.max(a.abs())


def test_replaced_model_and_eps_count(monkeypatch):
    from rdist_tensor_gb300 import gcp

    f0 = float(model("gaussian").step(300, 200))
    own, seen = gcp.sampled_model, []
    monkeypatch.setattr(gcp, "sampled_model", lambda idx, f: (seen.append(1), own(idx, f))[1])
    assert abs(float(model("gaussian").step(300, 200)) - f0) <= 1e-12 * abs(f0)
    assert seen == [1]
    monkeypatch.undo()
    p0 = float(model("poisson").step(300, 200))
    monkeypatch.setattr(gcp, "EPS", 0.5)
    m = model("poisson")
    p1 = float(m.step(300, 200))
    assert abs(p1 - p0) > 1e-3 * abs(p0)
