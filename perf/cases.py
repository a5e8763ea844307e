"""Performance cases: the work a user of this framework has it do, through its
public entry points, over the range of tensors, ranks, sample counts and
precisions it is used with.

Four kinds of pass:

  sweep   one sampled-ALS sweep (every mode updated once) of a session that
          holds its tensor: ``ALS_Optimizer.execute_sweeps(1, J, uniforms)``
          with either sampler in any of the three precisions.  This is the
          loop a decomposition spends its time in.
  setup   a new decomposition up to its first sampled update: the factors set,
          the session initialised (sorted copies, fibre tables, sampler
          state), one exact round (``-p exact``) and one sampled step.
  exact   one exact-ALS round and the exact fit after it (the ``-p exact``
          preprocessing and the accuracy epochs of ``decompose.py``).
  gcp     one gradient step of the generalized CP model on sampled entries.

A case is a plain dict; see ``listed`` for what each stands for and ``draw``
for the ranges.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from rdist_tensor_gb300 import gcp
from rdist_tensor_gb300.api import (AccumulatorStationary, CP_ARLS_LEV, ExactALS, Grid, LowRankTensor, STS_CP,
                                    SparseTensor, TensorGrid)


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def _case(kind, dims, nnz, R, J=0, sampler="", precision="", tensor="planted", loss="", name=None):
    c = {"kind": kind, "dims": "x".join(str(int(d)) for d in dims), "nnz": int(nnz), "R": int(R), "J": int(J),
         "sampler": sampler, "precision": precision, "tensor": tensor, "loss": loss}
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # The smallest decompositions (a first try, a test, an inner loop over
        # many small tensors): launches and latency are all of it.
        _case("sweep", (60, 50, 40), 4000, 6, 1000, "sts_cp", "fp64", name="sts_fp64_small"),
        # The reference's own arithmetic (the default precision) on the
        # 3-mode 2000^3 workload, at its ordinary rank and at a large one.
        _case("sweep", (2000, 2000, 2000), 2_000_000, 25, 65536, "sts_cp", "fp64", name="sts_fp64_r25"),
        _case("sweep", (2000, 2000, 2000), 2_000_000, 64, 1 << 18, "sts_cp", "fp64", name="sts_fp64_r64"),
        # The same arithmetic on a skewed 4-mode tensor with long and short
        # modes, a rank and a sample count that are no power of two.
        _case("sweep", (200_001, 50_000, 3_001, 99), 10_000_000, 100, 100_003, "sts_cp", "fp64", "zipf",
              name="sts_fp64_4mode"),
        # The mixed forms of the exact sampler: the 3-mode workload at R = 64
        # and the largest one, 5 modes at R = 128 with 2^19 samples a step.
        _case("sweep", (2000, 2000, 2000), 2_000_000, 64, 1 << 18, "sts_cp", "tf32", name="sts_tf32_r64"),
        _case("sweep", (1_000_000, 1_000_000, 100_000, 1_000, 100), 40_000_000, 128, 1 << 19, "sts_cp", "bf16", "zipf",
              name="sts_bf16_5mode"),
        # The approximate sampler: the 4-mode workload with 5e6-row modes in
        # its mixed form, and ragged sizes in the reference's arithmetic.
        _case("sweep", (5_000_000, 5_000_000, 20_000, 1_000), 40_000_000, 25, 1 << 17, "cp_arls_lev", "tf32", "zipf",
              name="arls_tf32_4mode"),
        _case("sweep", (12_007, 9_501, 777), 3_000_001, 45, 50_001, "cp_arls_lev", "fp64", "zipf",
              name="arls_fp64_odd"),
        # A new tensor: set-up, exact preprocessing and first sampled update.
        _case("setup", (300_000, 100_003, 5_000, 100), 20_000_000, 32, 1 << 16, "cp_arls_lev", "tf32", "zipf",
              name="setup_4mode"),
        # The exact preprocessing round and fit of the Zipf workloads.
        _case("exact", (100_000, 50_001, 1_000), 10_000_000, 32, tensor="zipf", name="exact_round"),
        # Gradient steps: the count-tensor workload, and a small FP64 model
        # with the other nonnegative loss.
        _case("gcp", (1_000_000, 1_000_000, 10_000), 10_000_000, 32, 1 << 17, precision="fp32", tensor="zipf",
              loss="poisson", name="gcp_fp32"),
        _case("gcp", (3_000, 2_001, 777), 200_000, 10, 1 << 13, precision="fp64", tensor="zipf", loss="bernoulli",
              name="gcp_fp64_small"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: an ALS sweep (most often), a new decomposition, an exact round or a
    gradient step, sizes log-uniform over the ranges of the listed ones."""
    what = rng.random()
    if what < 0.7:
        precision = rng.choice(("fp64", "fp64", "tf32", "bf16"))
        sampler = rng.choice(("sts_cp", "sts_cp", "cp_arls_lev"))
        R = _log_int(rng, 5, 128)
        if rng.random() < 0.5:
            dims = [_log_int(rng, 50, 2500) for _ in range(3)]
            nnz = min(int(0.25 * math.prod(dims)), max(20_000, dims[0] * dims[1] // 2, dims[0] * dims[2] // 2,
                                                       dims[1] * dims[2] // 2))
            tensor = "planted"
        else:
            N = rng.choice((3, 4, 4, 5))
            big = 200_000 if sampler == "sts_cp" else 2_000_000
            dims = [_log_int(rng, 5_000, big), _log_int(rng, 1_000, big)] + [_log_int(rng, 60, 5_000)
                                                                            for _ in range(N - 2)]
            nnz = _log_int(rng, 300_000, 10_000_000)
            tensor = "zipf"
        top = 1 << 18
        if precision == "fp64" and sampler == "sts_cp":
            # no more sampling work than the largest listed FP64 sweep
            top = max(4_000, min(top, int(100_003 * (100 / R) ** 2 / (2 if len(dims) > 4 else 1))))
        J = _log_int(rng, 2_000, top)
        return _case("sweep", dims, nnz, R, J, sampler, precision, tensor)
    if what < 0.8:
        dims = [_log_int(rng, 5_000, 300_000), _log_int(rng, 1_000, 100_000), _log_int(rng, 100, 5_000)]
        sampler = rng.choice(("sts_cp", "cp_arls_lev"))
        return _case("setup", dims, _log_int(rng, 200_000, 20_000_000), _log_int(rng, 5, 64), _log_int(rng, 2_000, 65536),
                     sampler, rng.choice(("fp64", "tf32")), "zipf")
    if what < 0.9:
        dims = [_log_int(rng, 2_000, 100_000), _log_int(rng, 500, 50_000), _log_int(rng, 100, 2_000)]
        if rng.random() < 0.5:
            dims.append(_log_int(rng, 50, 500))
        return _case("exact", dims, _log_int(rng, 100_000, 5_000_000), _log_int(rng, 5, 60), tensor="zipf")
    dims = [_log_int(rng, 2_000, 1_000_000), _log_int(rng, 1_000, 1_000_000), _log_int(rng, 100, 10_000)]
    return _case("gcp", dims, _log_int(rng, 200_000, 10_000_000), _log_int(rng, 4, 40), _log_int(rng, 4_000, 1 << 17),
                 precision=rng.choice(("fp32", "fp32", "fp64")), tensor="zipf",
                 loss=rng.choice(("poisson", "bernoulli", "gaussian")))


def _dims(case):
    return [int(d) for d in case["dims"].split("x")]


# ---------------------------------------------------------------------------
# inputs (plain torch, on the GPU)
# ---------------------------------------------------------------------------
def _generator(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1_000_003 + salt) % (1 << 62))
    return g


def _coordinates(case, seed):
    """nnz distinct coordinates, int32 [nnz, N]: uniform over the index space,
    or Zipf(1.1) in every mode (the count reached within a few rounds)."""
    dims, nnz = _dims(case), case["nnz"]
    g = _generator(seed, 1)
    dev = torch.device("cuda")
    if case["tensor"] == "planted":
        total = math.prod(dims)
        lin = torch.empty(0, dtype=torch.int64, device=dev)
        while lin.numel() < nnz:
            lin = torch.unique(torch.cat([lin, torch.randint(0, total, (int(1.2 * nnz) + 64,), generator=g, device=dev)]))
        lin = lin[torch.randperm(lin.numel(), generator=g, device=dev)[:nnz]]
        cols = []
        for d in reversed(dims):
            cols.append((lin % d).to(torch.int32))
            lin = lin // d
        return torch.stack(cols[::-1], dim=1).contiguous()
    cdfs = []
    for d in dims:
        c = np.cumsum(np.arange(1, d + 1, dtype=np.float64) ** -1.1)  # summed on the host, in order
        cdfs.append(torch.from_numpy(c / c[-1]).to(dev))
    mult = [int(m) | 1 for m in np.random.default_rng(12345).integers(1 << 40, 1 << 62, size=len(dims))]
    have = torch.empty((0, len(dims)), dtype=torch.int32, device=dev)
    for _ in range(6):
        m = int(1.3 * (nnz - have.shape[0])) + 1024
        cand = torch.stack([torch.searchsorted(cdfs[k], torch.rand(m, generator=g, device=dev, dtype=torch.float64),
                                               right=True).clamp_(max=dims[k] - 1).to(torch.int32)
                            for k in range(len(dims))], dim=1)
        have = torch.cat([have, cand])
        key = torch.zeros(have.shape[0], dtype=torch.int64, device=dev)  # a 64-bit hash of the coordinates
        for k in range(len(dims)):
            key = (key ^ (key >> 29)) * mult[k] + have[:, k].to(torch.int64) * mult[-1 - k]
        order = torch.sort(key, stable=True)
        first = torch.ones_like(key, dtype=torch.bool)
        first[1:] = order.values[1:] != order.values[:-1]
        have = have[torch.sort(order.indices[first]).values]
        if have.shape[0] >= nnz:
            break
    return have[:nnz].contiguous()


def _model_values(idx, factors):
    out = torch.empty(idx.shape[0], dtype=factors[0].dtype, device=idx.device)
    for a in range(0, idx.shape[0], 1 << 22):
        p = factors[0][idx[a:a + (1 << 22), 0].long()]
        for k in range(1, len(factors)):
            p = p * factors[k][idx[a:a + (1 << 22), k].long()]
        out[a:a + (1 << 22)] = p.sum(dim=1)
    return out


def _tensor(case, seed):
    """Coordinates and values: a planted nonnegative rank-10 model plus noise
    (uniform support), N(0, 1) values (Zipf support of the ALS cases) or
    planted counts (the gradient cases)."""
    dims = _dims(case)
    idx = _coordinates(case, seed)
    g = _generator(seed, 2)
    if case["kind"] == "gcp":
        A = [0.5 * torch.randn((d, 8), generator=g, device="cuda", dtype=torch.float32) ** 2 for d in dims]
        vals = torch.poisson(_model_values(idx, A), generator=g).clamp_(min=1.0)
        if case["loss"] == "bernoulli":
            vals = (vals > 0).to(vals.dtype)
        return idx, vals
    if case["tensor"] == "planted":
        A = [torch.randn((d, 10), generator=g, device="cuda", dtype=torch.float64).abs() for d in dims]
        return idx, _model_values(idx, A) + 0.1 * torch.randn(idx.shape[0], generator=g, device="cuda",
                                                              dtype=torch.float64)
    return idx, torch.randn(idx.shape[0], generator=g, device="cuda", dtype=torch.float32).to(torch.float64)


def _factors(case, seed):
    """N(0, 1) entries, columns of unit norm."""
    g = _generator(seed, 3)
    out = []
    for d in _dims(case):
        U = torch.randn((d, case["R"]), generator=g, device="cuda", dtype=torch.float64)
        out.append(U / torch.sqrt((U * U).sum(dim=0)))
    return out


def _uniforms(case, seed):
    """Uniforms of one sweep: N per-step blocks."""
    N, J = len(_dims(case)), case["J"]
    shape = (N, N, 2, J) if case["sampler"] == "sts_cp" else (N, N, J)
    return torch.rand(shape, generator=_generator(seed, 4), device="cuda", dtype=torch.float64)


def _gcp_dtype(case):
    return torch.float64 if case["precision"] == "fp64" else torch.float32


def _entry_counts(case):
    return case["J"] // 2, case["J"] - case["J"] // 2


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
def prepare(case, seed):
    dims = _dims(case)
    idx, vals = _tensor(case, seed)
    if case["kind"] == "gcp":
        model = gcp.GCP(idx, vals, dims, rank=case["R"], loss=case["loss"], dtype=_gcp_dtype(case), seed=int(seed))
        return {"kind": "gcp", "model": model, "counts": _entry_counts(case)}
    tg = TensorGrid(dims, Grid(np.ones(len(dims), dtype=np.int32)))
    st = SparseTensor(tg, idx, vals, "none")
    lr = LowRankTensor(case["R"], tg)
    start = _factors(case, seed)
    lr.set_factors(start)
    state = {"kind": case["kind"], "tensor": st, "lr": lr, "J": case["J"], "N": len(dims)}
    if case["kind"] == "exact":
        state["opt"] = ExactALS(st, lr)
        state["opt"].initialize_ground_truth_for_als()
        return state
    sampler = CP_ARLS_LEV(lr) if case["sampler"] == "cp_arls_lev" else STS_CP(lr)
    state["uniforms"] = _uniforms(case, seed)
    opt = AccumulatorStationary(st, lr, sampler, max_samples=case["J"], precision=case["precision"])
    state["opt"] = opt
    if case["kind"] == "setup":
        state["start"] = start
        return state
    opt.initialize_ground_truth_for_als()
    if case["tensor"] == "zipf":
        # the exact preprocessing round: from random factors the sampled
        # fibres of a skewed tensor are empty
        for n in range(len(dims)):
            opt.exact_step(n)
    return state


def run(state):
    if state["kind"] == "gcp":
        model = state["model"]
        f = model.step(*state["counts"])
        return {"objective": f, "gradients": [U.grad for U in model.factors]}
    opt, lr = state["opt"], state["lr"]
    if state["kind"] == "exact":
        for n in range(state["N"]):
            opt.execute_ALS_step(n)
        fit = opt.compute_exact_fit()
        return {"factors": [f.data for f in lr.factors], "sigma": lr.sigma, "fit": fit}
    if state["kind"] == "setup":
        lr.set_factors(state["start"])
        opt.initialize_ground_truth_for_als()
        for n in range(state["N"]):
            opt.exact_step(n)
        opt.execute_ALS_step(0, state["J"], state["uniforms"][0])
        out = {"factor": lr.factors[0].data, "sigma": lr.sigma, "norm": opt.tensor_norm}
        opt.deinitialize()
        return out
    opt.execute_sweeps(1, state["J"], state["uniforms"])
    return {"factors": [f.data for f in lr.factors], "sigma": lr.sigma}


# ---------------------------------------------------------------------------
# the work a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    dims, R, J, nnz = _dims(case), case["R"], case["J"], case["nnz"]
    N = len(dims)
    rows = sum(dims)
    if case["kind"] == "gcp":
        es = 8 if case["precision"] == "fp64" else 4
        # parameters and moments read and written, gradients written; the
        # sampled entries' coordinates, values and factor rows read
        return {"bytes": es * rows * R * 7 + J * (4 * N + 2 * es + N * R * es), "flops": J * R * (N * N + N) + 12 * rows * R}
    if case["kind"] == "exact":
        # per mode and for the fit: coordinates and values once, the factors
        # read and one written
        return {"bytes": (N + 1) * nnz * (4 * N + 8) + 8 * R * rows * (N + 2),
                "flops": float(nnz) * R * (N * N + N + 1) + 4.0 * R * R * rows}
    hit = J * (8 * R + 4 * N + 16)  # a step's samples, weights and design rows
    if case["sampler"] == "sts_cp":
        # one quadratic form per tree level of the N - 1 eigen and row trees
        levels = sum(math.log2(max(R, 2)) + math.log2(max(d / R, 1)) + 1 for d in dims) * (N - 1)
        flops = J * levels * R * (R + 1.0) + N * J * R * (R + N)
        uniforms = 2 * N * J * 8
    else:
        flops = N * J * R * (R + N) + 4.0 * R * R * min(rows, N * J)
        uniforms = N * J * 8
    if case["kind"] == "setup":
        # coordinates and values once, the per-mode sorted copies written once
        return {"bytes": (N + 1) * nnz * (4 * N + 8) + N * nnz * 12 + 8 * R * rows * (N + 2) + uniforms + hit,
                "flops": float(nnz) * R * N * N + flops / N + 4.0 * rows * R * R}
    touched = sum(min(d, J) for d in dims)
    return {"bytes": N * (uniforms + hit) + 16 * R * touched, "flops": flops}


# ---------------------------------------------------------------------------
# the same passes in 64 bits, plain torch
# ---------------------------------------------------------------------------
def _pinv(G, cut):
    lam, V = torch.linalg.eigh(G)
    inv = torch.where(lam > cut, 1.0 / lam, torch.zeros_like(lam))
    return (V * inv) @ V.T


def _off_mode_key(idx, dims, n):
    key = torch.zeros(idx.shape[0], dtype=torch.int64, device=idx.device)
    for k in range(len(dims)):
        if k != n:
            key = key * dims[k] + idx[:, k].long()
    return key


def _hadamard(grams, skip):
    out = torch.ones_like(grams[0])
    for k, G in enumerate(grams):
        if k != skip:
            out = out * G
    return out


def _normalised(U):
    sigma = torch.sqrt((U * U).sum(dim=0))
    return U / sigma, sigma


def _exact_mttkrp(dims, idx, vals, U, n):
    M = torch.zeros((dims[n], U[0].shape[1]), dtype=torch.float64, device="cuda")
    for a in range(0, idx.shape[0], 1 << 21):
        part = idx[a:a + (1 << 21)].long()
        p = vals[a:a + (1 << 21), None].clone().expand(-1, U[0].shape[1])
        for k in range(len(dims)):
            if k != n:
                p = p * U[k][part[:, k]]
        M.index_add_(0, part[:, n], p)
    return M


def _exact_als_mode(dims, idx, vals, U, n):
    grams = [u.T @ u for u in U]
    return _normalised(_exact_mttkrp(dims, idx, vals, U, n) @ _pinv(_hadamard(grams, n), 1e-11))


def _arls_draw(dims, U, grams, n, J, uni):
    s = torch.zeros((J, len(dims)), dtype=torch.int64, device="cuda")
    logw = torch.full((J,), -math.log(J), dtype=torch.float64, device="cuda")
    for k in range(len(dims)):
        if k == n:
            continue
        score = ((U[k] @ _pinv(grams[k], 1e-11)) * U[k]).sum(dim=1)
        total = score.sum()
        cdf = torch.cumsum(score / total, dim=0)
        s[:, k] = torch.searchsorted(cdf, uni[k].contiguous()).clamp_(max=dims[k] - 1)
        logw += torch.log(total) - torch.log(score[s[:, k]])
    return s, torch.exp(logw)


def _sts_draw(dims, U, grams, n, J, uni):
    N, R = len(dims), U[0].shape[1]
    chain, last = [None] * N, torch.ones_like(grams[0])
    for k in range(N - 1, -1, -1):
        if k != n:
            last = grams[k] * last
            chain[k] = last
    lam, V = torch.linalg.eigh(chain[1 if n == 0 else 0])
    W = torch.where(lam > 1e-8, V / torch.sqrt(lam.clamp(min=1e-300)), torch.zeros_like(V)).flip(1)
    Phi = W @ W.T
    rows_of = [None] * N + [W.T.contiguous()]
    for k in range(1, N):
        if k != n:
            lam, V = torch.linalg.eigh(chain[k] * Phi)
            rows_of[k] = (V * torch.sqrt(lam.clamp(min=0.0))).T.contiguous()
    s = torch.zeros((J, N), dtype=torch.int64, device="cuda")
    h = torch.ones((J, R), dtype=torch.float64, device="cuda")
    for k in range(N):
        if k == n:
            continue
        nxt = k + 1 if k + 1 != n else k + 2
        E = rows_of[min(nxt, N)]
        mass = torch.stack([((h * E[v]) @ grams[k] * (h * E[v])).sum(dim=1) for v in range(R)], dim=1)
        cum = torch.cumsum(mass, dim=1)
        v = torch.searchsorted(cum, (uni[k, 0] * cum[:, -1])[:, None]).clamp_(max=R - 1)[:, 0]
        x = h * E[v]
        step = max(1, (1 << 27) // dims[k])
        for a in range(0, J, step):
            cum = torch.cumsum((x[a:a + step] @ U[k].T) ** 2, dim=1)
            s[a:a + step, k] = torch.searchsorted(cum, (uni[k, 1, a:a + step] * cum[:, -1])[:, None]).clamp_(
                max=dims[k] - 1)[:, 0]
        h = h * U[k][s[:, k]]
    return s, R / (J * ((h @ Phi) * h).sum(dim=1))


def _sampled_mode(dims, idx, vals, U, grams, n, J, uni, sampler):
    s, w = (_sts_draw if sampler == "sts_cp" else _arls_draw)(dims, U, grams, n, J, uni)
    D = torch.ones((J, U[0].shape[1]), dtype=torch.float64, device="cuda")
    for k in range(len(dims)):
        if k != n:
            D = D * U[k][s[:, k]]
    P = _pinv((D * w[:, None]).T @ D, 1e-11)
    keys, order = torch.sort(_off_mode_key(idx, dims, n))
    uniq, inverse = torch.unique(_off_mode_key(s, dims, n), return_inverse=True)
    rows = torch.zeros((uniq.numel(), D.shape[1]), dtype=torch.float64, device="cuda")
    rows.index_add_(0, inverse, D * w[:, None])  # equal samples share one design row
    lo, hi = torch.searchsorted(keys, uniq), torch.searchsorted(keys, uniq, right=True)
    owner = torch.repeat_interleave(torch.arange(uniq.numel(), device="cuda"), hi - lo)
    starts = torch.cumsum(hi - lo, dim=0) - (hi - lo)
    nz = order[lo[owner] + torch.arange(owner.numel(), device="cuda") - starts[owner]]
    M = torch.zeros((dims[n], D.shape[1]), dtype=torch.float64, device="cuda")
    for a in range(0, nz.numel(), 1 << 21):
        part = nz[a:a + (1 << 21)]
        M.index_add_(0, idx[part, n].long(), rows[owner[a:a + (1 << 21)]] * vals[part, None])
    return _normalised(M @ P)


def _words(counter_low, counter, salt, seed):
    """Four 32-bit words of Philox4x32-10 (Salmon, Moraes, Dror, Shaw, 2011) as int64 tensors."""
    mask = 0xffffffff
    c = [counter_low & mask, counter_low >> 32, torch.full_like(counter_low, counter & mask),
         torch.full_like(counter_low, ((counter >> 32) ^ salt) & mask)]
    k0, k1 = seed & mask, (seed >> 32) & mask

    def mul(a, m):  # 32 x 32 -> (high, low), in pieces that stay below 2^63
        low, high = a * (m & 0xffff), a * (m >> 16)
        low = low + ((high & 0xffff) << 16)
        return ((high >> 16) + (low >> 32)) & mask, low & mask

    for _ in range(10):
        h0, l0 = mul(c[0], 0xD2511F53)
        h1, l1 = mul(c[2], 0xCD9E8D57)
        c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    return c


def _entries(case, idx, vals, seed):
    """The first step's stratified sample: uniform nonzeros, then uniform coordinates taken as zeros."""
    dims, (nz, z) = _dims(case), _entry_counts(case)
    j = torch.arange(nz + z, device="cuda")
    r0, r1 = _words(j, 0, 0x9E3779B9, seed), _words(j, 0, 0x7F4A7C15, seed)
    nnz = idx.shape[0]
    e = ((r0[0][:nz] % nnz) * ((1 << 32) % nnz) + r0[1][:nz]) % nnz  # 64 random bits modulo nnz
    words = r0 + r1
    zero = torch.stack([((words[k][nz:] << 21) ^ words[(k + 4) & 7][nz:]) % dims[k] for k in range(len(dims))], dim=1)
    rows = torch.cat([idx[e].long(), zero])
    x = torch.cat([vals[e].double(), torch.zeros(z, dtype=torch.float64, device="cuda")])
    total = math.prod(float(d) for d in dims)
    w = torch.cat([torch.full((nz,), nnz / nz, dtype=torch.float64, device="cuda"),
                   torch.full((z,), max(total - nnz, 0.0) / z, dtype=torch.float64, device="cuda")])
    return rows, x, w


def exact(case, seed):
    dims, N = _dims(case), len(_dims(case))
    idx, vals = _tensor(case, seed)
    if case["kind"] == "gcp":
        g = torch.Generator(device="cuda")
        g.manual_seed(int(seed))
        dt = _gcp_dtype(case)
        U = [torch.rand((d, case["R"]), generator=g, dtype=dt, device="cuda").mul_(0.5).double() for d in dims]
        rows, x, w = _entries(case, idx, vals, int(seed))
        gathered = [U[k][rows[:, k]] for k in range(N)]
        m = math.prod(gathered[1:], start=gathered[0]).sum(dim=1)
        eps = 1e-10
        if case["loss"] == "poisson":
            f, d = m - x * torch.log(m + eps), 1.0 - x / (m + eps)
        elif case["loss"] == "bernoulli":
            f, d = torch.log(m + 1.0) - x * torch.log(m + eps), 1.0 / (m + 1.0) - x / (m + eps)
        else:
            f, d = (x - m) ** 2, 2.0 * (m - x)
        grads = []
        for n in range(N):
            p = (w * d)[:, None]
            for k in range(N):
                if k != n:
                    p = p * gathered[k]
            grads.append(torch.zeros_like(U[n]).index_add_(0, rows[:, n], p))
        return {"objective": (w * f).sum(), "gradients": grads}
    U, sigma = _factors(case, seed), None
    if case["kind"] == "exact":
        for n in range(N):
            U[n], sigma = _exact_als_mode(dims, idx, vals, U, n)
        grams = [u.T @ u for u in U]
        model2 = (_hadamard(grams, -1) * torch.outer(sigma, sigma)).sum()
        m = _model_values(idx, [U[0] * sigma] + U[1:])
        fit = 1.0 - torch.sqrt(model2 + (vals * vals - 2.0 * vals * m).sum()) / torch.sqrt((vals * vals).sum())
        return {"factors": U, "sigma": sigma, "fit": float(fit)}
    if case["sampler"] == "sts_cp" and (case["precision"] != "fp64" or case["J"] * case["R"] * sum(dims) * N > 1e12):
        # the mixed forms draw other samples of the same distribution
        return None
    uni = _uniforms(case, seed)
    if case["tensor"] == "zipf":
        for n in range(N):
            U[n], sigma = _exact_als_mode(dims, idx, vals, U, n)
    if case["kind"] == "setup":
        U[0], sigma = _sampled_mode(dims, idx, vals, U, [u.T @ u for u in U], 0, case["J"], uni[0], case["sampler"])
        return {"factor": U[0], "sigma": sigma, "norm": float(torch.sqrt((vals * vals).sum()))}
    if case["precision"] != "fp64":
        # the first update only: the draws of the later ones follow scores
        # that the mixed forms hold to 32 bits, and are other samples
        U[0], sigma = _sampled_mode(dims, idx, vals, U, [u.T @ u for u in U], 0, case["J"], uni[0], case["sampler"])
        return {"factors": [U[0]] + [None] * (N - 1), "sigma": None}
    for n in range(N):
        U[n], sigma = _sampled_mode(dims, idx, vals, U, [u.T @ u for u in U], n, case["J"], uni[n], case["sampler"])
    return {"factors": U, "sigma": sigma}
