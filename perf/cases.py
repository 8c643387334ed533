"""Workloads of the fitting library for timing and numerical comparison.

Each case is one pass a program makes through the public Python API
(``fastpls_b200.api``), on host arrays as that API takes them:

* fits of one model (SIMPLS, PLS-SVD with LDA, OPLS, kernel PLS) with the
  exports and held-out predictions a program reads afterwards;
* predictions of new rows by a resident model;
* cross-validation of one response matrix, and cross-validation repeated over
  row permutations of the responses or labels;
* a truncated SVD.

``listed()`` are fixed sizes, ``draw`` gives others of the same ranges,
``exact`` restates the results in FP64 with plain torch. Inputs follow the
latent factor model of the library's benchmark: X = T W^T + noise with
decreasing factor scales, Y = T C + noise, labels = argmax(T C), drawn on the
GPU from the seed and handed over as host arrays.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from fastpls_b200 import api

DEV = "cuda" if torch.cuda.is_available() else "cpu"


# ---------------------------------------------------------------- cases
def _fit(n, p, q, a, bits, scaling="centering", name=None):
    return dict(kind="fit", n=n, p=p, q=q, a=a, bits=bits, scaling=scaling, name=name)


def listed():
    return [
        # one interactive fit of a small assay: launches, copies and host work
        _fit(97, 311, 1, 4, 64, name="fit_small"),
        # the fold fit of the benchmark (5000 x 10000, 10 folds) as a fit of its own
        _fit(4513, 10000, 3, 20, 32, name="fit_fold"),
        # many components on wide BF16 predictors, past the size one launch holds
        _fit(30011, 10000, 10, 50, 16, name="fit_bf16"),
        # a tall classification fit (more than 8 rows per predictor)
        dict(name="fit_classes", kind="classes", n=40003, p=500, classes=12, a=10, bits=32,
             scaling="autoscaling"),
        # PLS-SVD with the LDA head, labels of held-out rows along the prefixes
        dict(name="plssvd_lda", kind="plssvd", n=20000, p=10000, classes=10, a=9, bits=32,
             scaling="centering"),
        # new rows through a resident model along a component path
        dict(name="predict", kind="predict", rows=4001, p=4000, q=3, a=12, bits=32,
             scaling="autoscaling"),
        # ordinary 10-fold cross-validation of an autoscaled assay, predictions kept
        dict(name="cv", kind="cv", n=601, p=1500, q=2, a=8, folds=10, bits=64,
             scaling="autoscaling"),
        # the benchmark: 10 folds x (1 + 200) response permutations, path 1..20
        dict(name="perm", kind="perm", n=5000, p=10000, q=3, a=20, folds=10, perms=200, bits=32,
             scaling="centering"),
        # permutation test of a classifier on an ordinary assay
        dict(name="perm_classes", kind="permc", n=803, p=3001, classes=5, a=8, folds=7, perms=99,
             bits=32, scaling="centering"),
        # OPLS with two orthogonal filters
        dict(name="opls", kind="opls", n=1501, p=4000, q=1, a=4, north=2, bits=64,
             scaling="autoscaling"),
        # RBF kernel PLS with held-out predictions
        dict(name="kernel", kind="kernel", n=2001, p=1000, q=2, a=6, bits=32,
             scaling="autoscaling", kernel="rbf"),
        # truncated SVD of a tall matrix
        dict(name="svd", kind="svd", n=3001, p=1200, k=8, bits=64),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cost(case):
    w = work(case)
    return max(w["bytes"], w["flops"] / 50)


def draw(rng):
    cap = max(_cost(c) for c in listed())
    while True:
        kind = rng.choice(["fit", "classes", "plssvd", "predict", "cv", "perm", "permc", "opls",
                           "kernel", "svd"])
        scaling = rng.choice(["centering", "autoscaling"])
        bits = rng.choice([32, 64])
        if kind == "fit":
            bits = rng.choice([16, 32, 64])
            n, p = _log(rng, 50, 30000), _log(rng, 100, 20000)
            a = rng.randint(2, min({16: 50, 32: 20, 64: 10}[bits], n // 3, p // 3))
            c = _fit(n, p, rng.randint(1, 10), a, bits, scaling)
            del c["name"]
            big = n * p > {16: 3.0e8, 32: 1.0e8, 64: 4.0e7}[bits]
        elif kind == "classes":
            n, p, classes = _log(rng, 2000, 40000), _log(rng, 60, 2000), rng.randint(4, 16)
            c = dict(kind=kind, n=n, p=p, classes=classes, a=rng.randint(3, classes - 1),
                     bits=bits, scaling=scaling)
            big = n * p > 4.0e7
        elif kind == "plssvd":
            n, p, classes = _log(rng, 300, 20000), _log(rng, 500, 20000), rng.randint(3, 12)
            c = dict(kind=kind, n=n, p=p, classes=classes, a=rng.randint(2, classes - 1),
                     bits=bits, scaling=scaling)
            big = n * p > (2.0e8 if bits == 32 else 5.0e7)
        elif kind == "predict":
            c = dict(kind=kind, rows=_log(rng, 1, 4000), p=_log(rng, 200, 10000),
                     q=rng.randint(1, 8), a=rng.randint(2, 20), bits=bits, scaling=scaling)
            big = False
        elif kind == "cv":
            c = dict(kind=kind, n=_log(rng, 80, 1200), p=_log(rng, 100, 3000), q=rng.randint(1, 3),
                     a=rng.randint(3, 10), folds=rng.randint(5, 10), bits=bits, scaling=scaling)
            big = False
        elif kind == "perm":
            c = dict(kind=kind, n=_log(rng, 150, 5000), p=_log(rng, 200, 10000),
                     q=rng.randint(1, 3), a=rng.randint(4, 20), folds=rng.randint(5, 10),
                     perms=rng.randint(20, 200), bits=bits, scaling=scaling)
            big = scaling == "autoscaling" and c["n"] > 2500
        elif kind == "permc":
            c = dict(kind=kind, n=_log(rng, 150, 2000), p=_log(rng, 200, 5000),
                     classes=rng.randint(3, 6), a=rng.randint(3, 10), folds=rng.randint(5, 8),
                     perms=rng.randint(20, 150), bits=bits, scaling=scaling)
            big = False
        elif kind == "opls":
            c = dict(kind=kind, n=_log(rng, 100, 3000), p=_log(rng, 200, 8000),
                     q=rng.randint(1, 2), a=rng.randint(2, 5), north=rng.randint(1, 3), bits=bits,
                     scaling=scaling)
            big = False
        elif kind == "kernel":
            c = dict(kind=kind, n=_log(rng, 150, 2500), p=_log(rng, 50, 2000), q=rng.randint(1, 3),
                     a=rng.randint(2, 6), bits=32, scaling="autoscaling",
                     kernel=rng.choice(["rbf", "poly"]))
            big = False
        else:
            c = dict(kind=kind, n=_log(rng, 200, 4000), p=_log(rng, 100, 2000),
                     k=rng.randint(3, 12), bits=bits)
            big = False
        if not big and _cost(c) <= cap:
            return c


def _rows_new(case):
    """Held-out rows a fit case predicts afterwards."""
    return max(5, min(2000, case["n"] // 10))


def work(case):
    """Bytes: predictors, responses and results once. Flops: the products of
    the method in FP64 (cross-product, two per component, projections)."""
    k, es = case["kind"], case["bits"] // 8
    ro = 8 if case["bits"] == 64 else 4
    if k == "predict":
        m, p, q, a = case["rows"], case["p"], case["q"], case["a"]
        return {"bytes": m * p * es + ro * m * q * len(_prefixes(a)), "flops": 2 * m * p * a}
    n, p = case["n"], case["p"]
    if k == "svd":
        kk = case["k"]
        return {"bytes": n * p * es + 8 * kk * (n + p + 1), "flops": 4 * n * p * kk}
    q, a = case.get("q", case.get("classes", 0)), case["a"]
    inst = case.get("folds", 1) * (1 + case.get("perms", 0))
    if k in ("perm", "permc"):
        # one Gram, then two products with it per component and instance
        grams = case["folds"] if case["scaling"] == "autoscaling" else 1
        return {"bytes": n * p * es + n * q * es + 8 * (1 + case["perms"]) * a * 4,
                "flops": grams * n * (n + 1) * p + inst * a * 4 * n * n}
    if k == "cv":
        return {"bytes": n * p * es + n * q * es * (1 + a),
                "flops": case["folds"] * (2 * n * p * q + 4 * n * p * a)}
    new = _rows_new(case)
    out = ro * (p * a + n * a + q * a + new * q * len(_prefixes(a)))
    flops = 2 * n * p * q + 2 * new * p * a + (2 if k == "plssvd" else 4) * n * p * a
    if k == "opls":
        flops += case["north"] * (8 + 2 * q) * n * p
    if k == "kernel":
        flops = n * (n + 1) * p + 2 * new * n * p + 2 * n * n * q + 4 * n * n * a + 2 * new * n * a
        out = ro * (2 * n * a + q * a + new * q * len(_prefixes(a)))
    return {"bytes": (n + new) * p * es + n * q * ro + out, "flops": flops}


# ---------------------------------------------------------------- inputs
def _prefixes(a):
    return sorted({1, (a + 2) // 3, (2 * a + 2) // 3, a})


class _Draws:
    """The arrays of one case, drawn on the GPU from the seed."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEV).manual_seed(int(seed))

    def normal(self, *shape):
        return torch.randn(*shape, generator=self.g, device=DEV)

    def order(self, n):
        return torch.randperm(n, generator=self.g, device=DEV)


def _scales(k):
    """Decreasing factor scales, 1 down to 0.3."""
    return 0.3 ** (torch.arange(k, device=DEV, dtype=torch.float32) / k)


def _latent(d, n, p, k, noise=0.5):
    """Scores T (n x k, decreasing scales) and X^T (p x n)."""
    t = d.normal(n, k) * _scales(k)
    w = d.normal(p, k)
    xt = w @ t.T
    step = max(1, 200_000_000 // max(n, 1))
    for j in range(0, p, step):
        xt[j:j + step] += noise * d.normal(min(step, p - j), n)
    return t, xt


def _host(xt, bits):
    """The n x p column-major host matrix of X^T (p x n) in storage type."""
    if bits == 16:
        return xt.to(torch.bfloat16).view(torch.int16).cpu().numpy().view(np.uint16).T
    return xt.to(torch.float64 if bits == 64 else torch.float32).cpu().numpy().T


def _out_bits(bits):
    return 64 if bits == 64 else 32


def _folds(d, n, k):
    """Uneven folds: sizes spread by a few rows around n / k."""
    f = torch.empty(n, dtype=torch.int32, device=DEV)
    edges = [0] + [min(n - (k - i), max(i, i * n // k + (-1) ** i * (n // (40 * k)))) for i in range(1, k)] + [n]
    o = d.order(n)
    for i in range(k):
        f[o[edges[i]:edges[i + 1]]] = i + 1
    return f.cpu().numpy()


def _inputs(case, seed):
    d = _Draws(seed)
    kind, bits = case["kind"], case["bits"]
    s = {}
    if kind == "predict":
        n, new = 300, case["rows"]
    else:
        n = case["n"]
        new = _rows_new(case) if kind in ("fit", "classes", "plssvd", "opls", "kernel") else 0
    p = case["p"]
    if kind == "svd":
        _, xt = _latent(d, n, p, case["k"] + 4, noise=0.2)
        s["x"] = _host(xt, bits)
        return s
    a = case["a"]
    factors = {"perm": 10, "permc": case.get("classes", 0) + 2}.get(kind, a + case.get("north", 0) + 2)
    if kind in ("classes", "plssvd"):
        factors = case["classes"] + 4
    if kind == "kernel":
        factors = max(4, a)
    t, xt = _latent(d, n + new, p, factors, noise=0.3 if kind == "perm" else 0.5)
    if "classes" in case:
        c = d.normal(factors, case["classes"]) / _scales(factors)[:, None]
        s["labels"] = (torch.argmax(t @ c, dim=1)[:n] + 1).to(torch.int32).cpu().numpy()
    else:
        c = d.normal(factors, case["q"])
        y = t @ c + 0.1 * d.normal(n + new, case["q"])
        if kind == "kernel":
            y = y + 0.5 * (t[:, :1] ** 2)
        s["y"] = _host(y[:n].T.contiguous(), _out_bits(bits))
    s["x"] = _host(xt[:, :n].contiguous(), bits)
    if new:
        s["new"] = _host(xt[:, n:].contiguous(), bits)
    if "folds" in case:
        s["folds"] = _folds(d, n, case["folds"])
    if "perms" in case:
        s["perms"] = torch.stack([d.order(n) for _ in range(case["perms"])]).to(torch.int32).cpu().numpy()
    return s


def prepare(case, seed):
    s = _inputs(case, seed)
    s["case"] = case
    if case["kind"] == "predict":
        s["model"] = api.fit_resident(s["x"], s["y"], ncomp=case["a"], scaling=case["scaling"],
                                      precision=case["bits"])
    return s


# ---------------------------------------------------------------- one pass
def _read(model, s, a):
    out = {"R": model.weights(), "Q": model.loadings(), "T": model.scores(),
           "new": model.predict_path(s["new"], _prefixes(a))}
    model.close()
    return out


def run(s):
    c = s["case"]
    k = c["kind"]
    if k == "svd":
        u, d, v = api.fastsvd(s["x"], c["k"], precision=c["bits"])
        return {"u": u, "d": d, "v": v}
    a, sc, bits = c["a"], c["scaling"], c["bits"]
    path = list(range(1, a + 1))
    if k == "fit":
        return _read(api.fit_resident(s["x"], s["y"], ncomp=a, scaling=sc, precision=bits), s, a)
    if k == "classes":
        return _read(api.fit_resident(s["x"], labels=s["labels"], classes=c["classes"], ncomp=a,
                                      scaling=sc, precision=bits), s, a)
    if k == "plssvd":
        m = api.fit_resident(s["x"], labels=s["labels"], classes=c["classes"], ncomp=a,
                             scaling=sc, method="plssvd", precision=bits)
        labels = m.classify_path(s["new"], _prefixes(a), lda=True)
        return {"labels": labels, **_read(m, s, a)}
    if k == "predict":
        return {"new": s["model"].predict_path(s["new"], _prefixes(a))}
    if k == "cv":
        return api.cv_regression(s["x"], s["y"], s["folds"], path, scaling=sc, precision=bits,
                                 store_predictions=True)
    if k == "perm":
        return api.cv_permutation(s["x"], s["y"], s["folds"], s["perms"], path, scaling=sc,
                                  precision=bits)
    if k == "permc":
        return api.cv_permutation_classification(s["x"], s["labels"], c["classes"], s["folds"],
                                                 s["perms"], path, scaling=sc, precision=bits)
    if k == "opls":
        return _read(api.fit_resident(s["x"], s["y"], ncomp=a, scaling=sc, method="opls",
                                      north=c["north"], precision=bits), s, a)
    return _read(api.fit_resident(s["x"], s["y"], ncomp=a, scaling=sc, method="kernelpls",
                                  kernel=c["kernel"], precision=bits, degree=2, coef0=1.0), s, a)


# ---------------------------------------------------------------- FP64 results
def _f64(x):
    if x.dtype == np.uint16:
        return torch.from_numpy(np.ascontiguousarray(x.T).view(np.int16)).to(DEV).view(torch.bfloat16).double().T
    return torch.from_numpy(np.ascontiguousarray(x.T)).to(DEV).double().T


def _standard(x, scaling):
    mean = x.mean(0)
    scale = torch.ones_like(mean)
    if scaling == "autoscaling":
        scale = (x - mean).square().sum(0).div(max(x.shape[0] - 1, 1)).sqrt()
        scale = torch.where(scale > 0, scale, torch.ones_like(scale))
    return mean, scale


def _pairs(S):
    """Eigenvalues (decreasing) and vectors of S^T S, the largest entry of
    each vector positive. S: (B, p, q)."""
    lam, z = torch.linalg.eigh(S.mT @ S)
    lam, z = lam.flip(-1), z.flip(-1)
    top = z.gather(-2, z.abs().argmax(-2, keepdim=True))
    return lam, z * torch.sign(top)


def _simpls(xs, yc, a, block=1):
    """SIMPLS of standardised xs (n x p) on centred yc (B x n x q): R, Q, T
    (B x rows x a). block: directions taken from one decomposition."""
    S = xs.T @ yc
    S0 = S
    B, p, q = S.shape
    R, Q, T, V = (torch.zeros(B, m, a, dtype=torch.float64, device=xs.device)
                  for m in (p, q, xs.shape[0], p))
    use = j = 0
    for k in range(a):
        if j == use:
            use, j, Sb = min(block, a - k), 0, S
            lam, z = _pairs(S)
        r = (Sb @ z[..., j:j + 1])[..., 0] / lam[..., j:j + 1].sqrt()
        j += 1
        t = (xs @ r.T).T
        tn = t.norm(dim=-1, keepdim=True)
        r, t = r / tn, t / tn
        v = (xs.T @ t.T).T
        v = v - (V[..., :k] @ (V[..., :k].mT @ v[..., None]))[..., 0]
        v = v / v.norm(dim=-1, keepdim=True)
        R[..., k], T[..., k], V[..., k] = r, t, v
        Q[..., k] = (S0.mT @ r[..., None])[..., 0]
        S = S - v[..., None] @ (v[:, None, :] @ S)
    return R, Q, T


def _responses(s, case, rows=None):
    if "labels" in s:
        lab = torch.from_numpy(s["labels"]).to(DEV).long() - 1
        return torch.nn.functional.one_hot(lab, case["classes"]).double()
    return _f64(s["y"])


def _laid_out(R, Q, T, ymean, xnew, a, weights=None):
    """The outputs of _read, with per-prefix weights in the place of R Q^T."""
    t = xnew @ R
    new = [ymean + (t[:, :k] @ (weights[k] if weights else Q[:, :k].T)) for k in _prefixes(a)]
    return {"R": R, "Q": Q, "T": T, "new": torch.stack(new)}


def _host_all(out):
    return {k: None if v is None else v.cpu().numpy() for k, v in out.items()}


def _fold_paths(s, case, ys):
    """Per fold: held-out rows, held-out predictions (a x B x rows x q) and
    the training means (B x q) of the responses ys (B x n x q)."""
    x, folds = _f64(s["x"]), torch.from_numpy(s["folds"]).to(DEV)
    a = case["a"]
    for f in range(1, case["folds"] + 1):
        tr, te = (folds != f).nonzero()[:, 0], (folds == f).nonzero()[:, 0]
        mean, scale = _standard(x[tr], case["scaling"])
        xs = (x[tr] - mean) / scale
        ym = ys[:, tr].mean(1)
        q = ys.shape[-1]
        big = "classes" in case and a >= 4 and len(tr) * case["p"] * q >= 5e8
        R, Q, _ = _simpls(xs, ys[:, tr] - ym[:, None], a, min(a, q) if big else 1)
        t = torch.einsum("np,bpa->bna", (x[te] - mean) / scale, R)
        yield te, torch.cumsum(torch.einsum("bna,bqa->abnq", t, Q), 0) + ym[:, None], ym


def _metrics(s, case, ys):
    B, n, q = ys.shape
    sse = torch.zeros(B, case["a"], dtype=torch.float64, device=ys.device)
    fss = torch.zeros(B, 1, dtype=torch.float64, device=ys.device)
    pred = torch.zeros(case["a"], B, n, q, dtype=torch.float64, device=ys.device) if B == 1 else None
    for te, yh, ym in _fold_paths(s, case, ys):
        sse += (ys[:, te] - yh).square().sum((-1, -2)).T
        fss += (ys[:, te] - ym[:, None]).square().sum((-1, -2))[:, None]
        if pred is not None:
            pred[:, :, te] = yh
    total = (ys[0] - ys[0].mean(0)).square().sum()
    q2 = 1 - sse / fss
    return {"metrics": q2, "q2": q2, "rmsd": (sse / (n * q)).sqrt(), "observed_r2": 1 - sse / total,
            "status": None}, pred


def exact(case, seed):
    s = _inputs(case, seed)
    k = case["kind"]
    if k == "svd":
        return _host_all({"u": None, "d": torch.linalg.svdvals(_f64(s["x"]))[:case["k"]], "v": None})
    a = case["a"]
    y = _responses(s, case)
    if k == "cv":
        out, pred = _metrics(s, case, y[None])
        out = {key: v if v is None else v[0] for key, v in out.items()}
        return _host_all({**out, "predictions": pred[:, 0]})
    if k in ("perm", "permc"):
        rows = torch.cat([torch.arange(len(y))[None], torch.from_numpy(s["perms"]).long()]).to(DEV)
        ys = y[rows]
        if k == "perm":
            return _host_all(_metrics(s, case, ys)[0])
        hits = torch.zeros(len(ys), a, dtype=torch.float64, device=DEV)
        for te, yh, ym in _fold_paths(s, case, ys):
            yh = yh.masked_fill((ym <= 0)[None, :, None], -math.inf)
            hits += (yh.argmax(-1) == ys[:, te].argmax(-1)).double().sum(-1).T
        return _host_all({"accuracy": hits / len(y), "status": None})
    x, new = _f64(s["x"]), _f64(s["new"])
    mean, scale = _standard(x, case["scaling"])
    xs, xn = (x - mean) / scale, (new - mean) / scale
    ym = y.mean(0)
    yc = y - ym
    if k == "plssvd":
        S = xs.T @ yc
        lam, z = _pairs(S[None])
        sig, V = lam[0, :a].sqrt(), z[0, :, :a]
        R = S @ V / sig
        T = xs @ R
        W = {j: torch.linalg.solve(T[:, :j].T @ T[:, :j], sig[:j, None] * V[:, :j].T) for j in range(1, a + 1)}
        return _host_all({"labels": None, **_laid_out(R, V, T, ym, xn, a, W)})
    if k == "kernel":
        gamma = 1.0 / case["p"]

        def block(u):
            if case["kernel"] == "rbf":
                d2 = u.square().sum(1)[:, None] + xs.square().sum(1) - 2 * u @ xs.T
                return torch.exp(-gamma * d2.clamp(min=0))
            return (gamma * u @ xs.T + 1.0) ** 2
        K, Kn = block(xs), block(xn)
        col = K.mean(0)
        xs = K - K.mean(1)[:, None] - col + col.mean()
        xn = Kn - Kn.mean(1)[:, None] - col + col.mean()
    filters = []
    for _ in range(case.get("north", 0) if k == "opls" else 0):
        S = xs.T @ yc
        lam, z = _pairs(S[None])
        w = S @ z[0, :, 0] / lam[0, 0].sqrt()
        t = xs @ w
        load = xs.T @ t / (t @ t)
        wo = load - (w @ load) / (w @ w) * w
        wo = wo / wo.norm()
        to = xs @ wo
        po = xs.T @ to / (to @ to)
        xs = xs - torch.outer(to, po)
        filters.append((wo, po))
    n, p = xs.shape
    big = k == "classes" and a >= 4 and n * p * case["classes"] >= 5e8
    R, Q, T = (m[0] for m in _simpls(xs, yc[None], a, min(a, case["classes"]) if big else 1))
    for wo, po in reversed(filters):
        R = R - torch.outer(wo, po @ R)
    if k == "predict":
        return _host_all({"new": _laid_out(R, Q, T, ym, xn, a)["new"]})
    return _host_all(_laid_out(R, Q, T, ym, xn, a))
