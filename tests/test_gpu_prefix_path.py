"""Predictions along a component path: every prefix from one pass over the
scores, projections at the widths where the product changes kernel.

Tolerance: FP64 sums of K products differ by at most 2 (K + 2) u sum |a||b|
between two orders (u = 2^-53); FP32 results add one rounding."""
import numpy as np
import pytest

from fastpls_b200 import api, workloads as W
from oracle import pls_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [64, 32, 16])
@pytest.mark.parametrize("rows,p,q,a", [(1, 65, 1, 1), (127, 64, 2, 2), (129, 1025, 3, 3),
                                        (513, 333, 4, 33), (64, 2500, 5, 66)])
def test_every_prefix_matches_products_of_the_exports(rows, p, q, a, precision):
    n = 260
    x, y = W.latent_regression(n + rows, p, q, 12, 0.5, rows + p, dtype=np.float32)
    y = y.astype(np.float64 if precision == 64 else np.float32)
    xs = api.to_bf16(x) if precision == 16 else x.astype(y.dtype)
    a = min(a, p)
    m = api.fit_resident(np.asfortranarray(xs[:n]), y[:n], ncomp=a, precision=precision, scaling="autoscaling")
    got = m.predict_path(np.asfortranarray(xs[n:]), list(range(1, a + 1)))
    scores = m.project(np.asfortranarray(xs[n:]), a)
    R, Q = m.weights().astype(np.float64), m.loadings().astype(np.float64)
    mu, sd, ym = (m.export(f).astype(np.float64) for f in (3, 4, 5))
    m.close()
    v = (api.from_bf16(xs[n:]).reshape(rows, p) if precision == 16 else xs[n:]).astype(np.float64)
    z = (v - mu) / sd
    t = z @ R
    u = 2.0 ** -53 if precision == 64 else 2.0 ** -23
    # projection: raw X and offset sums, and (FP32) rounded exports
    bound_t = 8 * (p + 4) * 2.0 ** -53 * ((np.abs(v) + np.abs(mu)) / sd) @ np.abs(R) + 4 * u * np.abs(z) @ np.abs(R) + 8 * u * (np.abs(mu) / sd) @ np.abs(R)
    assert np.all(np.abs(scores - t) <= bound_t)
    for k in range(1, a + 1):
        want = ym + t[:, :k] @ Q[:, :k].T
        bound = bound_t[:, :k] @ np.abs(Q[:, :k]).T + 8 * u * (np.abs(ym) + np.abs(t[:, :k]) @ np.abs(Q[:, :k]).T) \
            + 4 * (k + 2) * 2.0 ** -53 * (np.abs(t[:, :k]) @ np.abs(Q[:, :k]).T)
        assert np.all(np.abs(got[k - 1] - want) <= bound)


@pytest.mark.parametrize("classes,a", [(3, 2), (12, 11), (40, 39)])
@pytest.mark.parametrize("method", ["simpls", "plssvd"])
def test_lda_and_response_paths(method, classes, a):
    """LDA terms of all prefixes in one launch (more than 32 of them too),
    labels and responses in FP64 and FP32."""
    x, lab = W.latent_classification(700, 150, classes, classes + 3, 0.6, 31 + classes, dtype=np.float64)
    ok = np.bincount(lab, minlength=classes + 1)[1:] > 1
    keep = ok[lab - 1]
    levels, codes = np.unique(lab[keep], return_inverse=True)
    x, lab, classes = np.asfortranarray(x[keep]), (codes + 1).astype(np.int32), len(levels)
    a = min(a, classes - 1)
    pre = list(range(1, a + 1))
    m = api.fit_resident(x, labels=lab, classes=classes, ncomp=a, method=method, precision=64)
    labels, resp = m.classify_path(x, pre, lda=True, responses=True)
    disc = m.predict_path(x, pre, lda=True)
    plain = m.classify_path(x, pre)
    T = m.scores()
    assert np.array_equal(resp, m.predict_path(x, pre))
    m.close()
    lda = O.lda_train(T, lab, classes, pre)
    for j in range(a):
        want = O.lda_discriminants(lda[j], T)
        # one factorisation against another: the condition number of the
        # ridged covariance times a few roundings
        assert np.allclose(disc[j], want, rtol=1e-8, atol=1e-8 * np.abs(want).max())
        gap = np.sort(want, axis=1)
        clear = gap[:, -1] - gap[:, -2] > 1e-7 * np.abs(want).max()
        assert np.array_equal(labels[j][clear, 0], want.argmax(1)[clear] + 1)
        assert np.array_equal(plain[j][:, 0], resp[j].argmax(1) + 1)
