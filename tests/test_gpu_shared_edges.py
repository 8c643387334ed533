"""Orders at which a block's dynamic shared memory is just below 48 KB but not
with its kernel's static arrays beside it: the eigenproblems of PLS-SVD
(2 m^2 doubles, m = 55) and of a sketch (fastsvd, 55 columns)."""
import numpy as np
import pytest

from fastpls_b200 import api, workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [53, 54, 55, 56])
def test_plssvd_responses(m):
    x, y = W.latent_regression(200, 90, m, 60, 0.5, m, dtype=np.float64)
    model = api.fit_resident(x, y, ncomp=3, method="plssvd", precision=64)
    R, Q = model.weights(), model.loadings()
    model.close()
    u, s, vt = np.linalg.svd((x - x.mean(0)).T @ (y - y.mean(0)), full_matrices=False)
    # an eigenvector of S^T S: m 2^-53 s_0^2 over the gap of the squares
    gap = np.min(s[:3] ** 2 - s[1:4] ** 2) / s[0] ** 2
    tol = 1e3 * m * 2.0 ** -53 / gap
    sign = np.sign((u[:, :3] * R).sum(0))
    assert np.max(np.abs(Q * sign - vt[:3].T)) <= tol
    assert np.max(np.abs(R * sign - u[:, :3])) <= tol * s[0] / s[2]


@pytest.mark.parametrize("k", [20, 21, 22, 23])
def test_sketch_columns(k):
    rng = np.random.default_rng(k)
    qa, _ = np.linalg.qr(rng.standard_normal((300, 200)))
    qb, _ = np.linalg.qr(rng.standard_normal((200, 200)))
    s = 100.0 * 0.8 ** np.arange(200) + 1e-3
    u, d, v = api.fastsvd((qa * s) @ qb.T, k, oversample=32, power=4)
    # subspace iteration: the sketch's first dropped factor enters as (s_l / s_k)^9
    l = k + 33
    tol = 1e3 * l * 2.0 ** -53 * (s[0] / s[k - 1]) + 10 * (s[l] / s[k - 1]) ** 9
    assert np.max(np.abs(d - s[:k])) <= tol * s[0]
