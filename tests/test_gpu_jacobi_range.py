"""Responses of very different scales: the Gram of X^T Yc mixes a pair of
entries whose squares underflow (or overflow) with ordinary ones, and the
cyclic Jacobi sweeps over it stay finite and right.

Reference: the SVD of X^T Yc with each response brought to a common scale is
not the same problem, so the leading triplets are taken from numpy's SVD of
the unscaled matrix; the small responses (2^-280: squares of their Gram
entries below 2^-1074) change nothing in them beyond rounding."""
import numpy as np
import pytest

from fastpls_b200 import api, workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q,small", [(4, 2), (5, 3), (9, 4), (20, 7)])
@pytest.mark.parametrize("exponent", [-280, -300, -400])
def test_small_responses_beside_ordinary_ones(q, small, exponent):
    n, p, k = 120, 60, q - small
    x, y = W.latent_regression(n, p, q, q + 2, 0.5, 9 * q + small, dtype=np.float64)
    y = y.copy(order="F")
    # not the last columns alone: pairs of small ones meet in every round
    tiny = np.arange(q)[::-1][:2 * small:2] if 2 * small <= q else np.arange(q)[-small:]
    y[:, tiny] = np.ldexp(y[:, tiny], exponent)
    m = api.fit_resident(x, y, ncomp=k, method="plssvd", precision=64)
    R, Q, pred = m.weights(), m.loadings(), m.predict_path(x[:20], [1, k])
    m.close()
    assert np.isfinite(R).all() and np.isfinite(Q).all() and np.isfinite(pred).all()
    S = (x - x.mean(0)).T @ (y - y.mean(0))
    u, s, vt = np.linalg.svd(S, full_matrices=False)
    # FP64 eigenproblem of S^T S: errors of a vector m 2^-53 s_0^2 / gap of
    # squares; the leading factors here are separated by more than 1e-3
    gap = np.min(np.abs(s[:k] ** 2 - np.append(s[1:k], 0.0) ** 2)) / s[0] ** 2
    tol = 1e3 * q * 2.0 ** -53 / gap
    sign = np.sign((u[:, :k] * R).sum(0))
    assert np.max(np.abs(R * sign - u[:, :k])) <= tol * s[0] / s[k - 1]
    assert np.max(np.abs(Q * sign - vt[:k].T)) <= tol
