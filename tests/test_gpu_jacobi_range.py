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


@pytest.mark.parametrize("exponent", [-450, -300, -210, 210, 300])
@pytest.mark.parametrize("q", [3, 12, 40])
def test_plssvd_of_scaled_responses(q, exponent):
    """A power of two on the responses leaves the directions alone: the squares
    of the Gram's entries vanish or pass the range, the entries do not."""
    n, p, k = 120, 60, min(q, 5)
    x, y = W.latent_regression(n, p, q, q + 2, 0.5, q, dtype=np.float64)
    got = []
    for z in (y, np.ldexp(y, exponent)):
        m = api.fit_resident(x, np.asfortranarray(z), ncomp=k, method="plssvd", precision=64)
        got.append((m.weights(), m.loadings(), m.predict_path(x[:9], [1, k])))
        m.close()
    (R0, Q0, y0), (R1, Q1, y1) = got
    # exact scaling up to the rounding of values that leave the normal range
    assert np.max(np.abs(R1 - R0)) <= 1e-12
    assert np.max(np.abs(Q1 - Q0)) <= 1e-12
    assert np.max(np.abs(np.ldexp(y1, -exponent) - y0)) <= 1e-12 * np.max(np.abs(y0))


@pytest.mark.parametrize("exponent", [-300, -210, 210])
def test_svd_of_scaled_matrices(exponent):
    x = np.random.default_rng(2).standard_normal((90, 50)) * 0.7 ** np.arange(50)
    u0, d0, v0 = api.fastsvd(x, 4)
    u, d, v = api.fastsvd(np.ldexp(x, exponent), 4)
    assert np.max(np.abs(np.ldexp(d, -exponent) - d0)) <= 1e-12 * d0[0]
    assert np.max(np.abs(u - u0)) <= 1e-9 and np.max(np.abs(v - v0)) <= 1e-9
