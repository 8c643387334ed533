"""fastsvd over sketch widths: the l x l factorisation at warp and row edges."""
import numpy as np
import pytest

from fastpls_b200 import api

pytestmark = pytest.mark.gpu


# widths l = min(k + 1 + oversample, n, p): 6 .. 120
@pytest.mark.parametrize("n,p,k,oversample", [(6, 9, 2, 32), (400, 300, 1, 29), (400, 300, 1, 30),
                                              (400, 300, 1, 31), (301, 200, 30, 32), (33, 500, 5, 40),
                                              (300, 260, 80, 38)])
def test_sketch_widths(n, p, k, oversample):
    rng = np.random.default_rng(n + p + k)
    r = min(n, p)
    qa, _ = np.linalg.qr(rng.standard_normal((n, r)))
    qb, _ = np.linalg.qr(rng.standard_normal((p, r)))
    s = 100.0 * 0.8 ** np.arange(r) + 1e-3
    x = (qa * s) @ qb.T
    u, d, v = api.fastsvd(x, k, oversample=oversample, power=4, seed=3)
    # subspace iteration with 4 rounds: components below the sketch enter as
    # (s_l / s_k)^9; the rest is rounding, l * 2^-53 * s_1 / s_k on vectors
    l = min(k + 1 + oversample, r)
    tail = (s[l] / s[k - 1]) ** 9 if l < r else 0.0
    tol = 1e3 * l * 2.0 ** -53 * (s[0] / s[k - 1]) + 10 * tail
    assert np.max(np.abs(d - s[:k])) <= tol * s[0]
    assert np.max(np.abs(u.T @ u - np.eye(k))) <= tol
    assert np.max(np.abs(v.T @ v - np.eye(k))) <= max(tol, 1e3 * l * 2.0 ** -53 * (s[0] / s[k - 1]) ** 2)
    assert np.linalg.norm(x @ v - u * d) <= tol * s[0] * np.sqrt(k)


def test_sketch_beyond_one_block_is_refused():
    """120 columns: the small eigenproblem's 2 l^2 doubles and its static
    arrays pass one block's shared memory; the call reports it."""
    with pytest.raises(api._lib.FastplsError):
        api.fastsvd(np.random.default_rng(1).standard_normal((300, 260)), 80, oversample=39, power=4)
