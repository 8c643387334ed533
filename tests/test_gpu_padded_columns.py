"""Resident training predictors with padded columns (row counts from 8192 that
are not a multiple of 8): the same model as the padded-free equivalent, every
storage type alike, all methods and exports that read the predictors again."""
import numpy as np
import pytest

from fastpls_b200 import api, workloads as W
from oracle import pls_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8191, 8192, 8193, 8199, 9001])
@pytest.mark.parametrize("method", ["simpls", "plssvd", "opls"])
def test_row_counts_around_the_padding(n, method):
    p, q, a = 61, 3, 3
    x, y = W.latent_regression(n, p, q, 5, 0.4, n, dtype=np.float64)
    kw = {"north": 1} if method == "opls" else {}
    m = api.fit_resident(x, y, ncomp=a, method=method, precision=64, scaling="autoscaling", **kw)
    got = m.predict_path(x[:50], [1, a])
    P, ss = m.export(6), m.export(7)
    T = m.scores()
    m.close()
    if method == "plssvd":
        ref = O.plssvd_fit(x, y, prefixes=[1, a], scaling=2)
        want = [O.plssvd_predict(ref, x[:50], j) for j in range(2)]
    else:
        ref = (O.opls_fit(x, y, ncomp=a, scaling=2, north=1) if method == "opls"
               else O.simpls_fit(x, y, ncomp=a, scaling=2))
        f = O.opls_predict if method == "opls" else O.simpls_predict
        want = [f(ref, x[:50], k) for k in (1, a)]
    for j in range(2):
        assert O.rel_err(got[j], want[j]) < 1e-9
    if method != "opls":
        xs = (x - x.mean(0)) / x.std(0, ddof=1)
        assert O.rel_err(P, xs.T @ T / np.sum(T * T, axis=0)) < 1e-9
        assert abs(ss[a] - (n - 1) * p) < 1e-8 * n * p


@pytest.mark.parametrize("n,p", [(9003, 700), (40961, 1800)])
def test_storage_types_agree(n, p):
    """One launch and (past 2^26 elements) the per-kernel loop, BF16 against
    FP32 storage of the same values, bit for bit."""
    x, y = W.latent_regression(n, p, 2, 6, 0.5, 5, dtype=np.float32)
    bits = api.to_bf16(x)
    m16 = api.fit_resident(bits, y, ncomp=5, precision=16)
    m32 = api.fit_resident(np.asfortranarray(api.from_bf16(bits).reshape(x.shape)), y, ncomp=5, precision=32)
    for f in range(8):
        assert np.array_equal(m16.export(f), m32.export(f)), f
    m16.close()
    m32.close()
