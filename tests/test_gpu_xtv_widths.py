"""X^T V at widths and row counts whose row chunk, rounded up to 128 rows, needs
more than 64 KB of shared memory for the staged columns of V (66.5 to 76.8 KB
on 148 SMs): the variance export (V = the scores) and the OPLS filter's
X^T Yc (V = the responses).

Tolerance: an FP64 sum of n products differs by at most 2 (n + 2) u sum |a||b|
between two orders (u = 2^-53); standardising subtracts mean * sum t and
divides, the numpy side the other way round: 8 (n + 8) u covers both."""
import numpy as np
import pytest

from fastpls_b200 import api, workloads as W
from oracle import pls_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,p,a", [(2400, 3168, 24), (5000, 1600, 25), (7700, 2400, 11), (40000, 1100, 5)])
@pytest.mark.parametrize("precision", [32, 64])
def test_variance_loadings(n, p, a, precision):
    x, y = W.latent_regression(n, p, 3, 12, 0.5, n + a, dtype=np.float64 if precision == 64 else np.float32)
    m = api.fit_resident(x, y, ncomp=a, precision=precision)
    P, T, mean, scale = m.export(6), m.scores(), m.export(3), m.export(4)
    m.close()
    x64, T = x.astype(np.float64), T.astype(np.float64)
    xs = (x64 - mean.astype(np.float64)) / scale.astype(np.float64)
    den = (T * T).sum(0)
    u = 2.0 ** -53 if precision == 64 else 2.0 ** -23  # exports are rounded to FP32
    bound = 8 * (n + 8) * 2.0 ** -53 * ((np.abs(x64) + np.abs(mean)).T @ np.abs(T)) / den
    bound += 8 * u * (np.abs(x64) + np.abs(mean)).T @ np.abs(T) / den
    assert np.all(np.abs(P - xs.T @ T / den) <= bound)


@pytest.mark.parametrize("n,p,q", [(2400, 3168, 24), (3500, 3168, 17)])
def test_opls_filter(n, p, q):
    x, y = W.latent_regression(n, p, q, 6, 0.5, n + q, dtype=np.float64)
    m = api.fit_resident(x, y, ncomp=2, method="opls", north=1)
    ref = O.opls_fit(x, y, ncomp=2, scaling=1, north=1)
    got = m.predict_path(x[:50], [1, 2])
    m.close()
    for j, k in enumerate([1, 2]):
        assert O.rel_err(got[j], O.opls_predict(ref, x[:50], k)) < 1e-10  # as in test_gpu_special.py
