"""FP64 tensor-core GEMM: tile edges, odd strides, K slices, operand layouts.

Tolerance: |fl(sum) - sum| <= (K + 2) u sum |a||b| per entry for any order of
an FP64 sum of K products (u = 2^-53), once for the device and once for
numpy."""
import numpy as np
import pytest

from fastpls_b200 import api

pytestmark = pytest.mark.gpu


def _bound(a, b):
    return 2.0 * (a.shape[1] + 2) * 2.0 ** -53 * (np.abs(a) @ np.abs(b))


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("m,k,n", [(1, 1, 1), (127, 17, 33), (129, 16, 31), (65, 15, 64),
                                   (33, 5003, 9), (2001, 130, 41), (64, 4096, 64),
                                   (300, 1027, 300), (700, 64, 5), (5, 64, 700)])
def test_gemm_shapes(m, k, n, precision):
    rng = np.random.default_rng(m * 7 + k + n)
    dt = np.float64 if precision == 64 else np.float32
    a = rng.standard_normal((m, k)).astype(dt)
    b = rng.standard_normal((k, n)).astype(dt)
    got = api.cuda_gemm(a, b, precision=precision)
    a, b = a.astype(np.float64), b.astype(np.float64)
    want = a @ b
    bound = _bound(a, b)
    if precision == 32:  # the result is returned in FP32
        bound = bound + 2.0 ** -23 * np.abs(want)
    assert np.all(np.abs(got - want) <= bound)


@pytest.mark.parametrize("units,feats", [(31, 900), (64, 64), (65, 129), (200, 2003), (513, 40)])
def test_symmetric_product_odd_sizes(units, feats):
    """fastcor without b: A A^T over the lower tiles, mirrored."""
    rng = np.random.default_rng(units)
    x = rng.standard_normal((units, feats))
    got = api.fastcor(x)
    z = x - x.mean(1, keepdims=True)
    z /= np.linalg.norm(z, axis=1, keepdims=True)
    assert np.array_equal(got, got.T)
    # centring and scaling add a few roundings per entry of z: 8 u |z| each
    assert np.all(np.abs(got - z @ z.T) <= _bound(z, z.T) + 16 * 2.0 ** -53 * (np.abs(z) @ np.abs(z.T)) * 2)


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("n,p", [(1201, 63), (2500, 128), (4003, 251)])
def test_transposed_gram_of_tall_predictors(n, p, precision):
    """The cached-Gram classification fit (X^T X in K slices): orthonormal
    training scores and loadings equal to the FP64 products."""
    rng = np.random.default_rng(p)
    dt = np.float64 if precision == 64 else np.float32
    t = rng.standard_normal((n, 12))
    x = np.asfortranarray((t @ rng.standard_normal((12, p)) + 0.5 * rng.standard_normal((n, p))).astype(dt))
    labels = np.argmax(t @ rng.standard_normal((12, 10)), axis=1).astype(np.int32) + 1
    m = api.fit_resident(x, labels=labels, classes=10, ncomp=8, precision=precision)
    assert m.controls()["predictor_crossprod_cache"] == 1
    R, T = m.weights().astype(np.float64), m.scores().astype(np.float64)
    m.close()
    xs = x.astype(np.float64) - x.astype(np.float64).mean(0)
    tol = 1e-9 if precision == 64 else 1e-5
    assert np.max(np.abs(T.T @ T - np.eye(8))) < tol
    assert np.linalg.norm(xs @ R - T) < tol * np.linalg.norm(T)
