"""For fewer than 2^24 elements of new rows a prefix asked for alone has the bits
of the same prefix in a longer path, whatever the number of rows and components:
the scores are one product with K in slices of 256 predictors. (Larger inputs
take a form that depends on the number of components.)"""
import numpy as np
import pytest

from fastpls_b200 import api, workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method,precision", [("simpls", 64), ("simpls", 32), ("simpls", 16), ("plssvd", 32),
                                              ("opls", 64)])
@pytest.mark.parametrize("rows,p,q,a", [(1, 300, 3, 2), (129, 1025, 4, 4), (700, 513, 20, 18), (4001, 257, 2, 2),
                                        (65, 5000, 70, 66)])
def test_prefix_alone_equals_path(method, precision, rows, p, q, a):
    n = 240
    x, y = W.latent_regression(n + rows, p, q, 30, 0.5, rows + p, dtype=np.float64 if precision == 64 else np.float32)
    xs = api.to_bf16(x) if precision == 16 else x
    m = api.fit_resident(np.asfortranarray(xs[:n]), np.asfortranarray(y[:n]), ncomp=a, method=method,
                         scaling="autoscaling", precision=precision)
    new = np.asfortranarray(xs[n:])
    path = m.predict_path(new, list(range(1, a + 1)))
    scores = m.project(new, a)
    for k in sorted({1, 2, (a + 1) // 2, max(1, a - 1), a}):
        assert np.array_equal(m.predict_path(new, [k])[0], path[k - 1]), k
        assert np.array_equal(m.project(new, k), scores[:, :k]), k
    m.close()
