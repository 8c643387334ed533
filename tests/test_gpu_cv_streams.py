"""Cross-validation with and without lanes beside the main stream: SIMPLS folds
in one persistent launch and PLS-SVD folds (no lane), SIMPLS folds whose
component loops are kernels (lanes: more than 32 responses, the cached Gram).
Each matches the oracle and repeats bit for bit."""
import numpy as np
import pytest

from fastpls_b200 import api, workloads as W
from oracle import pls_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method,n,p,q,a,folds", [("simpls", 246, 62, 2, 3, 5), ("plssvd", 288, 40, 4, 2, 30),
                                                   ("simpls", 90, 50, 40, 5, 9), ("simpls", 60, 40, 33, 2, 60)])
def test_folds_match_the_oracle(method, n, p, q, a, folds):
    x, y = W.latent_regression(n, p, q, 6, 0.5, n + q, dtype=np.float64)
    f = (np.arange(n, dtype=np.int32) * 7919 % folds) + 1
    pre = list(range(1, a + 1))
    got = [api.cv_regression(x, y, f, pre, method=method, store_predictions=True) for _ in range(3)]
    ref = O.cv_regression(x, y, f, pre, scaling=1, family=3 if method == "simpls" else 1, store_predictions=True)
    assert O.rel_err(got[0]["predictions"], ref["predictions"]) < 1e-9
    for g in got[1:]:
        assert np.array_equal(g["predictions"], got[0]["predictions"])


def test_gram_route_folds():
    x, lab = W.latent_classification(900, 60, 3, 12, 0.5, 9, dtype=np.float64)
    f = (np.arange(900) % 5 + 1).astype(np.int32)
    got = [api.cv_classification(x, lab, 3, f, [2, 8], store_scores=True) for _ in range(3)]
    ref = O.cv_classification(x, lab, 3, f, [2, 8], head=0)
    assert np.allclose(got[0]["metrics"], ref["metrics"])
    for g in got[1:]:
        assert np.array_equal(g["scores"], got[0]["scores"])
