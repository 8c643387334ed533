"""Cross-validation in batches of folds: more folds than lanes and than one
launch holds, empty folds, classes missing from a training fold. Against the
oracle at the tolerances of test_gpu_cv.py (FP64 products: 1e-9)."""
import numpy as np
import pytest

from fastpls_b200 import api, workloads as W
from oracle import pls_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method,family", [("simpls", 3), ("plssvd", 1)])
@pytest.mark.parametrize("n,p,folds,skip", [(41, 29, 41, ()), (230, 700, 23, (5,)), (700, 1400, 2, ()),
                                            (900, 900, 11, (1, 11)), (12, 5, 1, ())])
def test_regression_folds(n, p, folds, skip, method, family):
    x, y = W.latent_regression(n, p, 3, 4, 0.4, n + p, dtype=np.float64)
    f = (np.arange(n, dtype=np.int32) * 7919 % folds) + 1
    for s in skip:      # a fold number that holds out no row
        f[f == s] = s - 1 if s > 1 else 2
    if folds == 1:      # two folds, the first empty
        f = np.where(np.arange(n) < 5, 2, 3).astype(np.int32)
    pre = [1, 2, 3]
    got = api.cv_regression(x, y, f, pre, method=method, scaling=2, store_predictions=True)
    ref = O.cv_regression(x, y, f, pre, scaling=2, family=family, store_predictions=True)
    for key in ("q2", "rmsd", "observed_r2"):
        assert np.allclose(got[key], ref[key], rtol=1e-9, atol=1e-11), key
    assert O.rel_err(got["predictions"], ref["predictions"]) < 1e-9
    assert np.array_equal(got["status"], ref["status"])


@pytest.mark.parametrize("lda", [False, True])
@pytest.mark.parametrize("n,folds", [(120, 31), (260, 9)])
def test_classification_folds_with_missing_classes(n, folds, lda):
    x, lab = W.latent_classification(n, 80, 4, 3, 0.5, n, dtype=np.float64)
    f = (np.arange(n, dtype=np.int32) % folds) + 1
    f[lab == 4] = 3                      # class 4 is held out whole by fold 3
    pre = [1, 2, 3]
    got = api.cv_classification(x, lab, 4, f, pre, lda=lda, store_predictions=True, store_scores=True)
    ref = O.cv_classification(x, lab, 4, f, pre, head=int(lda), store_predictions=True)
    assert np.array_equal(got["predictions"], ref["predictions"])
    assert np.allclose(got["metrics"], ref["metrics"])
    assert np.array_equal(got["status"], ref["status"])
    # fold 3's scores of the class its training rows lack stay zero
    assert not got["scores"][:, f == 3, 3].any() and got["scores"][:, f == 3, :3].any()


def test_a_rank_error_follows_the_folds_before_it():
    x, y = W.latent_regression(30, 40, 1, 3, 0.4, 3, dtype=np.float64)
    f = np.ones(30, dtype=np.int32)
    f[:4] = 2                            # fold 1 leaves 4 training rows
    with pytest.raises(api._lib.FastplsError, match="exceeds a fold rank"):
        api.cv_regression(x, y, f, [1, 2, 6])
