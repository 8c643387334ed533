"""Plain cross-validation gives the same bits whatever memory is free: the
free memory decides how many folds are resident at a time, not how a fold's
sums are split."""
import numpy as np
import pytest

from fastpls_b200 import api, workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,n,p,folds", [(64, 601, 1500, 10), (32, 401, 2000, 9)])
def test_bits_do_not_follow_free_memory(precision, n, p, folds):
    torch = pytest.importorskip("torch")
    x, y = W.latent_regression(n, p, 2, 5, 0.4, n + p, dtype=np.float64 if precision == 64 else np.float32)
    f = (np.arange(n, dtype=np.int32) * 7919 % folds) + 1
    lab = (1 + (y[:, 0] > 0) + (y[:, 1] > 0)).astype(np.int32)
    pre = list(range(1, 7))

    def both():
        r = api.cv_regression(x, y, f, pre, precision=precision, store_predictions=True)
        c = api.cv_classification(x, lab, 3, f, pre, precision=precision, store_scores=True)
        return r["predictions"], r["q2"], r["rmsd"], c["scores"], c["metrics"]

    roomy = both()
    free, _ = torch.cuda.mem_get_info()
    # a quarter of what stays free holds 3 to 5 folds of 64 MB and more
    ballast = torch.empty(max(0, free - 1400 * 2 ** 20), dtype=torch.uint8, device="cuda")
    try:
        tight = both()
    finally:
        del ballast
        torch.cuda.empty_cache()
    for a, b in zip(roomy, tight):
        assert np.array_equal(a, b)
