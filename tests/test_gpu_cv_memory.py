"""Plain cross-validation gives the same bits whatever memory is free: the
free memory decides how many folds are resident at a time, not how a fold's
sums are split."""
import os
import subprocess
import sys

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


CHILD = """
import numpy as np, torch
from fastpls_b200 import api, workloads as W

def both(n, p):
    x, y = W.latent_regression(n, p, 2, 5, 0.4, 3, dtype=np.float64)
    f = (np.arange(n, dtype=np.int32) % 10) + 1
    lab = (1 + (y[:, 0] > 0)).astype(np.int32)
    r = api.cv_regression(x, y, f, [1, 3], precision=64, store_predictions=True)
    c = api.cv_classification(x, lab, 2, f, [1, 3], precision=64, store_predictions=True, store_scores=True)
    return r["predictions"], r["q2"], r["status"], c["scores"], c["predictions"], c["metrics"], c["status"]

both(60, 40)  # modules loaded
free, _ = torch.cuda.mem_get_info()
ballast = torch.empty(free - FREE_MB * 2 ** 20, dtype=torch.uint8, device="cuda")
tight = both(4000, 4000)  # before the library's pool holds any memory of that size
del ballast
torch.cuda.empty_cache()
for a, b in zip(tight, both(4000, 4000)):
    assert np.array_equal(a, b)
print("same")
"""


@pytest.mark.parametrize("free_mb", [900, 600])
def test_a_batch_without_memory_is_taken_in_parts(free_mb):
    """Ten folds of 4000 x 4000 FP64 (128 MB of training and held-out rows each,
    beside X) where two to five fit: the batch is halved until it fits, with
    the bits of the whole one. In a process of its own, whose memory pool is
    still empty."""
    pytest.importorskip("torch")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    done = subprocess.run([sys.executable, "-c", CHILD.replace("FREE_MB", str(free_mb))], cwd=root,
                          capture_output=True, text=True, timeout=300)
    assert done.returncode == 0 and "same" in done.stdout, done.stdout + done.stderr


def test_one_class_folds_are_counted_once():
    n = 90
    x, _ = W.latent_regression(n, 30, 1, 3, 0.4, 5, dtype=np.float64)
    lab = np.ones(n, dtype=np.int32)
    lab[:20] = 2
    f = np.where(np.arange(n) < 20, 1, 2 + np.arange(n) % 4).astype(np.int32)  # fold 1 holds class 2 out whole
    got = api.cv_classification(x, lab, 2, f, [1, 2], precision=64, store_predictions=True)
    assert got["status"][0] == 4 and np.all(got["status"][1:] == 1)
    assert np.all(got["predictions"][:20] == 1)
    want = (got["predictions"] == lab[:, None]).mean(0)
    assert np.allclose(got["metrics"], want, rtol=0, atol=1e-15)
