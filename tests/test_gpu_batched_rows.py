"""The batched deflation at the edges of its block shapes: rows of one warp, of
whole blocks and one past them, the largest single sweep (2560 rows) and the
first size that takes two; the score kernel's row and block variants likewise,
against the oracle."""
import numpy as np
import pytest

from fastpls_b200 import api, workloads as W
from oracle import pls_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q", [1, 3, 9])
@pytest.mark.parametrize("n", [31, 160, 161, 769, 1025, 2560, 2561, 5121])
def test_deflation_row_edges(n, q):
    p = 120
    x, y = W.latent_regression(n, p, q, 4, 0.3, 71, dtype=np.float64)
    folds = W.uneven_folds(n, 4, 71)
    perms = W.permutations(n, 1, 71)
    pre = [1, 2, 5]
    got = api.cv_permutation(x, y, folds, perms, pre, precision=64, digits=0)
    for b in range(2):
        yb = y if b == 0 else y[perms[b - 1]]
        ref = O.cv_regression(x, yb, folds, pre, family=3)
        # the tolerance of the engine's other FP64 comparisons
        for key in ("q2", "rmsd", "observed_r2"):
            assert np.allclose(got[key][b], ref[key], rtol=1e-9, atol=1e-11), (b, key)
