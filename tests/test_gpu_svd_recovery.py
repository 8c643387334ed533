"""fastsvd at the widest sketch one block's eigenproblem holds (119 columns):
wider requests name the limit, and a recovery that reaches it goes on with
power steps.

The audit accepts triplets with a relative residual of at most 1e-2, and a
singular value differs from the exact one by no more than its residual."""
import numpy as np
import pytest

from fastpls_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,p,k,oversample", [(300, 260, 80, 39), (400, 300, 119, 0), (300, 260, 60, 120)])
def test_wider_sketches_name_the_limit(n, p, k, oversample):
    with pytest.raises(api._lib.FastplsError, match="sketch too wide for one block"):
        api.fastsvd(np.random.default_rng(1).standard_normal((n, p)), k, oversample=oversample, power=4)


@pytest.mark.parametrize("k", [20, 40])
def test_recovery_at_the_widest_sketch(k):
    x = np.random.default_rng(1).standard_normal((400, 300))  # flat spectrum: the first attempts fail the audit
    u, d, v, info = api.fastsvd(x, k, oversample=0, power=0, audit=True)
    assert info["certified"] and info["attempts"] > 3
    assert k + 1 + info["effective_oversample"] == 119
    s = np.linalg.svd(x, compute_uv=False)[:k]
    assert info["triplet_residual"] <= 1e-2
    assert np.max(np.abs(d - s)) <= 1e-2 * s[0]
    assert np.max(np.abs(u.T @ u - np.eye(k))) <= 1e-10
