"""An LDA path that is refused (its widest prefix passes one block's shared
memory: 2 k^2 + c k doubles) leaves nothing behind: later paths of the same
model give what a fresh model gives, and the refused prefix stays refused."""
import numpy as np
import pytest

from fastpls_b200 import api, workloads as W

pytestmark = pytest.mark.gpu


def _model():
    x, lab = W.latent_classification(300, 200, 6, 5, 0.6, 17, dtype=np.float64)
    return x, api.fit_resident(x, labels=lab, classes=6, ncomp=120, precision=64)


@pytest.mark.parametrize("path", [[1, 3, 120], [2, 5, 7, 120], [120]])
def test_prefixes_of_a_refused_path(path):
    x, fresh = _model()
    want = fresh.predict_path(x, [1, 2, 3, 5, 7], lda=True)
    labels = fresh.classify_path(x, [1, 2, 3, 5, 7], lda=True)
    fresh.close()
    x, m = _model()
    for _ in range(2):
        with pytest.raises(api._lib.FastplsError):
            m.predict_path(x, path, lda=True)
    assert np.array_equal(m.predict_path(x, [1, 2, 3, 5, 7], lda=True), want)
    assert np.array_equal(m.classify_path(x, [1, 2, 3, 5, 7], lda=True), labels)
    with pytest.raises(api._lib.FastplsError):
        m.classify_path(x, path, lda=True)
    m.close()
