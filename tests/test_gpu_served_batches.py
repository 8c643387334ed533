"""Queued fits of ordinary sizes still share persistent launches: a fit alone
takes no more CTAs than leave room for others. Each served fit has the bits of
the same fit alone."""
import numpy as np
import pytest

from fastpls_b200 import api, workloads as W

pytestmark = pytest.mark.gpu


# fits per launch of 296 co-resident CTAs: four up to 2.4e6 elements, three at 3e6, two at 4e6
@pytest.mark.parametrize("n,p,per_launch", [(541, 1500, 4), (700, 2500, 4), (1000, 3000, 3), (1600, 2500, 2)])
def test_fits_per_launch(n, p, per_launch):
    count = 6
    data = [W.latent_regression(n, p, 2, 4, 0.4, 40 + i, dtype=np.float32) for i in range(count)]
    big = W.latent_regression(6000, 12000, 3, 4, 0.4, 39, dtype=np.float32)
    srv = api.Server(workers=1)
    blocker = srv.submit_fit(*big, ncomp=40)  # keeps the worker busy while the others queue
    tickets = [srv.submit_fit(x, y, ncomp=5) for x, y in data]
    for t in [blocker] + tickets:
        srv.wait(t)
    stats = srv.batch_stats()
    got = [srv.wait(srv.submit_predict(t, data[i][0][:11], [1, 5]))[0] for i, t in enumerate(tickets)]
    srv.close()
    # a last batch of one fit is not counted as a batch
    assert stats["launches"] <= -(-count // per_launch) and stats["fits"] >= count - 1, stats
    for i, (x, y) in enumerate(data):
        m = api.fit_resident(x, y, ncomp=5, precision=32)
        assert np.array_equal(got[i], m.predict_path(x[:11], [1, 5]))
        m.close()
