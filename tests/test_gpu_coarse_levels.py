"""The initialisation's coarse levels, whose rows' other weights are looked up:
coarse rows of each tier (up to 128, up to 1024 and more entries), with and without
hubs. The initial embedding equals the oracle's bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k,hub", [(700, 2, False), (3000, 4, True), (20000, 12, False),
                                     (60000, 30, False), (20000, 8, True)])
def test_coarse_rows(ctx, oracle, n, k, hub):
    rng = np.random.default_rng(n + k)
    idx = ((np.arange(n)[:, None] + rng.integers(1, n, (n, k))) % n).astype(np.uint32)
    if hub:
        idx[1:, 0] = 0
    dist = np.sort(rng.uniform(0.05, 1.0, (n, k)).astype(np.float32), axis=1)
    g = ctx.fuzzy_set(idx, dist, float(k), True)
    ip, ix, w = g.export()
    for x in (None, rng.standard_normal((n, 5)).astype(np.float32)):
        got = ctx.label_propagation_init(g, 3, x, seed=11)
        ref = oracle.lp_init(ip, ix, w, 3, x, 11)
        assert np.array_equal(got.view(np.uint32), ref.view(np.uint32))
