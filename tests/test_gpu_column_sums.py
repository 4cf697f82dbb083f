"""GPU check of the centring's column sums where their path changes: the values
equal the oracle's serial sums bit for bit (so no tolerance)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ring_knn(n, k, seed):
    """Near neighbours on a ring with a few far ones, distances ascending."""
    rng = np.random.default_rng(seed)
    step = np.sort(rng.choice(np.arange(1, 4 * k), size=(n, k), replace=True), axis=1)
    step[:, -1] = rng.integers(1, n, n)
    idx = ((np.arange(n)[:, None] + step) % n).astype(np.uint32)
    return idx, np.sort(rng.uniform(0.05, 1.0, (n, k)).astype(np.float32), axis=1)


# the last size without chunks, sizes with one value, a part of a group and a whole group
# above it, one chunk after the serial head and a value more, and several
@pytest.mark.parametrize("n", [8192, 8193, 8203, 8208, 16384, 16385, 50001])
@pytest.mark.parametrize("dim", [1, 3, 16])
def test_centring(ctx, oracle, n, dim):
    idx, dist = _ring_knn(n, 8, seed=n)
    g = ctx.fuzzy_set(idx, dist, 8.0, True)
    ip, ix, w = g.export()
    x = np.random.default_rng(dim).standard_normal((n, 6)).astype(np.float32) + np.float32(0.3)
    got = ctx.label_propagation_init(g, dim, x, seed=7)
    ref = oracle.lp_init(ip, ix, w, dim, x, 7)
    assert np.array_equal(got.view(np.uint32), ref.view(np.uint32))
