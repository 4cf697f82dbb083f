"""GPU checks of the row grouping, the scan and the radix sort at the sizes where
their paths change: results equal the oracle's bit for bit (whole numbers and
f32 sums in the same order, so no tolerance)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _hub_knn(n, k, hubs, seed):
    """Random kNN lists in which hub h (rows 0..) is listed by about hubs[h] rows."""
    rng = np.random.default_rng(seed)
    idx = np.zeros((n, k), np.uint32)
    for i in range(n):
        c = rng.choice(n - 1, size=k, replace=False)
        idx[i] = c + (c >= i)
    for h, m in enumerate(hubs):
        for i in rng.choice(np.arange(len(hubs), n), size=min(m, n - len(hubs)), replace=False):
            if h not in idx[i]:
                idx[i, rng.integers(k)] = h
    dist = np.sort(rng.uniform(0.05, 1.0, (n, k)).astype(np.float32), axis=1)
    return idx, dist


# row lengths around a warp's 32, 64 and 128 entries, the middle rows' 256, 512 and 1024, and
# the long rows' second and third chunk
@pytest.mark.parametrize("hubs", [(20, 21, 22, 23), (52, 53, 54, 55), (116, 117, 118, 119),
                                  (244, 245, 500, 501), (1010, 1011, 1012, 1013, 1014, 1015),
                                  (2030, 2050, 2100, 3000)])
def test_rows_of_every_tier(ctx, oracle, hubs):
    n, k = 3200, 12
    idx, dist = _hub_knn(n, k, hubs, seed=len(hubs) + hubs[0])
    g = ctx.fuzzy_set(idx, dist, float(k), True)
    ip, ix, w = g.export()
    part, parts = ctx.label_prop_partition(g, 40, 20, seed=3)
    want, wparts = oracle.lp_partition(ip, ix, w, 40, 20, 3)
    assert parts == wparts and np.array_equal(part, want)
    x = np.random.default_rng(1).standard_normal((n, 24)).astype(np.float32)
    for dim in (2, 16):
        got = ctx.label_propagation_init(g, dim, x, seed=5)
        ref = oracle.lp_init(ip, ix, w, dim, x, 5)
        assert np.array_equal(got.view(np.uint32), ref.view(np.uint32))


# one tile of the sort, its edges, and the scan's change from one block to the look-back
@pytest.mark.parametrize("n,k", [(1365, 3), (4095, 1), (4096, 1), (4097, 1), (8191, 2),
                                 (16383, 1), (16384, 1), (16385, 1), (20481, 2)])
def test_sort_and_scan_edges(ctx, oracle, n, k):
    rng = np.random.default_rng(n)
    idx = rng.integers(0, n, (n, k)).astype(np.uint32)
    dist = np.sort(rng.uniform(0.05, 1.0, (n, k)).astype(np.float32), axis=1)
    got = ctx.fuzzy_set(idx, dist, float(k), True).export()
    ref = oracle.fuzzy_set(idx, dist, float(k), True)
    assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1])
    assert np.array_equal(got[2].view(np.uint32), ref[2].view(np.uint32))
