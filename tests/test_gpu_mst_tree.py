"""build_mst at the sizes where the tree changes shape: one leaf, the first inner
level, a block's 4096 points, the first radix-sorted level, and the change from
one to two groups of five levels. Edges and weights equal the oracle's bit for bit
(the tree only prunes)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _points(n, dim, kind, seed):
    rng = np.random.default_rng(seed)
    if kind == "grid":  # many equal distances, duplicated points
        return rng.integers(0, 4, (n, dim)).astype(np.float32)
    c = rng.standard_normal((7, dim)) * 4.0
    x = c[rng.integers(0, 7, n)] + 0.2 * rng.standard_normal((n, dim))
    far = rng.random(n) < 0.03
    x[far] = rng.standard_normal((int(far.sum()), dim)) * 6.0
    return x.astype(np.float32)


@pytest.mark.parametrize("n", [2, 31, 32, 33, 64, 65, 1024, 1025, 4096, 4097, 8193, 32769])
@pytest.mark.parametrize("dim,k,kind", [(3, 5, "blobs"), (8, 40, "blobs"), (2, 5, "grid"),
                                        (16, 33, "grid")])
def test_mst_equals_oracle_at_tree_edges(ctx, oracle, n, dim, k, kind):
    if n > 9000 and (dim > 8 or k > 5):
        pytest.skip("covered at the smaller sizes")
    x = _points(n, dim, kind, seed=n + dim)
    u, v, w = ctx.build_mst(x, k)
    ru, rv, rw = oracle.build_mst(x, k)
    assert np.array_equal(u, ru) and np.array_equal(v, rv)
    assert np.array_equal(w.view(np.uint32), rw.view(np.uint32))
