"""build_mst where late rounds search for the points of a leaf together: the sizes
at which that begins and goes from half to whole leaves on 152 multiprocessors, a
part-filled last leaf, each padded dimension, and equal distances. Edges and
weights equal the oracle's bit for bit (which points search together decides
nothing)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HALF = 152 * 32 * 32  # points from which half leaves are searched for together
WHOLE = 4 * HALF


def _points(n, dim, kind, seed):
    rng = np.random.default_rng(seed)
    if kind == "grid":  # few distances, many of them equal
        return rng.integers(0, 700, (n, dim)).astype(np.float32)
    c = rng.standard_normal((12, dim)) * 3.0
    x = c[rng.integers(0, 12, n)] + 0.3 * rng.standard_normal((n, dim))
    far = rng.random(n) < 0.02
    x[far] = rng.standard_normal((int(far.sum()), dim)) * 5.0
    return x.astype(np.float32)


@pytest.mark.parametrize("n,dim,k,kind", [
    (HALF - 31, 3, 5, "blobs"), (HALF, 3, 5, "blobs"), (HALF + 17, 2, 5, "grid"),
    (HALF + 1, 8, 5, "blobs"), (HALF, 9, 2, "blobs"), (WHOLE - 31, 2, 5, "blobs"),
    (WHOLE + 5, 2, 5, "blobs"), (WHOLE + 1, 4, 0, "grid")])
def test_points_searched_for_together(ctx, oracle, n, dim, k, kind):
    x = _points(n, dim, kind, seed=n % 97 + dim)
    u, v, w = ctx.build_mst(x, k)
    ru, rv, rw = oracle.build_mst(x, k)
    assert np.array_equal(u, ru) and np.array_equal(v, rv)
    assert np.array_equal(w.view(np.uint32), rw.view(np.uint32))
