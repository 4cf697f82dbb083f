"""build_mst's merge in one block at its edges: the first round has as many
components as points, so 2,048 points are merged in one block from the start and
2,049 after one round. Long pick chains, pairs, ties and equal points. Edges and
weights equal the oracle's bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _points(n, kind):
    rng = np.random.default_rng(n)
    i = np.arange(n, dtype=np.float64)
    if kind == "chain":  # gaps grow: each point picks the one before it
        x = np.stack([np.cumsum(1.0 + i / n), np.zeros(n)], 1)
    elif kind == "pairs":
        x = np.stack([i // 2 * 3.0 + i % 2 * rng.uniform(0.5, 1.0, n), rng.uniform(0, 0.1, n)], 1)
    elif kind == "ties":
        x = rng.integers(0, 60, (n, 2))
    else:
        x = np.ones((n, 2))
    return x[rng.permutation(n)].astype(np.float32)


@pytest.mark.parametrize("n", [2, 3, 1023, 2047, 2048, 2049, 4099])
@pytest.mark.parametrize("kind", ["chain", "pairs", "ties", "equal"])
def test_merge_edges(ctx, oracle, n, kind):
    x = _points(n, kind)
    for k in (0, 3):
        u, v, w = ctx.build_mst(x, k)
        ru, rv, rw = oracle.build_mst(x, k)
        assert np.array_equal(u, ru) and np.array_equal(v, rv)
        assert np.array_equal(w.view(np.uint32), rw.view(np.uint32))
