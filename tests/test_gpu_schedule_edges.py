"""The epoch schedule, its slots and the epoch kernel where their forms change:
32-epoch words, negative counts of two and four bits and beyond, chunks of 1024
entries, tiles of 4 to 32 nodes. Embeddings and schedule counts equal the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(ctx, n, k, hubs=0, seed=0):
    rng = np.random.default_rng(seed)
    idx = (np.arange(n)[:, None] + rng.integers(1, n, (n, k))) % n
    if hubs:  # rows of a few thousand entries next to each other: several chunks per tile
        idx[:, 0] = np.where(np.arange(n) < hubs, idx[:, 0], rng.integers(0, hubs, n))
    dist = np.sort(rng.uniform(0.05, 1.0, (n, k)).astype(np.float32), axis=1)
    return ctx.fuzzy_set(idx.astype(np.uint32), dist, float(k), True)


def _check(ctx, oracle, g, dim, ne, rate, seed=7):
    import evoc_gb300 as E
    p = E.EvocEmbeddingParams(n_epochs=ne, negative_sample_rate=rate)
    plan = ctx.plan(g, dim, p, seed=seed)
    got = plan.debug_run(None, 0, ne)
    ref, st = oracle.evoc_embedding(*g.export(), dim, n_epochs=ne, negative_sample_rate=rate,
                                    seed=seed, want_stats=True)
    assert np.array_equal(got.view(np.uint32), ref.view(np.uint32))
    assert np.array_equal(plan.stats(), st)
    plan.free()


@pytest.mark.parametrize("ne", [1, 2, 31, 32, 33, 63, 64, 65, 96, 97, 127, 128, 129])
def test_epoch_counts(ctx, oracle, ne):
    _check(ctx, oracle, _graph(ctx, 333, 6, seed=ne), 4, ne, 1.0)


@pytest.mark.parametrize("ne", [50, 100])
@pytest.mark.parametrize("rate", [0.0, 0.3, 1.0, 2.5, 2.6, 4.5, 6.0, 12.0, 22.0, 40.0])
def test_negative_counts(ctx, oracle, ne, rate):
    _check(ctx, oracle, _graph(ctx, 400, 5, seed=3), 8, ne, rate)


@pytest.mark.parametrize("ne,rate", [(50, 1.0), (100, 5.0)])
@pytest.mark.parametrize("dim", [2, 8, 16])
def test_hub_tiles(ctx, oracle, ne, rate, dim):
    _check(ctx, oracle, _graph(ctx, 5000, 4, hubs=3, seed=1), dim, ne, rate)


# each side of the sizes at which tiles grow (152 SMs: 25,536, 51,072 and 102,144 nodes)
@pytest.mark.parametrize("n", [1, 3, 33, 25_535, 25_536, 51_071, 51_073, 102_143, 102_150])
def test_tile_sizes(ctx, oracle, n):
    if n < 33:
        k = 1
        idx = ((np.arange(n)[:, None] + 1) % n).astype(np.uint32)
        g = ctx.fuzzy_set(idx, np.full((n, k), 0.5, np.float32), 1.0, True)
    else:
        g = _graph(ctx, n, 3, seed=2)
    if g.nnz == 0:
        return
    _check(ctx, oracle, g, 8, 12, 1.0)


def test_general_graphs_share_the_schedule(ctx, oracle):
    """Directed lists, duplicates and self loops: lists of their own, the same schedule."""
    rng = np.random.default_rng(5)
    n = 700
    deg = rng.integers(0, 9, n)
    ip = np.concatenate([[0], np.cumsum(deg)])
    ix = rng.integers(0, n, ip[-1]).astype(np.uint32)
    w = rng.uniform(0.01, 1.0, ip[-1]).astype(np.float32)
    g = ctx.graph_from_csr(ip, ix, w)
    for ne, rate in ((50, 1.0), (70, 3.0), (140, 1.0)):
        _check(ctx, oracle, g, 4, ne, rate)
