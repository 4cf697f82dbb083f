"""Epochs and label rounds that start while the one before ends: every run of a
plan (the first launches its epochs, the later replay a graph) and every number
of nodes per warp give the oracle's results, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(ctx, n, k, seed=0):
    rng = np.random.default_rng(seed)
    idx = ((np.arange(n)[:, None] + rng.integers(1, n, (n, k))) % n).astype(np.uint32)
    dist = np.sort(rng.uniform(0.05, 1.0, (n, k)).astype(np.float32), axis=1)
    return ctx.fuzzy_set(idx, dist, float(k), True)


# fewer tiles than warps on the chip (some warps have none), about as many, and several each
@pytest.mark.parametrize("n,k,dim", [(3, 1, 2), (33, 3, 4), (700, 6, 16), (20000, 8, 8),
                                     (70000, 4, 4)])
def test_runs_of_one_plan(ctx, oracle, n, k, dim):
    import torch
    import evoc_gb300 as E
    g = _graph(ctx, n, k, seed=n)
    ne = 31
    plan = ctx.plan(g, dim, E.EvocEmbeddingParams(n_epochs=ne), seed=5)
    ref = oracle.evoc_embedding(*g.export(), dim, n_epochs=ne, seed=5)
    ref = ref[0] if isinstance(ref, tuple) else ref
    out = torch.empty(n, dim, dtype=torch.float32, device="cuda")

    def run_equals():
        out.zero_()
        torch.cuda.synchronize()
        plan.run_device(None, out.data_ptr())
        return np.array_equal(out.cpu().numpy().view(np.uint32), ref.view(np.uint32))

    assert all([run_equals() for _ in range(3)])
    plan.set_config(1, 4, 2)  # another launch shape: the graph is made again
    assert all([run_equals() for _ in range(2)])
    plan.free()


# a warp takes 1 to 32 nodes: both sides of each change on 152 multiprocessors
@pytest.mark.parametrize("npw", [2, 4, 8, 16, 32])
def test_nodes_per_warp(ctx, oracle, npw):
    for n in (152 * 12 * npw - 1, 152 * 12 * npw):
        g = _graph(ctx, n, 5, seed=npw)
        got, parts = ctx.label_prop_partition(g, n // 9, 20, seed=3)
        want, wparts = oracle.lp_partition(*g.export(), n // 9, 20, 3)
        assert parts == wparts and np.array_equal(got, want)


# pointers from outlier to earlier outlier: chains within, at and beyond one pass
@pytest.mark.parametrize("n", [40, 65, 66, 67, 130, 5000])
def test_outlier_chains(ctx, oracle, n):
    adj = [[(j, 0.3) for j in (i - 1, i + 1) if 0 <= j < n] for i in range(n)]
    g = ctx.graph_from_adjacency(adj)
    for seed in (1, 2):
        got, parts = ctx.label_prop_partition(g, 1, 20, seed)
        want, wparts = oracle.lp_partition(*g.export(), 1, 20, seed)
        assert parts == wparts and np.array_equal(got, want)
