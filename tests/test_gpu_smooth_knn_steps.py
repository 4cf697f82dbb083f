"""smooth_knn_dist where its evaluations are skipped or cannot be: sigma and rho
equal the oracle's bit for bit after any number of steps, and the step count is
the number of steps the oracle takes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rows(kind, n, k, seed):
    rng = np.random.default_rng(seed)
    d = rng.uniform(0.1, 1.0, (n, k))
    if kind == "spread":  # scales from row to row over thirty decades
        d *= 10.0 ** rng.uniform(-15, 15, (n, 1))
    elif kind == "tail":
        d = np.exp(3.0 * rng.standard_normal((n, k)))
    elif kind == "ties":  # many zeros after rho, equal rows, integers
        d = rng.integers(0, 4, (n, k)).astype(float)
        d[: n // 4] = 2.0
    elif kind == "extreme":  # nothing to certify: overflowing sums, infinities, denormals
        d *= 3e38
        d[::3, -1] = np.inf
        d[1::3] *= 1e-44 / 3e38
    return np.sort(d.astype(np.float32), axis=1)


@pytest.mark.parametrize("kind", ["plain", "spread", "tail", "ties", "extreme"])
@pytest.mark.parametrize("k", [1, 2, 15, 31, 33, 100])
def test_sigma_after_any_number_of_steps(ctx, oracle, kind, k):
    d = _rows(kind, 257, k, seed=k)
    for target in (1, 2, k, 3 * k, 1 << 20):
        for n_iter in (0, 1, 7, 64, 200):
            for lc in (1.0, 0.0) if n_iter == 64 else (1.0,):
                s, r = ctx.smooth_knn_dist(d, target, lc, n_iter)
                rs, rr = oracle.smooth_knn_dist(d, target, lc, n_iter)
                assert np.array_equal(s.view(np.uint32), rs.view(np.uint32)), (target, n_iter, lc)
                assert np.array_equal(r.view(np.uint32), rr.view(np.uint32))


@pytest.mark.parametrize("kind", ["plain", "tail"])
def test_step_count(ctx, oracle, kind):
    d = _rows(kind, 100, 15, seed=3)
    after = [oracle.smooth_knn_dist(d, 15, 1.0, t)[0] for t in range(66)]
    # a step that converges leaves sigma as it was; every other step changes it
    want = sum(next((t + 1 for t in range(64) if after[t + 1][i] == after[t][i]), 64)
               for i in range(len(d)))
    ctx.smooth_knn_dist(d, 15, 1.0, 64)
    assert ctx.smooth_knn_steps() == want


@pytest.mark.parametrize("k", [1, 15, 16, 17, 31, 32, 33])
def test_forward_lists_of_every_width(ctx, oracle, k):
    """Self loops, repeated columns and short rows around the 16 and 32 lane groups."""
    rng = np.random.default_rng(k)
    n = 1001
    idx = rng.integers(0, 60 if k < 33 else n, (n, k)).astype(np.uint32)
    idx[:, k // 2] = np.arange(n)
    for i in range(0, n, 5):
        idx[i, rng.integers(1, k + 1):] = 0xFFFFFFFF
    dist = np.sort(rng.uniform(0.05, 1.0, (n, k)).astype(np.float32), axis=1)
    got = ctx.fuzzy_set(idx, dist, float(k), True).export()
    ref = oracle.fuzzy_set(idx, dist, float(k), True)
    assert all(np.array_equal(a.view(np.uint8), np.asarray(b).view(np.uint8))
               for a, b in zip(got, ref))
