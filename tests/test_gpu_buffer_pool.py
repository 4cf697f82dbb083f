"""Device buffers are kept between calls, one pool per context: calls of changing
sizes, contexts side by side in threads, and a context after another's end give
the results of a fresh context, bit for bit."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = ((300, 5), (5000, 12), (40, 3), (5200, 12), (20000, 8), (300, 5))


def _problem(n, k):
    rng = np.random.default_rng(n * 31 + k)
    idx = ((np.arange(n)[:, None] + rng.integers(1, n, (n, k))) % n).astype(np.uint32)
    return idx, np.sort(rng.uniform(0.05, 1.0, (n, k)).astype(np.float32), axis=1)


def _run(c, n, k):
    idx, dist = _problem(n, k)
    g = c.fuzzy_set(idx, dist, float(k), True)
    init = c.label_propagation_init(g, 4, None, seed=2)
    out = c.embed(g, 4, init=init, seed=3)
    u, v, w = c.build_mst(out, 3)
    g.free()
    return np.concatenate([init.ravel().view(np.uint32), out.ravel().view(np.uint32),
                           u.astype(np.uint32), v.astype(np.uint32), w.view(np.uint32)])


def test_changing_sizes_threads_and_contexts():
    import evoc_gb300 as E
    fresh = {}
    for size in set(SIZES):
        c = E.Context(0)
        fresh[size] = _run(c, *size)
        c.close()
    failures = []

    def worker(order):
        try:
            c = E.Context(0)
            for i in order:
                if not np.array_equal(_run(c, *SIZES[i]), fresh[SIZES[i]]):
                    failures.append(SIZES[i])
            c.close()
        except Exception as e:  # reported by the assertion below
            failures.append(e)

    threads = [threading.Thread(target=worker, args=(o,))
               for o in ((0, 1, 2, 3, 4, 5), (4, 3, 5, 1, 0, 2), (2, 4, 1, 5, 3, 0))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures
