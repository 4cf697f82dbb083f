"""Which form of the schedule a plan takes, by its stages (EVOC_TRACE): bit planes below a
negative rate of 11.25, the recurrence per entry from there on, never one after the other."""
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
PKG = Path(__file__).resolve().parents[1] / "evoc-rs_gb300"
RATES = (1.0, 3.0, 11.2, 11.25, 11.9, 12.0, 15.0, 25.0)
CODE = """
import sys, numpy as np, evoc_gb300 as E
n, k = 3000, 6
rng = np.random.default_rng(4)
idx = ((np.arange(n)[:, None] + rng.integers(1, n, (n, k))) % n).astype(np.uint32)
dist = np.sort(rng.uniform(0.05, 1.0, (n, k)).astype(np.float32), axis=1)
c = E.Context(0)
g = c.fuzzy_set(idx, dist, float(k), True)
sys.stderr.write("plan\\n")
c.plan(g, 4, E.EvocEmbeddingParams(n_epochs=100, negative_sample_rate=RATE), seed=3)
"""


@pytest.mark.parametrize("rate", RATES)
def test_one_pass_only(rate):
    r = subprocess.run([sys.executable, "-c", CODE.replace("RATE", str(rate))], cwd=PKG,
                       capture_output=True, text=True, timeout=300,
                       env={**os.environ, "EVOC_TRACE": "1"})
    assert r.returncode == 0, r.stderr
    stages = r.stderr.split("plan\n", 1)[1]
    planes, entries = stages.count("schedule masks"), stages.count("count pass")
    assert (planes, entries) == ((1, 0) if rate < 11.25 else (0, 1)), stages


@pytest.mark.parametrize("rate", RATES)
def test_embedding(ctx, oracle, rate):
    import evoc_gb300 as E
    rng = np.random.default_rng(4)
    n, k = 500, 6
    idx = ((np.arange(n)[:, None] + rng.integers(1, n, (n, k))) % n).astype(np.uint32)
    g = ctx.fuzzy_set(idx, np.sort(rng.uniform(0.05, 1.0, (n, k)).astype(np.float32), axis=1),
                      float(k), True)
    plan = ctx.plan(g, 4, E.EvocEmbeddingParams(n_epochs=40, negative_sample_rate=rate), seed=7)
    got = plan.debug_run(None, 0, 40)
    ref, st = oracle.evoc_embedding(*g.export(), 4, n_epochs=40, negative_sample_rate=rate, seed=7,
                                    want_stats=True)
    assert np.array_equal(got.view(np.uint32), ref.view(np.uint32))
    assert np.array_equal(plan.stats(), st)
    plan.free()
