"""Choices of the epoch-kernel tuner kept in a file: a plan of the same shape takes
them, but not those of a version that launched the epochs differently."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
PKG = Path(__file__).resolve().parents[1] / "evoc-rs_gb300"
CODE = """
import sys, numpy as np, evoc_gb300 as E
n, k = 700, 5
rng = np.random.default_rng(1)
idx = ((np.arange(n)[:, None] + rng.integers(1, n, (n, k))) % n).astype(np.uint32)
dist = np.sort(rng.uniform(0.05, 1.0, (n, k)).astype(np.float32), axis=1)
c = E.Context(0)
plan = c.plan(c.fuzzy_set(idx, dist, float(k), True), 8, E.EvocEmbeddingParams(n_epochs=10), seed=3)
print(plan.autotune() if sys.argv[1] == "tune" else plan.info()["warps_per_block"])
"""


def _run(what, cache):
    r = subprocess.run([sys.executable, "-c", CODE, what], capture_output=True, text=True,
                       timeout=300, cwd=PKG, env={**os.environ, "EVOC_TUNE_CACHE": str(cache)})
    assert r.returncode == 0, r.stderr
    return r.stdout.strip()


def test_entries_of_another_version_are_ignored(tmp_path):
    kept = tmp_path / "kept.txt"
    _run("tune", kept)
    (line,) = kept.read_text().splitlines()
    key = line.split()[0]
    shape = key[key.index("d8_"):]
    default = int(_run("info", tmp_path / "none.txt"))
    other = 4 if default != 4 else 1
    cache = tmp_path / "cache.txt"
    for k, want in ((shape, default), ("v1_" + shape, default), (key, other)):
        cache.write_text(f"{k} 0 {other} 0 0.01\n")
        assert int(_run("info", cache)) == want, k
