"""The build script written out in INTEGRATION.md compiles what build.py compiles, with
the same flags: a library of fewer sources does not load."""
import re
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
sys.path.insert(0, str(ROOT / "evoc-rs_gb300"))


def test_build_script_matches_the_library():
    import build as B
    text = (ROOT / "INTEGRATION.md").read_text()
    count, names = re.search(r"const SOURCES: \[&str; (\d+)\] = \[(.*?)\];", text, re.S).groups()
    sources = re.findall(r'"([^"]+)"', names)
    assert sorted(sources) == sorted(B.SOURCES) and int(count) == len(sources)
    assert sorted(p.name for p in B.CSRC.glob("*.cu")) == sorted(sources)
    args = re.search(r"\.args\(\[(\"-O3\".*?)\]\)", text, re.S).group(1)
    assert re.findall(r'"([^"]+)"', args) == [*B.NVCC_FLAGS, "-c"]
    arch = re.search(r"let arch = \[(.*?)\];", text).group(1)
    assert re.findall(r'"([^"]+)"', arch) == B.ARCH
