"""The epoch kernels keep everything in their registers: the compiler reports no spills."""
import re
import subprocess
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
sys.path.insert(0, str(ROOT / "evoc-rs_gb300"))


def test_epoch_kernels_do_not_spill(tmp_path):
    import build as B
    r = subprocess.run([B.nvcc(), *B.ARCH, *B.NVCC_FLAGS, "-Xptxas", "-v", "-c",
                        str(B.CSRC / "embed.cu"), "-o", str(tmp_path / "embed.o")],
                       capture_output=True, text=True, check=True)
    spills = {}
    for name, stores, loads in re.findall(
            r"Function properties for (\S+)\n\s*\d+ bytes stack frame, (\d+) bytes spill stores, "
            r"(\d+) bytes spill loads", r.stderr):
        if "k_epoch_slot" in name:
            spills[name] = (int(stores), int(loads))
    assert len(spills) == 24  # three row widths, four variants, one epoch or all
    assert not any(a or b for a, b in spills.values()), spills
