"""Launches that start while the one before them still runs: what that one writes is
not read-only while they are resident, so no such parameter may be const __restrict__
(the compiler may then read it by ld.global.nc, or ahead of the wait)."""
import re
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parents[1] / "evoc-rs_gb300" / "csrc"
# parameters that the overlapped launches hand to each other
HANDED_ON = {"k_lp_iter_rows": {"in", "prev_changed", "mark"},
             "k_lp_iter_long": {"in", "longs", "n_long"},
             "k_epoch_slot": set()}  # a struct: rows and moments by load_row<..., true>


def _overlapped_kernels():
    """name -> (parameter list, body) of every kernel with a griddepcontrol.wait."""
    found = {}
    for path in CSRC.glob("*.cu"):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"__global__ void (?:__launch_bounds__\(.*?\)\s*)?(\w+)\(([^{;]*)\)\s*\{", text, re.S):
            end = text.find("\n}", m.end())
            if "griddepcontrol.wait" in text[m.end():end]:
                found[m.group(1)] = (m.group(2), text[m.end():end])
    return found


def test_nothing_handed_on_is_read_as_constant():
    kernels = _overlapped_kernels()
    assert set(kernels) == set(HANDED_ON)
    for name, handed in HANDED_ON.items():
        params, body = kernels[name]
        for p in handed:
            decl = next(d for d in params.split(",") if re.search(rf"\b{p}\s*$", d))
            assert "__restrict__" not in decl, (name, decl.strip())
            plain = re.findall(rf"(?<![\w.]){p}\[|\*{p}\b(?!\s*,)|__ldg\({p}\b", body)
            assert not plain, (name, p, plain)


def test_epochs_read_rows_in_program_order():
    """Rows and moments go from epoch to epoch, by launches that overlap or across the
    barrier of one: read by load_l2 or ldcg8 (volatile, after the wait), not by an
    intrinsic that the compiler may treat as a function of its address."""
    text = re.sub(r"//[^\n]*", "", (CSRC / "embed.cu").read_text())
    assert "__ldcg(" not in text
    device = (CSRC / "evoc_device.cuh").read_text()
    for body in re.findall(r"load_l2\(const [^{]*\{(.*?)\n\}", device, re.S):
        assert "asm volatile" in body and '"memory"' in body and "ld.global.cg" in body


@pytest.mark.gpu
def test_rounds_with_hubs_repeat(ctx, oracle):
    """Short and long rows, labels spreading over many rounds, again and again."""
    rng = np.random.default_rng(11)
    n, hubs = 30_000, 6
    idx = (np.arange(n)[:, None] + rng.integers(1, n, (n, 4))) % n
    idx[:, 0] = np.where(np.arange(n) < hubs, idx[:, 0], rng.integers(0, hubs, n))
    dist = np.sort(rng.uniform(0.05, 1.0, (n, 4)).astype(np.float32), axis=1)
    g = ctx.fuzzy_set(idx.astype(np.uint32), dist, 4.0, True)
    for parts, rounds in ((50, 60), (3000, 20)):
        want, wparts = oracle.lp_partition(*g.export(), parts, rounds, 5)
        for _ in range(40):
            got, nparts = ctx.label_prop_partition(g, parts, rounds, 5)
            assert nparts == wparts and np.array_equal(got, want)
    g.free()


@pytest.mark.gpu
def test_last_overlapped_and_first_serial_size(ctx, oracle):
    """A round of one wave of blocks (6 per multiprocessor, 8 warps of 32 nodes) and of more."""
    import torch
    one_wave = torch.cuda.get_device_properties(0).multi_processor_count * 6 * 8 * 32
    for n in (one_wave, one_wave + 1):
        rng = np.random.default_rng(n)
        idx = ((np.arange(n)[:, None] + rng.integers(1, n, (n, 4))) % n).astype(np.uint32)
        dist = np.sort(rng.uniform(0.05, 1.0, (n, 4)).astype(np.float32), axis=1)
        g = ctx.fuzzy_set(idx, dist, 4.0, True)
        want, wparts = oracle.lp_partition(*g.export(), 2000, 20, 5)
        for _ in range(5):
            got, nparts = ctx.label_prop_partition(g, 2000, 20, 5)
            assert nparts == wparts and np.array_equal(got, want)
        g.free()
