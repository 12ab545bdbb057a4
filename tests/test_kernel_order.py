"""Order of memory accesses in the kernels, read off their sources: what a
missing fence or barrier breaks shows up by timing only, so no run can be
relied on to fail for it."""
from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "master_b200" / "csrc"


def source(name: str) -> str:
    text = (CSRC / name).read_text()
    return re.sub(r"//[^\n]*", "", text)


@pytest.mark.parametrize("name,waits", [("conv_plane.cuh", 3), ("wgrad_plane.cuh", 3)])
def test_tensor_memory_is_touched_only_after_a_fence_behind_the_wait(name, waits):
    """Each wait of the issuer and of the epilogue (operands landed, an
    accumulator full or free again) is followed by
    tcgen05.fence::after_thread_sync on every path to the next MMA or TMEM load:
    in the same block or outside it, not under a further condition."""
    text = source(name)
    found = list(re.finditer(r"mbar_wait\(&(full|accfull|accfree)\[", text))
    assert len(found) == waits
    for m in found:
        depth = 0
        for t in re.finditer(r"[{}]|fence_after_sync\(\)|mma_bf16\w*\(|tmem_ld\w*\(", text[m.end():]):
            if t.group() == "{":
                depth += 1
            elif t.group() == "}":
                depth = max(depth - 1, 0)
            elif t.group().startswith("fence"):
                if depth <= 0:
                    break
            else:
                pytest.fail(f"{name}: {t.group()} after the wait on {m.group(1)} without a fence between")
        else:
            pytest.fail(f"{name}: no fence after the wait on {m.group(1)}")


def test_one_lane_reads_and_writes_a_cells_state():
    """The generic cell pass: a cell's collision state is read, selected on and
    written by one lane, and the warp learns the pair count from it. (Read
    by every lane, the state could be written before a late lane had read it.)"""
    text = source("engine.cuh")
    body = text[text.index("pass_kernel(PassParams P)"):text.index("pass_walls_kernel(PassParams P)")]
    uses = [m.start() for m in re.finditer(r"P\.cells\.state\[a\]", body)]
    assert len(uses) == 2
    for at in uses:
        opened, depth = at, 0  # the innermost block that is open here
        while depth <= 0:
            opened -= 1
            depth += {"{": 1, "}": -1}.get(body[opened], 0)
        assert re.search(r"if \(collide && lane == 0\) $", body[:opened]), body[opened - 60:at]
    assert re.search(r"pairs = __shfl_sync\(0xffffffffu, pairs, 0\)", body[uses[0]:uses[1]])
