"""What the compiler reported for the default FP32-mixed stage kernels (no GPU needed)."""

from __future__ import annotations

import os
import re

import pytest

REPORT = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cfd_demo_b200", "ptxas_report.txt")


def _spills(pattern):
    text = open(REPORT).read()
    found = re.findall(r"Compiling entry function '([^']*)'[^\n]*\n[^\n]*\n\s+\d+ bytes stack frame, (\d+) bytes spill stores, "
                       r"(\d+) bytes spill loads", text)
    return {name: (int(a), int(b)) for name, a, b in found if re.search(pattern, name)}


@pytest.mark.skipif(not os.path.exists(REPORT), reason="the library was not built in this tree")
@pytest.mark.parametrize("shape", [
    r"stage_tile_kernelIfLi[012]ELi[012]ELi32ELb0ELi8E",  # tiles of 32, the default
    r"stage_tile_kernelIfLi[012]ELi[012]ELi64ELb1ELi4ELb1ELb1ELb1ELb0ELb0E",  # tiles of 64, the default of large unlimited steps
    r"stage_pair_kernelIfLi[012]ELi[012]E",
])
def test_default_fp32_stage_kernels_do_not_spill(shape):
    """The rare positivity repair is a call from the middle of their epilogue; what it keeps in registers
    must not push the hot path's values out to memory."""
    spills = _spills(shape)
    assert len(spills) >= 9
    assert {n: s for n, s in spills.items() if s != (0, 0)} == {}


@pytest.mark.skipif(not os.path.exists(REPORT), reason="the library was not built in this tree")
@pytest.mark.parametrize("real,blocks", [("d", 3), ("f", 4)])
def test_persistent_batch_kernels_leave_room_for_their_blocks(real, blocks):
    """Static shared memory beside the stage tile of 64 elements (state rows, staged base rows in FP32,
    traces, geometry, integer rows) must not cost an SM one of the blocks the kernel is built for: 228 KB
    an SM, 1 KB of them taken by each block."""
    size, row = (8, 68) if real == "d" else (4, 72)
    tile = size * (60 * row + (60 * 64 + 16 if real == "f" else 0) + 64 * 64 + 13 * row) + 4 * 64 * 4
    text = open(REPORT).read()
    found = re.findall(r"Compiling entry function '(\w*batch_persistent_kernelI" + real + r"\w*)'(?:[^\n]*\n){3}[^\n]*?(\d+) bytes smem",
                       text)
    assert len(found) == 15
    for name, static in found:
        assert blocks * (tile + int(static) + 1024) <= 228 * 1024, name
