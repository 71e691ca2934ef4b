"""Sizes of the tile kernel's buffers (no GPU), compiled with g++ from tests/cpp/tile_layout_check.cpp
against the package's internal header, and which expressions index them."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "biwfa_gpu_pii2025_gb300" / "csrc"


@pytest.fixture(scope="module")
def facts(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    exe = tmp_path_factory.mktemp("tile_layout") / "tile_layout_check"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I", str(CSRC),
                    str(ROOT / "tests" / "cpp" / "tile_layout_check.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout
    return [line.split("\t") for line in out.strip().splitlines()]


def test_rows_of_the_widest_ring_lie_in_64_bits(facts):
    """Unit penalties accept plen + tlen up to 2^26 - 17, whose rings have 2^27 diagonals."""
    rows = [(int(f[1]), int(f[2])) for f in facts if f[0] == "row"]
    assert len(rows) == 36
    for row, at in rows:
        assert at == row * (2 ** 27 + 64)
    assert rows[-1][1] > 2 ** 31


def test_ring_rows_are_reached_through_the_64_bit_offset():
    for name in ("biwfa_tiles.cuh", "biwfa_tile_kernel.cuh"):
        for line in (CSRC / name).read_text().splitlines():
            if re.search(r"rdata \+", line):
                assert "wfg_tile_row" in line, (name, line)


def test_nulls_stay_negative_over_the_longest_search():
    """A null grows by at most 17 a row (one and a window of 16 matches); a search has at most half of the
    largest accepted score (2^26) in rows, plus the score scope, and adds two nulls and a diagonal."""
    null = -5 * 2 ** 27
    text = (CSRC / "wfg_internal.h").read_text()
    assert "#define WFG_TILE_NULL (-(5 << 27))" in text
    assert "constexpr int kTNull = WFG_TILE_NULL;" in (CSRC / "biwfa_tiles.cuh").read_text()
    assert null + 17 * (2 ** 25 + 64) < 0 and 2 * null - 2 ** 27 >= -2 ** 31


def test_leaf_blocks_cover_their_rows(facts):
    """Block b holds rows 4b + 1 .. 4b + 4; the blocks lie end to end, in multiples of four ints. One
    component: row t spans t / lo diagonals on each side; gap-affine (lo 0): see row_lo and row_hi."""
    end = {}
    for lo, b, at, n in (map(int, f[1:]) for f in facts if f[0] == "leaf"):
        assert at == end.get(lo, 4) and n % 4 == 0 and at % 4 == 0
        end[lo] = at + 4 * (1 if lo else 3) * n
        t = 4 * b + 4
        if lo:
            first = -4 * (b // lo) - 4
            assert first <= -(t // lo) and t // lo < first + n
        else:
            for cb, low, high in (("M", -(t - 3), t - 3), ("I", min(0, 5 - t), t), ("D", -t, max(0, t - 5))):
                first = -4 * b if cb == "I" else -4 * b - 4
                assert first <= low and high < first + n, (b, cb)


def test_planned_leaf_store_holds_unlike_pairs(facts):
    """Rows of a leaf of two unlike sequences, the most that a window of plen + tlen bases has (up to the
    largest leaf score), against the words planned for a batch of just that length: the tiles' blocks
    end in the plan, so such a pair never runs out of leaf store in the last pass."""
    blocks = {(int(f[1]), int(f[2])): (int(f[3]), int(f[4])) for f in facts if f[0] == "leaf"}
    plans = [tuple(map(int, f[1:])) for f in facts if f[0] == "plan"]
    assert len(plans) == 3 * 9 * (1 + 4 * 4)
    for g, lo, lx, total, words in plans:
        for plen in {1, 2, 3, 5, total // 4, total // 2}:
            tlen = total - plen
            if plen < 1 or tlen < 1 or max(plen, tlen) > 100:  # the whole pair is a leaf up to 100 bases
                continue
            least, diff = min(plen, tlen), abs(plen - tlen)
            rows = lx * least + lo * diff if lo else 2 * least + 3 + diff
            at, n = blocks[lo, (rows + 3) // 4]
            assert at <= words, (g, lo, lx, plen, tlen)
