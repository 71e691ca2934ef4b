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
