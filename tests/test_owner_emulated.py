"""Owned passes (csrc/owner_pass.cuh) of one block, run on the CPU: a thread per
CUDA thread, barriers for the warp collectives (tests/emulation), and a graph that
counts every lookup outside of it."""
from __future__ import annotations

import re
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
EMU = ROOT / "tests" / "emulation"

# The accesses that are inline PTX, as C++.
HOST = {
    "void pool_entry": "{ u = kNoEntry; w = 0.0f; if (e < len) { int2 x; std::memcpy(&x, g_smem + at + OFF, 8);"
                       " u = static_cast<unsigned>(x.x); std::memcpy(&w, &x.y, 4); } }",
    "float gather": "{ return u == kNoEntry ? 0.0f : src[u & ~kUnmarkable]; }",
    "void mark": "{ if (moved && !(u & kUnmarkable)) marks[u] = 1; }",
}


def host_source() -> str:
    src = (ROOT / "labelpropcuda_gb300" / "csrc" / "owner_pass.cuh").read_text()
    for name, body in HOST.items():
        at = re.search(re.escape(name) + r"\(", src)
        assert at, name
        begin = end = src.index("{", at.end())
        depth = 0
        while True:
            depth += {"{": 1, "}": -1}.get(src[end], 0)
            end += 1
            if depth == 0:
                break
        assert "asm volatile" in src[begin:end], name
        src = src[:begin] + body + src[end:]
    assert "asm" not in src
    return src.replace('#include "common.cuh"', '#include "warps.h"').replace(
        "__cvta_generic_to_shared(&s.pool(0))", "(reinterpret_cast<unsigned char *>(&s.pool(0)) - g_smem)")


@pytest.fixture(scope="module")
def block(tmp_path_factory):
    d = tmp_path_factory.mktemp("owner")
    (d / "owner_pass.cuh").write_text(host_source())
    exe = d / "owner_block"
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-pthread", "-Wno-unknown-pragmas", f"-I{d}",
                    f"-I{EMU}", str(EMU / "owner_block.cpp"), "-o", str(exe)], check=True)
    return lambda *a: subprocess.run([str(exe), *a], check=True, capture_output=True, text=True, timeout=120).stdout


def test_partial_tile_beyond_the_pool(block):
    """40 rows of 5 and of 30 entries, room for 100 entries: the lanes after the last
    vertex look nothing up."""
    assert block("remainder") == "outside 0 wrong 0\n"


def test_rows_keep_no_count_that_can_run_over(block):
    """A row whose visit counter would run over is not taken for one listed as a
    row of more than 32 entries."""
    assert block("counter") == "outside 0 wrong 0 label 7.0\n"


def test_short_long_and_wide_rows(block):
    """Labels, marks and row counts of passes over rows of 0 to 290 entries, with room
    for none, some and all of them, listed and by tiles, marked and dense."""
    assert block("mixed") == "outside 0 wrong 0\n"


def test_shared_memory_of_a_launch(block):
    assert block("shared") == "wrong 0\n"
