"""The constant tables that kernels read 16 bytes at a time are declared with that alignment (a
device variable is placed by its type's alignment alone)."""
import os
import subprocess

SOURCE = """
#include "poseidon2_tc.cuh"
#include "poseidon2_warp.cuh"
static_assert(alignof(kb::P2TcTab<16>) % 16 == 0 && alignof(kb::P2TcTab<24>) % 16 == 0, "B operands");
static_assert(offsetof(kb::P2TcTab<24>, w) % 16 == 0, "B operands");
static_assert(alignof(kb::P2WarpConsts) % 16 == 0, "warp permutation's constants");
"""


def test_tables_read_in_pieces_of_16_bytes(tmp_path):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    src = tmp_path / "align.cpp"
    src.write_text("#include <cstddef>\n" + SOURCE)
    r = subprocess.run(["g++", "-std=c++17", "-fsyntax-only", "-I", os.path.join(root, "whirlaway_b200", "csrc"), str(src)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
