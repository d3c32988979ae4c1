"""Bounds that planning keeps its launches within, computed on the host from the library's own header."""
import os
import subprocess

from conftest import ROOT

PROGRAM = r"""
#include <cstdio>
#include "internal.h"
int main() {
    for (int dend = 3; dend <= beep::kMaxQ; ++dend)
        for (int en = 0; en < 2; ++en)
            for (unsigned grid : {1u, 148u, 1184u, 65536u}) {
                const uint32_t parts = beep::walk_parts(dend, en != 0);
                std::printf("%d %d %u %u %u\n", dend, en, grid, parts, beep::cursor_items(parts, grid));
            }
}
"""


def test_medium_cursor_cannot_wrap(tmp_path):
    """A launch's cursor counts its items times the parts of each, then one draw a block: below 2^32 for the longest
    list that planning puts in one launch, which is also as long as that allows."""
    src, exe = tmp_path / "bounds.cpp", tmp_path / "bounds"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "beep_b200", "csrc"), "-I", "/usr/local/cuda/include",
                    "-c", str(src), "-o", str(exe) + ".o"], check=True)
    # (the header's inline functions name CUDA calls that this program never makes)
    subprocess.run(["g++", str(exe) + ".o", "-o", str(exe), "-Wl,--unresolved-symbols=ignore-all"], check=True)
    lines = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.splitlines()
    assert len(lines) == 8 * 2 * 4
    for line in lines:
        dend, en, grid, parts, items = map(int, line.split())
        assert parts == (1 if en or dend < 6 else 8 if dend == 6 else 32)
        assert items * parts + grid < 1 << 32 <= (items + 1) * parts + grid + 1
