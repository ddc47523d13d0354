"""How a staged copy is split: lanes (host threads) and slot sizes over all sizes.

Two lanes are slower than one: the single helper thread often wakes late (257 x 257 states 370
against 258 us in, 310 against 210 us out).  From 16 MiB on a lane's slots are 1 MiB: with half of
that, states of 700 x 700 to 900 x 900 vertices came in up to 30 % slower.
"""
import os
import shutil
import subprocess

import pytest

from tensum_b200 import build

PROGRAM = """
#include "tg_stage.h"
#include <cstdio>
#include <cstdlib>
int main(int argc, char** argv) {
  for (int i = 1; i < argc; ++i) {
    const size_t b = std::strtoull(argv[i], nullptr, 10);
    std::printf("%d %zu\\n", tg::Stager::lanes_for(b), tg::Stager::slot_for(b));
  }
}
"""
MIB = 1 << 20


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_lanes_and_slots(tmp_path):
    cuda = os.path.join(os.path.dirname(os.path.dirname(build.nvcc())), "include")
    (tmp_path / "rule.cc").write_text(PROGRAM)
    exe = tmp_path / "rule"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", build.CSRC, "-I", cuda, "-o", str(exe), str(tmp_path / "rule.cc")],
                   check=True)
    sizes = [40, MIB - 8, MIB, 2 * MIB - 8, 2 * MIB, 40 * 229 * 229, 40 * 257 * 257, 3 * MIB - 8, 3 * MIB, 40 * 300 * 300,
             8 * MIB, 16 * MIB - 8, 16 * MIB, 40 * 700 * 700, 32 * MIB, 40 * 1025 * 1025, 1 << 40]
    out = subprocess.run([str(exe), *map(str, sizes)], check=True, capture_output=True, text=True).stdout.split("\n")
    for b, line in zip(sizes, out):
        lanes, slot = map(int, line.split())
        assert lanes != 2 and lanes == (1 if b < 3 * MIB else min(8, b // MIB)), b
        assert slot == (MIB if b >= 16 * MIB else MIB // 2), b
