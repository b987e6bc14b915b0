"""The rule that gives the verify attention's blocks their ring (csrc/attention_ring.hpp): a kernel for every choice, more blocks on an
SM only where more have tokens, and the ring that is the faster one at the sizes its comment names."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
PROGRAM = r"""
#include <cstdio>
#include "attention_ring.hpp"
using namespace ei;
int main() {
  for (int warps = 1; warps <= 7; ++warps)
    for (int tiles = 1; tiles <= 40; ++tiles)
      for (int blocks = 0; blocks <= 8192; ++blocks) {
        const int b = attention_buffers(warps, blocks, tiles, 148);
        const bool ok = (b == 3 && warps == 1) || b == 4 || b == 6;
        // Not known, or no more than two an SM: the deepest ring where blocks of it come in twos, but for short chunks of one warp.
        const bool few = blocks > 296 || warps > 2 || (warps == 1 && tiles <= 4) || b == 6;
        if (!ok || !few) return std::printf("%d warps, %d blocks, %d tiles: %d\n", warps, blocks, tiles, b), 1;
      }
  const int measured[][4] = {{1, 472, 8, 3}, {1, 256, 16, 6}, {1, 0, 8, 6}, {1, 0, 4, 3}, {2, 512, 4, 4}, {2, 512, 8, 6}, {2, 256, 8, 6}, {2, 4000, 8, 4},
                             {3, 512, 8, 4}, {4, 1, 1, 4}, {5, 64, 16, 6}, {7, 256, 8, 6}};
  for (const auto& m : measured)
    if (attention_buffers(m[0], m[1], m[2], 148) != m[3]) return std::printf("%d warps, %d blocks\n", m[0], m[1]), 1;
  return 0;
}
"""


def test_every_ring_is_one_of_the_kernels(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    (tmp_path / "ring.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(ROOT / "edge-infer_b200" / "csrc"), str(tmp_path / "ring.cpp"), "-o",
                    str(tmp_path / "ring")], check=True)
    result = subprocess.run([str(tmp_path / "ring")], capture_output=True, text=True)
    assert result.returncode == 0, result.stdout
