"""The ring of the BF16 weight-streaming kernel (csrc/dense_ring.hpp) for every K slice and shared-memory limit: whole
phases, within the limit, at least two of them, and refused exactly where not even two single tiles fit. The kernel steps
through its barriers and tiles by whole phases, so a ring that is no multiple of them would be left and never wrapped."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

PROGRAM = r"""
#include <cstdio>
#include "dense_ring.hpp"
using namespace ei;
int main() {
  for (int parts = 1; parts <= 16; ++parts)
    for (size_t limit = 20 * 1024; limit <= 227 * 1024; limit += 256) {
      const DenseRing r = dense_ring(parts, limit);
      const size_t single = dense_layout(DenseLaunch{2, dense_units_box(parts), 0, 0}).total;
      const size_t total = dense_layout(DenseLaunch{r.stages, dense_units_box(parts), 0, 0}).total;
      bool ok = (r.tiles == 0) == (single > limit);
      if (r.tiles)
        ok = ok && r.stages % r.tiles == 0 && r.stages >= 2 * r.tiles && r.stages <= kDenseMaxStages && total <= limit &&
             r.tiles * parts <= kDenseWarps && (r.tiles == 1 || r.tiles == 2 || r.tiles == 4);
      if (!ok) {
        std::printf("%d parts, %zu bytes: %d tiles, %d stages\n", parts, limit, r.tiles, r.stages);
        return 1;
      }
    }
  for (int parts = 1; parts <= 16; ++parts) std::printf("%d ", dense_ring(parts, 227 * 1024).tiles);
  return 0;
}
"""


def test_ring_is_whole_phases_within_the_limit(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    source, binary = tmp_path / "ring.cpp", tmp_path / "ring"
    source.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", str(ROOT / "edge-infer_b200" / "csrc"), str(source), "-o", str(binary)],
                   check=True)
    result = subprocess.run([str(binary)], capture_output=True, text=True)
    assert result.returncode == 0, result.stdout
    # The device's own limit holds the widest form of every slice.
    assert result.stdout.split() == ["4"] * 4 + ["2"] * 4 + ["1"] * 8
