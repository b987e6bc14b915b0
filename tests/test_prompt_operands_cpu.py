"""Where an int4 prompt tile's dequantised weights stand (csrc/prompt_choice.hpp): beside the accumulators in tensor memory wherever
two operands fit there, with rings that fit shared memory and keep what the kernel relies on."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
PROGRAM = r"""
#include <cstdio>
#include "prompt_choice.hpp"
using namespace ei;
int main() {
  for (int tiles = 1; tiles <= 2; ++tiles)
    for (int columns = 16; columns <= kPromptMaxColumns; columns += 16) {
      PromptTile given{1, tiles, columns, 0, 0, 0};
      if (!prompt_rings(true, given)) continue;
      const PromptTile t = prompt_tensor_operands(given);
      const int used = tiles * columns + t.w_stages * kPromptWeightColumns;
      const bool room = tiles * columns + 2 * kPromptWeightColumns <= kPromptTmemColumns;
      const bool ok = t.tensor_operands == room && (!t.tensor_operands || used <= kPromptTmemColumns) && t.w_stages >= 2 &&
                      t.w_stages <= kPromptWorkerWarps / kPromptTeamWarps && t.raw_stages % t.w_stages == 0 &&
                      t.raw_stages >= t.w_stages && t.raw_stages <= kPromptMaxStages && t.x_stages >= t.w_stages &&
                      t.x_stages >= given.x_stages && t.x_stages <= kPromptMaxStages &&
                      prompt_ring_bytes(t) + kPromptSharedExtra <= kPromptSharedLimit;
      if (!ok) {
        std::printf("%d x %d: rings %d %d %d, tensor %d\n", tiles, columns, t.x_stages, t.w_stages, t.raw_stages, t.tensor_operands);
        return 1;
      }
    }
  return 0;
}
"""


def test_operands_and_rings_fit(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    (tmp_path / "operands.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(ROOT / "edge-infer_b200" / "csrc"), str(tmp_path / "operands.cpp"), "-o",
                    str(tmp_path / "operands")], check=True)
    result = subprocess.run([str(tmp_path / "operands")], capture_output=True, text=True)
    assert result.returncode == 0, result.stdout
