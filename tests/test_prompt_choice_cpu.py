"""The shapes that the prompt GEMM's host side chooses (csrc/prompt_choice.hpp), over sizes from one row to the largest: the
rings fit, hold what the kernel relies on, and every token, feature and input belongs to a block."""
import shutil
import subprocess
from pathlib import Path

import pytest

from test_prompt_tiles_gpu import BLOCKS

ROOT = Path(__file__).resolve().parents[1]

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include "prompt_choice.hpp"
using namespace ei;
int check() {
  const int features[] = {16, 144, 272, 1024, 3584, 4608, 12288, 24592, 152064};
  const int inputs[] = {64, 128, 192, 896, 1024, 2304, 4096, 18944};
  for (int awq = 0; awq < 2; ++awq)
    for (int n : features)
      for (int k : inputs)
        for (int rows = 1; rows <= 6000; rows += rows < 600 ? 1 : 97)
          for (int store = 0; store < 2; ++store) {
            if (awq && k % 128) continue;
            const size_t room = size_t(1 + rows % 17) * rows * n * sizeof(float);
            const PromptShapes shapes(awq, rows, n, k, 148);
            const int ksplit = shapes.ksplit(store, room);
            const PromptTile t = shapes.best(ksplit, ksplit > 1 || !store, false).tile;
            const int groups = (rows + t.token_tiles * t.columns - 1) / (t.token_tiles * t.columns);
            bool ok = t.columns >= 16 && t.columns % 16 == 0 && t.columns <= kPromptMaxColumns && groups <= 65535 &&
                      t.feature_tiles >= 1 && t.feature_tiles <= (awq ? 1 : 2) && t.token_tiles >= 1 && t.token_tiles <= 2 &&
                      t.feature_tiles * t.token_tiles * t.columns <= kPromptTmemColumns;
            ok = ok && t.x_stages >= 2 && t.x_stages <= kPromptMaxStages && t.x_stages >= t.w_stages &&
                 prompt_ring_bytes(t) + kPromptSharedExtra <= kPromptSharedLimit;
            if (awq)
              ok = ok && t.w_stages >= 2 && t.w_stages * kPromptTeamWarps <= kPromptWorkerWarps &&
                   t.raw_stages >= t.w_stages && t.raw_stages % t.w_stages == 0 && t.raw_stages <= kPromptMaxStages;
            else
              ok = ok && t.w_stages == t.x_stages;
            ok = ok && ksplit >= 1 && ksplit <= 16 && (ksplit == 1 || (k % 128 == 0 && ksplit <= k / 128 &&
                 size_t(ksplit) * rows * n * sizeof(float) <= room));
            if (!ok) {
              std::printf("awq %d, %d x %d, %d rows: %d x %d x %d, rings %d %d %d, %d slices\n", awq, n, k, rows,
                          t.feature_tiles, t.token_tiles, t.columns, t.x_stages, t.w_stages, t.raw_stages, ksplit);
              return 1;
            }
          }
  return 0;
}
int main(int argc, char** argv) {
  if (argc == 1) return check();
  // awq rows features inputs slices -> the tile and the rings
  int v[5];
  for (int i = 0; i < 5; ++i) v[i] = std::atoi(argv[1 + i]);
  const PromptShapes shapes(v[0], v[1], v[2], v[3], 148);
  const int ksplit = v[4] ? shapes.ksplit(true, size_t(v[4]) * v[1] * v[2] * sizeof(float)) : 1;
  const PromptTile t = shapes.best(ksplit, ksplit > 1, false).tile;
  std::printf("%d %d %d %d %d %d %d\n", t.feature_tiles, t.token_tiles, t.columns, t.x_stages, t.w_stages, t.raw_stages, ksplit);
  return 0;
}
"""


@pytest.fixture(scope="module")
def choice(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    folder = tmp_path_factory.mktemp("choice")
    source, binary = folder / "choice.cpp", folder / "choice"
    source.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(ROOT / "edge-infer_b200" / "csrc"), str(source), "-o",
                    str(binary)], check=True)

    def run(*args):
        return subprocess.run([str(binary), *map(str, args)], capture_output=True, text=True)
    return run


def test_every_choice_fits_the_kernel(choice):
    result = choice()
    assert result.returncode == 0, result.stdout


@pytest.mark.parametrize("awq,rows,n,k,slices,block", BLOCKS)
def test_blocks_that_the_gpu_tests_are_about(choice, awq, rows, n, k, slices, block):
    assert tuple(int(v) for v in choice(awq, rows, n, k, slices).stdout.split()) == block
