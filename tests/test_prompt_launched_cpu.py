"""The tiles that prompt projections are launched with (csrc/prompt_choice.hpp: the shape chosen and, for int4, where its operands
stand): those that the GPU tests are about, every depth of the rings that int4 blocks of two token tiles get among them, and for
BF16 gate and up projections no second fetch of large weights that one feature tile would spare."""
import shutil
import subprocess
from pathlib import Path

import pytest

from test_prompt_gated_gpu import GATED
from test_prompt_tiles_gpu import BLOCKS

ROOT = Path(__file__).resolve().parents[1]
PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <set>
#include <tuple>
#include "prompt_choice.hpp"
using namespace ei;
// Rings and places of the operands of every int4 block of two token tiles.
int rings() {
  std::set<std::tuple<int, int, int, int>> seen;
  for (int n = 144; n <= 40000; n += 272)
    for (int rows = 33; rows <= 2048; rows += 3) {
      const PromptTile t = prompt_tensor_operands(PromptShapes(true, rows, n, 896, 148).best(1, false, false).tile);
      if (t.token_tiles == 2) seen.insert({t.x_stages, t.w_stages, t.raw_stages, int(t.tensor_operands)});
    }
  for (const auto& [x, w, raw, tensor] : seen) std::printf("%d %d %d %d ", x, w, raw, tensor);
  return 0;
}
int main(int argc, char** argv) {
  if (argc == 1) return rings();
  // awq rows features inputs gated -> the tile, its rings and the groups of tokens
  int v[5];
  for (int i = 0; i < 5; ++i) v[i] = std::atoi(argv[1 + i]);
  PromptTile t = PromptShapes(v[0], v[1], v[2], v[3], 148, v[4]).best(1, false, false).tile;
  if (v[0]) t = prompt_tensor_operands(t);
  const int tokens = t.token_tiles * t.columns;
  std::printf("%d %d %d %d %d %d %d %d\n", t.feature_tiles, t.token_tiles, t.columns, t.x_stages, t.w_stages, t.raw_stages,
              int(t.tensor_operands), (v[1] + tokens - 1) / tokens);
  return 0;
}
"""


@pytest.fixture(scope="module")
def launched(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    folder = tmp_path_factory.mktemp("launched")
    source, binary = folder / "launched.cpp", folder / "launched"
    source.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(ROOT / "edge-infer_b200" / "csrc"), str(source), "-o",
                    str(binary)], check=True)

    def run(*args):
        return tuple(int(v) for v in subprocess.run([str(binary), *map(str, args)], capture_output=True, text=True).stdout.split())
    return run


@pytest.mark.parametrize("awq,rows,hidden,ffn,block", GATED)
def test_gated_blocks(launched, awq, rows, hidden, ffn, block):
    assert launched(awq, rows, 2 * ffn, hidden, 1)[:7] == block


def test_int4_blocks_of_two_token_tiles(launched):
    """In the order of the GPU test's int4 blocks: the rings they are launched with, and no others exist."""
    expected = [(3, 2, 2, 0), (3, 2, 4, 1), (3, 3, 6, 1), (4, 4, 8, 1), (4, 4, 8, 1), (5, 4, 8, 1)]
    blocks = [b for b in BLOCKS if b[0] and not b[4]]
    assert [launched(1, rows, n, k, 0)[3:7] for _, rows, n, k, _, _ in blocks] == expected
    every = launched()
    assert {every[i:i + 4] for i in range(0, len(every), 4)} == set(expected)


@pytest.mark.parametrize("rows", [257, 290, 320, 333, 400])
def test_large_gated_weights_are_fetched_once(launched, rows):
    """37888 x 3584: 272 MB, twice what L2 holds. A tile each for gate and up leaves room for 256 tokens a block."""
    assert launched(0, rows, 37888, 3584, 1)[7] == 1
