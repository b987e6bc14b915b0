// Ring of K and V tiles of the verify attention (attention.cu): how many buffers a block gets. Plain C++ without CUDA, so that the
// rule can be checked on its own.
#pragma once

namespace ei {

// Three buffers (blocks of one warp, four of them on an SM), four (two tiles; three blocks of two warps on an SM, of three and four
// warps two, for their registers) or six (three tiles, at most two blocks on an SM). `live_blocks`: blocks of the grid that have
// tokens, 0 if the caller does not know; `tiles`: 64-token tiles of a block's chunk.
//
// More blocks on an SM hide one another's chains of loads and arithmetic, but only if there are that many; a deeper ring hides
// the loads of one. Calls of 32 heads behind 8 KV heads, us, six buffers -> fewer:
//   one warp (4 rows), 472 live blocks (30 011 tokens) 34.9 -> 30.8, 256 (32 000 of 65 536) 32.8 -> 36.1, but chunks of up to
//   four tiles are at most 2 % slower with any number of live blocks (4000 of 16 384 13.5 -> 12.4);
//   two warps (6 rows), 512 live blocks of 4 tiles 26.2 -> 24.4, of 8 tiles 37.0 -> 38.3, 256 (16 000 of 32 768) 21.6 -> 24.7,
//   thousands (64 sessions, whole step) 11 245 -> 10 892;
//   three and four warps 44.2 -> 42.7 (9 rows, 32 768 tokens) and never slower; five to seven have an SM each for their registers:
//   within 1 %, but 34.9 -> 35.9 at 8000 of 65 536 (28 heads behind 4, 10 rows).
constexpr int attention_buffers(int warps, int live_blocks, int tiles, int multiprocessors) {
  if (warps >= 5) return 6;
  if (warps >= 3) return 4;
  if (warps == 1 && tiles <= 4) return 3;
  if (live_blocks <= 2 * multiprocessors) return 6;
  if (warps == 1) return 3;
  const bool second_wave_of_few = live_blocks > 3 * multiprocessors && live_blocks <= 4 * multiprocessors;
  return second_wave_of_few && tiles >= 8 ? 6 : 4;
}

}  // namespace ei
