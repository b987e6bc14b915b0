// Shared-memory ring of the BF16 weight-streaming kernel (dense_tma.cuh): its layout and the rule that sizes it. Plain C++
// without CUDA, so that the rule can be checked on its own over every K and shared-memory limit.
#pragma once

#include <cstddef>
#include <cstdint>

namespace ei {

constexpr int kDenseMaxStages = 12;
constexpr int kDenseWarps = 16;
constexpr int kDenseWarpInputs = 256;  // inputs of the slice one warp owns: four 64-input units
constexpr int kDensePartBlock = 136;   // floats of partial sums per warp and phase

struct DenseLaunch {
  int stages;           // tiles in flight per block, a multiple of the tiles per phase
  int units_box;        // 64-input units the weight box covers (<= 64)
  uint32_t wait_limit;  // polls before a wait gives up (0: kAwqWaitLimit)
  uint32_t extra_tx;    // test hook: bytes the first copy is expected to deliver beyond what it does (0 in production)
};

struct DenseLayout {
  int tile_bytes;
  size_t stage_offset, part_offset, barrier_offset, total;
};
constexpr DenseLayout dense_layout(const DenseLaunch& cfg) {
  DenseLayout l{};
  l.tile_bytes = cfg.units_box * 1024;
  l.stage_offset = 0;
  l.part_offset = size_t(cfg.stages) * l.tile_bytes;
  l.barrier_offset = l.part_offset + size_t(2) * kDenseWarps * kDensePartBlock * sizeof(float);
  l.total = l.barrier_offset + 128 + 1024;  // + slack to reach a 1024-byte boundary
  return l;
}

constexpr int dense_units_box(int parts) { return parts * 4 < 64 ? parts * 4 : 64; }

struct DenseRing {
  int tiles, stages;  // tiles per phase, tiles in flight; tiles == 0: not even two tiles fit
};
// Ring for slices of at most `parts` x 256 inputs within `limit` bytes of shared memory. Tiles side by side: as many as
// the sixteen warps hold at one warp per 256 inputs, as long as two phases of them fit (with one phase in the ring the
// refill's latency would be paid per phase); otherwise fewer. The kernel steps through the ring by whole phases, so the
// stages are a multiple of the tiles. At the device's own 227 KB every slice gets the widest form.
constexpr DenseRing dense_ring(int parts, size_t limit) {
  for (int tiles = parts <= kDenseWarps / 4 ? 4 : parts <= kDenseWarps / 2 ? 2 : 1; tiles >= 1; tiles /= 2) {
    int stages = kDenseMaxStages / tiles * tiles;
    while (stages >= 2 * tiles && dense_layout(DenseLaunch{stages, dense_units_box(parts), 0, 0}).total > limit)
      stages -= tiles;
    if (stages >= 2 * tiles) return DenseRing{tiles, stages};
  }
  return DenseRing{0, 0};
}

}  // namespace ei
