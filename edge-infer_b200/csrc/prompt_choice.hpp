// Shape of a prompt GEMM launch (prompt_gemm.cuh): the tile of a block, the depths of its rings and the K split, chosen from
// an estimate of what a K block costs. Plain C++ without CUDA, so that the choice can be checked on its own.
#pragma once

#include <algorithm>
#include <cstddef>

namespace ei {

constexpr int kPromptFeatures = 128;   // features per feature tile = M of one MMA
constexpr int kPromptMaxColumns = 256; // tokens per token tile = N of one MMA, at most
constexpr int kPromptTmemColumns = 512;
constexpr int kPromptBlockK = 64;      // inputs per stage: one 128-byte swizzle row of BF16
constexpr int kPromptMaxStages = 8;
constexpr int kPromptWorkerWarps = 16;
constexpr int kPromptTeamWarps = 4;    // int4: a team of warps dequantises a K block of the one feature tile
constexpr int kPromptWeightBytes = kPromptFeatures * kPromptBlockK * 2;             // 16 KiB BF16 operand per feature tile
constexpr int kPromptRawBytes = kPromptFeatures * (kPromptBlockK / 2);              // 4 KiB of int4 per feature tile
constexpr int kPromptWeightColumns = kPromptBlockK / 2;  // of tensor memory, for the int4 operand of a K block
constexpr size_t kPromptSharedExtra = 1024 /* alignment */ + 512;
constexpr size_t kPromptSharedLimit = 227 * 1024;

// Shape of a block: feature tiles of 128, token tiles of `columns` (a multiple of 16).
struct PromptTile {
  int feature_tiles, token_tiles, columns;
  int x_stages, w_stages;  // K blocks of activations and of BF16 weights in the rings (x_stages >= w_stages)
  int raw_stages;          // int4: K blocks of packed weights; a multiple of w_stages
  bool tensor_operands = false;  // int4: the dequantised weights stand in tensor memory, not in shared memory
};

// Bytes of the rings: activations, weight operands, packed int4 weights (every stage a multiple of 1024).
constexpr int prompt_ring_bytes(const PromptTile& t) {
  return t.x_stages * t.token_tiles * t.columns * kPromptBlockK * 2 +
         t.feature_tiles * ((t.tensor_operands ? 0 : t.w_stages * kPromptWeightBytes) + t.raw_stages * kPromptRawBytes);
}

// The best shape of a launch and what it is estimated to cost, in SM cycles.
struct PromptChoice {
  PromptTile tile{};
  double cycles = 0.0;
};

// Depths of the rings. BF16: as many stages as fit. int4: two rounds of packed weights and as many operand buffers as
// there are teams, as long as that leaves three stages of activations, and no fewer than operand buffers (the kernel's
// rings rely on that); then fewer.
inline bool prompt_rings(bool awq, PromptTile& t) {
  const int room = int(kPromptSharedLimit - kPromptSharedExtra);
  const int x = t.token_tiles * t.columns * kPromptBlockK * 2;
  if (!awq) {
    t.x_stages = t.w_stages = std::min(kPromptMaxStages, room / (x + t.feature_tiles * kPromptWeightBytes));
    t.raw_stages = 0;
    return t.x_stages >= 2;
  }
  for (int wanted = 3; wanted >= 2; --wanted)
    for (t.w_stages = kPromptWorkerWarps / kPromptTeamWarps; t.w_stages >= 2; --t.w_stages)
      for (int rounds = 2; rounds >= 1; --rounds) {
        t.raw_stages = rounds * t.w_stages;
        t.x_stages = 0;
        t.x_stages = std::min(kPromptMaxStages, (room - prompt_ring_bytes(t)) / x);
        if (t.x_stages >= std::max(wanted, t.w_stages)) return true;
      }
  return false;
}

// An int4 tile with its operands in the columns of tensor memory that the accumulators leave, where those are enough for two, and
// the rings as deep as the shared memory so freed allows. Up to 448 tokens; 480 keep theirs in shared memory.
inline PromptTile prompt_tensor_operands(const PromptTile& tile) {
  PromptTile t = tile;
  t.tensor_operands = true;
  const int room = int(kPromptSharedLimit - kPromptSharedExtra), tokens = t.token_tiles * t.columns;
  for (t.w_stages = kPromptWorkerWarps / kPromptTeamWarps; t.w_stages >= 2; --t.w_stages) {
    if (tokens + t.w_stages * kPromptWeightColumns > kPromptTmemColumns) continue;
    for (int rounds = 2; rounds >= 1; --rounds) {
      t.raw_stages = rounds * t.w_stages;
      t.x_stages = 0;
      t.x_stages = std::min(kPromptMaxStages, (room - prompt_ring_bytes(t)) / (tokens * kPromptBlockK * 2));
      if (t.x_stages >= std::max(t.w_stages, tile.x_stages)) return t;
    }
  }
  return tile;
}

// The shapes considered for a problem, each with what its estimate needs at any K split: searched once and compared at every
// split. (Searched again for every split, a BF16 1024 x 3072 call of 64 rows with scratch took 13.1 us of host time; 12.3
// so, and 11.7 when there was no choice to make.)
class PromptShapes {
 public:
  // int4 takes one feature tile: two of them dequantise the weights of 256 features per K block, which at 128-240 columns
  // took 1500-1900 cycles where one tile with as many accumulator columns takes 1226.
  // `gated`: a block computes gate and up features side by side, half a tile of each or, where it takes two tiles, one of each.
  PromptShapes(bool awq, int rows, int N, int K, int multiprocessors, bool gated = false)
      : awq_(awq), gated_(gated), rows_(rows), n_(N), k_(K), multiprocessors_(multiprocessors) {
    for (int feature_tiles = 1; feature_tiles <= (awq ? 1 : 2); ++feature_tiles)
      for (int token_tiles = 1; token_tiles <= 2; ++token_tiles) {
        const int most = std::min(kPromptMaxColumns, kPromptTmemColumns / (feature_tiles * token_tiles) / 16 * 16);
        const int fewest = (rows + most * token_tiles - 1) / (most * token_tiles);
        for (int groups = fewest, last = 0; groups < fewest + 4; ++groups) {
          const int parts = groups * token_tiles;
          PromptTile t{feature_tiles, token_tiles, std::max(16, ((rows + parts - 1) / parts + 15) / 16 * 16), 0, 0, 0};
          if (t.columns == last || t.columns > most || !prompt_rings(awq, t)) continue;
          last = t.columns;
          add(t);
        }
      }
  }

  // The best of them for a K split of `ksplit` slices. `partial`: the sums leave in FP32; `store`: one more kernel then
  // makes the BF16 result of them.
  PromptChoice best(int ksplit, bool partial, bool store) const {
    PromptChoice result;
    const int k_blocks = (k_ / kPromptBlockK + ksplit - 1) / ksplit;
    const double more = split_cycles(ksplit, partial, store);
    for (int i = 0; i < count_; ++i) {
      const Shape& s = shapes_[i];
      const long long waves = (s.blocks * ksplit + multiprocessors_ - 1) / multiprocessors_;
      double cycles = 2500.0 + waves * (k_blocks * s.block + s.fixed);
      const bool pair = gated_ && s.tile.feature_tiles == 2;
      if (pair) cycles *= kPairedTiles;
      cycles = std::max(cycles, s.memory) + more;
      if (s.tile.x_stages < 3) cycles *= 1.25;  // two stages do not hide a copy's latency
      const bool better = cycles < result.cycles || (pair && cycles == result.cycles && result.tile.feature_tiles == 1);
      if (!result.tile.columns || better) result = PromptChoice{s.tile, cycles};
    }
    return result;
  }

  // K slices worth using, none of them shorter than four K blocks, within `partial_bytes` of FP32 sums.
  int ksplit(bool store, size_t partial_bytes) const {
    if (k_ % 128) return 1;
    int chosen = 1;
    double cycles = best(1, !store, store).cycles;
    for (int ksplit = 2; ksplit <= 16 && k_ / ksplit >= 4 * kPromptBlockK; ++ksplit) {
      if (size_t(ksplit) * rows_ * n_ * sizeof(float) > partial_bytes) break;
      if (split_cycles(ksplit, true, store) >= cycles * 0.97) break;  // no shape can make up for it, nor for more slices
      const double c = best(ksplit, true, store).cycles;
      if (c < cycles * 0.97) {
        cycles = c;
        chosen = ksplit;
      }
    }
    return chosen;
  }

 private:
  struct Shape {
    PromptTile tile;
    long long blocks;             // of the grid, per K slice
    double block, fixed, memory;  // cycles of a K block, of a block beside those, and of the weights' way from HBM
  };

  // Estimated SM cycles of a launch: waves x (K blocks x the slowest of a K block's resources + the fixed part), plus
  // what a split of K costs. Per K block: the tensor pipe needs columns / 2 cycles per MMA; shared memory is charged the
  // copies in, the dequantised weights in and, per MMA, 4 KB of weights and 32 bytes per column out, 128 bytes a cycle;
  // an SM receives about 75 bytes a cycle from L2; a tile of 128 x 64 int4 weights takes about 520 cycles to dequantise.
  // Fixed: about 5000 cycles to start, fill the rings and leave, and about 6 per accumulator column. This is an empirical
  // cost that orders shapes, not a bandwidth limit: the charge for shared memory is above most measured K blocks (cycles at
  // 1.9 GHz, estimate in brackets: BF16 128 x 96 380 (448), 256 x 112 813 (848), 128 x 240 796 (736); int4 128 x 112 541
  // (520), 128 x 256 721 (800), 128 x 320 1005-1050 (1056), 128 x 416 1226 (1248)), and launches with FP32 sums come out up
  // to a quarter above their time. Over 332 sizes with every shape and split timed, the one chosen here takes 2.5 % longer
  // than the best in the geometric mean, 27 % at most (int4 3584 x 3584 at 512 rows, 25.8 us for 20.3). Constants fitted to
  // those times leave 1.5 %. The int4 times are of the kernel with its operands in shared memory, and so are the charges: tiles of
  // up to 448 tokens, whose operands stand in tensor memory now, are cheaper than this says and 480 tokens are not.
  void add(const PromptTile& t) {
    const int tokens = t.token_tiles * t.columns, mmas = t.feature_tiles * t.token_tiles * (kPromptBlockK / 16);
    const double operand = t.feature_tiles * double(awq_ ? kPromptRawBytes : kPromptWeightBytes);
    const double copied = tokens * kPromptBlockK * 2.0 + operand;
    const double written = copied + (awq_ ? t.feature_tiles * double(kPromptWeightBytes) : 0.0);
    const double tensor = mmas * t.columns / 2.0;
    const double shared = (written + mmas * (kPromptFeatures * 32.0 + t.columns * 32.0)) / 128.0;
    const int features = kPromptFeatures * t.feature_tiles, groups = (rows_ + tokens - 1) / tokens;
    Shape& s = shapes_[count_++];
    s.tile = t;
    s.blocks = (long long)((n_ + features - 1) / features) * groups;
    s.block = std::max({tensor, shared, copied / 75.0, awq_ ? 520.0 * t.feature_tiles : 0.0});
    s.fixed = 2500.0 + 6.0 * t.feature_tiles * tokens;
    // Weights beyond what L2 keeps come from HBM (about 3400 bytes a cycle) once per group of tokens: the vocabulary head
    // of the 7B shape over 320 rows takes 321 us in one group of two token tiles, 418 us in two groups.
    const double weights = double(n_) * k_ * (awq_ ? 0.5 : 2.0);
    s.memory = (weights > 64e6 ? groups : 1) * weights / 3400.0 + 4000.0;
  }

  double split_cycles(int ksplit, bool partial, bool store) const {
    double cycles = 0.0;
    if (partial) cycles += double(ksplit) * rows_ * n_ * 8.0 / 3000.0;  // FP32 sums out and in again, through L2
    if (store && ksplit > 1) cycles += 4000.0;                          // one more kernel
    return cycles;
  }

  // BF16 gate and up rows in a feature tile each are charged this share of the estimate against half a tile each, whose warps
  // have to exchange their values (half the units a block, so twice the blocks), and they win where both wait for HBM. Fitted
  // between the sizes where one or the other is faster; a layer of a prompt, whole tiles -> half tiles, us: 6144 x 1024 at 33
  // rows 39.2 -> 38.2, at 256 49.2 -> 47.7, but at 700 65.8 -> 68.6 (*); 12288 x 2048 at 40 rows 53.0 -> 49.6, at 128 59.9 ->
  // 57.4, but at 200 66.0 -> 70.0 (*); 37888 x 3584 at 320 rows, where whole tiles take two groups of tokens and fetch the
  // weights twice, 220 -> 195, but at 33 112 -> 118.6 (*). (*: with one kernel for both, about 1 us slower.) Over those, 17920 x 1536, 19456 x 2560 and 24576 x 4096 at 33 to 2040 rows the projection
  // and units chosen here take 1 to 10 % off a layer with a kernel of its own for the units, and are slower nowhere.
  static constexpr double kPairedTiles = 0.85;

  bool awq_, gated_;
  int rows_, n_, k_, multiprocessors_, count_ = 0;
  Shape shapes_[16];
};

}  // namespace ei
