// BF16 small-M GEMM fed by TMA: out[M,N] = x[M,K] * W[N,K]^T (+ bias), M <= 16, K a multiple of 256.
//
// Same skeleton as the int4 kernel (awq_tma.cuh) without the dequantisation: a tile is 8 output features over
// one K slice of up to 4096 inputs, brought into shared memory by one tiled TMA copy (rank-3 map
// [unit of 64 inputs][row][128 bytes], 128-byte swizzle, 64 KiB for a full slice) through a ring of stages on
// mbarriers with bounded waits. A warp owns 256 inputs of the slice; its activation fragments
// are loaded once, 64 contiguous bytes per row and load, and stay in registers (the register-prefetching
// kernel in smallm_gemm.cuh keeps them in shared memory and reads them again for every MMA, which at more
// than 8 rows costs a quarter of the HBM rate on the vocabulary head). The loop is 8 128-bit shared-memory
// loads and 16 mma.sync.m16n8k16 per tile and warp; a lane's 16-byte chunk feeds two MMAs, and because the
// activation fragments take their inputs from the same positions, any fixed assignment of a chunk's eight
// inputs to MMA k-slots is valid. Per phase the warps add their partial accumulators through shared memory
// in a fixed order; K beyond 4096 is split over blocks (ksplit) that write FP32 partials.
//
// A slice of at most 2048 (1024) inputs needs eight (four) of the sixteen warps: two (four) tiles then go side by side
// (kTiles), so that a phase - one barrier, one reduction, one epilogue - covers as many tiles and no warp idles. What
// bounds the projections of a small decoder at one row is latency, not bytes: the 1024-input projections of the 0.6B
// model are 3 to 5 tiles per block, each formerly a phase of its own with a quarter of the warps at work. Measured, with the
// first few tiles of the ring requested ahead: one token of that model 837 -> 799 us, of the 1024-wide layered decoder
// 932 -> 905 us (four tiles); two tiles instead of one, a step of four layers of 1280 inputs 163 -> 153 us at one row and
// 192 -> 180 at eight, of 2048 inputs 212 -> 200 at one row and 229 -> 216 at five. With the whole ring requested ahead and a
// refill that asks for less: 764 and 863 us for those two tokens.
#pragma once

#include <cuda.h>

#include "awq_tma.cuh"
#include "dense_ring.hpp"

namespace ei {

static_assert(kDenseWarps == kGemmWarps, "the ring is laid out for the block of these kernels");

// kTiles (1, 2, 4): tiles per phase, kGemmWarps / kTiles warps each.
template <bool kHigh, int kTiles>
__global__ void __launch_bounds__(kGemmThreads, 1)
    dense_tma_kernel(const __grid_constant__ CUtensorMap weights, const GemmParams p, const DenseLaunch cfg) {
  constexpr int kBlock = kDensePartBlock;
  constexpr int kTileWarps = kGemmWarps / kTiles;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((1024u - (smem_address(smem_raw) & 1023u)) & 1023u);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
  const int slice = blockIdx.x % p.ksplit;
  const int group = blockIdx.x / p.ksplit;
  const int groups = gridDim.x / p.ksplit;
  // Slices in steps of one warp's 256 inputs.
  const int parts_total = p.K / kDenseWarpInputs;
  const int part_begin = int((long long)slice * parts_total / p.ksplit);
  const int parts = int((long long)(slice + 1) * parts_total / p.ksplit) - part_begin;
  const int tiles = p.N / 8;
  const bool pair = p.epilogue == kEpiSiluPair;
  const int chunks = pair ? tiles / 2 : tiles;
  const int per_chunk = pair ? 2 : 1;
  const int item_begin = int((long long)group * chunks / groups) * per_chunk;
  const int item_end = int((long long)(group + 1) * chunks / groups) * per_chunk;
  const int item_count = item_end - item_begin;
  auto tile_of = [&](int item) -> int { return pair ? (item >> 1) + (item & 1) * (tiles / 2) : item; };

  const DenseLayout layout = dense_layout(cfg);
  unsigned char* stages = smem + layout.stage_offset;
  float* part = reinterpret_cast<float*>(smem + layout.part_offset);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + layout.barrier_offset);
  volatile int* failed = reinterpret_cast<volatile int*>(full + kDenseMaxStages);  // set by a thread whose wait ran out
  const uint32_t wait_limit = cfg.wait_limit ? cfg.wait_limit : kAwqWaitLimit;

  auto issue = [&](int index) {
    if (index >= item_count) return;
    const int slot = index % cfg.stages;
    mbarrier_expect_tx(&full[slot], uint32_t(layout.tile_bytes) + (index == 0 ? cfg.extra_tx : 0u));
    tma_load_3d(stages + size_t(slot) * layout.tile_bytes, &weights, 0, tile_of(item_begin + index) * 8,
                part_begin * 4, &full[slot]);
  };
  if (threadIdx.x == 0) {
    for (int s = 0; s < cfg.stages; ++s) mbarrier_init(&full[s], 1);
    *failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    // Weights do not depend on the preceding kernel: the whole ring is requested now and streams while that kernel runs.
    // (With one tile now and the rest behind the activation loads a step of eight layers of 4096 takes 759 us at 8 rows and
    // 804 at 16, instead of 733 and 768; of 2048 350.5 instead of 340.1 at one row, 411.7 instead of 407.6 at 16.)
    for (int index = 0; index < cfg.stages; ++index) issue(index);
  }
  __syncthreads();  // barriers initialised: synchronise while the block would wait for its predecessor anyway
  grid_dependency_wait();
  grid_launch_dependents();

  // A fragments of this warp's 256 inputs: cell (unit u, half h) of lane (g, c) holds inputs
  // [64 u + 32 h + 8 c, + 8) of rows g and g + 8: the four lanes of a row read 64 contiguous bytes per load.
  const int mine = warp / kTileWarps, part_of_tile = warp % kTileWarps;  // tile of the phase, inputs of the slice
  const bool live = part_of_tile < parts;
  uint4 lo[8], hi[8];
  {
    const int k = (part_begin + (live ? part_of_tile : 0)) * kDenseWarpInputs + c * 8;
#pragma unroll
    for (int cell = 0; cell < 8; ++cell) {
      lo[cell] = make_uint4(0, 0, 0, 0);
      hi[cell] = make_uint4(0, 0, 0, 0);
      if (live && g < p.M) lo[cell] = *reinterpret_cast<const uint4*>(p.x + size_t(g) * p.x_stride + k + cell * 32);
      if (kHigh && live && g + 8 < p.M)
        hi[cell] = *reinterpret_cast<const uint4*>(p.x + size_t(g + 8) * p.x_stride + k + cell * 32);
    }
  }

  // Reduction role of this thread: element e of the phase's output unit `unit` (a tile, or a gate and an up tile),
  // share q of `shares` of its partials; the shares are neighbouring lanes.
  const int units = kTiles == 1 ? 1 : pair ? kTiles / 2 : kTiles, shares = 4 / units;
  const int unit = threadIdx.x / (128 * shares), e = (threadIdx.x / shares) & 127, q = threadIdx.x & (shares - 1);
  const int rl = e >> 2, reg = e & 3;
  const int row = (rl >> 2) + (reg >= 2 ? 8 : 0);
  const int col = (rl & 3) * 2 + (reg & 1);
  float best_value = -INFINITY;
  int best_index = 0x7fffffff;
  float gate_sum = 0.0f;  // fused SwiGLU, one tile per phase: the gate tile's sum waits here for the up tile

  // Rows g of the warp's four units in a staged tile [unit][row][128 B]; 16-byte chunk j of row r sits at
  // chunk (j ^ r), and bits 4-6 of lane_base hold g, so chunk (4 h + c) of unit u is at
  // (lane_base + u * 1024) ^ ((4 h + c) << 4).
  const uint32_t stages_address = smem_address(stages);
  const uint32_t lane_base = uint32_t(part_of_tile * 4096 + g * 128 + (g << 4));
  auto shared_u128 = [](uint32_t address) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(address));
    return v;
  };

  int slot = 0;
  uint32_t parity = 0;
  // Giving up is the block's decision: a thread whose wait ran out raises the flag before the phase's block-wide
  // barrier; every thread reads it after the barrier and acts on it at the top of the next phase.
  int gave_up = 0, tiles_done = 0;
  for (int index = 0, phase = 0; index < item_count && !gave_up; index += kTiles, phase ^= 1) {
    const bool here = index + mine < item_count;
    const bool ok = !here || mbarrier_wait(&full[slot + mine], parity, wait_limit);
    if (!ok) *failed = 1;
    float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f}, other[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (live && here && ok) {
      const uint32_t tile_address = stages_address + uint32_t(slot + mine) * uint32_t(layout.tile_bytes) + lane_base;
      uint4 w[8];
#pragma unroll
      for (int cell = 0; cell < 8; ++cell)
        w[cell] = shared_u128((tile_address + uint32_t(cell >> 1) * 1024u) ^ uint32_t((((cell & 1) << 2) + c) << 4));
#pragma unroll
      for (int cell = 0; cell < 8; ++cell) {
        if (kHigh) {
          mma_bf16_16816(acc, lo[cell].x, hi[cell].x, lo[cell].y, hi[cell].y, w[cell].x, w[cell].y);
          mma_bf16_16816(other, lo[cell].z, hi[cell].z, lo[cell].w, hi[cell].w, w[cell].z, w[cell].w);
        } else {
          mma_bf16_16816(acc, lo[cell].x, 0u, lo[cell].y, 0u, w[cell].x, w[cell].y);
          mma_bf16_16816(other, lo[cell].z, 0u, lo[cell].w, 0u, w[cell].z, w[cell].w);
        }
      }
      acc[0] += other[0]; acc[1] += other[1]; acc[2] += other[2]; acc[3] += other[3];
    }
    slot += kTiles;
    if (slot == cfg.stages) {
      slot = 0;
      parity ^= 1;
    }
    float* part_phase = part + size_t(phase) * kGemmWarps * kBlock;
    *reinterpret_cast<float4*>(part_phase + warp * kBlock + lane * 4) = make_float4(acc[0], acc[1], acc[2], acc[3]);
    __syncthreads();
    // Every warp has finished reading these stages: refill them with the tiles `stages` ahead. Not after a wait that ran
    // out: a barrier whose phase has not completed cannot be armed again, nor could the drain below tell its copies apart.
    // (Of one tile a phase this thread's own wait tells.)
    if (threadIdx.x == 0 && index + cfg.stages < item_count && (kTiles == 1 ? ok : !*failed))
      for (int t = 0; t < kTiles; ++t) issue(index + cfg.stages + t);
    gave_up = *failed;
    tiles_done = index + kTiles;

    // Fixed-order reduction: share q adds the partials of its tile's warps q, q + shares, ... in that order and the
    // shares are combined by shuffles, so an output sees the same additions in every run.
    auto total_of = [&](int tile) {
      const float* src = part_phase + size_t(tile) * kTileWarps * kBlock + e;
      float sum = 0.0f;
      if (shares == 4) {
#pragma unroll
        for (int w = 0; w < kTileWarps; w += 4) sum += src[size_t(w + q) * kBlock];
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
      } else if (shares == 2) {
#pragma unroll
        for (int w = 0; w < kTileWarps; w += 2) sum += src[size_t(w + q) * kBlock];
      } else {
#pragma unroll
        for (int w = 0; w < kTileWarps; ++w) sum += src[size_t(w) * kBlock];
      }
      if (shares >= 2) sum += __shfl_xor_sync(0xffffffffu, sum, 1);
      return sum;
    };
    auto store_pair = [&](int n, float gate, float up) {  // n: feature of the up half
      const int out_n = n - p.N / 2;
      if (p.bias) {
        gate += __bfloat162float(p.bias[out_n]);
        up += __bfloat162float(p.bias[n]);
      }
      p.out[size_t(row) * p.out_stride + out_n] = __float2bfloat16_rn(gated_pair_value(p.glu, p.glu_limit, gate, up));
    };
    const int first = pair && kTiles > 1 ? unit * 2 : unit;  // first tile of this thread's unit
    float sum = total_of(first), up_sum = 0.0f;
    if (pair && kTiles > 1) up_sum = total_of(first + 1);
    const int item = item_begin + index + first;
    if (q == 0 && row < p.M && index + first < item_count) {
      const int n = tile_of(item) * 8 + col;
      if (pair) {
        if (kTiles > 1)
          store_pair(tile_of(item + 1) * 8 + col, sum, up_sum);
        else if ((item & 1) == 0)
          gate_sum = sum;
        else
          store_pair(n, gate_sum, sum);
      } else if (p.epilogue == kEpiPartial) {
        p.partial[(size_t(slice) * p.M + row) * p.N + n] = sum;
      } else {
        if (p.bias) sum += __bfloat162float(p.bias[n]);
        const bf16 rounded = __float2bfloat16_rn(activated_value(p.activation, sum));
        p.out[size_t(row) * p.out_stride + n] = rounded;
        if (p.epilogue == kEpiArgmax) {
          float value = __bfloat162float(rounded);
          if (isnan(value)) value = -INFINITY;
          if (value > best_value || (value == best_value && n < best_index)) {
            best_value = value;
            best_index = n;
          }
        }
      }
    }
  }

  if (gave_up) {
    if (threadIdx.x == 0) {
      if (p.status) atomicOr(p.status, 4);
      // A block never leaves while a copy into its shared memory may be in flight: give every tile still in
      // the ring (the phase that gave up and the `stages` tiles requested from there on, of one tile a phase also the one
      // requested after it; if it was not, the parity asked for is that of a phase long past) its chance to land (bounded
      // again).
      const int requested = tiles_done - (kTiles == 1 ? 0 : kTiles) + cfg.stages;
      for (int back = max(0, tiles_done - kTiles); back < min(item_count, requested); ++back)
        mbarrier_wait(&full[back % cfg.stages], uint32_t((back / cfg.stages) & 1), wait_limit);
    }
    __syncthreads();
    return;
  }

  if (p.epilogue == kEpiArgmax) {
    // An element owner always sees the same output row; warp r folds the 8 owners of row r in each unit.
    __syncthreads();
    float* values = part;
    int* indices = reinterpret_cast<int*>(part + 128 * kTiles);
    if (q == 0) {
      values[unit * 128 + e] = best_value;
      indices[unit * 128 + e] = best_index;
    }
    __syncthreads();
    float bv = -INFINITY;
    int bi = 0x7fffffff;
    if (lane < 8 * kTiles) {
      const int owner = (lane >> 3) * 128 + ((warp & 7) * 4 + ((lane >> 1) & 3)) * 4 + (warp >= 8 ? 2 : 0) + (lane & 1);
      bv = values[owner];
      bi = indices[owner];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float value = __shfl_xor_sync(0xffffffffu, bv, o);
      const int index = __shfl_xor_sync(0xffffffffu, bi, o);
      if (value > bv || (value == bv && index < bi)) {
        bv = value;
        bi = index;
      }
    }
    if (lane == 0) {
      p.best_value[blockIdx.x * 16 + warp] = bv;
      p.best_index[blockIdx.x * 16 + warp] = bi;
    }
  }
}

}  // namespace ei
