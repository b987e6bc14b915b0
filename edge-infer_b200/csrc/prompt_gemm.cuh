// Prompt (prefill) GEMM for sm_100a on the 5th-generation tensor cores: out[T,N] = x[T,K] * W[N,K]^T (+ bias) for
// T in the hundreds or thousands, W int4 (AWQ, group 128) or BF16.
//
// With many rows the projection is no longer bound by weight bytes but by arithmetic, so the small-M streaming
// kernels (one pass over the weights per 16 rows) are the wrong tool: here every weight is dequantised once per
// 256 tokens and multiplied on tcgen05.
//
// The features are the M of the MMA (128 per tile, one or two tiles per block) and the tokens its N: a block owns
// feature_tiles x 128 features (int4: 128) and token_tiles x columns tokens (columns a multiple of 16, at most 256; at
// most 512 accumulator columns in all). So a tile is cut to the rows there are - 333 tokens are two tiles of 176, 320 are
// one pass over the weights with two tiles of 160 - where a tile of 128 tokens as M would leave up to 127 of them empty
// and dequantise the weights once more. The host chooses the shape from the cost of a K block (prompt_choice.hpp).
// A block walks K in blocks of 64 inputs through rings of their own for activations, weights and, int4, packed weights (a
// ring's depth has to hide its own latency only: a copy's for activations and packed weights, the way from a free operand
// buffer through conversion and MMA for the dequantised ones):
//   * two threads (warps 16 and 19) issue the TMA copies, one those of the weights and one those of the activations: the
//     activations as [columns tokens][64 inputs] BF16 boxes with the 128-byte swizzle (the K-major operand layout of
//     tcgen05.mma), BF16 weights as [128 features][64 inputs] swizzled boxes, int4 weights as raw [128 rows][32 bytes]
//     boxes. The weights of the ring's first round are requested before the kernel waits for its predecessor, which does
//     not write them;
//   * for int4, teams of four of warps 0-15 turn the raw boxes into the BF16 operand, a row per lane of tensor memory, in the
//     columns that the accumulators leave: team j of w_stages every w_stages-th K block, with the exact dequantisation of the
//     small-M kernels (dequant_pair: round_bf16((w - z) * scale)); they arrive on the K block's `ready` barrier when their
//     stores have completed. Shared memory is what a K block of many tokens is bound by (activations in, operands out): an
//     operand in shared memory cost 128 cycles of stores (twice that while rows r and r + 4 met in a bank) and 32 a MMA of
//     loads. 8B int4, 2048 rows: 30.4 ms with the conflict, 29.2 without, 28.5 from tensor memory; batches of 64 x 5 rows, 7B
//     int4: 9.45, 9.40, 9.24 (each row of figures in turn on one GPU; the batch takes 9.2 to 9.9 ms from GPU to GPU);
//   * one warp or, with more than one accumulator, two (warps 17 and 18) issue, per K block, feature tile and token
//     tile, four tcgen05.mma (M 128, N columns, K 16) that accumulate in tensor memory, and commit the K block's `empty`
//     barrier, which hands both operands' buffers back;
//   * after the last K block warps 0-15 read the accumulators with tcgen05.ld (warp w: features 32 (w % 4) ..., every
//     fourth group of 16 tokens from w / 4). A lane is a feature, so the bias is one register and a token's 32 features
//     leave a warp as one 128-byte line of FP32 sums or, after an exchange between neighbouring lanes, as 64 bytes of
//     BF16. For a projection whose sum the residual + norm kernel finishes the FP32 partial sums are stored, K split
//     over blockIdx.z so that few tiles still fill the SMs.
// What bounds it, by leaving parts out in copies of the kernel: for small tiles the instruction chain of the warp that
// issues the MMAs. With one lane walking the issuing loop a K block of a 128-feature tile took 575 (BF16) and 800 (int4)
// cycles at any number of tokens; with warp-uniform descriptors, one barrier and one commit per K block it takes 380 and
// 540-560 at up to 160 tokens. Above that it grows with the tile (int4 721 at 256 columns, 1005-1050 at 320, 1226 at 416,
// counted at 1.9 GHz while the operands stood in shared memory), and launches that fill the chip run at the rate its power
// sustains: 320 rows of 37888 x 3584 in 64-68 us, where the sustained cuBLAS rate gives 62-65. Measured, int4, per launch, first form (tiles of 128 tokens as M, 256
// features) -> this one: 37888 x 3584, 320 rows 105 -> 66 us; 24576 x 4096, 2048 rows 344-357 -> 297-331 us (over GPUs);
// BF16: 4096 x 2048, 333 rows 15 -> 9.9 us.
// kGated: the gate and up projection of a feed-forward, whose gated units are all that leaves. Their own kernel cost a launch
// and the pairs' way out and back (6 us at 333 x 12288, 25-37 us at 2048 x 24576); in the epilogue, which nothing overlaps, the
// units take some 15 us of the latter's 314 (the projection alone 300). Whole prompts, separate -> here, each in turn on one GPU:
// 1.7B, 333 rows 2.31 -> 2.18 ms; 8B int4, 2048 rows 30.8 -> 30.5; 1500 rows of the 2048-wide join decoder 8.02 -> 7.67; a batch
// of 64 x 5 rows, 7B int4 9.80 -> 9.57. prompt_choice.hpp has more sizes, and where BF16 takes half tiles.
// (An int4 tile of 480 tokens leaves no columns: its operands stand in shared memory, swizzled, K-major, as BF16 ones do.)
// Rows beyond T and features beyond N are zero-filled by TMA and masked in the epilogue.
//
// Every wait on an mbarrier is bounded. A role whose wait runs out raises a flag in shared memory that every
// other wait polls, so all roles leave their loops. When all have, one thread waits (bounded) for the MMAs issued and the
// copies in flight (prompt_drain), sets bit 2 of GemmParams::status, and the tensor memory is freed before the block
// returns.
#pragma once

#include "awq_tma.cuh"
#include "prompt_choice.hpp"

namespace ei {

constexpr int kPromptThreads = (kPromptWorkerWarps + 4) * 32;

struct PromptMaps {
  CUtensorMap x;        // bf16 [T][K], box [columns][64], 128-byte swizzle
  CUtensorMap weights;  // int4: u32 [N][K/8], box [128][8]; BF16: bf16 [N][K], box [128][64], 128-byte swizzle
};

struct PromptShared {
  // Both operands of a K block are there / have been read, in a ring as long as that of the activations: one wait and
  // one commit per K block, because the warp that issues the MMAs is what bounds a small tile.
  uint64_t ready[kPromptMaxStages], empty[kPromptMaxStages];
  uint64_t raw_full[kPromptMaxStages], raw_empty[kPromptMaxStages];  // packed int4 weights
  uint64_t done;
  uint32_t tmem_base;
  volatile int abort;
  // Where the roles stopped, for prompt_drain: K blocks that the activations' and the weights' copy thread requested, and
  // the first K block of its team that a dequantising warp did not hand over.
  int issued[2], left[kPromptWorkerWarps];
};
static_assert(sizeof(PromptShared) <= kPromptSharedExtra - 1024, "the block's state lies behind the rings");

// ---- tcgen05 wrappers ----------------------------------------------------------------------------------------
__device__ __forceinline__ void tmem_alloc(uint32_t* shared_result, uint32_t columns) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_address(shared_result)),
               "r"(columns)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t address, uint32_t columns) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(address), "r"(columns) : "memory");
}
__device__ __forceinline__ void tcgen05_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tcgen05_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tcgen05_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_address(bar))
               : "memory");
}
// D[tmem_d] (+)= A * B^T, both operands K-major in shared memory, FP32 accumulation. The operands' descriptors are given
// by their low words; the high word is the same for every K-major 128-byte-swizzled operand.
__device__ __forceinline__ void umma_bf16_ss(uint32_t tmem_d, uint32_t desc_a, uint32_t desc_b, uint32_t desc_high,
                                             uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "mov.b64 a, {%1, %3};\n\t"
      "mov.b64 b, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %4, p;\n\t}"
      :
      : "r"(tmem_d), "r"(desc_a), "r"(desc_b), "r"(desc_high), "r"(idesc), "r"(accumulate)
      : "memory");
}
// The loads, stores and waits of tensor memory are instructions of a whole warp that has not parted: each helper brings the
// warp together first, since the code ahead of it may have lanes that store, arrive or take one more trip than others.
__device__ __forceinline__ void tmem_load16(uint32_t address, float (&v)[16]) {
  uint32_t r[16];
  __syncwarp();
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
      "[%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(address)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// The same with A in tensor memory: a row per lane, two inputs per column.
__device__ __forceinline__ void umma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint32_t desc_b, uint32_t desc_high, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 b;\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "mov.b64 b, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %4, p;\n\t}"
      :
      : "r"(tmem_d), "r"(tmem_a), "r"(desc_b), "r"(desc_high), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ void tmem_store16(uint32_t address, const uint32_t (&r)[16]) {
  __syncwarp();
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};" ::
          "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
      "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(address)
      : "memory");
}
__device__ __forceinline__ void tmem_stored() {
  __syncwarp();
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_load8(uint32_t address, float (&v)[8]) {
  uint32_t r[8];
  __syncwarp();
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(address)
               : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

// Shared-memory matrix descriptor of a K-major, 128-byte-swizzled operand: rows 128 bytes apart, groups of eight
// rows 1024 bytes apart; bits [46,48) carry the descriptor version of this architecture, bits [61,64) the swizzle.
__device__ __forceinline__ uint32_t umma_desc_low(uint32_t shared_address) {
  return ((shared_address & 0x3ffffu) >> 4) | (1u << 16);
}
constexpr uint32_t kUmmaDescHigh = uint32_t(1024 >> 4) | (1u << 14) | (2u << 29);
// Instruction descriptor: D FP32, A and B BF16, both K-major, M = 128, N = `columns`.
__device__ __forceinline__ uint32_t prompt_instruction(int columns) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t(columns) >> 3) << 17) | ((uint32_t(kPromptFeatures) >> 4) << 24);
}

// Bounded wait that also gives up as soon as another role of the block has.
__device__ __forceinline__ bool prompt_wait(PromptShared* sh, uint64_t* bar, uint32_t parity, uint32_t limit) {
  if (mbarrier_test_wait(bar, parity)) return true;
  for (uint32_t polls = 0; polls < limit; ++polls) {
    if (mbarrier_try_wait(bar, parity)) return true;
    if (sh->abort) return false;
  }
  sh->abort = 1;
  return false;
}
// 1 in one lane of a converged warp.
__device__ __forceinline__ uint32_t elect_one() {
  uint32_t elected;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(elected));
  return elected;
}
__device__ __forceinline__ void mbarrier_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_address(bar)) : "memory");
}
// Takes `bytes` off what the current phase still expects, as a copy that delivers them would.
__device__ __forceinline__ void mbarrier_complete_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.complete_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_address(bar)), "r"(bytes) : "memory");
}

// After every role has left, one of them early: waits until nothing writes into the block's shared or tensor memory any
// more. A K block's `ready` also counts arrivals that the roles which left still owe (of the other copy thread, of the
// dequantising warps); they are made up for here, so that its phase completes on the bytes of its copies alone and every
// wait ends when they have landed. Without that the int4 form's activations could only be waited for by letting the limit
// run out, once per stage. The bytes that the test hook expects beyond the first copy's are taken off first.
template <bool kAwq>
__device__ __forceinline__ void prompt_drain(PromptShared* sh, const PromptTile& tile, uint32_t extra_tx, uint32_t limit) {
  auto landed = [&](uint64_t* bar, int kb, int stages) {
    for (uint32_t polls = 0; polls < limit; ++polls)
      if (mbarrier_try_wait(bar, (kb / stages) & 1)) return;
  };
  landed(&sh->done, 0, 1);
  if (extra_tx) mbarrier_complete_tx(kAwq ? &sh->raw_full[0] : &sh->ready[0], extra_tx);
  const int stages = tile.x_stages, activations = sh->issued[0], weights = sh->issued[1];
  if (kAwq)
    for (int kb = max(0, weights - tile.raw_stages); kb < weights; ++kb)
      landed(&sh->raw_full[kb % tile.raw_stages], kb, tile.raw_stages);
  const int last = kAwq ? activations : max(activations, weights);
  for (int kb = max(0, last - stages); kb < last; ++kb) {
    uint64_t* const bar = &sh->ready[kb % stages];
    int owed = 0;
    if (kAwq) {
      const int* const left = sh->left + kb % tile.w_stages * kPromptTeamWarps;
      for (int w = 0; w < kPromptTeamWarps; ++w) owed += left[w] <= kb;
    } else {
      owed = (activations <= kb) + (weights <= kb);
    }
    for (; owed > 0; --owed) mbarrier_arrive(bar);
    landed(bar, kb, stages);
  }
}

// The gated units of kWords pairs of gate and up values, which replace the gates. Values travel as BF16 pairs, which take half
// the conversions of single ones: the epilogue of 128 x 416 sums is bound by its instructions (two of which per unit are
// those of the exponential and the reciprocal). The SiLU's branches for tiny and very negative gates are taken only where one
// of the values needs them. The gates of tokens and units that do not exist (from value `live` on) are zeros, which would take
// all lanes into those branches (0.4 to 0.5 us of a layer at 33 or 56 rows of 24576 x 4096 and 257 or 333 of 12288 x 2048).
template <int kWords>
__device__ __forceinline__ void gated_units(int glu, float limit, int live, uint32_t (&gate)[kWords], const uint32_t (&up)[kWords]) {
  if (live <= 0) return;
  if (live < 2 * kWords) {
    const uint32_t one = 0x3f80u;
#pragma unroll
    for (int i = 0; i < kWords; ++i) {
      if (2 * i >= live) gate[i] = one | (one << 16);
      else if (2 * i + 1 >= live) gate[i] = (gate[i] & 0xffffu) | (one << 16);
    }
  }
  float least = INFINITY, lowest = INFINITY;
#pragma unroll
  for (int i = 0; i < kWords; ++i) {
    least = fminf(least, fminf(fabsf(bf16_lo(gate[i])), fabsf(bf16_hi(gate[i]))));
    lowest = fminf(lowest, fminf(bf16_lo(gate[i]), bf16_hi(gate[i])));
  }
  if (glu == kGluClamped) {
#pragma unroll
    for (int i = 0; i < kWords; ++i)
      gate[i] = pack_bf16(clamped_glu_value(bf16_lo(gate[i]), bf16_lo(up[i]), limit),
                          clamped_glu_value(bf16_hi(gate[i]), bf16_hi(up[i]), limit));
  } else if (silu_is_rare(least) || silu_is_rare(lowest)) {
#pragma unroll
    for (int i = 0; i < kWords; ++i)
      gate[i] = pack_bf16(silu_multiply_value(bf16_lo(gate[i]), bf16_lo(up[i])),
                          silu_multiply_value(bf16_hi(gate[i]), bf16_hi(up[i])));
  } else {
#pragma unroll
    for (int i = 0; i < kWords; ++i) {
      auto silu = [](float x) { return __fdividef(x, 1.0f + __expf(-x)); };  // silu_value's main branch
      const uint32_t a = pack_bf16(silu(bf16_lo(gate[i])), silu(bf16_hi(gate[i])));
      const uint32_t signs = a ^ up[i];  // a zero of the product's sign, as in multiply_activated
      gate[i] = pack_bf16(__fmaf_ieee_rn(bf16_lo(a), bf16_lo(up[i]), __uint_as_float((signs << 16) & 0x80000000u)),
                          __fmaf_ieee_rn(bf16_hi(a), bf16_hi(up[i]), __uint_as_float(signs & 0x80000000u)));
    }
  }
}

// Where a block has its gate and up rows: in the halves of its one feature tile, or (BF16) in a tile each. Instances of their own:
// one kernel that asked at run time took 1 us of 38 more a layer at 33 rows of 6144 x 1024.
enum PromptGate { kUngated, kHalfTiles, kWholeTiles };

template <bool kAwq, int kGate, bool kTensorOperands>
__global__ void __launch_bounds__(kPromptThreads, 1)
    prompt_gemm_kernel(const __grid_constant__ PromptMaps maps, const GemmParams p) {
  extern __shared__ unsigned char prompt_smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(prompt_smem_raw) + 1023) &
                                                         ~uintptr_t(1023));
  const int columns = p.prompt.columns, block_tokens = p.prompt.token_tiles * columns;
  PromptShared* sh = reinterpret_cast<PromptShared*>(smem + prompt_ring_bytes(p.prompt));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // kGated: the block's rows are n0 ... of the gate and, from `pairs` on, as many of the up projection; the epilogue leaves
  // their gated units. The one feature tile's first and second half are gate and up, or (BF16) the first and second tile.
  constexpr bool kGated = kGate != kUngated;
  const int pairs = p.N / 2;
  const int n0 = blockIdx.x * (kPromptFeatures * p.prompt.feature_tiles / (kGated ? 2 : 1)), t0 = blockIdx.y * block_tokens;
  const int feature_tiles =
      kGated ? p.prompt.feature_tiles : min(p.prompt.feature_tiles, (p.N - n0 + kPromptFeatures - 1) / kPromptFeatures);
  const int token_tiles = min(p.prompt.token_tiles, (p.M - t0 + columns - 1) / columns);
  // K slice of this block (blockIdx.z of p.ksplit): whole quantisation groups, i.e. pairs of K blocks.
  const int slice = blockIdx.z;
  const int pairs_total = p.K / (2 * kPromptBlockK);
  const int kb_begin = p.ksplit > 1 ? int((long long)slice * pairs_total / p.ksplit) * 2 : 0;
  const int kb_end = p.ksplit > 1 ? int((long long)(slice + 1) * pairs_total / p.ksplit) * 2 : p.K / kPromptBlockK;
  const int k_blocks = kb_end - kb_begin;
  const uint32_t limit = p.wait_limit ? p.wait_limit : kAwqWaitLimit;
  const int issuers = min(2, p.prompt.feature_tiles * p.prompt.token_tiles);  // warps that issue MMAs

  if (threadIdx.x == 0) {
    for (int s = 0; s < kPromptMaxStages; ++s) {
      mbarrier_init(&sh->ready[s], kAwq ? 1 + kPromptTeamWarps : 2);
      mbarrier_init(&sh->empty[s], issuers);
      mbarrier_init(&sh->raw_full[s], 1);
      mbarrier_init(&sh->raw_empty[s], kPromptTeamWarps);
    }
    mbarrier_init(&sh->done, issuers);
    sh->abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kPromptWorkerWarps + 1) tmem_alloc(&sh->tmem_base, kPromptTmemColumns);
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem = sh->tmem_base;

  const int tile_bytes = columns * kPromptBlockK * 2;  // activations of one token tile
  const int x_bytes = p.prompt.token_tiles * tile_bytes, w_bytes = p.prompt.feature_tiles * kPromptWeightBytes;
  const int raw_bytes = p.prompt.feature_tiles * kPromptRawBytes;
  unsigned char* const x_ring = smem;
  unsigned char* const w_ring = x_ring + p.prompt.x_stages * x_bytes;
  unsigned char* const raw_ring = kTensorOperands ? w_ring : w_ring + p.prompt.w_stages * w_bytes;
  const uint32_t w_tmem = tmem + kPromptTmemColumns - p.prompt.w_stages * kPromptWeightColumns;  // int4: the operands

  if (warp == kPromptWorkerWarps || warp == kPromptWorkerWarps + 3) {
    // ---- copy threads: one for the weights, one for the activations ----
    const bool weights = warp == kPromptWorkerWarps;
    const int stages = !weights ? p.prompt.x_stages : kAwq ? p.prompt.raw_stages : p.prompt.w_stages;
    uint64_t* const full = weights && kAwq ? sh->raw_full : sh->ready;
    uint64_t* const empty = weights && kAwq ? sh->raw_empty : sh->empty;
    auto request = [&](int kb, int s) {
      if (weights) {
        mbarrier_expect_tx(&full[s], uint32_t(feature_tiles) * (kAwq ? kPromptRawBytes : kPromptWeightBytes) +
                                         (kb == 0 ? p.fault_tx : 0u));
        for (int f = 0; f < feature_tiles; ++f) {
          if (kAwq) {
            unsigned char* const to = raw_ring + s * raw_bytes + f * kPromptRawBytes;
            const int word = (kb_begin + kb) * (kPromptBlockK / 8);
            tma_load_2d(to, &maps.weights, word, n0 + f * kPromptFeatures, &full[s]);
            if (kGated) tma_load_2d(to + kPromptRawBytes / 2, &maps.weights, word, pairs + n0, &full[s]);
          } else {
            unsigned char* const to = w_ring + s * w_bytes + f * kPromptWeightBytes;
            const int input = (kb_begin + kb) * kPromptBlockK;
            tma_load_2d(to, &maps.weights, input, n0 + (kGated ? f * pairs : f * kPromptFeatures), &full[s]);
            if (kGate == kHalfTiles) tma_load_2d(to + kPromptWeightBytes / 2, &maps.weights, input, pairs + n0, &full[s]);
          }
        }
      } else {
        mbarrier_expect_tx(&full[s], uint32_t(token_tiles * tile_bytes));
        for (int mt = 0; mt < token_tiles; ++mt)
          tma_load_2d(x_ring + s * x_bytes + mt * tile_bytes, &maps.x, (kb_begin + kb) * kPromptBlockK, t0 + mt * columns,
                      &full[s]);
      }
    };
    const int early = min(stages, k_blocks);
    if (weights && lane == 0)
      for (int kb = 0; kb < early; ++kb) request(kb, kb);
    grid_dependency_wait();
    grid_launch_dependents();
    if (lane == 0) {
      if (!weights)
        for (int kb = 0; kb < early; ++kb) request(kb, kb);
      int issued = early, slot = 0;
      uint32_t parity = 0;
      for (int kb = early; kb < k_blocks; ++kb) {
        if (!prompt_wait(sh, &empty[slot], parity, limit)) break;
        request(kb, slot);
        issued = kb + 1;
        if (++slot == stages) {
          slot = 0;
          parity ^= 1;
        }
      }
      sh->issued[weights ? 1 : 0] = issued;
    }
  } else if (warp > kPromptWorkerWarps) {
    // ---- MMA warps: warp i issues for the accumulators i, i + issuers, ... (feature tile major). The whole warp walks
    // the loop and one elected lane issues, so that descriptors and counters are warp-uniform values. ----
    grid_dependency_wait();
    grid_launch_dependents();
    const int mine = __shfl_sync(0xffffffffu, warp - (kPromptWorkerWarps + 1), 0);
    if (mine < issuers) {
      const uint32_t leader = elect_one();
      const uint32_t instruction = prompt_instruction(columns);
      const int live = feature_tiles * token_tiles, second = mine + issuers;  // at most two accumulators per warp
      const int f0 = mine / token_tiles, m0 = mine - f0 * token_tiles, f1 = second / token_tiles, m1 = second - f1 * token_tiles;
      const uint32_t a0 = kTensorOperands ? w_tmem : umma_desc_low(smem_address(w_ring) + f0 * kPromptWeightBytes);
      const uint32_t b0 = umma_desc_low(smem_address(x_ring) + m0 * tile_bytes);
      const uint32_t a1 = kTensorOperands ? w_tmem : umma_desc_low(smem_address(w_ring) + f1 * kPromptWeightBytes);
      const uint32_t b1 = umma_desc_low(smem_address(x_ring) + m1 * tile_bytes);
      const uint32_t d0 = tmem + f0 * block_tokens + m0 * columns, d1 = tmem + f1 * block_tokens + m1 * columns;
      const uint32_t w_step = kTensorOperands ? kPromptWeightColumns : uint32_t(w_bytes) >> 4, x_step = uint32_t(x_bytes) >> 4;
      auto multiply = [&](uint32_t d, uint32_t a, uint32_t b, int j, uint32_t accumulate) {
        if (kTensorOperands)
          umma_bf16_ts(d, a + j * 8, b + j * 2, kUmmaDescHigh, instruction, accumulate);
        else
          umma_bf16_ss(d, a + j * 2, b + j * 2, kUmmaDescHigh, instruction, accumulate);
      };
      int w_slot = 0, slot = 0;
      uint32_t parity = 0, w_at = 0, x_at = 0;
      for (int kb = 0; kb < k_blocks; ++kb) {
        if (!__all_sync(0xffffffffu, prompt_wait(sh, &sh->ready[slot], parity, limit))) break;
        tcgen05_fence_after();
        if (leader) {
          if (mine < live) {
#pragma unroll
            for (int j = 0; j < kPromptBlockK / 16; ++j)  // 16 inputs = 32 bytes further along the swizzled row
              multiply(d0, a0 + w_at, b0 + x_at, j, j > 0 ? 1u : uint32_t(kb));
          }
          if (second < live) {
#pragma unroll
            for (int j = 0; j < kPromptBlockK / 16; ++j)
              multiply(d1, a1 + w_at, b1 + x_at, j, j > 0 ? 1u : uint32_t(kb));
          }
          tcgen05_commit(&sh->empty[slot]);
        }
        w_at += w_step;
        x_at += x_step;
        if (++w_slot == p.prompt.w_stages) {
          w_slot = 0;
          w_at = 0;
        }
        if (++slot == p.prompt.x_stages) {
          slot = 0;
          x_at = 0;
          parity ^= 1;
        }
      }
      if (leader) tcgen05_commit(&sh->done);  // arrives when every MMA issued so far has completed
    }
  } else {
    // ---- workers: dequantisation (int4 only), then the epilogue ----
    if (kAwq) {
      // Team j of w_stages converts K blocks j, j + w_stages, ... into operand buffer j, from the raw buffers j, j +
      // w_stages, ...: every buffer belongs to one team, so no team can miss a phase of its barriers. A thread owns one
      // row: 64 inputs = 32 raw bytes = eight 16-byte chunks of the operand row.
      const int teams = p.prompt.w_stages, team = warp / kPromptTeamWarps, row = threadIdx.x & (kPromptFeatures - 1);
      const int first_up = kPromptFeatures / 2;
      const int live_row = min(kGated && row >= first_up ? pairs + n0 + row - first_up : n0 + row, p.N - 1);
      const bf16* scales = p.scales + size_t(live_row) * p.padded_groups;
      const int32_t* zeros = p.zeros + size_t(live_row) * p.zero_stride;
      // Scales and zero points are requested one of the team's K blocks before they are used.
      uint32_t scale_next = 0, zero_next = 0, zero_shift = 0;
      auto request = [&](int kb) {
        const int g = (kb_begin + kb) >> 1;  // 128 inputs per group, 64 per K block
        scale_next = __bfloat16_as_ushort(scales[g]);
        zero_next = uint32_t(zeros[g >> 3]);
        zero_shift = (g & 7) * 4;
      };
      const int end = team < teams ? k_blocks : 0;
      if (team < end) request(team);
      const uint32_t operand = w_tmem + team * kPromptWeightColumns + (uint32_t(warp & 3) * 32 << 16);
      unsigned char* const operand_row = w_ring + team * w_bytes + row * 128;
      // Rows 4-7 of eight read their halves in the other order, so that the eight lanes of a load hit distinct banks, and change
      // them back in registers.
      const unsigned char* const raw_row = raw_ring + row * 32;
      const int first_half = (row & 4) * 4;
      // K block kb takes the operand buffer that K block kb - teams leaves; the MMAs complete in order and the ring of
      // `empty` is at least as long as that of the operands, so the phase waited for is the next one to complete.
      int raw_slot = team, ready_slot = team, left_slot = team;
      uint32_t raw_parity = 0, left_parity = 0;
      int kb = team;
      for (; kb < end; kb += teams) {
        const uint32_t scale2 = scale_next * 0x10001u, zero2 = (0x4300u | ((zero_next >> zero_shift) & 15u)) * 0x10001u;
        if (kb + teams < end) request(kb + teams);
        // The loop is left by whole warps: the barriers and the votes below are warp-wide.
        if (!__all_sync(0xffffffffu, prompt_wait(sh, &sh->raw_full[raw_slot], raw_parity, limit))) break;
        const uint4 raw0 = *reinterpret_cast<const uint4*>(raw_row + raw_slot * raw_bytes + first_half);
        const uint4 raw1 = *reinterpret_cast<const uint4*>(raw_row + raw_slot * raw_bytes + 16 - first_half);
        const bool second = row & 4;  // the second half came first
        const uint32_t words[8] = {second ? raw1.x : raw0.x, second ? raw1.y : raw0.y, second ? raw1.z : raw0.z, second ? raw1.w : raw0.w,
                                   second ? raw0.x : raw1.x, second ? raw0.y : raw1.y, second ? raw0.z : raw1.z, second ? raw0.w : raw1.w};
        if (kb != team) {  // the buffer is fresh in the team's first round
          if (!__all_sync(0xffffffffu, prompt_wait(sh, &sh->empty[left_slot], left_parity, limit))) break;
          left_slot += teams;
          if (left_slot >= p.prompt.x_stages) {
            left_slot -= p.prompt.x_stages;
            left_parity ^= 1;
          }
        }
        if (kTensorOperands) tcgen05_fence_after();
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          uint32_t o[16];
#pragma unroll
          for (int w = 0; w < 4; ++w) {
            // dequant_pair gives (k, k + 4) pairs; the operand wants the eight inputs of a word in order.
            const uint32_t word = words[half * 4 + w];
            const uint32_t p0 = dequant_pair(word, zero2, scale2);
            const uint32_t p1 = dequant_pair(word >> 4, zero2, scale2);
            const uint32_t p2 = dequant_pair(word >> 8, zero2, scale2);
            const uint32_t p3 = dequant_pair(word >> 12, zero2, scale2);
            o[4 * w] = __byte_perm(p0, p1, 0x5410);
            o[4 * w + 1] = __byte_perm(p2, p3, 0x5410);
            o[4 * w + 2] = __byte_perm(p0, p1, 0x7632);
            o[4 * w + 3] = __byte_perm(p2, p3, 0x7632);
          }
          if (kTensorOperands) {
            tmem_store16(operand + half * 16, o);
          } else {
#pragma unroll
            for (int w = 0; w < 4; ++w)
              *reinterpret_cast<uint4*>(operand_row + (((half * 4 + w) ^ (row & 7)) << 4)) =
                  make_uint4(o[4 * w], o[4 * w + 1], o[4 * w + 2], o[4 * w + 3]);
          }
        }
        if (kTensorOperands) {
          tmem_stored();
          tcgen05_fence_before();
        } else {
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
        __syncwarp();
        if (lane == 0) {
          mbarrier_arrive(&sh->ready[ready_slot]);
          mbarrier_arrive(&sh->raw_empty[raw_slot]);
        }
        ready_slot += teams;
        if (ready_slot >= p.prompt.x_stages) ready_slot -= p.prompt.x_stages;
        raw_slot += teams;
        if (raw_slot >= p.prompt.raw_stages) {
          raw_slot = team;
          raw_parity ^= 1;
        }
      }
      if (lane == 0) sh->left[warp] = kb;
    }
    // The dequantisation above reads weights only; the outputs below may be read by the predecessor.
    grid_dependency_wait();
    grid_launch_dependents();
    // ---- epilogue ----
    const bool complete = __all_sync(0xffffffffu, prompt_wait(sh, &sh->done, 0, limit) && !sh->abort);
    tcgen05_fence_after();
    const int quarter = warp & 3;
    const int tokens = min(token_tiles * columns, p.M - t0);  // live ones of this block
    constexpr int kEpilogueStep = kPromptWorkerWarps / 4 * 16;
    const uint32_t lane_base = tmem + (uint32_t(quarter * 32) << 16);
    const bool odd = lane & 1;
    // Two neighbouring lanes (features) exchange one of two tokens' values, so that each stores a pair of features.
    auto store_pairs = [&](const float (&v)[16], int token, int first_feature) {
#pragma unroll
      for (int i = 0; i < 16; i += 2) {
        const float other = __shfl_xor_sync(0xffffffffu, odd ? v[i] : v[i + 1], 1);
        const uint32_t packed = odd ? pack_bf16(other, v[i + 1]) : pack_bf16(v[i], other);
        const int mine = token + i + (odd ? 1 : 0);
        if (mine < p.M && first_feature < p.N)
          *reinterpret_cast<uint32_t*>(p.out + size_t(mine) * p.out_stride + first_feature) = packed;
      }
    };
    // The same for pairs of two tokens' values.
    const uint32_t own_halves = odd ? 0x3276u : 0x5410u;
    auto store_words = [&](const auto& words, int token, int first_unit) {
#pragma unroll
      for (int i = 0; i < int(sizeof(words) / sizeof(uint32_t)); ++i) {
        const uint32_t other = __shfl_xor_sync(0xffffffffu, words[i], 1);
        const int mine = token + 2 * i + (odd ? 1 : 0);
        if (mine < p.M && first_unit < pairs)
          *reinterpret_cast<uint32_t*>(p.out + size_t(mine) * p.out_stride + first_unit) = __byte_perm(words[i], other, own_halves);
      }
    };
    if (kGate == kWholeTiles && complete) {
      // A lane has a unit's gate in one accumulator and its up value in the other.
      const int unit = n0 + quarter * 32 + lane;
      const float gate_bias = p.bias && unit < pairs ? __bfloat162float(p.bias[unit]) : 0.0f;
      const float up_bias = p.bias && unit < pairs ? __bfloat162float(p.bias[pairs + unit]) : 0.0f;
#pragma unroll 1
      for (int c = (warp >> 2) * 16; c < tokens; c += kEpilogueStep) {
        float gate[16], up[16];
        tmem_load16(lane_base + c, gate);
        tmem_load16(lane_base + block_tokens + c, up);
        uint32_t gates[8], ups[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          gates[i] = pack_bf16(gate[2 * i] + gate_bias, gate[2 * i + 1] + gate_bias);
          ups[i] = pack_bf16(up[2 * i] + up_bias, up[2 * i + 1] + up_bias);
        }
        gated_units(p.glu, p.glu_limit, unit < pairs ? p.M - (t0 + c) : 0, gates, ups);
        store_words(gates, t0 + c, unit & ~1);
      }
    } else if (kGate == kHalfTiles) {
      // A unit's gate is in lane l of the first two quarters, its up value in the same lane two quarters on: the two warps
      // hand one another half the tokens of each group of 16 through the rings, which nothing uses any more, and each
      // finishes the other half.
      const bool has_up = quarter >= 2;
      const int unit = n0 + (quarter & 1) * 32 + lane;
      const float bias = p.bias && unit < pairs ? __bfloat162float(p.bias[has_up ? pairs + unit : unit]) : 0.0f;
      uint4* const sent = reinterpret_cast<uint4*>(smem) + warp * 32 + lane;
      const uint4* const received = reinterpret_cast<const uint4*>(smem) + (warp ^ 2) * 32 + lane;
      const int mine = has_up ? 8 : 0;
      if (complete) {
#pragma unroll 1
        for (int c = (warp >> 2) * 16, at = 0; c < tokens; c += kEpilogueStep, at += kPromptWorkerWarps * 32) {
          float v[8];
          tmem_load8(lane_base + c + (8 - mine), v);
          sent[at] = make_uint4(pack_bf16(v[0] + bias, v[1] + bias), pack_bf16(v[2] + bias, v[3] + bias),
                                pack_bf16(v[4] + bias, v[5] + bias), pack_bf16(v[6] + bias, v[7] + bias));
        }
      }
      __syncwarp();  // as for tensor memory
      asm volatile("bar.sync %0, 64;" ::"r"(1 + (warp >> 2) * 2 + (warp & 1)) : "memory");
      if (complete) {
#pragma unroll 1
        for (int c = (warp >> 2) * 16, at = 0; c < tokens; c += kEpilogueStep, at += kPromptWorkerWarps * 32) {
          float v[8];
          tmem_load8(lane_base + c + mine, v);
          const uint4 others = received[at];
          const uint32_t words[4] = {others.x, others.y, others.z, others.w};
          uint32_t gates[4], ups[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint32_t own = pack_bf16(v[2 * i] + bias, v[2 * i + 1] + bias);
            gates[i] = has_up ? words[i] : own;
            ups[i] = has_up ? own : words[i];
          }
          gated_units(p.glu, p.glu_limit, unit < pairs ? p.M - (t0 + c + mine) : 0, gates, ups);
          store_words(gates, t0 + c + mine, unit & ~1);
        }
      }
    } else if (!kGated && complete) {
      for (int f = 0; f < feature_tiles; ++f) {
        const int feature = n0 + f * kPromptFeatures + quarter * 32 + lane;
        const float bias = p.bias && feature < p.N ? __bfloat162float(p.bias[feature]) : 0.0f;
#pragma unroll 1
        for (int c = (warp >> 2) * 16; c < tokens; c += kEpilogueStep) {
          float v[16];
          tmem_load16(lane_base + f * block_tokens + c, v);
          if (p.epilogue == kEpiPartial) {
            if (feature < p.N) {
              float* dst = p.partial + (size_t(slice) * p.M + t0 + c) * p.N + feature;
#pragma unroll
              for (int i = 0; i < 16; ++i)
                if (t0 + c + i < p.M) dst[size_t(i) * p.N] = v[i];
            }
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = activated_value(p.activation, v[i] + bias);
            store_pairs(v, t0 + c, feature & ~1);
          }
        }
      }
    }
  }
  tcgen05_fence_before();
  __syncthreads();
  if (sh->abort) {  // no role is left to raise it: block-uniform
    if (threadIdx.x == 0) {
      prompt_drain<kAwq>(sh, p.prompt, p.fault_tx, limit);
      if (p.status) atomicOr(p.status, 4);
    }
    __syncthreads();
  }
  tcgen05_fence_after();
  if (warp == kPromptWorkerWarps + 1) {
    __syncwarp();
    tmem_dealloc(tmem, kPromptTmemColumns);
  }
}

}  // namespace ei
