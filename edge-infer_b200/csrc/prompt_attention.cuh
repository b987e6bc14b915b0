// Causal attention of many query rows (a prompt segment) on the 5th-generation tensor cores.
//
// A block owns 256 stacked query rows (row x query head of one KV head) as two tiles of 128 and walks the history in tiles
// of 64 tokens. Per tile and query tile: scores S = Q K^T into tensor memory (both operands from shared memory, K as the
// cache's rows stand there), a thread per query row takes the row's 64 scores out, keeps its running maximum and sum, and
// puts the weights back as BF16 into the place the scores had, from where they are the A operand of O += P V (V token-major
// in shared memory is that product's N-major B operand, so nothing is transposed). Scores have two places, so a tile's
// S is computed while the previous one's weights are made; the two query tiles' softmax shares the SM.
//
// Roles of the twelve warps: 0-3 and 4-7 the softmax of one query tile each (a warp reads the 32 lanes of tensor memory that
// its place in the four allows), 8 the TMA copies, 9 and 10 the MMAs of one query tile each, 11 the tensor memory.
//
// The plan is the published one of attention on this generation of tensor cores (FlashAttention-3, arXiv 2407.08608: two query tiles
// whose softmax take turns; FlashAttention-4: weights back through tensor memory, outputs rescaled only beyond a slack).
//
// What bounds it: the chain scores, softmax, product of each query tile, of which two share an SM. 2048 rows of 32 heads behind 8
// KV heads, counters of one launch: tensor pipe 42 % of the SM's active cycles, special functions 32 %, issue slots 47 %, 95
// thousand cycles for the 32 tiles of the longest blocks, some 2900 a tile (where 256 x 64 exponentials at 16 a cycle are 1024 and
// the MMAs 1100). On mma.sync, where a tile's MMAs take their scheduler's issue slots, that layer took 129 us; it takes 60. Whole
// prompts, mma.sync -> this (weights relative to a lagging maximum then): that shape (36 layers, int4) 33.0 -> 30.7 ms; 333 rows
// of 16 heads behind 8 (28 layers) 2.39 -> 2.32; 1500 rows of 16 behind 8 (14 layers of 128 / 128 wide heads) 8.30 -> 8.00; 2048
// rows of 16 heads of 192 / 128 (9 layers) 10.43 -> 10.15. A block costs some 4 to 5 us to start and to leave, so that short
// prompts of the layered designs stay on mma.sync (sized_attention.cu).
//
// kKeys: 128 or 192 values a key. kSplit: weights keep 16 significant bits, as two BF16 terms, one product each.
//
// Every wait is bounded. A role whose wait runs out raises `abort`, which every other wait polls; when all roles have left,
// one thread waits (bounded) for the copies and MMAs in flight, the status bit is raised and the tensor memory freed.
#pragma once

#include "prompt_gemm.cuh"

namespace ei {

constexpr int kPaTile = 64;        // tokens
constexpr int kPaRows = 128;       // stacked query rows of a tile
constexpr int kPaThreads = 384;
constexpr float kPaSlack = 8.0f;     // powers of two
constexpr int kPaTileBytes = kPaTile * 128;  // 64 values of 64 tokens

template <int kKeys>
struct PaLayout {
  static constexpr int kStages = kKeys == 128 ? 4 : 3;
  static constexpr int kKeyBytes = kKeys / 64 * kPaTileBytes, kStageBytes = kKeyBytes + 2 * kPaTileBytes;
  static constexpr int kQueryBytes = kKeys / 64 * kPaRows * 128;  // of one query tile
  static constexpr size_t kTotal = size_t(2) * kQueryBytes + size_t(kStages) * kStageBytes + 1024 /* alignment */ + 512;
};

struct PaShared {
  uint64_t full[4], empty[4];         // K / V stages
  uint64_t queries[2];                // a query tile is in shared memory
  uint64_t scores[2][2], weights[2][2];  // [query tile][place]: S computed, P written
  uint64_t added[2];                  // O holds the tile's product
  uint64_t turns[4][2];               // [warp of four][query tile]: the other tile's warp has made its weights
  uint64_t done;                      // every MMA issued has completed
  uint32_t tmem_base;
  volatile int abort;
  int issued, query_tiles;            // tiles of keys and values, of queries whose copies were requested
};

// 16 columns of the warp's 32 lanes, without waiting for them.
__device__ __forceinline__ void tmem_request16(uint32_t address, uint32_t (&r)[16]) {
  __syncwarp();
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
      "[%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(address)
      : "memory");
}
// Waits for the loads requested; the registers pass through so that nothing reads them earlier.
__device__ __forceinline__ void tmem_loaded(uint32_t (&r)[16]) {
  __syncwarp();
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]),
                 "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])::"memory");
}
// Two FP32 operations in one instruction.
__device__ __forceinline__ float2 fma_pair(float2 a, float2 b, float2 c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(r)
      : "l"(*reinterpret_cast<uint64_t*>(&a)), "l"(*reinterpret_cast<uint64_t*>(&b)), "l"(*reinterpret_cast<uint64_t*>(&c)));
  return *reinterpret_cast<float2*>(&r);
}
__device__ __forceinline__ float2 add_pair(float2 a, float2 b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(*reinterpret_cast<uint64_t*>(&a)), "l"(*reinterpret_cast<uint64_t*>(&b)));
  return *reinterpret_cast<float2*>(&r);
}

// What differs between the callers: where queries come from, how K and V tiles are requested, what becomes of a finished row.
//   int offset, rows, group, kv_head;                       position of row 0, query rows, query heads per KV head
//   float exponent_scale;                                   scores times this are exponents of two
//   bool copied_queries;                                    the group divides 128: a query tile is a box of the queries' map
//   void request_queries(unsigned char* to, int part, int first_row, uint64_t* bar)   64 values of 128 stacked rows
//   const bf16* query(int row, int head_of_group)           otherwise the softmax threads load their rows
//   void request(unsigned char* keys, unsigned char* values, int token, uint64_t* bar)
// `query_tiles` (1 or 2): query tiles of a block.
//   void finish(int row, int head_of_group, float maximum, float sum, Load load)
// with `load(d, v)`: outputs [16 d, 16 d + 16) of the row into v[16] (called by whole warps, `live` tells which lanes store).
// Map of the queries [rows][kv_heads * group * keys] for boxes of 64 values of 128 stacked rows. (Loaded by the threads a
// tile's queries took 5 us; a copy takes one.)
inline bool encode_query_map(CUtensorMap* map, const void* q, int rows, int stride, int group, int kv_heads, int keys) {
  if (kPaRows % group || stride % 8 || (reinterpret_cast<uintptr_t>(q) & 15)) return false;
  const cuuint64_t dims[5] = {64, cuuint64_t(group), cuuint64_t(rows), cuuint64_t(keys / 64), cuuint64_t(kv_heads)};
  const cuuint64_t strides[4] = {cuuint64_t(keys) * 2, cuuint64_t(stride) * 2, 128, cuuint64_t(group) * keys * 2};
  const cuuint32_t box[5] = {64, cuuint32_t(group), cuuint32_t(kPaRows / group), 1, 1};
  encode_map(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, q, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B, "queries");
  return true;
}
// Query tiles a block takes: two share the keys and values they read, but where two would leave half of the chip idle the
// steps of one are shorter (two tiles' exponentials share an SM's 16 a cycle).
inline int pa_query_tiles(int kv_heads, int stacked, int multiprocessors) {
  return kv_heads * ((stacked + 2 * kPaRows - 1) / (2 * kPaRows)) * 2 <= multiprocessors ? 1 : 2;
}

template <int kKeys, bool kSplit, typename Caller>
__device__ __forceinline__ void prompt_attention_block(const Caller& caller, int block, int query_tiles, uint32_t limit,
                                                       uint32_t fault_tx, int* status) {
  using Layout = PaLayout<kKeys>;
  extern __shared__ unsigned char pa_smem_raw[];
  unsigned char* smem = pa_smem_raw + ((1024u - (smem_address(pa_smem_raw) & 1023u)) & 1023u);
  unsigned char* const stages = smem + 2 * Layout::kQueryBytes;
  PaShared* sh = reinterpret_cast<PaShared*>(stages + size_t(Layout::kStages) * Layout::kStageBytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int stacked = caller.rows * caller.group, first_row = block * query_tiles * kPaRows;
  // Tiles that a query tile's last row sees.
  auto tiles_of = [&](int tile) {
    const int first = first_row + tile * kPaRows;
    if (tile >= query_tiles || first >= stacked) return 0;
    return (caller.offset + min(stacked - 1, first + kPaRows - 1) / caller.group + kPaTile) / kPaTile;
  };
  const int tiles[2] = {tiles_of(0), tiles_of(1)}, most = max(tiles[0], tiles[1]);
  const int length = caller.offset + min(stacked - 1, first_row + query_tiles * kPaRows - 1) / caller.group + 1;  // tokens this block may see

  if (threadIdx.x == 0) {
    for (int s = 0; s < Layout::kStages; ++s) {
      mbarrier_init(&sh->full[s], 1);
      mbarrier_init(&sh->empty[s], 2);
    }
    for (int i = 0; i < 2; ++i) {
      mbarrier_init(&sh->queries[i], caller.copied_queries ? 1 : 4);
      mbarrier_init(&sh->added[i], 1);
      for (int b = 0; b < 2; ++b) {
        mbarrier_init(&sh->scores[i][b], 1);
        mbarrier_init(&sh->weights[i][b], 4);
      }
    }
    for (int w = 0; w < 4; ++w)
      for (int i = 0; i < 2; ++i) mbarrier_init(&sh->turns[w][i], 1);
    mbarrier_init(&sh->done, 2);
    sh->abort = 0;
    sh->issued = sh->query_tiles = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 11) tmem_alloc(&sh->tmem_base, 512);
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem = sh->tmem_base;
  // Queries, and the keys and values of the segment, come from the preceding kernel.
  grid_dependency_wait();
  grid_launch_dependents();
  auto wait = [&](uint64_t* bar, uint32_t parity) {
    if (mbarrier_test_wait(bar, parity)) return true;
    for (uint32_t polls = 0; polls < limit; ++polls) {
      if (mbarrier_try_wait(bar, parity)) return true;
      if (sh->abort) return false;
    }
    sh->abort = 1;
    return false;
  };

  if (warp < 8) {
    // ---- softmax: thread = query row ----
    const int tile = warp >> 2, row_of_tile = threadIdx.x & (kPaRows - 1);
    const int index = first_row + tile * kPaRows + row_of_tile;
    const bool live = tile < query_tiles && index < stacked;
    const int row = live ? index / caller.group : 0, head = live ? index - row * caller.group : 0;
    if (!caller.copied_queries) {
      unsigned char* const own = smem + tile * Layout::kQueryBytes + row_of_tile * 128;
      const bf16* q = caller.query(row, head);
#pragma unroll 1
      for (int part = 0; part < kKeys / 64; ++part) {
        uint4 held[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) held[i] = live ? reinterpret_cast<const uint4*>(q + part * 64)[i] : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int i = 0; i < 8; ++i) *reinterpret_cast<uint4*>(own + part * kPaRows * 128 + ((i ^ (row_of_tile & 7)) << 4)) = held[i];
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbarrier_arrive(&sh->queries[tile]);
    }
    const uint32_t lanes = uint32_t((warp & 3) * 32) << 16;
    const uint32_t outputs = tmem + lanes + tile * 256 + 128;
    const int last = caller.offset + row;  // last token the row sees
    float maximum = -INFINITY, sum = 0.0f;
    const bool taking_turns = tiles[1] > 0;  // then tiles[1] >= tiles[0] > 0
    bool ok = true;
    for (int t = 0; t < tiles[tile]; ++t) {
      const int place = t & 1, first = t * kPaTile;
      const uint32_t at = tmem + lanes + tile * 256 + place * 64;
      ok = __all_sync(0xffffffffu, wait(&sh->scores[tile][place], (t >> 1) & 1));
      if (!ok) break;
      tcgen05_fence_after();
      uint32_t s[4][16];
#pragma unroll
      for (int i = 0; i < 4; ++i) tmem_request16(at + i * 16, s[i]);
#pragma unroll
      for (int i = 0; i < 4; ++i) tmem_loaded(s[i]);
      // Causal mask, and beyond the history, where the copy brought whatever the cache holds.
      if (first + kPaTile - 1 > caller.offset) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (first + i * 16 + j > last) s[i][j] = 0xff800000u;
        }
      }
      float tops[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        tops[i] = __uint_as_float(s[i][0]);
#pragma unroll
        for (int j = 1; j < 16; ++j) tops[i] = fmaxf(tops[i], __uint_as_float(s[i][j]));
      }
      const float top = fmaxf(fmaxf(tops[0], tops[1]), fmaxf(tops[2], tops[3]));
      // The weights are powers relative to `maximum`. In one BF16 term they follow the row's true maximum at once, so that its
      // largest weight is exactly 1: relative to an older maximum it would be rounded, the sum would not, and a row that one
      // token dominates would come out 2^-8 off (errors of the last row's logits against 64 bits, 1.7B, 333 rows, eight seeds:
      // 0.01318 lagging, 0.01288 so; 2.183 -> 2.200 ms, and 8B int4, 2048 rows within the noise at 28.8). In two terms they may
      // lag it by kPaSlack: a weight may then reach 2^kPaSlack, sums and products keep their relative precision, and the
      // outputs are hardly ever taken out of tensor memory to be rescaled.
      const bool moved = !kSplit ? top > maximum
                                 : maximum == -INFINITY ? top != -INFINITY : (top - maximum) * caller.exponent_scale > kPaSlack;
      const float previous = maximum;
      if (moved) maximum = top;
      // A row with nothing visible yet keeps -inf; 0 as the exponent's base then makes every weight 0.
      const float base = maximum == -INFINITY ? 0.0f : maximum, shift = -base * caller.exponent_scale;
      const float rescale = moved ? power_of_two((previous - base) * caller.exponent_scale) : 1.0f;
      // The exponentials of the two query tiles take turns, warp by warp (the two warps of a pair share a scheduler and its
      // four exponentials a cycle): while one is at them the other fetches scores, looks for the maximum and hands over.
      if (taking_turns && (tile == 0 ? t > 0 : t < tiles[0])) {
        ok = __all_sync(0xffffffffu, wait(&sh->turns[warp & 3][tile], tile == 0 ? (t - 1) & 1 : t & 1));
        if (!ok) break;
      }
      uint32_t lead[2][16], rest[2][16];
      float2 parts[4] = {};
      const float2 scales = make_float2(caller.exponent_scale, caller.exponent_scale), shifts = make_float2(shift, shift);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
          const float2 x = fma_pair(make_float2(__uint_as_float(s[i][j]), __uint_as_float(s[i][j + 1])), scales, shifts);
          const float2 w = make_float2(power_of_two(x.x), power_of_two(x.y));
          parts[i] = add_pair(parts[i], w);
          const uint32_t both = pack_bf16(w.x, w.y);
          lead[i >> 1][(i & 1) * 8 + j / 2] = both;
          if (kSplit) rest[i >> 1][(i & 1) * 8 + j / 2] = pack_bf16(w.x - bf16_lo(both), w.y - bf16_hi(both));
        }
      }
      if (taking_turns) {
        __syncwarp();
        if (lane == 0) mbarrier_arrive(&sh->turns[warp & 3][tile ^ 1]);
      }
      const float2 total = add_pair(add_pair(parts[0], parts[1]), add_pair(parts[2], parts[3]));
      sum = sum * rescale + (total.x + total.y);
      // The weights take the scores' place: first the leading terms, behind them what those leave.
#pragma unroll
      for (int i = 0; i < 2; ++i) tmem_store16(at + i * 16, lead[i]);
      if (kSplit) {
#pragma unroll
        for (int i = 0; i < 2; ++i) tmem_store16(at + 32 + i * 16, rest[i]);
      }
      if (t > 0) {
        ok = __all_sync(0xffffffffu, wait(&sh->added[tile], (t - 1) & 1));
        if (!ok) break;
        if (__any_sync(0xffffffffu, moved)) {
          tcgen05_fence_after();
#pragma unroll
          for (int i = 0; i < 8; i += 2) {
            uint32_t a[16], b[16];
            tmem_request16(outputs + i * 16, a);
            tmem_request16(outputs + i * 16 + 16, b);
            tmem_loaded(a);
            tmem_loaded(b);
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              a[j] = __float_as_uint(__uint_as_float(a[j]) * rescale);
              b[j] = __float_as_uint(__uint_as_float(b[j]) * rescale);
            }
            tmem_store16(outputs + i * 16, a);
            tmem_store16(outputs + i * 16 + 16, b);
          }
        }
      }
      if (length - first < kPaTile) {
        // Values beyond the history are cleared: a non-finite leftover must not pass through a zero weight. (Both query
        // tiles' warps do it before they hand over their weights, with the same zeros.)
        const int have = length - first;
        ok = __all_sync(0xffffffffu, wait(&sh->full[t % Layout::kStages], (t / Layout::kStages) & 1));
        if (!ok) break;
        unsigned char* values = stages + size_t(t % Layout::kStages) * Layout::kStageBytes + Layout::kKeyBytes;
        for (int i = row_of_tile; i < (kPaTile - have) * 16; i += kPaRows)
          *reinterpret_cast<uint4*>(values + (i & 1) * kPaTileBytes + (have + (i >> 4)) * 128 + ((i >> 1) & 7) * 16) = make_uint4(0, 0, 0, 0);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      }
      tmem_stored();
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbarrier_arrive(&sh->weights[tile][place]);
    }
    if (tiles[tile] > 0) {
      ok = ok && __all_sync(0xffffffffu, wait(&sh->added[tile], (tiles[tile] - 1) & 1));
      if (ok) {
        tcgen05_fence_after();
        caller.finish(live, row, head, maximum, sum, [&](int d, float (&v)[16]) { tmem_load16(outputs + d * 16, v); });
      }
    }
  } else if (warp == 8) {
    // ---- copies ----
    if (lane == 0) {
      if (caller.copied_queries)
        for (int tile = 0; tile < 2 && tiles_of(tile) > 0; ++tile) {
          mbarrier_expect_tx(&sh->queries[tile], uint32_t(Layout::kQueryBytes));
          for (int part = 0; part < kKeys / 64; ++part)
            caller.request_queries(smem + tile * Layout::kQueryBytes + part * kPaRows * 128, part, (first_row + tile * kPaRows) / caller.group,
                                   &sh->queries[tile]);
          sh->query_tiles = tile + 1;
        }
      for (int t = 0; t < most; ++t) {
        const int s = t % Layout::kStages;
        if (t >= Layout::kStages && !wait(&sh->empty[s], (t / Layout::kStages - 1) & 1)) break;
        unsigned char* const keys = stages + size_t(s) * Layout::kStageBytes;
        mbarrier_expect_tx(&sh->full[s], uint32_t(Layout::kStageBytes) + (t == 0 ? fault_tx : 0u));
        caller.request(keys, keys + Layout::kKeyBytes, t * kPaTile, &sh->full[s]);
        sh->issued = t + 1;
      }
    }
  } else if (warp < 11) {
    // ---- MMAs of one query tile ----
    const int tile = warp - 9, n = tiles[tile];
    const uint32_t leader = elect_one();
    constexpr uint32_t kScores = (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(kPaTile >> 3) << 17) | (uint32_t(kPaRows >> 4) << 24);
    // The values' 128 columns are N-major: bit 16.
    constexpr uint32_t kOutputs = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | (uint32_t(128 >> 3) << 17) | (uint32_t(kPaRows >> 4) << 24);
    const uint32_t query_desc = umma_desc_low(smem_address(smem) + tile * Layout::kQueryBytes);
    const uint32_t outputs = tmem + tile * 256 + 128;
    auto score = [&](int t) {
      const int s = t % Layout::kStages;
      if (!__all_sync(0xffffffffu, wait(&sh->full[s], (t / Layout::kStages) & 1))) return false;
      tcgen05_fence_after();
      if (leader) {
        const uint32_t keys = umma_desc_low(smem_address(stages) + s * Layout::kStageBytes);
#pragma unroll
        for (int k = 0; k < kKeys / 16; ++k)
          umma_bf16_ss(tmem + tile * 256 + (t & 1) * 64, query_desc + (k >> 2) * (kPaRows * 128 >> 4) + (k & 3) * 2,
                       keys + (k >> 2) * (kPaTileBytes >> 4) + (k & 3) * 2, kUmmaDescHigh, kScores, k > 0 ? 1u : 0u);
        tcgen05_commit(&sh->scores[tile][t & 1]);
      }
      return true;
    };
    bool ok = n == 0 || (__all_sync(0xffffffffu, wait(&sh->queries[tile], 0)) && score(0));
    for (int t = 0; t < n && ok; ++t) {
      if (t + 1 < n) ok = score(t + 1);
      ok = ok && __all_sync(0xffffffffu, wait(&sh->weights[tile][t & 1], (t >> 1) & 1));
      if (!ok) break;
      tcgen05_fence_after();
      if (leader) {
        const int s = t % Layout::kStages;
        // 64 values of a token are a 128-byte row; the other 64 values' rows kPaTileBytes on; eight tokens 1024 bytes.
        const uint32_t values = (((smem_address(stages) + s * Layout::kStageBytes + Layout::kKeyBytes) & 0x3ffffu) >> 4) |
                                (uint32_t(kPaTileBytes >> 4) << 16);
        const uint32_t weights = tmem + tile * 256 + (t & 1) * 64;
#pragma unroll
        for (int k = 0; k < kPaTile / 16; ++k)
          umma_bf16_ts(outputs, weights + k * 8, values + k * (16 * 128 >> 4), kUmmaDescHigh, kOutputs, k > 0 ? 1u : uint32_t(t));
        if (kSplit) {
#pragma unroll
          for (int k = 0; k < kPaTile / 16; ++k)
            umma_bf16_ts(outputs, weights + 32 + k * 8, values + k * (16 * 128 >> 4), kUmmaDescHigh, kOutputs, 1u);
        }
        tcgen05_commit(&sh->empty[s]);
        tcgen05_commit(&sh->added[tile]);
      }
    }
    // Tiles that only the other query tile sees: each is given back when it is there, not earlier, so that an arrival
    // cannot count for the stage's previous tile.
    for (int t = n; t < most && ok; ++t) {
      ok = __all_sync(0xffffffffu, wait(&sh->full[t % Layout::kStages], (t / Layout::kStages) & 1));
      if (ok && leader) mbarrier_arrive(&sh->empty[t % Layout::kStages]);
    }
    if (leader) tcgen05_commit(&sh->done);
  }
  tcgen05_fence_before();
  __syncthreads();
  if (sh->abort) {  // no role is left to raise it: block-uniform
    if (threadIdx.x == 0) {
      for (uint32_t polls = 0; polls < limit && !mbarrier_try_wait(&sh->done, 0); ++polls) {
      }
      for (int tile = 0; tile < sh->query_tiles; ++tile)
        for (uint32_t polls = 0; polls < limit && !mbarrier_try_wait(&sh->queries[tile], 0); ++polls) {
        }
      // The bytes that the test hook expects beyond the first copy's are taken off, so that its phase completes.
      if (fault_tx) mbarrier_complete_tx(&sh->full[0], fault_tx);
      for (int t = max(0, sh->issued - Layout::kStages); t < sh->issued; ++t)
        for (uint32_t polls = 0; polls < limit && !mbarrier_try_wait(&sh->full[t % Layout::kStages], (t / Layout::kStages) & 1); ++polls) {
        }
      if (status) atomicOr(status, 4);
    }
    __syncthreads();
  }
  tcgen05_fence_after();
  if (warp == 11) {
    __syncwarp();
    tmem_dealloc(tmem, 512);
  }
}

}  // namespace ei
