// Host side of the prompt GEMM: eligibility, tensor maps, launch.
#include "prompt_gemm.cuh"

#include <algorithm>
#include <stdexcept>

namespace ei {

namespace {
bool aligned_16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
}  // namespace

bool prompt_gemm_eligible(bool awq, int group_size, int N, int K, const void* x, int x_stride, const void* out,
                          int out_stride) {
  if (N < 16 || N % 16 || K < kPromptBlockK || K % kPromptBlockK) return false;
  if (awq && (group_size != 128 || K % 128)) return false;
  return aligned_16(x) && x_stride % 8 == 0 && aligned_16(out) && out_stride % 8 == 0;
}

namespace {

constexpr size_t kPromptSharedLimit = 227 * 1024;

struct PromptChoice {
  PromptTile tile{};
  double cycles = 0.0;
};

// Estimated SM cycles of a launch: waves x (K blocks x the slowest of a K block's resources + the fixed part), plus
// what a split of K costs. Per K block: the tensor pipe needs columns / 2 cycles per MMA; shared memory moves the
// copies in, the dequantised weights in and, per MMA, 4 KB of weights and 32 bytes per column out, 128 bytes a cycle;
// an SM receives about 75 bytes a cycle from L2; a tile of 128 x 64 int4 weights takes about 520 cycles to dequantise.
// Fixed: about 5000 cycles to start, fill the rings and leave, and about 6 per accumulator column. (Measured per K block,
// cycles at 1.9 GHz: BF16 128 x 96 380, 256 x 112 813, 128 x 240 796; int4 128 x 112 541, 128 x 320 1005-1050, 128 x 416
// 1226, 128 x 256 721.)
double prompt_cycles(bool awq, const PromptTile& t, int ksplit, int rows, int N, int K, bool partial, bool store,
                     int multiprocessors) {
  const int tokens = t.token_tiles * t.columns, mmas = t.feature_tiles * t.token_tiles * (kPromptBlockK / 16);
  const double operand = t.feature_tiles * double(awq ? kPromptRawBytes : kPromptWeightBytes);
  const double copied = tokens * kPromptBlockK * 2.0 + operand;
  const double written = copied + (awq ? t.feature_tiles * double(kPromptWeightBytes) : 0.0);
  const double tensor = mmas * t.columns / 2.0;
  const double shared = (written + mmas * (kPromptFeatures * 32.0 + t.columns * 32.0)) / 128.0;
  const double block = std::max({tensor, shared, copied / 75.0, awq ? 520.0 * t.feature_tiles : 0.0});
  const int features = kPromptFeatures * t.feature_tiles;
  const long long blocks = (long long)((N + features - 1) / features) * ((rows + tokens - 1) / tokens) * ksplit;
  const long long waves = (blocks + multiprocessors - 1) / multiprocessors;
  const int k_blocks = (K / kPromptBlockK + ksplit - 1) / ksplit;
  double cycles = 2500.0 + waves * (k_blocks * block + 2500.0 + 6.0 * t.feature_tiles * tokens);
  // Weights beyond what L2 keeps come from HBM (about 3400 bytes a cycle) once per group of tokens: the vocabulary head
  // of the 7B shape over 320 rows takes 321 us in one group of two token tiles, 418 us in two groups.
  const double weights = double(N) * K * (awq ? 0.5 : 2.0);
  const int passes = weights > 64e6 ? (rows + tokens - 1) / tokens : 1;
  cycles = std::max(cycles, passes * weights / 3400.0 + 4000.0);
  if (partial) cycles += double(ksplit) * rows * N * 8.0 / 3000.0;  // FP32 sums out and in again, through L2
  if (store && ksplit > 1) cycles += 4000.0;                        // one more kernel
  return cycles;
}

// Depths of the rings. BF16: as many stages as fit. int4: two rounds of packed weights and as many operand buffers as
// there are teams, as long as that leaves three stages of activations, and no fewer than operand buffers (the kernel's
// rings rely on that); then fewer.
bool prompt_rings(bool awq, PromptTile& t) {
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

// The best shape for a given K split. int4 takes one feature tile: two of them dequantise the weights of 256 features
// per K block, which at 128-240 columns took 1500-1900 cycles where one tile with as many accumulator columns takes 1226.
PromptChoice prompt_choice(bool awq, int rows, int N, int K, int epilogue, bool store, int ksplit, int multiprocessors) {
  PromptChoice best;
  for (int feature_tiles = 1; feature_tiles <= (awq ? 1 : 2); ++feature_tiles)
    for (int token_tiles = 1; token_tiles <= 2; ++token_tiles) {
      const int most = std::min(kPromptMaxColumns, kPromptTmemColumns / (feature_tiles * token_tiles) / 16 * 16);
      const int fewest = (rows + most * token_tiles - 1) / (most * token_tiles);
      for (int groups = fewest; groups < fewest + 4; ++groups) {
        const int parts = groups * token_tiles;
        PromptChoice c;
        c.tile.feature_tiles = feature_tiles;
        c.tile.token_tiles = token_tiles;
        c.tile.columns = std::max(16, ((rows + parts - 1) / parts + 15) / 16 * 16);
        if (c.tile.columns > most || !prompt_rings(awq, c.tile)) continue;
        c.cycles = prompt_cycles(awq, c.tile, ksplit, rows, N, K, epilogue == kEpiPartial, store, multiprocessors);
        if (c.tile.x_stages < 3) c.cycles *= 1.25;  // two stages do not hide a copy's latency
        if (!best.tile.columns || c.cycles < best.cycles) best = c;
      }
    }
  return best;
}

}  // namespace

int prompt_gemm_ksplit(bool awq, int rows, int N, int K, bool store, int multiprocessors, size_t partial_bytes) {
  if (K % 128) return 1;
  int best = 1;
  double cycles = prompt_choice(awq, rows, N, K, store ? kEpiStore : kEpiPartial, store, 1, multiprocessors).cycles;
  for (int ksplit = 2; ksplit <= 16 && K / ksplit >= 4 * kPromptBlockK; ++ksplit) {
    if (size_t(ksplit) * rows * N * sizeof(float) > partial_bytes) break;
    const double c = prompt_choice(awq, rows, N, K, kEpiPartial, store, ksplit, multiprocessors).cycles;
    if (c < cycles * 0.97) {
      cycles = c;
      best = ksplit;
    }
  }
  return best;
}

void launch_prompt_gemm(bool awq, const GemmParams& p, cudaStream_t stream, bool pdl) {
  if (p.M < 1) throw std::invalid_argument("prompt GEMM needs at least one row");
  static thread_local int configured_device = -1, multiprocessors = 0;
  int device = 0;
  EI_CUDA(cudaGetDevice(&device));
  if (configured_device != device) {
    EI_CUDA(cudaDeviceGetAttribute(&multiprocessors, cudaDevAttrMultiProcessorCount, device));
    EI_CUDA(cudaFuncSetAttribute(prompt_gemm_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 int(kPromptSharedLimit)));
    EI_CUDA(cudaFuncSetAttribute(prompt_gemm_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 int(kPromptSharedLimit)));
    configured_device = device;
  }
  const int ksplit = p.epilogue == kEpiPartial ? std::max(1, p.ksplit) : 1;
  if (p.epilogue != kEpiStore && p.epilogue != kEpiPartial)
    throw std::invalid_argument("prompt GEMM stores BF16 outputs or FP32 partial sums");
  if (ksplit > 1 && (p.K % 128 || ksplit > p.K / 128)) throw std::invalid_argument("prompt GEMM: K split too fine");
  if (p.epilogue == kEpiPartial && (!p.partial || (reinterpret_cast<uintptr_t>(p.partial) & 15) || p.N % 4))
    throw std::invalid_argument("prompt GEMM: partial sums need a 16-byte aligned buffer");
  GemmParams q = p;
  q.ksplit = ksplit;
  q.prompt = prompt_choice(awq, p.M, p.N, p.K, p.epilogue, false, ksplit, multiprocessors).tile;
  PromptMaps maps{};
  {
    const cuuint64_t dims[2] = {cuuint64_t(p.K), cuuint64_t(p.M)};
    const cuuint64_t strides[1] = {cuuint64_t(p.x_stride) * 2};
    const cuuint32_t box[2] = {kPromptBlockK, cuuint32_t(q.prompt.columns)};
    encode_map(&maps.x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, p.x, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B,
               "prompt activations");
  }
  if (awq) {
    if (!aligned_16(p.qweight) || (p.K / 8) % 4) throw std::invalid_argument("prompt GEMM: packed weight rows must be 16-byte aligned");
    const cuuint64_t dims[2] = {cuuint64_t(p.K / 8), cuuint64_t(p.N)};
    const cuuint64_t strides[1] = {cuuint64_t(p.K / 8) * 4};
    const cuuint32_t box[2] = {kPromptBlockK / 8, kPromptFeatures};
    encode_map(&maps.weights, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, p.qweight, dims, strides, box,
               CU_TENSOR_MAP_SWIZZLE_NONE, "prompt int4 weights");
  } else {
    if (!aligned_16(p.w) || p.ldw % 8) throw std::invalid_argument("prompt GEMM: weight rows must be 16-byte aligned");
    const cuuint64_t dims[2] = {cuuint64_t(p.K), cuuint64_t(p.N)};
    const cuuint64_t strides[1] = {cuuint64_t(p.ldw) * 2};
    const cuuint32_t box[2] = {kPromptBlockK, kPromptFeatures};
    encode_map(&maps.weights, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, p.w, dims, strides, box,
               CU_TENSOR_MAP_SWIZZLE_128B, "prompt weights");
  }
  const int tokens = q.prompt.token_tiles * q.prompt.columns, features = kPromptFeatures * q.prompt.feature_tiles;
  const size_t shared = size_t(prompt_ring_bytes(q.prompt)) + kPromptSharedExtra;
  const dim3 grid((p.N + features - 1) / features, (p.M + tokens - 1) / tokens, ksplit);
  if (awq)
    launch(prompt_gemm_kernel<true>, grid, dim3(kPromptThreads), shared, stream, pdl, maps, q);
  else
    launch(prompt_gemm_kernel<false>, grid, dim3(kPromptThreads), shared, stream, pdl, maps, q);
}

}  // namespace ei
