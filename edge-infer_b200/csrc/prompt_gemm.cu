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

int prompt_gemm_ksplit(bool awq, int rows, int N, int K, bool store, int multiprocessors, size_t partial_bytes) {
  return PromptShapes(awq, rows, N, K, multiprocessors).ksplit(store, partial_bytes);
}

void launch_prompt_gemm(bool awq, const GemmParams& p, cudaStream_t stream, bool pdl) {
  if (p.M < 1) throw std::invalid_argument("prompt GEMM needs at least one row");
  static thread_local int configured_device = -1, multiprocessors = 0;
  int device = 0;
  EI_CUDA(cudaGetDevice(&device));
  if (configured_device != device) {
    EI_CUDA(cudaDeviceGetAttribute(&multiprocessors, cudaDevAttrMultiProcessorCount, device));
    for (const auto kernel : {prompt_gemm_kernel<true, kUngated, false>, prompt_gemm_kernel<true, kUngated, true>,
                              prompt_gemm_kernel<true, kHalfTiles, false>, prompt_gemm_kernel<true, kHalfTiles, true>,
                              prompt_gemm_kernel<false, kUngated, false>, prompt_gemm_kernel<false, kHalfTiles, false>,
                              prompt_gemm_kernel<false, kWholeTiles, false>})
      EI_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kPromptSharedLimit)));
    configured_device = device;
  }
  const int ksplit = p.epilogue == kEpiPartial ? std::max(1, p.ksplit) : 1;
  const bool gated = p.epilogue == kEpiSiluPair;
  if (p.epilogue != kEpiStore && p.epilogue != kEpiPartial && !gated)
    throw std::invalid_argument("prompt GEMM stores BF16 outputs, gated units or FP32 partial sums");
  if (ksplit > 1 && (p.K % 128 || ksplit > p.K / 128)) throw std::invalid_argument("prompt GEMM: K split too fine");
  if (p.epilogue == kEpiPartial && (!p.partial || (reinterpret_cast<uintptr_t>(p.partial) & 15) || p.N % 4))
    throw std::invalid_argument("prompt GEMM: partial sums need a 16-byte aligned buffer");
  GemmParams q = p;
  q.ksplit = ksplit;
  q.prompt = PromptShapes(awq, p.M, p.N, p.K, multiprocessors, gated).best(ksplit, p.epilogue == kEpiPartial, false).tile;
  if (awq) q.prompt = prompt_tensor_operands(q.prompt);
  const bool halves = gated && q.prompt.feature_tiles == 1;  // gate and up rows share a tile and come as a box each
  const cuuint32_t rows_of_box = halves ? kPromptFeatures / 2 : kPromptFeatures;
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
    const cuuint32_t box[2] = {kPromptBlockK / 8, rows_of_box};
    encode_map(&maps.weights, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, p.qweight, dims, strides, box,
               CU_TENSOR_MAP_SWIZZLE_NONE, "prompt int4 weights");
  } else {
    if (!aligned_16(p.w) || p.ldw % 8) throw std::invalid_argument("prompt GEMM: weight rows must be 16-byte aligned");
    const cuuint64_t dims[2] = {cuuint64_t(p.K), cuuint64_t(p.N)};
    const cuuint64_t strides[1] = {cuuint64_t(p.ldw) * 2};
    const cuuint32_t box[2] = {kPromptBlockK, rows_of_box};
    encode_map(&maps.weights, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, p.w, dims, strides, box,
               CU_TENSOR_MAP_SWIZZLE_128B, "prompt weights");
  }
  const int tokens = q.prompt.token_tiles * q.prompt.columns, features = kPromptFeatures * q.prompt.feature_tiles;
  const size_t shared = size_t(prompt_ring_bytes(q.prompt)) + kPromptSharedExtra;
  const dim3 grid((p.N + features - 1) / features, (p.M + tokens - 1) / tokens, ksplit);
  const bool tensor = q.prompt.tensor_operands;
  const auto kernel = !awq    ? (halves ? prompt_gemm_kernel<false, kHalfTiles, false>
                                 : gated ? prompt_gemm_kernel<false, kWholeTiles, false>
                                         : prompt_gemm_kernel<false, kUngated, false>)
                      : gated ? (tensor ? prompt_gemm_kernel<true, kHalfTiles, true> : prompt_gemm_kernel<true, kHalfTiles, false>)
                              : (tensor ? prompt_gemm_kernel<true, kUngated, true> : prompt_gemm_kernel<true, kUngated, false>);
  launch(kernel, grid, dim3(kPromptThreads), shared, stream, pdl, maps, q);
}

}  // namespace ei
