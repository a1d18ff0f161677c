// Instantiations and host-side dispatch of the single-CTA points of 128 and 256 channels of the tensor-core convolution kernel
// (conv_tc_kernel.cuh) with sixteen epilogue warps.  A translation unit of its own so that it compiles beside the others.
#include "conv_tc_kernel.cuh"

namespace gieb {
namespace {

#define GIEB_TC_DISPATCH(FN, ...) \
  switch (tile_m / 128 * 100000 + tile_n * 100 + tile_k) { \
    case 1 * 100000 + 128 * 100 + 16: GIEB_TC_EITHER(FN, 128, 16, 1, 16, false, false, __VA_ARGS__); \
    case 2 * 100000 + 128 * 100 + 16: GIEB_TC_EITHER(FN, 128, 16, 2, 16, false, false, __VA_ARGS__); \
    case 1 * 100000 + 128 * 100 + 32: GIEB_TC_EITHER(FN, 128, 32, 1, 16, false, false, __VA_ARGS__); \
    case 2 * 100000 + 128 * 100 + 32: GIEB_TC_EITHER(FN, 128, 32, 2, 16, false, false, __VA_ARGS__); \
    case 1 * 100000 + 128 * 100 + 64: GIEB_TC_EITHER(FN, 128, 64, 1, 16, false, false, __VA_ARGS__); \
    case 2 * 100000 + 128 * 100 + 64: GIEB_TC_EITHER(FN, 128, 64, 2, 16, false, false, __VA_ARGS__); \
    case 1 * 100000 + 256 * 100 + 16: GIEB_TC_EITHER(FN, 256, 16, 1, 16, false, false, __VA_ARGS__); \
    case 2 * 100000 + 256 * 100 + 16: GIEB_TC_EITHER(FN, 256, 16, 2, 16, false, false, __VA_ARGS__); \
    case 1 * 100000 + 256 * 100 + 32: GIEB_TC_EITHER(FN, 256, 32, 1, 16, false, false, __VA_ARGS__); \
    case 2 * 100000 + 256 * 100 + 32: GIEB_TC_EITHER(FN, 256, 32, 2, 16, false, false, __VA_ARGS__); \
    case 1 * 100000 + 256 * 100 + 64: GIEB_TC_EITHER(FN, 256, 64, 1, 16, false, false, __VA_ARGS__); \
    case 2 * 100000 + 256 * 100 + 64: GIEB_TC_EITHER(FN, 256, 64, 2, 16, false, false, __VA_ARGS__); \
    default: return cudaErrorInvalidValue; \
  }

}  // namespace

cudaError_t conv_tc_wide16_prepare(int tile_m, int tile_n, int tile_k, bool general, size_t smem_bytes) {
  GIEB_TC_DISPATCH(prepare_point, smem_bytes)
}

cudaError_t conv_tc_wide16_launch(int tile_m, int tile_n, int tile_k, bool general, const CUtensorMap& tm_act, const CUtensorMap& tm_wgt,
                              const CUtensorMap& tm_out, const CUtensorMap& tm_res, const ConvTcParams& p, dim3 grid, size_t smem_bytes,
                              cudaStream_t stream) {
  GIEB_TC_DISPATCH(launch_point, tm_act, tm_wgt, tm_out, tm_res, p, grid, smem_bytes, stream)
}

}  // namespace gieb
