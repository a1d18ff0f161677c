// Instantiations and host-side dispatch of the CTA-pair points of the tensor-core convolution kernel
// (conv_tc_kernel.cuh with PAIR = true): 256-pixel x tile_n-channel tiles computed by clusters of two CTAs with
// tcgen05.mma.cta_group::2.  A translation unit of its own so that it compiles beside the single-CTA points.
#include "conv_tc_kernel.cuh"

namespace gieb {
namespace {

// 64-column tiles drain with 8 epilogue warps, wider ones with 16 (a CTA of a pair always has its SM to itself).
#define GIEB_TC_PAIR_DISPATCH(FN, ...)                                  \
  switch (tile_n * 100 + tile_k) {                                      \
    case 64 * 100 + 16: GIEB_TC_EITHER(FN, 64, 16, 1, 8, true, false, __VA_ARGS__); \
    case 64 * 100 + 32: GIEB_TC_EITHER(FN, 64, 32, 1, 8, true, false, __VA_ARGS__); \
    case 64 * 100 + 64: GIEB_TC_EITHER(FN, 64, 64, 1, 8, true, false, __VA_ARGS__); \
    case 128 * 100 + 16: GIEB_TC_EITHER(FN, 128, 16, 1, 16, true, false, __VA_ARGS__); \
    case 128 * 100 + 32: GIEB_TC_EITHER(FN, 128, 32, 1, 16, true, false, __VA_ARGS__); \
    case 128 * 100 + 64: GIEB_TC_EITHER(FN, 128, 64, 1, 16, true, false, __VA_ARGS__); \
    case 256 * 100 + 16: GIEB_TC_EITHER(FN, 256, 16, 1, 16, true, false, __VA_ARGS__); \
    case 256 * 100 + 32: GIEB_TC_EITHER(FN, 256, 32, 1, 16, true, false, __VA_ARGS__); \
    case 256 * 100 + 64: GIEB_TC_EITHER(FN, 256, 64, 1, 16, true, false, __VA_ARGS__); \
    default: return cudaErrorInvalidValue;                              \
  }

}  // namespace

int conv_tc_pair_epi_warps(int tile_n) { return tile_n >= 128 ? 16 : 8; }

cudaError_t conv_tc_pair_prepare(int tile_n, int tile_k, bool general, size_t smem_bytes) { GIEB_TC_PAIR_DISPATCH(prepare_point, smem_bytes) }

cudaError_t conv_tc_pair_launch(int tile_n, int tile_k, const CUtensorMap& tm_act, const CUtensorMap& tm_wgt, const CUtensorMap& tm_out,
                                const CUtensorMap& tm_res, const ConvTcParams& p, dim3 grid, size_t smem_bytes, cudaStream_t stream) {
  const bool general = conv_tc_general(p, tile_k);
  GIEB_TC_PAIR_DISPATCH(launch_point, tm_act, tm_wgt, tm_out, tm_res, p, grid, smem_bytes, stream)
}

}  // namespace gieb
