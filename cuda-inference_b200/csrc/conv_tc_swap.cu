// Instantiations and host-side dispatch of the transposed-accumulator points of the tensor-core convolution kernel
// (conv_tc_kernel.cuh with SWAP = true): NCHW output written by TMA stores.  A translation unit of its own so that it
// compiles beside the others.
#include "conv_tc_kernel.cuh"

namespace gieb {
namespace {

#define GIEB_TC_SWAP_DISPATCH(FN, ...)                                                        \
  switch (tile_m / 128 * 100000 + tile_n * 100 + tile_k) {                                    \
    case 1 * 100000 + 128 * 100 + 16: return FN<128, 16, 1, 8, false, true, false, false>(__VA_ARGS__); \
    case 2 * 100000 + 128 * 100 + 16: return FN<128, 16, 2, 8, false, true, false, false>(__VA_ARGS__); \
    case 1 * 100000 + 128 * 100 + 32: return FN<128, 32, 1, 8, false, true, false, false>(__VA_ARGS__); \
    case 2 * 100000 + 128 * 100 + 32: return FN<128, 32, 2, 8, false, true, false, false>(__VA_ARGS__); \
    case 1 * 100000 + 128 * 100 + 64: GIEB_TC_EITHER(FN, 128, 64, 1, 8, false, true, __VA_ARGS__); \
    case 2 * 100000 + 128 * 100 + 64: GIEB_TC_EITHER(FN, 128, 64, 2, 8, false, true, __VA_ARGS__); \
    case 1 * 100000 + 256 * 100 + 16: return FN<256, 16, 1, 8, false, true, false, false>(__VA_ARGS__); \
    case 2 * 100000 + 256 * 100 + 16: return FN<256, 16, 2, 8, false, true, false, false>(__VA_ARGS__); \
    case 1 * 100000 + 256 * 100 + 32: return FN<256, 32, 1, 8, false, true, false, false>(__VA_ARGS__); \
    case 2 * 100000 + 256 * 100 + 32: return FN<256, 32, 2, 8, false, true, false, false>(__VA_ARGS__); \
    case 1 * 100000 + 256 * 100 + 64: GIEB_TC_EITHER(FN, 256, 64, 1, 8, false, true, __VA_ARGS__); \
    case 2 * 100000 + 256 * 100 + 64: GIEB_TC_EITHER(FN, 256, 64, 2, 8, false, true, __VA_ARGS__); \
    default: return cudaErrorInvalidValue;                                                    \
  }

}  // namespace

cudaError_t conv_tc_swap_prepare(int tile_m, int tile_n, int tile_k, bool general, size_t smem_bytes) {
  GIEB_TC_SWAP_DISPATCH(prepare_point, smem_bytes)
}

cudaError_t conv_tc_swap_launch(int tile_m, int tile_n, int tile_k, const CUtensorMap& tm_act, const CUtensorMap& tm_wgt,
                                const CUtensorMap& tm_out, const ConvTcParams& p, dim3 grid, size_t smem_bytes, cudaStream_t stream) {
  const bool general = conv_tc_general(p, tile_k);  // (NCHW output: only a partial last slab asks for it, at tile_k 64)
  GIEB_TC_SWAP_DISPATCH(launch_point, tm_act, tm_wgt, tm_out, tm_out, p, grid, smem_bytes, stream)
}

}  // namespace gieb
