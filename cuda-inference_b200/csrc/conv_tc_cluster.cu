// Instantiations and host-side dispatch of the points of the tensor-core convolution kernel (conv_tc_kernel.cuh) that sum the split-K
// slices of a tile inside a cluster.
#include "conv_tc_kernel.cuh"

namespace gieb {
namespace {

// (only a tile_k of 64 has partial last slabs; rows that TMA cannot store are nothing to these kernels)
#define GIEB_TC_CLUSTER_POINTS(FN, BN, EW, ...) \
  case EW * 100000 + BN * 100 + 16: return FN<BN, 16, 1, EW, false, false, false, true>(__VA_ARGS__); \
  case EW * 100000 + BN * 100 + 32: return FN<BN, 32, 1, EW, false, false, false, true>(__VA_ARGS__); \
  case EW * 100000 + BN * 100 + 64: \
    return tail ? FN<BN, 64, 1, EW, false, false, true, true>(__VA_ARGS__) : FN<BN, 64, 1, EW, false, false, false, true>(__VA_ARGS__);

#define GIEB_TC_CLUSTER_DISPATCH(FN, ...) \
  switch (epi_warps * 100000 + tile_n * 100 + tile_k) { \
    GIEB_TC_CLUSTER_POINTS(FN, 32, 8, __VA_ARGS__) \
    GIEB_TC_CLUSTER_POINTS(FN, 64, 8, __VA_ARGS__) \
    GIEB_TC_CLUSTER_POINTS(FN, 128, 8, __VA_ARGS__) \
    GIEB_TC_CLUSTER_POINTS(FN, 256, 8, __VA_ARGS__) \
    GIEB_TC_CLUSTER_POINTS(FN, 256, 16, __VA_ARGS__) \
    default: return cudaErrorInvalidValue; \
  }

}  // namespace

cudaError_t conv_tc_cluster_prepare(int tile_n, int tile_k, int epi_warps, bool tail, size_t smem_bytes) {
  GIEB_TC_CLUSTER_DISPATCH(prepare_point, smem_bytes)
}

cudaError_t conv_tc_cluster_launch(int tile_n, int tile_k, int epi_warps, const CUtensorMap& tm_act, const CUtensorMap& tm_wgt, const ConvTcParams& p,
                                   dim3 grid, size_t smem_bytes, cudaStream_t stream) {
  const bool tail = tile_k == 64 && p.last_ksteps != 4;
  GIEB_TC_CLUSTER_DISPATCH(launch_point, tm_act, tm_wgt, tm_act, tm_act, p, grid, smem_bytes, stream)
}

}  // namespace gieb
