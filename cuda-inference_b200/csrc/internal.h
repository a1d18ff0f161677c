// Internal interfaces between the C ABI layer (api.cu) and the kernel translation units.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace gieb {

// Device-status codes ORed into a plan's status word by a kernel that gave up on a bounded wait.
enum : uint32_t {
  kStatusProducerTimeout = 1u << 0,
  kStatusMmaTimeout = 1u << 1,
  kStatusEpilogueTimeout = 1u << 2,
};

constexpr int kNumSms = 148;       // streaming multiprocessors of the one supported target (B200): grids are sized in multiples of it
constexpr int kTileM = 128;        // output pixels per CTA tile = TMEM lanes = UMMA M
constexpr int kMaxStages = 8;
constexpr size_t kCtaSmemLimit = 232448;  // 227 KiB opt-in limit of dynamic shared memory per CTA
constexpr int kProducerWarps = 3;  // warps 0..2 issue the TMA loads, slab by slab in turn
// warp 3: MMA issuer and TMEM owner; warps 4..11 (4..19 with 16 epilogue warps): epilogue
static_assert((kProducerWarps + 1) % 4 == 0, "epilogue warp w must sit on TMEM lane quarter w % 4");

// Division by a run-time constant as multiply-high + shift (round-up reciprocal method): exact for 0 <= n < 2^31 and
// 1 <= d < 2^31.  The host builds it once per launch; a device-side divide costs a few cycles instead of ~150.
struct FastDiv {
  uint32_t d, mul, shr;
#if defined(__CUDACC__)
  __host__ __device__
#endif
  static FastDiv make(int divisor) {
    FastDiv f;
    f.d = uint32_t(divisor);
    if (divisor <= 1) {
      f.mul = 0;
      f.shr = 0;
    } else {
      uint32_t lg = 0;  // ceil(log2(d))
      while ((1ull << lg) < uint64_t(f.d)) ++lg;
      const uint32_t p = 31 + lg;
      f.mul = uint32_t(((1ull << p) + f.d - 1) / f.d);
      f.shr = p - 32;
    }
    return f;
  }
#if defined(__CUDACC__)
  __device__ __forceinline__ int div(int n) const { return d == 1 ? n : int(__umulhi(uint32_t(n), mul) >> shr); }
  __device__ __forceinline__ void divmod(int n, int& q, int& r) const {
    q = div(n);
    r = n - q * int(d);
  }
#endif
  int div_host(int n) const { return d == 1 ? n : int((uint64_t(uint32_t(n)) * mul >> 32) >> shr); }
};

#if defined(__CUDACC__)
// Launch with programmatic stream serialization: the grid may be scheduled before the previous kernel of the stream
// has finished; the kernel orders itself with ptx::grid_dep_wait().  Works under stream capture (the edge becomes a
// programmatic dependency of the graph).
// GIEB_DISABLE_PDL=1 in the environment launches every kernel fully serialised (a debugging aid).
bool pdl_enabled();
bool prefetch_enabled();

template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl_cluster(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                      unsigned cluster_x, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  unsigned n = 0;
  if (pdl_enabled()) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  if (cluster_x > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = cluster_x;
    attr[n].val.clusterDim.y = 1;
    attr[n].val.clusterDim.z = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
}
template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
  return launch_pdl_cluster(kernel, grid, block, smem, stream, 1u, static_cast<Args&&>(args)...);
}
#endif

// Everything the tensor-core kernel needs besides the two tensor maps.  Plain data, passed by value.
struct ConvTcParams {
  int m_total;        // GEMM rows: B * P * Q output pixels (modes 0, 1) or box-numbered rows (mode 2)
  int64_t y_elems;    // B * O * P * Q
  int out_channels;   // O (GEMM N)
  int out_h, out_w;   // P, Q
  int pq;             // P * Q
  int kernel_w;       // S (taps are enumerated r-major: tap = r * S + s)
  int c_padded;       // channels of the NHWC copy / prepacked weights
  int kb_per_tap;     // ceil(c_padded / BK)
  int last_ksteps;    // 16-channel steps of a tap's last slab: its columns beyond c_padded (the next tap's) are not multiplied
  int total_kb;       // R * S * kb_per_tap reduction slabs
  int kb_per_split;   // slabs per split-K slice
  int tiles_m, tiles_n;  // tile grid over (pixels, output channels)
  int num_tiles;      // tiles_m * tiles_n * split_k: the list every persistent CTA walks with stride gridDim.x
  int stride_h, stride_w, pad_h, pad_w;
  int stages;
  int relu, has_bias, is_bf16, bias_fp32;
  // 1: FP32 storage computed as TF32 (kind::tf32).  Tile and padding quantities (BK, c_padded, kb_per_tap) stay in
  // 2-byte units, i.e. twice the FP32 element counts; TMA coordinates along channels are halved; Y is float.
  int is_tf32;
  int is_fp8;            // FP8 E4M3 operands (kind::f8f6f4), FP16 output: channel coordinates are twice the 2-byte-unit counts
  // How the activation operand reaches shared memory:
  //   0  im2col-mode TMA over the channel-padded NHWC copy (any kernel / stride / padding)
  //   1  tiled TMA over the same copy seen as the matrix [pixels][c_padded] (1x1, stride 1, pad 0)
  //   2  tiled TMA straight from the caller's NCHW tensor, pixels contiguous (MN-major operand; 1x1, stride 1,
  //      pad 0, H*W % 8 == 0, 16-byte aligned x): no repack of the activations at all.  Rows of the GEMM are then
  //      numbered in 64-pixel boxes that never straddle an image: m_total = batch * boxes_per_image * 64.
  int a_mode;
  int boxes_per_image;  // mode 2: ceil(H*W / 64)
  uint32_t idesc;
  // > 1: split-K slices of one tile form a thread-block cluster (cluster rank = slice) and are summed through
  // distributed shared memory; blockIdx.x = tile * cluster_split + slice, one tile per CTA, `partial` unused.
  int cluster_split;
  FastDiv fd_cluster;
  FastDiv fd_tiles_mn, fd_tiles_n, fd_pq, fd_out_w, fd_kb_per_tap, fd_kernel_w, fd_boxes;  // reciprocals of the fields above
  const void* bias;
  const void* residual;  // optional tensor of the output's shape, layout and type, added before the activation
  int out_nhwc;          // 0: y (and residual, partials) are NCHW; 1: channel-contiguous [B][P][Q][O]
  int out_rows;          // channel-contiguous output goes through shared memory and leaves row by row: 2 = in channel pairs, 1 = singly
  int epi_boxes;         // 2 KiB staging boxes per epilogue warp: 1, or one per chunk that a warp owns (a residual needs those)
  int out_tma, res_tma;  // channel-contiguous output leaves through TMA stores / the residual arrives through TMA loads
  // Transposed-accumulator kernels: swap_tma = y may be written by TMA stores over its {P*Q, O, N} view (16-byte aligned y,
  // P*Q % 8 == 0); out_vec = pixels per store (4, 2 or 1) of the path that handles everything else (a unit that crosses
  // into the next image, or an unaligned y): needs P*Q % out_vec == 0 and y aligned to 2 * out_vec bytes.
  int swap_tma, out_vec;
  void* y;            // output in the storage type (split_k == 1 or cluster reduction)
  float* partial;     // [splits][B*O*P*Q] FP32 partial sums in the output's element order (workspace reduction), else null
  uint32_t* status;
  long long wait_limit;  // SM cycles a device-side wait may last before its role gives up and reports to *status
  int res_vec;           // transposed-accumulator epilogue: the residual may be read as 16-byte vectors (pointer 16-byte aligned)
  uint32_t debug_skip;   // test hook, 0 in production: bit 0 = the producers load nothing, bit 1 = the MMA warp issues nothing
};

// Everything conv_halo_kernel needs besides the tensor maps (see conv_halo.cu for the padded grid and the halo tile).
struct ConvHaloParams {
  const void* bias;      // or null
  const void* residual;  // or null; shape, layout and type of y
  void* y;
  uint32_t* status;
  long long wait_limit;
  int batch;
  int out_channels, out_h, out_w, pq;
  int kernel_w, taps, stride_h, stride_w, pad_h, pad_w;
  int hs, ws;            // rows and columns of the padded grid per image
  int rows_total;        // batch * hs * ws
  int phases, phases_w;  // phases of a halo tile (1 at stride 1)
  int halo_rows;         // rows of one phase in shared memory
  uint32_t a_stage_bytes;
  int a_stages, b_stages;
  int resident;          // the weights of a tile fit b_stages and are the same for all tiles of a CTA: loaded once
  // a phase is `boxes` boxes of box_h padded rows (box_rows = box_h * ws grid rows, box_bytes = 128 * box_rows)
  int boxes, box_h, box_rows;
  uint32_t box_bytes;
  int row_elems;                          // elements of a 128-byte row: 64, or 32 (TF32) or 128 (FP8)
  int c_blocks, last_ksteps;              // blocks of row_elems channels; MMA steps (32 bytes) of the last one
  int taps_per_load, tap_groups;          // filter taps per weight load, loads per channel block
  int total_loads, loads_per_split;       // the reduction in weight loads
  int tiles_n, num_tiles, split;
  int out_nhwc, out_cells, out_rows;      // channel-contiguous output: 16-byte cells allowed; 2 = else channel pairs, 1 = singly
  int relu, is_bf16, is_tf32, is_fp8, bias_fp32;
  uint32_t idesc, debug_skip;
  FastDiv fd_split, fd_tiles_n, fd_groups, fd_kernel_w, fd_ws, fd_hs, fd_gpo, fd_boxes, fd_box_rows;
};
size_t conv_halo_smem_bytes(int tile_n, bool pair, int workers, int taps_per_load, int a_stages, size_t a_stage_bytes, int b_stages, bool staging);
cudaError_t conv_halo_prepare(int tile_n, int workers, bool pair, size_t smem);
cudaError_t conv_halo_launch(int tile_n, int workers, bool pair, const CUtensorMap& tm_act, const CUtensorMap& tm_wgt,
                             const ConvHaloParams& p, dim3 grid, size_t smem, cudaStream_t stream);

// Everything conv_image_kernel needs (see conv_image.cu for strips, positions and groups).
struct ConvImageParams {
  const void* x;         // NCHW, 16-bit
  const void* w;         // OIHW, or [O][R][T * 8] as the plan converts them (prepacked, 16-byte aligned)
  const void* bias;      // or null
  const void* residual;  // or null; shape and layout of y
  void* y;
  uint32_t* status;
  long long wait_limit;
  int channels, in_h, in_w;
  int out_channels, out_h, out_w, pq;
  int kernel_h, kernel_w, stride_h, pad_h;
  int left, shift;                        // positions left of column 0, first tap within the window
  int pitch, segments;                    // positions per strip, in runs of 32
  int group_rows, group_in_rows, rows_per_phase;  // output rows of a group, input rows they read, ceil(group_in_rows / stride_h)
  int groups_per_image, groups;
  uint32_t strip_stage_bytes;
  int words;                              // x may be read as aligned 32-bit column pairs
  int prepacked, is_bf16, bias_fp32, relu;
  int out_nhwc, out_cells;                // channel-contiguous output; in aligned 16-byte cells
  uint32_t idesc, debug_skip;
  FastDiv fd_groups_per_image, fd_pitch, fd_stride_h, fd_segments, fd_cells;  // fd_cells: kernel_h * T
};
constexpr int kImageTileN = 64;                  // output channels of a tile
constexpr int kImageThreads = 32 * (4 + 1 + 8);  // warps that load the image, issue the MMAs, drain the accumulators
// t_positions: positions per window, 2, 4 or 8
size_t conv_image_smem_bytes(int kernel_h, int t_positions, size_t strip_stage_bytes, bool staging);
cudaError_t conv_image_prepare(int t_positions);
cudaError_t conv_image_launch(int t_positions, const ConvImageParams& p, dim3 grid, size_t smem, cudaStream_t stream);

// tile_m is 128 or 256 output pixels per CTA (one or two TMEM accumulators sharing each weight tile).
// pair: the tile belongs to a CTA pair (tile_m = 256), each CTA stages 128 activation rows and tile_n / 2 weight rows.
// epilogue_bytes: staging of the epilogue behind the ring (TMA-store boxes, or the NCHW transposition tiles).
size_t conv_tc_smem_bytes(int tile_m, int tile_n, int tile_k, int stages, size_t epilogue_bytes, bool pair = false);
int conv_tc_epilogue_boxes(int tile_n, int epi_warps);  // chunks of 32 channels one epilogue warp owns per 128 pixels
// epi_warps: 8, or 16 for CTAs that have an SM to themselves (tile_n >= 128 only)
int conv_tc_threads(int epi_warps);
// general: the kernels with partial last slabs and row-wise output (see conv_tc_kernel); a launch takes them when it needs them
bool conv_tc_general(const ConvTcParams& p, int tile_k);
cudaError_t conv_tc_prepare(int tile_m, int tile_n, int tile_k, int epi_warps, bool general, size_t smem_bytes);  // opt in to large dynamic shared memory
// tm_out / tm_res: the output and the residual as 2-D tensors {channels, pixels} with a 32 x 32 box and 64-byte swizzle;
// read only when p.out_tma / p.res_tma are set.
cudaError_t conv_tc_launch(int tile_m, int tile_n, int tile_k, int epi_warps, const CUtensorMap& tm_act, const CUtensorMap& tm_wgt,
                           const CUtensorMap& tm_out, const CUtensorMap& tm_res, const ConvTcParams& p, dim3 grid, size_t smem_bytes,
                           cudaStream_t stream);
// (their points of 128 and 256 channels with 8 and with 16 epilogue warps, translation units of their own)
cudaError_t conv_tc_wide_prepare(int tile_m, int tile_n, int tile_k, bool general, size_t smem_bytes);
cudaError_t conv_tc_wide_launch(int tile_m, int tile_n, int tile_k, bool general, const CUtensorMap& tm_act, const CUtensorMap& tm_wgt,
                              const CUtensorMap& tm_out, const CUtensorMap& tm_res, const ConvTcParams& p, dim3 grid, size_t smem_bytes,
                              cudaStream_t stream);
cudaError_t conv_tc_wide16_prepare(int tile_m, int tile_n, int tile_k, bool general, size_t smem_bytes);
cudaError_t conv_tc_wide16_launch(int tile_m, int tile_n, int tile_k, bool general, const CUtensorMap& tm_act, const CUtensorMap& tm_wgt,
                              const CUtensorMap& tm_out, const CUtensorMap& tm_res, const ConvTcParams& p, dim3 grid, size_t smem_bytes,
                              cudaStream_t stream);

// CTA-pair points (tcgen05.mma.cta_group::2): tile_m = 256, tile_n 64 / 128 / 256; `grid` = 2 x the number of pairs.
int conv_tc_pair_epi_warps(int tile_n);
cudaError_t conv_tc_pair_prepare(int tile_n, int tile_k, bool general, size_t smem_bytes);
cudaError_t conv_tc_pair_launch(int tile_n, int tile_k, const CUtensorMap& tm_act, const CUtensorMap& tm_wgt, const CUtensorMap& tm_out,
                                const CUtensorMap& tm_res, const ConvTcParams& p, dim3 grid, size_t smem_bytes, cudaStream_t stream);

// Points whose split-K slices are summed inside a cluster: tile_m = 128, `grid` = tiles x p.cluster_split.  tail: partial last slabs.
cudaError_t conv_tc_cluster_prepare(int tile_n, int tile_k, int epi_warps, bool tail, size_t smem_bytes);
cudaError_t conv_tc_cluster_launch(int tile_n, int tile_k, int epi_warps, const CUtensorMap& tm_act, const CUtensorMap& tm_wgt, const ConvTcParams& p,
                                   dim3 grid, size_t smem_bytes, cudaStream_t stream);

// Transposed-accumulator points (lane = output channel): NCHW output through TMA stores; tile_n 128 or 256, 16-bit types, 8 epilogue warps.
// tm_out: y as the 3-D tensor {P*Q, O, N} with a 32-pixel x 32-channel box and 64-byte swizzle (read when p.swap_tma).
cudaError_t conv_tc_swap_prepare(int tile_m, int tile_n, int tile_k, bool general, size_t smem_bytes);
cudaError_t conv_tc_swap_launch(int tile_m, int tile_n, int tile_k, const CUtensorMap& tm_act, const CUtensorMap& tm_wgt,
                                const CUtensorMap& tm_out, const ConvTcParams& p, dim3 grid, size_t smem_bytes, cudaStream_t stream);

// Sum of split-K partials + bias (+ residual) + ReLU + one rounding; `total` = B*O*P*Q elements in the output's order.
cudaError_t splitk_reduce_launch(const float* partial, int splits, int64_t total, int out_channels, int pq,
                                 const void* bias, int bias_fp32, int relu, int out_type, const void* residual, int out_nhwc,
                                 void* y, cudaStream_t stream);  // out_type: 0 fp16, 1 bf16, 2 fp32

#if defined(__CUDACC__)
// Launches blocks of 256 threads with shared memory nobody uses (beyond `fixed` declared bytes and `dynamic` needed ones), so that an SM
// takes no more of them than an even share.  Programmatic launches begin while the kernel ahead still holds most SMs: blocks that need
// next to nothing all pile up on the few it leaves idle, eight at a time, and are still at it there when the others are free.
// It is for one stream: 12 layers take 0.92 of the time without it.  Where another stream's kernel holds the machine, blocks that need not
// wait for one of their own stream could all run on its idle SMs at once, and now wait for a place each: the same layer in two streams
// takes 1.08 times as long, in three 1.10 (8 x 512 -> 512 at 14 x 14, 3x3, 25.6 and 30.0 us, 7 x 7 of one image 13.3 and 15.4), while 66
// pairs of different layers take 0.995, 16 of them over 3 % longer.  Blocks kept apart by threads and registers that idle, which leave
// shared memory to the other stream, cost two streams as much (30.0 and 29.9 us); two to an SM, 25.7, take most of the gain away.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl_spread(void (*kernel)(KArgs...), unsigned blocks, size_t fixed, size_t dynamic, cudaStream_t stream, Args&&... args) {
  const size_t share = (blocks + kNumSms - 1) / kNumSms, total = 233472 / (share + 1) + 128;  // of an SM's 228 KiB; a block takes 1 KiB besides
  size_t smem = dynamic;
  if (share < 8 && total > 1024 + fixed + dynamic) smem = (total - 1024 - fixed) / 128 * 128;
  if (fixed + smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kCtaSmemLimit - fixed));
    if (e != cudaSuccess) return e;
  }
  return launch_pdl(kernel, dim3(blocks), dim3(256), smem, stream, static_cast<Args&&>(args)...);
}
#endif
// The two repacks of repack_pair_launch where both are small (repack_direct.cu); false: not for these.  Either source may be null;
// the second is filters of 9 taps or 1.
bool repack_direct_launch(const void* src_a, void* dst_a, int batch_a, int ch_a, int hw_a, int cp_a, const void* src_b, void* dst_b, int batch_b,
                          int ch_b, int hw_b, int cp_b, cudaStream_t stream, cudaError_t* status);
// 16-bit [B][C][HW] -> [B][HW][Cp] (zero-filled channel padding).
cudaError_t repack_launch(const void* src, void* dst, int batch, int channels, int hw, int c_padded, cudaStream_t stream);
// FP32, two tensors in one launch: [batch][channels][hw] -> [batch][hw][c_padded], every value rounded to TF32 (ties away);
// c_padded counts FP32 elements (a multiple of 8).
cudaError_t repack_tf32_pair_launch(const void* src_a, void* dst_a, int batch_a, int ch_a, int hw_a, int cp_a, const void* src_b,
                                    void* dst_b, int batch_b, int ch_b, int hw_b, int cp_b, cudaStream_t stream);
// 1-byte elements (FP8), two tensors in one launch: [batch][channels][hw] -> [batch][hw][c_padded], zero-padded channels;
// c_padded counts elements (a multiple of 32); destinations 16-byte aligned.
cudaError_t repack_bytes_pair_launch(const void* src_a, void* dst_a, int batch_a, int ch_a, int hw_a, int cp_a, const void* src_b,
                                     void* dst_b, int batch_b, int ch_b, int hw_b, int cp_b, cudaStream_t stream);
// Two repacks (activations + weights) in ONE launch; src_b == nullptr runs only the first.
// Column-pair gather (row gather for stride_w = 2 and <= 4 channels): X3[n][h][positions][8], W3[o][r][t_positions * 8].
cudaError_t gather_pairs_launch(const void* x, void* x3, int batch, int channels, int h, int w, int positions, int left, int t_positions,
                                int shift, const void* wsrc, void* w3, int out_channels, int kernel_h, int kernel_w, cudaStream_t stream);
// Activations of a strided 1x1 convolution: only the pixels it reads, [batch][out_h * out_w][c_padded]; optionally the
// 1x1 filters in the same launch.
cudaError_t repack_subsampled_launch(const void* x, void* xn, int batch, int channels, int h, int w, int out_h, int out_w, int stride_h,
                                     int stride_w, int c_padded, const void* wsrc, void* wdst, int out_channels, cudaStream_t stream);
cudaError_t repack_pair_launch(const void* src_a, void* dst_a, int batch_a, int ch_a, int hw_a, int cp_a, const void* src_b,
                               void* dst_b, int batch_b, int ch_b, int hw_b, int cp_b, cudaStream_t stream);

// Row gather for convolutions with few input channels (16-bit types, bit-exact):
//   x2[n][h][q][s*C + c] = x[n][c][h][q*stride_w - pad_w + s]   (c2 = padded S*C elements per position, zero-filled)
//   w2[o][r][s*C + c]    = w[o][c][r][s]
// x == nullptr gathers only the weights, wsrc == nullptr only the activations.  x2 needs 16-byte alignment.
cudaError_t gather_rows_launch(const void* x, void* x2, int batch, int channels, int h, int w, int q, int kernel_w, int stride_w,
                               int pad_w, int c2, const void* wsrc, void* w2, int out_channels, int kernel_h, cudaStream_t stream);

// FP32 SIMT implicit GEMM straight from NCHW.
struct Fp32Shape {
  int batch, c, h, w, o, r, s, stride_h, stride_w, pad_h, pad_w, out_h, out_w;
};
// The kernel, the tile and the CTAs of a cluster that split the reduction of a tile:
struct Fp32Choice {
  int wide;            // 1: conv_fp32_wide.cu (thread tiles of 16 x 8)
  int tile_p, tile_o;  // output pixels and channels of a tile
  int slices;
};
Fp32Choice conv_fp32_choose(const Fp32Shape& g);
size_t conv_fp32_smem_bytes(const Fp32Choice& ch, const Fp32Shape& g);  // dynamic, for tensors on 16-byte boundaries
size_t conv_fp32_wide_smem_bytes(int tile_p);
cudaError_t conv_fp32_wide_prepare(const Fp32Choice& ch, const Fp32Shape& g);
cudaError_t conv_fp32_launch(const Fp32Choice& ch, const Fp32Shape& g, const void* x, const void* w, const void* bias, void* y, int relu,
                             cudaStream_t stream);
cudaError_t conv_fp32_wide_launch(const Fp32Choice& ch, const Fp32Shape& g, const void* x, const void* w, const void* bias, void* y, int relu,
                                  cudaStream_t stream);
cudaError_t rmsnorm_launch(int rows, int hidden, float eps, int dtype, int gamma_fp32, const void* x, const void* gamma,
                           void* y, const void* res_in, void* res_out, cudaStream_t stream);

cudaError_t bias_act_launch(int precision, int64_t total, int channels, int hw, const void* bias, int relu, void* y,
                            cudaStream_t stream);
cudaError_t maxpool2d_launch(int precision, int batch, int channels, int h, int w, int k, int stride, int pad, const void* x,
                             void* y, cudaStream_t stream);
// [B][H][W][C] tensors, C % 8 == 0, 16-bit types.
cudaError_t maxpool2d_nhwc_launch(int precision, int batch, int channels, int h, int w, int k, int stride, int pad, const void* x,
                                  void* y, cudaStream_t stream);
cudaError_t add_relu_launch(int precision, int relu, const void* a, const void* b, void* y, int64_t n, cudaStream_t stream);

}  // namespace gieb
