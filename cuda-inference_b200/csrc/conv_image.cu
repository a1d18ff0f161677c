// First layers over images (at most 4 channels, horizontal stride 2, even width) on the sm_100a tensor cores, straight from the
// caller's NCHW tensor in one launch.
//
// A row of the image is kept in shared memory as a strip of positions: position i holds the column pair (2 (i - left),
// 2 (i - left) + 1) of all channels, 8 values = 16 bytes.  The window of output column q is then the T adjacent positions
// q .. q + T - 1, so an unswizzled K-major descriptor whose rows are 16 bytes apart reads the OVERLAPPING windows of 128 output
// pixels straight from the strip (ptx::smem_desc_kmajor_plain).  A CTA takes `group_rows` output rows of one image at a time: the
// input rows they read become strips one behind the other, the rows that are stride_h apart next to each other, so that GEMM row
// pr * pitch + q is output pixel (p0 + pr, q) for every filter row, each of which starts at another strip.  (pitch = out_w + T - 1
// positions: the T - 1 rows between two output rows are no output pixels.)
//   * warps 0-3 load the image with 4-byte loads (coalesced along the columns), interleave the channels and write the strips, two
//     buffers in turn; warp 4 issues the MMAs (128 pixels x 64 channels, R * T / 2 instructions of 16 values); warps 5-12 drain the
//     accumulators, four of which stand in tensor memory.  The filters are laid out once per CTA.
//   * channel-contiguous output: a warp owns 32 pixels x 64 channels, staged in shared memory and written as whole 128-byte rows.
// It takes the place of a gather launch into a copy of the image in this layout, and of a convolution on it whose tiles held one
// output row each.  What bounds it: the instructions of loads and epilogue and the stores of the output (64-byte runs per channel in
// NCHW); the tensor pipe is a fifth busy.  7x7/2, 3 -> 64 channels, FP16, NCHW, with the two launches and so: one image of 64 x 64
// 8.4 and 5.8 us, 4 x 224 x 224 12.3 and 9.2, 32 x 224 x 224 45.3 and 33.3, 128 x 224 x 224 157 and 101, 57 x 144 x 144 43.4 and 22.6.
// Every window written out (64-byte rows, swizzled) instead of overlapping ones took four times the shared-memory stores and 178 us
// for the 128 images.
#include "conv_tc_kernel.cuh"

namespace gieb {
namespace {

constexpr int kGatherWarps = 4, kImageWorkers = 8;
static_assert(kImageThreads == 32 * (kGatherWarps + 1 + kImageWorkers), "warps of a CTA");
constexpr int kImageSlots = 4;                       // accumulators of 64 columns
constexpr uint32_t kImageCtrl = 1024;                // 64 bias values, barriers, TMEM address slot
constexpr int kImageCols = kImageTileN;

// The words of C channels at one column pair (low half: even column) as the 8 values of a position: the channels of the even
// column, those of the odd one, zeros.
template <int C>
__device__ __forceinline__ uint4 position_of(const uint32_t (&w)[C]) {
  if constexpr (C == 1) return make_uint4(w[0], 0u, 0u, 0u);
  else if constexpr (C == 2) return make_uint4(__byte_perm(w[0], w[1], 0x5410), __byte_perm(w[0], w[1], 0x7632), 0u, 0u);
  else if constexpr (C == 3)
    return make_uint4(__byte_perm(w[0], w[1], 0x5410), __byte_perm(w[2], w[0], 0x7610), __byte_perm(w[1], w[2], 0x7632), 0u);
  else
    return make_uint4(__byte_perm(w[0], w[1], 0x5410), __byte_perm(w[2], w[3], 0x5410), __byte_perm(w[0], w[1], 0x7632),
                      __byte_perm(w[2], w[3], 0x7632));
}

template <int T>
__global__ void __launch_bounds__(kImageThreads, 2) conv_image_kernel(const __grid_constant__ ConvImageParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  float* bias_s = reinterpret_cast<float*>(smem);
  uint64_t* s_full = reinterpret_cast<uint64_t*>(smem + 256);  // [2] strips written
  uint64_t* s_empty = s_full + 2;                              // [2] strips read
  uint64_t* acc_full = s_empty + 2;                            // [kImageSlots]
  uint64_t* acc_empty = acc_full + kImageSlots;                // [kImageSlots]
  uint64_t* w_full = acc_empty + kImageSlots;                  // filters and bias laid out
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(w_full + 1);
  uint32_t* strip_of = tmem_slot + 1;  // [kernel_h + 1] first position of a filter row's strip within a stage
  uint8_t* w_base = smem + kImageCtrl;  // [r][64 channels][T * 16 bytes], swizzled by that width
  uint8_t* strip_base = w_base + size_t(p.kernel_h) * T * (kImageCols * 16);
  uint8_t* stage_base = strip_base + 2 * size_t(p.strip_stage_bytes);  // (channel-contiguous output: 4 KiB per worker warp)

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = int(blockIdx.y) * kImageCols;

  if (threadIdx.x == kImageThreads - 32) {
    for (int b = 0; b < 2; ++b) {
      ptx::mbar_init(&s_full[b], kGatherWarps);
      ptx::mbar_init(&s_empty[b], 1);
    }
    for (int b = 0; b < kImageSlots; ++b) {
      ptx::mbar_init(&acc_full[b], 1);
      ptx::mbar_init(&acc_empty[b], 4);  // the four warps that drain it
    }
    ptx::mbar_init(w_full, kImageWorkers);
    ptx::fence_mbar_init();
  }
  if (warp == 0)
    for (int r = lane; r < p.kernel_h; r += 32) {
      const int q = p.fd_stride_h.div(r);
      strip_of[r] = uint32_t(((r - q * p.stride_h) * p.rows_per_phase + q) * p.pitch);
    }
  if (warp == kGatherWarps) ptx::tmem_alloc_then_signal(tmem_slot, kImageSlots * kImageCols);
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(tmem_slot);

  if (warp < kGatherWarps) {
    // ---------------- image rows -> strips ----------------
    int st = 0;
    uint32_t phase = 0;
    ptx::grid_dep_wait();
    auto run = [&](auto c_tag, auto words_tag) {
      constexpr int C = decltype(c_tag)::value;
      constexpr bool WORDS = decltype(words_tag)::value;
      const uint16_t* x = static_cast<const uint16_t*>(p.x);
      const int64_t plane = int64_t(p.in_h) * p.in_w;
      const int pairs = p.in_w >> 1;
      for (int g = blockIdx.x; g < p.groups; g += gridDim.x) {
        const int img = p.fd_groups_per_image.div(g), p0 = (g - img * p.groups_per_image) * p.group_rows;
        const bool ok = ptx::mbar_wait(&s_empty[st], phase ^ 1u, p.status, kStatusProducerTimeout, p.wait_limit);
        if (!__all_sync(0xffffffffu, ok)) return;
        uint8_t* dst0 = strip_base + size_t(st) * p.strip_stage_bytes;
        const uint16_t* src0 = x + int64_t(img) * C * plane;
        const int h0 = p0 * p.stride_h - p.pad_h;
        const int units = p.group_in_rows * p.segments;  // runs of 32 positions
        constexpr int U = 8;                             // runs in flight
        for (int u0 = warp; u0 < units; u0 += U * kGatherWarps) {
          uint32_t v[U][C];
          int at[U];
#pragma unroll
          for (int k = 0; k < U; ++k) {
            const int u = u0 + k * kGatherWarps, j = p.fd_segments.div(u), i = (u - j * p.segments) * 32 + lane;
            const int h = h0 + j, pair = i - p.left, q = p.fd_stride_h.div(j);
            at[k] = u < units && i < p.pitch ? ((j - q * p.stride_h) * p.rows_per_phase + q) * p.pitch + i : -1;
            const bool in = at[k] >= 0 && h >= 0 && h < p.in_h && pair >= 0 && pair < pairs;
            const uint16_t* s = src0 + (in ? int64_t(h) * p.in_w + 2 * pair : 0);
#pragma unroll
            for (int c = 0; c < C; ++c) {
              v[k][c] = 0u;
              if (in) v[k][c] = WORDS ? *reinterpret_cast<const uint32_t*>(s + c * plane) : uint32_t(s[c * plane]) | (uint32_t(s[c * plane + 1]) << 16);
            }
          }
#pragma unroll
          for (int k = 0; k < U; ++k)
            if (at[k] >= 0) *reinterpret_cast<uint4*>(dst0 + size_t(at[k]) * 16) = position_of<C>(v[k]);
        }
        ptx::fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&s_full[st]);
        if (++st == 2) { st = 0; phase ^= 1u; }
      }
    };
    auto with_words = [&](auto c_tag) {
      if (p.words) run(c_tag, std::integral_constant<bool, true>{});
      else run(c_tag, std::integral_constant<bool, false>{});
    };
    if (p.debug_skip & 1u) {
    } else if (p.channels == 1) with_words(std::integral_constant<int, 1>{});
    else if (p.channels == 2) with_words(std::integral_constant<int, 2>{});
    else if (p.channels == 3) with_words(std::integral_constant<int, 3>{});
    else with_words(std::integral_constant<int, 4>{});
  } else if (warp == kGatherWarps) {
    // ---------------- MMA issuer ----------------
    int st = 0, tcount = 0;
    uint32_t phase = 0;
    bool alive = !(p.debug_skip & 2u);
    const uint64_t a_desc0 = ptx::smem_desc_kmajor_plain(0, 16, 128), b_desc0 = ptx::smem_desc_kmajor<T * 16>(0);
    const uint32_t b_lo0 = ptx::smem_u32(w_base) >> 4;
    if (alive) {
      const bool ok = ptx::mbar_wait(w_full, 0, p.status, kStatusMmaTimeout, p.wait_limit);
      alive = __all_sync(0xffffffffu, ok);
    }
    for (int g = blockIdx.x; alive && g < p.groups; g += gridDim.x) {
      const int img = p.fd_groups_per_image.div(g), p0 = (g - img * p.groups_per_image) * p.group_rows;
      const int rows = min(p.group_rows, p.out_h - p0);
      const int tiles = ((rows - 1) * p.pitch + p.out_w + kTileM - 1) / kTileM;
      const bool in = ptx::mbar_wait(&s_full[st], phase, p.status, kStatusMmaTimeout, p.wait_limit);
      if (!__all_sync(0xffffffffu, in)) break;
      const uint32_t a_lo0 = (ptx::smem_u32(strip_base) + uint32_t(st) * p.strip_stage_bytes) >> 4;
      for (int i = 0; i < tiles; ++i, ++tcount) {
        const int slot = tcount & (kImageSlots - 1);
        const bool ok = ptx::mbar_wait(&acc_empty[slot], ((tcount / kImageSlots) & 1) ^ 1u, p.status, kStatusMmaTimeout, p.wait_limit);
        if (!__all_sync(0xffffffffu, ok)) { alive = false; break; }
        ptx::tc_fence_after_sync();
        if (ptx::elect_one()) {
          const uint32_t acc = tmem_base + uint32_t(slot) * kImageCols;
          const uint32_t a_tile = a_lo0 + uint32_t(i * kTileM);
          uint32_t b_lo = b_lo0, next = strip_of[0];
          for (int r = 0; r < p.kernel_h; ++r) {
            const uint64_t ad = a_desc0 | uint64_t((a_tile + next) & 0x3fffu), bd = b_desc0 | uint64_t(b_lo & 0x3fffu);
            next = strip_of[r + 1];  // (one beyond the last: inside the control block, not used)
            b_lo += kImageCols * T;
#pragma unroll
            for (int k = 0; k < T; k += 2) ptx::mma_f16_ss(acc, ad + k, bd + k, p.idesc, k != 0 || r != 0);
          }
          ptx::mma_commit(&acc_full[slot]);
          if (i + 1 == tiles) ptx::mma_commit(&s_empty[st]);
        }
        __syncwarp();
      }
      if (++st == 2) { st = 0; phase ^= 1u; }
    }
  } else {
    // ---------------- workers: filters and bias, then the accumulators ----------------
    const int we = warp - kGatherWarps - 1, quad = warp & 3, eg = we >> 2;
    const int et = threadIdx.x - 32 * (kGatherWarps + 1);
    ptx::grid_dep_wait();
    {
      // 16-byte cell t of channel row o and filter row r: a warp takes the cells of a channel side by side, which lie side by side in
      // memory too (with a channel per lane the loads of 128 CTAs took ~6 us); rows are T cells, swizzled
      const int per_row = p.kernel_h * T, cells = per_row * kImageCols, rs = p.kernel_h * p.kernel_w;
      const uint16_t* w = static_cast<const uint16_t*>(p.w);
      auto fill = [&](auto c_tag) {
        constexpr int C = decltype(c_tag)::value;  // (0: converted weights)
#pragma unroll 4
        for (int idx = et; idx < cells; idx += 32 * kImageWorkers) {
          const int row = p.fd_cells.div(idx), rt = idx - row * per_row, r = rt / T, t = rt & (T - 1), o = n0 + row;
          uint4 v = make_uint4(0u, 0u, 0u, 0u);
          if constexpr (C == 0) {
            if (o < p.out_channels) v = reinterpret_cast<const uint4*>(w)[(int64_t(o) * p.kernel_h + r) * T + t];
          } else {
            // (the pair of taps of a channel, as the pair of columns of a position)
            const int s = 2 * t - p.shift;
            const uint16_t* src = w + (int64_t(o) * C * p.kernel_h + r) * p.kernel_w + s;
            const bool even = o < p.out_channels && s >= 0 && s < p.kernel_w, odd = o < p.out_channels && s + 1 >= 0 && s + 1 < p.kernel_w;
            uint32_t e[C];
#pragma unroll
            for (int c = 0; c < C; ++c) {
              uint32_t lo = 0u, hi = 0u;
              if (even) lo = src[c * rs];
              if (odd) hi = src[c * rs + 1];
              e[c] = lo | (hi << 16);
            }
            v = position_of<C>(e);
          }
          constexpr int kShift = T == 8 ? 0 : (T == 4 ? 1 : 2);
          *reinterpret_cast<uint4*>(w_base + (size_t(r * kImageCols + row) * T + (t ^ ((row >> kShift) & (T - 1)))) * 16) = v;
        }
      };
      if (p.prepacked) fill(std::integral_constant<int, 0>{});
      else if (p.channels == 1) fill(std::integral_constant<int, 1>{});
      else if (p.channels == 2) fill(std::integral_constant<int, 2>{});
      else if (p.channels == 3) fill(std::integral_constant<int, 3>{});
      else fill(std::integral_constant<int, 4>{});
      if (et < kImageCols) {
        float b = 0.f;
        const int oc = n0 + et;
        if (p.bias != nullptr && oc < p.out_channels)
          b = p.bias_fp32 ? static_cast<const float*>(p.bias)[oc]
                          : (p.is_bf16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(p.bias)[oc]) : __half2float(static_cast<const __half*>(p.bias)[oc]));
        bias_s[et] = b;
      }
      ptx::fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(w_full);
      asm volatile("bar.sync 1, %0;" ::"n"(32 * kImageWorkers) : "memory");  // (the bias values)
    }
    uint8_t* box = stage_base + size_t(we) * 4096;
    const int64_t cstride = p.out_nhwc ? 1 : p.pq;
    int tcount = 0;
    bool alive = true;
    for (int g = blockIdx.x; alive && g < p.groups; g += gridDim.x) {
      const int img = p.fd_groups_per_image.div(g), p0 = (g - img * p.groups_per_image) * p.group_rows;
      const int rows = min(p.group_rows, p.out_h - p0);
      const int tiles = ((rows - 1) * p.pitch + p.out_w + kTileM - 1) / kTileM;
      for (int i = 0; i < tiles; ++i, ++tcount) {
        if ((tcount & 1) != eg) continue;
        const int slot = tcount & (kImageSlots - 1);
        // GEMM row -> pixel of the output plane (-1: none)
        auto pixel = [&](int m) {
          const int pr = p.fd_pitch.div(m), q = m - pr * p.pitch;
          return pr < rows && q < p.out_w ? (p0 + pr) * p.out_w + q : -1;
        };
        const int m0 = i * kTileM + quad * 32;
        const int pix = pixel(m0 + lane);
        const bool m_ok = pix >= 0;
        const int64_t base = p.out_nhwc ? (int64_t(img) * p.pq + pix) * p.out_channels + n0 : (int64_t(img) * p.out_channels + n0) * p.pq + pix;
        const bool ok = ptx::mbar_wait(&acc_full[slot], (tcount / kImageSlots) & 1, p.status, kStatusEpilogueTimeout, p.wait_limit);
        if (!__all_sync(0xffffffffu, ok)) { alive = false; break; }
        ptx::tc_fence_after_sync();
        const bool some = __any_sync(0xffffffffu, m_ok);
        const uint32_t acc = tmem_base + uint32_t(slot) * kImageCols + (uint32_t(quad * 32) << 16);
        auto drained = [&]() {
          ptx::tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(&acc_empty[slot]);
        };
        const int chunks = !some ? 0 : (n0 + 32 < p.out_channels ? 2 : 1);
        if (chunks == 0) drained();
        auto with_type = [&](auto&& f) {
          if (p.is_bf16) f(static_cast<__nv_bfloat16*>(p.y), static_cast<const __nv_bfloat16*>(p.residual));
          else f(static_cast<__half*>(p.y), static_cast<const __half*>(p.residual));
        };
        if (p.out_cells) {
          // 16-byte cells of whole rows: eight lanes per pixel, four pixels per instruction
          const int cell = lane & 7;
          const bool cell_ok = n0 + cell * 8 < p.out_channels;
          uint4* cells = reinterpret_cast<uint4*>(box + (cell >> 2) * 2048);
          auto each_row = [&](auto&& f) {
#pragma unroll
            for (int it = 0; it < 8; ++it) {
              const int r = it * 4 + (lane >> 3), px = __shfl_sync(0xffffffffu, pix, r);
              const int at = r * 4 + ((cell & 3) ^ ((r >> 1) & 3));
              if (px >= 0 && cell_ok) f(cells[at], (int64_t(img) * p.pq + px) * p.out_channels + n0 + cell * 8);
            }
          };
          if (chunks != 0) {
            if (p.residual != nullptr) each_row([&](uint4& c, int64_t off) { c = *reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(p.residual) + off); });
            __syncwarp();
            for (int chunk = 0; chunk < chunks; ++chunk) {
              uint32_t v[32];
              ptx::tmem_ld_32x32b_x32(acc + uint32_t(chunk * 32), v);
              ptx::tmem_ld_wait();
              if (chunk + 1 == chunks) drained();
              if (p.is_bf16) chunk_to_staging<__nv_bfloat16>(v, bias_s + chunk * 32, box + chunk * 2048, lane, p.relu, p.residual != nullptr);
              else chunk_to_staging<__half>(v, bias_s + chunk * 32, box + chunk * 2048, lane, p.relu, p.residual != nullptr);
            }
            __syncwarp();
            each_row([&](uint4& c, int64_t off) { *reinterpret_cast<uint4*>(static_cast<uint16_t*>(p.y) + off) = c; });
            __syncwarp();
          }
        } else {
          for (int chunk = 0; chunk < chunks; ++chunk) {
            uint32_t v[32];
            ptx::tmem_ld_32x32b_x32(acc + uint32_t(chunk * 32), v);
            ptx::tmem_ld_wait();
            if (chunk + 1 == chunks) drained();
            if (m_ok) {
              const int nvalid = min(32, p.out_channels - (n0 + chunk * 32));
              const int64_t off = base + int64_t(chunk * 32) * cstride;
              with_type([&](auto* yp, auto* rp) { store_chunk<true>(v, bias_s + chunk * 32, yp + off, rp != nullptr ? rp + off : nullptr, cstride, nvalid, p.relu); });
            }
          }
        }
      }
    }
  }

  ptx::tc_fence_before_sync();
  __syncthreads();
  if (warp == kGatherWarps) {
    ptx::tc_fence_after_sync();
    ptx::tmem_dealloc(tmem_base, kImageSlots * kImageCols);
  }
}

}  // namespace

size_t conv_image_smem_bytes(int kernel_h, int t_positions, size_t strip_stage_bytes, bool staging) {
  return kImageCtrl + size_t(kernel_h) * t_positions * (kImageCols * 16) + 2 * strip_stage_bytes + (staging ? size_t(kImageWorkers) * 4096 : 0);
}

cudaError_t conv_image_prepare(int t_positions) {
  // (the limit belongs to the function and is replaced by each call: every plan sets the same one, so that none lowers another's)
  const auto set = [&](auto kernel) { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kCtaSmemLimit)); };
  return t_positions == 2 ? set(conv_image_kernel<2>) : (t_positions == 4 ? set(conv_image_kernel<4>) : set(conv_image_kernel<8>));
}

cudaError_t conv_image_launch(int t_positions, const ConvImageParams& p, dim3 grid, size_t smem, cudaStream_t stream) {
  const auto go = [&](auto kernel) { return launch_pdl(kernel, grid, dim3(kImageThreads), smem, stream, p); };
  return t_positions == 2 ? go(conv_image_kernel<2>) : (t_positions == 4 ? go(conv_image_kernel<4>) : go(conv_image_kernel<8>));
}

}  // namespace gieb
