// Convolution on the sm_100a tensor cores with every activation fetched once per channel block instead of once per filter tap.
//
// The im2col-mode kernels (conv_tc_kernel.cuh) load one 128-pixel slab per (channel block, tap): a 3x3 layer pulls its
// activations through L2 nine times, and since an SM receives ~74 B/clk that bounds their main loop.  Here the GEMM rows are
// numbered on a padded grid instead of the output pixels: row (n * Hs + p) * Ws + q is output pixel (n, p, q) for p < P, q < Q
// and nothing otherwise.  On that grid the input element of tap (r, s) lies a CONSTANT number of rows further for every row
// (r * Ws + s at stride 1), so one shared-memory tile of the 128 rows and the (R - 1) * Ws + S - 1 after them x 64 channels
// (the halo tile: K-major, 128-byte swizzle) feeds all the taps, each through a descriptor that starts at another row.  Rows of
// the grid that are no output pixel cost 4 % of the MMA work on 56 x 56 maps, 15 % on 14 x 14, 31 % on 7 x 7.
//   * Strides: the rows of one tap are stride apart, so the tile is kept as stride_h * stride_w phases, each a halo tile of its
//     own; tap (r, s) reads phase (r % stride_h, s % stride_w) from row (r / stride_h) * Ws + s / stride_w on.
//   * Neighbouring grid rows and images share their padding at stride 1: Ws = W + pad, Hs = H + pad.
// Channel-contiguous activations (the caller's own, or the repacked copy of NCHW tensors) arrive by TMA: one box per padded row
// of the grid (or group of rows of one image), whose columns and rows outside the image read as zeros, which IS the padding.
// Weights arrive by TMA as [taps per load][channels][64] boxes, and stay in shared memory for all tiles of a CTA when they fit.
// Accumulators are double-buffered in tensor memory.  With few output tiles the reduction is split over the CTAs of a
// cluster; pairs of CTAs compute 256-row tiles with tcgen05.mma.cta_group::2 where the weights are many (see resolve_halo in
// api.cu for the choices).
// What bounds it: the shared-memory reads of the MMAs (128 B/clk: 48 cycles for 128 x 64 x 16, ~60 where the operand starts at
// a row that is no multiple of 8) for narrow tiles, the tensor pipe for 256 columns; ~230 cycles around each elected block of
// instructions and ~600 between tiles (clock stamps).  Measured against the slab kernels: 512 -> 512,
// 7 x 7, 3x3, one image 14.7 -> 12.3 us; 304 -> 32, 40 x 40, 3x3 11.4 -> 9.7; 256 -> 60, 76 x 40, 3x3 18.4 -> 14.9;
// 109 x 64 -> 64, 70 x 70, 3x3 68.7 -> 57.1; 256 -> 256, 14 x 14, 3x3, 32 images 15.8 -> 15.4; long reductions over 256-column
// pair tiles are as fast on the slab kernels and stay there.
#include "conv_tc_kernel.cuh"

namespace gieb {
namespace {

// [0,2048): 32 bias values per worker warp; [2048,3072): mbarriers + TMEM address slot
constexpr uint32_t kHaloCtrl = 3072;

// A staged chunk (layout of chunk_to_staging) to or from channel-contiguous rows in 16-byte cells: four lanes take the 64 bytes
// of a row, eight rows per instruction.  rows[i]: offset of row 8 i + lane / 4 of this warp in cells (~0: no output pixel).
template <bool LOAD, typename T>
__device__ __forceinline__ void staging_cells(uint8_t* box, int lane, T* gmem, const uint32_t (&rows)[4], uint32_t chunk_cells) {
  uint4* g = reinterpret_cast<uint4*>(gmem) + chunk_cells + (lane & 3);
#pragma unroll
  for (int it = 0; it < 4; ++it) {
    const int r = it * 8 + (lane >> 2), q = lane & 3;
    uint4* cell = reinterpret_cast<uint4*>(box + r * 64 + ((q ^ ((r >> 1) & 3)) << 4));
    if (rows[it] == ~0u) continue;
    if (LOAD) *cell = g[rows[it]];
    else g[rows[it]] = *cell;
  }
}

// NW worker warps (8 or 16); PAIR as in conv_tc_kernel.  Warps: 0 and 2 load weights, 1 loads activations, 3 issues the MMAs.
template <int BN, int NW, bool PAIR>
__global__ void __launch_bounds__(32 * (kProducerWarps + 1 + NW), NW == 16 ? 1 : 2)
conv_halo_kernel(const __grid_constant__ CUtensorMap tm_act, const __grid_constant__ CUtensorMap tm_wgt,
                 const __grid_constant__ ConvHaloParams p) {
  constexpr int B_ROWS = PAIR ? BN / 2 : BN;  // weight rows this CTA loads per tap
  constexpr uint32_t TAP_BYTES = B_ROWS * 128;
  constexpr uint32_t TMEM_COLS = 2 * BN < 32 ? 32 : 2 * BN;
  constexpr int EG = NW / 4;                  // worker warps per TMEM lane quarter

  // (Pairs take the alignment of the declaration; single CTAs round up by hand: what the compiler makes of either is 1 % faster
  // there, 3x3 14x14 b32 15.1 and 15.35 us, 70 -> 64 at 65x65, 76 images 97.2 and 96.2.)
  extern __shared__ __align__(PAIR ? 1024 : 16) uint8_t smem_raw[];
  uint8_t* smem = PAIR ? smem_raw : smem_raw + ((1024u - (ptx::smem_u32(smem_raw) & 1023u)) & 1023u);
  float* bias_s = reinterpret_cast<float*>(smem);  // [NW][32]
  uint64_t* b_full = reinterpret_cast<uint64_t*>(smem + 2048);
  uint64_t* b_empty = b_full + kMaxStages;
  uint64_t* a_full = b_empty + kMaxStages;
  uint64_t* a_empty = a_full + kMaxStages;
  uint64_t* acc_full = a_empty + kMaxStages;  // [2]
  uint64_t* acc_empty = acc_full + 2;         // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  uint32_t* tap_row = tmem_slot + 4;          // [up to 64] first row of a tap's operand within the halo tile, in 16-byte units
  uint8_t* a_base = smem + kHaloCtrl;
  uint8_t* b_base = a_base + size_t(p.a_stages) * p.a_stage_bytes;
  const uint32_t b_stage_bytes = uint32_t(p.taps_per_load) * TAP_BYTES;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool cluster = !PAIR && p.split > 1;
  const uint32_t pair_rank = PAIR ? ptx::cluster_ctarank() : 0u;  // 0 = leader (issues the MMAs), 1 = peer
  const bool leader = pair_rank == 0;
  const int tile_first = PAIR ? int(blockIdx.x >> 1) : int(blockIdx.x);
  const int tile_step = PAIR ? int(gridDim.x >> 1) : int(gridDim.x);

  if (warp == 0) {
    if (lane == 0) {
      ptx::prefetch_tensormap(&tm_wgt);
      ptx::prefetch_tensormap(&tm_act);
    }
    constexpr int kBars = 4 * kMaxStages + 4;
    for (int b = lane; b < kBars; b += 32) {
      const bool is_acc_empty = b >= 4 * kMaxStages + 2;  // one arrival per worker warp (of both CTAs of a pair)
      ptx::mbar_init(&b_full[b], is_acc_empty ? (PAIR ? 2 * NW : NW) : 1);
    }
    ptx::fence_mbar_init();
  }
  if (warp == 2) {
    for (int tap = lane; tap < p.taps; tap += 32) {
      const int r = p.fd_kernel_w.div(tap), sx = tap - r * p.kernel_w;
      int row = r * p.ws + sx;
      if (p.phases > 1)  // strides are 1 or 2
        row = ((r & (p.stride_h - 1)) * p.phases_w + (sx & (p.stride_w - 1))) * p.halo_rows + (r >> (p.stride_h - 1)) * p.ws + (sx >> (p.stride_w - 1));
      tap_row[tap] = uint32_t(row) * 8u;
    }
  }
  if (warp == kProducerWarps) {
    if constexpr (PAIR) {
      ptx::tmem_alloc_pair(tmem_slot, TMEM_COLS);
      ptx::tmem_relinquish_pair();
    } else {
      ptx::tmem_alloc(tmem_slot, TMEM_COLS);
      ptx::tmem_relinquish();
    }
    ptx::grid_dep_launch();  // (behind the allocation: see conv_tc_kernel)
  }
  ptx::tc_fence_before_sync();
  if constexpr (PAIR) ptx::cluster_sync_all();
  else __syncthreads();
  ptx::tc_fence_after_sync();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(tmem_slot);

  // Work of a tile: loads [i0, i1) of the (channel block, tap group) list.
  struct Tile { int m0, n0, i0, i1; };
  auto decode = [&](int tile) {
    Tile t;
    int z = 0, rest = tile;
    if (cluster) {  // slices of a tile sit side by side in one cluster
      rest = p.fd_split.div(tile);
      z = tile - rest * p.split;
    }
    const int m_blk = p.fd_tiles_n.div(rest);
    t.n0 = (rest - m_blk * p.tiles_n) * BN;
    t.m0 = PAIR ? m_blk * (2 * kTileM) + int(pair_rank) * kTileM : m_blk * kTileM;
    t.i0 = z * p.loads_per_split;
    t.i1 = min(p.total_loads, t.i0 + p.loads_per_split);
    return t;
  };

  if (warp == 1) {
    // ---------------- activation producer: lane l loads box l, l + 32, .. of a halo tile ----------------
    const int lane_units = p.phases * p.boxes;
    const uint32_t full0 = PAIR ? ptx::map_to_cta(ptx::smem_u32(&a_full[0]), 0u) : 0u;
    int as = 0;
    uint32_t aphase = 0;
    bool alive = !(p.debug_skip & 1u);
    ptx::grid_dep_wait();
    for (int tile = tile_first; alive && tile < p.num_tiles; tile += tile_step) {
      const Tile t = decode(tile);
      const int box0 = p.fd_box_rows.div(t.m0);  // first box of the grid the tile touches
      // The leader's instructions address both CTAs of a pair alike: each shifts its boxes so that its first grid row lands
      // on row box_rows - 1.
      const uint32_t shift = PAIR ? uint32_t(p.box_rows - 1 - (t.m0 - box0 * p.box_rows)) * 128u : 0u;
      const int cb_end = p.fd_groups.div(t.i1 - 1);
      for (int cb = p.fd_groups.div(t.i0); cb <= cb_end; ++cb) {
        const bool ok = ptx::mbar_wait(&a_empty[as], aphase ^ 1u, p.status, kStatusProducerTimeout, p.wait_limit);
        if (!__all_sync(0xffffffffu, ok)) { alive = false; break; }
        if (lane == 0 && leader) ptx::mbar_arrive_expect_tx(&a_full[as], (PAIR ? 2u : 1u) * uint32_t(lane_units) * p.box_bytes);
        __syncwarp();
        for (int u = lane; u < lane_units; u += 32) {
          int ph = 0, k = u;
          if (p.phases > 1) {
            ph = p.fd_boxes.div(u);
            k = u - ph * p.boxes;
          }
          const int pa = p.phases_w == 2 ? ph >> 1 : ph, pb = p.phases_w == 2 ? ph & 1 : 0;  // phase (row, column)
          const int prow = (box0 + k) * p.box_h, img = p.fd_hs.div(prow), pp = prow - img * p.hs;
          uint8_t* dst = a_base + size_t(as) * p.a_stage_bytes + (uint32_t(ph * p.halo_rows) * 128u + shift + uint32_t(k) * p.box_bytes);
          const int c = cb * p.row_elems, w = pb - p.pad_w, h = pp * p.stride_h + pa - p.pad_h;
          if constexpr (PAIR) ptx::tma_load_4d_pair(dst, &tm_act, full0 + uint32_t(as) * 8u, c, w, h, img);
          else ptx::tma_load_4d(dst, &tm_act, &a_full[as], c, w, h, img);
        }
        __syncwarp();
        if (++as == p.a_stages) { as = 0; aphase ^= 1u; }
      }
    }
    if (cluster) {
      ptx::cluster_sync_all();
      ptx::cluster_sync_all();
    }
  } else if (warp < kProducerWarps) {
    // ---------------- weight producers: the CTA's loads in turn (one TMA instruction keeps its warp busy ~350 cycles) ----
    bool alive = lane == 0 && !(p.debug_skip & 1u);
    const uint32_t full0 = PAIR ? ptx::map_to_cta(ptx::smem_u32(&b_full[0]), 0u) : 0u;
    int s = warp >> 1, skip = warp >> 1;
    uint32_t phase = 0;
    ptx::grid_dep_wait();
    // (weights that stay: the first tile's loads are the only ones)
    for (int tile = tile_first; alive && tile < p.num_tiles && !(p.resident && tile != tile_first); tile += tile_step) {
      const Tile t = decode(tile);
      int i = t.i0 + skip;
      for (; i < t.i1; i += 2) {
        if (!ptx::mbar_wait(&b_empty[s], phase ^ 1u, p.status, kStatusProducerTimeout, p.wait_limit)) { alive = false; break; }
        const int cb = p.fd_groups.div(i);
        const int tap = (i - cb * p.tap_groups) * p.taps_per_load;
        uint8_t* dst = b_base + size_t(s) * b_stage_bytes;
        if constexpr (PAIR) {
          if (leader) ptx::mbar_arrive_expect_tx(&b_full[s], 2u * b_stage_bytes);
          ptx::tma_load_3d_pair(dst, &tm_wgt, full0 + uint32_t(s) * 8u, cb * p.row_elems, t.n0 + int(pair_rank) * B_ROWS, tap);
        } else {
          ptx::mbar_arrive_expect_tx(&b_full[s], b_stage_bytes);
          ptx::tma_load_3d(dst, &tm_wgt, &b_full[s], cb * p.row_elems, t.n0, tap);
        }
        s += 2;
        while (s >= p.b_stages) { s -= p.b_stages; phase ^= 1u; }
      }
      skip = i - t.i1;
    }
    __syncwarp();
    if (cluster) {
      ptx::cluster_sync_all();
      ptx::cluster_sync_all();
    }
  } else if (warp == kProducerWarps) {
    // ---------------- MMA issuer: converged warp, one elected lane issues ----------------
    // A lone warp pays for every dependent instruction in full, so the issue sequence is kept down to a table look-up and a few
    // additions on the low words of the descriptors per tap (with divisions and per-tap row arithmetic a load cost ~400 cycles
    // before its first instruction).  The MMA kind and whether the last channel block is a partial one are compile-time.
    const uint32_t idesc = p.idesc;
    const int taps_per_load = p.taps_per_load, tap_groups = p.tap_groups, a_stages = p.a_stages, b_stages = p.b_stages;
    const uint32_t a_step = p.a_stage_bytes >> 4, b_step = b_stage_bytes >> 4;
    const uint64_t desc0 = ptx::smem_desc_kmajor<128>(0);  // everything but the address
    const uint32_t a_lo0 = ptx::smem_u32(a_base) >> 4, b_lo0 = ptx::smem_u32(b_base) >> 4;
    const bool resident = p.resident != 0;
    auto run = [&](auto kind_tag, auto tail_tag) {
      constexpr int KIND = decltype(kind_tag)::value;  // 0 kind::f16, 1 kind::tf32, 2 kind::f8f6f4
      constexpr bool TAIL = decltype(tail_tag)::value;
      int bs = 0, as = 0, tcount = 0;
      uint32_t bphase = 0, aphase = 0;
      bool alive = leader && !(p.debug_skip & 2u);
      // first grid row of a tile within its halo tile (boxes hold whole padded rows)
      auto first_row = [&](const Tile& t) { return PAIR ? p.box_rows - 1 : t.m0 - p.fd_box_rows.div(t.m0) * p.box_rows; };
      Tile t = decode(tile_first);
      int row0 = first_row(t);
      for (int tile = tile_first; alive && tile < p.num_tiles; tile += tile_step, ++tcount) {
        const int buf = tcount & 1;
        int cb = cluster ? p.fd_groups.div(t.i0) : 0;
        int tg = t.i0 - cb * tap_groups;
        const bool wait_b = !(resident && tcount > 0);  // (weights that stay have arrived once and for all)
        const uint32_t acc = tmem_base + buf * BN;
        const bool drained = ptx::mbar_wait(&acc_empty[buf], ((tcount >> 1) & 1) ^ 1u, p.status, kStatusMmaTimeout, p.wait_limit);
        bool need_a = true;
        uint32_t accumulate = 0;
        for (int i = t.i0; i < t.i1;) {
          bool ok = drained;
          if (need_a) ok = ok && ptx::mbar_wait(&a_full[as], aphase, p.status, kStatusMmaTimeout, p.wait_limit);
          if (wait_b) ok = ok && ptx::mbar_wait(&b_full[bs], bphase, p.status, kStatusMmaTimeout, p.wait_limit);
          if (!__all_sync(0xffffffffu, ok)) { alive = false; break; }
          // Loads that follow each other in the ring and have landed as well go out in one elected block (the wait / vote / fence
          // sequence between blocks costs as much as four instructions): all of a channel block when the weights stay, else two.
          int n = 1;
          const int room = min(min(tap_groups - tg, t.i1 - i), b_stages - bs);
          if (!wait_b) n = room;
          else if (room > 1 && __all_sync(0xffffffffu, ptx::mbar_try_wait(&b_full[bs + 1], bphase))) n = 2;
          ptx::tc_fence_after_sync();
          const int ksteps = !TAIL || cb + 1 != p.c_blocks ? 4 : p.last_ksteps;
          const bool last = i + n == t.i1, block_done = tg + n == tap_groups || last;
          const uint32_t a_lo = a_lo0 + uint32_t(as) * a_step + uint32_t(row0) * 8u;
          uint32_t b_lo = b_lo0 + uint32_t(bs) * b_step;
          const uint32_t* row = tap_row + tg * taps_per_load;
          if (ptx::elect_one()) {
            uint32_t next = row[0];
            const int taps_now = n * taps_per_load;
            for (int tt = 0; tt < taps_now; ++tt) {
              const uint64_t ad = desc0 | uint64_t((a_lo + next) & 0x3fffu), bd = desc0 | uint64_t(b_lo & 0x3fffu);
              next = row[tt + 1];  // (one beyond the last tap: inside the control block, not used)
              b_lo += TAP_BYTES >> 4;
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                if (TAIL && k >= ksteps) break;
                const bool acc_in = k != 0 || accumulate != 0;
                if constexpr (PAIR && KIND == 2) ptx::mma_f8_ss_pair(acc, ad + 2 * k, bd + 2 * k, idesc, acc_in);
                else if constexpr (PAIR) ptx::mma_f16_ss_pair(acc, ad + 2 * k, bd + 2 * k, idesc, acc_in);
                else if constexpr (KIND == 2) ptx::mma_f8_ss(acc, ad + 2 * k, bd + 2 * k, idesc, acc_in);
                else if constexpr (KIND == 1) ptx::mma_tf32_ss(acc, ad + 2 * k, bd + 2 * k, idesc, acc_in);
                else ptx::mma_f16_ss(acc, ad + 2 * k, bd + 2 * k, idesc, acc_in);
              }
              accumulate = 1;
            }
            if constexpr (PAIR) {
              if (!resident) ptx::mma_commit_pair(&b_empty[bs], 3);
              if (!resident && n > 1) ptx::mma_commit_pair(&b_empty[bs + 1], 3);
              if (block_done) ptx::mma_commit_pair(&a_empty[as], 3);
              if (last) ptx::mma_commit_pair(&acc_full[buf], 3);
            } else {
              if (!resident) ptx::mma_commit(&b_empty[bs]);
              if (!resident && n > 1) ptx::mma_commit(&b_empty[bs + 1]);
              if (block_done) ptx::mma_commit(&a_empty[as]);
              if (last) ptx::mma_commit(&acc_full[buf]);
            }
          }
          __syncwarp();
          accumulate = 1;
          need_a = block_done;
          if (block_done && ++as == a_stages) { as = 0; aphase ^= 1u; }
          i += n;
          if ((bs += n) == b_stages) { bs = 0; bphase ^= 1u; }
          if ((tg += n) == tap_groups) { tg = 0; ++cb; }
        }
        if (tile + tile_step < p.num_tiles) {  // (the tensor core is still at work on this tile)
          t = decode(tile + tile_step);
          row0 = first_row(t);
        }
        if (resident) bs = 0;
      }
    };
    auto with_tail = [&](auto kind_tag) {
      if (p.last_ksteps != 4) run(kind_tag, std::integral_constant<bool, true>{});
      else run(kind_tag, std::integral_constant<bool, false>{});
    };
    if (p.is_fp8) with_tail(std::integral_constant<int, 2>{});
    else if (!PAIR && p.is_tf32) with_tail(std::integral_constant<int, PAIR ? 0 : 1>{});
    else with_tail(std::integral_constant<int, 0>{});
    if (cluster) {
      ptx::cluster_sync_all();
      ptx::cluster_sync_all();
    }
  } else {
    // ---------------- epilogue: drain accumulators ----------------
    const int we = warp - kProducerWarps - 1;  // index among the worker warps
    const int quad = warp & 3, par = we >> 2;
    const uint32_t acc_empty0 = PAIR ? ptx::map_to_cta(ptx::smem_u32(&acc_empty[0]), 0u) : 0u;
    ptx::grid_dep_wait();

    // grid row -> (image, pixel of the output plane); false: no output pixel
    auto out_pixel = [&](int g, int& img, int& pix) {
      const int prow = p.fd_ws.div(g), q = g - prow * p.ws;
      img = p.fd_hs.div(prow);
      const int pp = prow - img * p.hs;
      pix = pp * p.out_w + q;
      const bool ok = g < p.rows_total && q < p.out_w && pp < p.out_h && img < p.batch;
      if (!ok) img = pix = 0;
      return ok;
    };
    auto bias_at = [&](int oc) {
      if (p.bias == nullptr || oc >= p.out_channels) return 0.f;
      if (p.bias_fp32) return static_cast<const float*>(p.bias)[oc];
      return p.is_bf16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(p.bias)[oc]) : __half2float(static_cast<const __half*>(p.bias)[oc]);
    };
    auto with_type = [&](auto&& f) {
      if (!PAIR && p.is_tf32) f(static_cast<float*>(p.y), static_cast<float*>(const_cast<void*>(p.residual)));
      else if (p.is_bf16) f(static_cast<__nv_bfloat16*>(p.y), static_cast<__nv_bfloat16*>(const_cast<void*>(p.residual)));
      else f(static_cast<__half*>(p.y), static_cast<__half*>(const_cast<void*>(p.residual)));
    };
    const int64_t cstride = p.out_nhwc ? 1 : p.pq;
    // Drains the accumulator of a tile (complete: acc_full has been waited for).  Warps drain on their own: the bias values of
    // a chunk pass through a corner of shared memory that belongs to the warp, and so do the rows of channel-contiguous output.
    // What does not need the accumulator is prepared before it is waited for.
    constexpr int CPW = BN / 32 / EG > 0 ? BN / 32 / EG : 1;  // chunks per warp: 1 or 2
    struct Out { int64_t base; bool ok; float bv[CPW]; uint32_t rows[4]; };
    auto prepare_out = [&](const Tile& t) {
      Out o;
      int img, pix;
      o.ok = out_pixel(t.m0 + quad * 32 + lane, img, pix);
      o.base = p.out_nhwc ? (int64_t(img) * p.pq + pix) * p.out_channels + t.n0 : (int64_t(img) * p.out_channels + t.n0) * p.pq + pix;
#pragma unroll
      for (int c = 0; c < CPW; ++c) o.bv[c] = bias_at(t.n0 + (par + EG * c) * 32 + lane);
      if (p.out_cells) {
#pragma unroll
        for (int it = 0; it < 4; ++it) {
          const bool ok = out_pixel(t.m0 + quad * 32 + it * 8 + (lane >> 2), img, pix);
          o.rows[it] = ok ? uint32_t(((int64_t(img) * p.pq + pix) * p.out_channels + t.n0) >> 3) : ~0u;
        }
      }
      return o;
    };
    float* bias_w = bias_s + we * 32;
    uint8_t* box = b_base + size_t(p.b_stages) * b_stage_bytes + size_t(we) * 2048;  // (p.out_nhwc)
    auto drain = [&](const Tile& t, int buf, const Out& o) {
      ptx::tc_fence_after_sync();
      const uint32_t acc = tmem_base + buf * BN + (uint32_t(quad * 32) << 16);
      const bool m_ok = o.ok;
      float bv = o.bv[0];
#pragma unroll 1
      for (int chunk = par; chunk < BN / 32; chunk += EG) {
        if (t.n0 + chunk * 32 >= p.out_channels) break;  // warp-uniform
        const int nvalid = min(32, p.out_channels - (t.n0 + chunk * 32));
        const int64_t off = o.base + int64_t(chunk * 32) * cstride;
        uint32_t v[32];
        ptx::tmem_ld_32x32b_x32(acc + uint32_t(chunk * 32), v);
        __syncwarp();
        bias_w[lane] = bv;
        bv = o.bv[CPW - 1];
        with_type([&](auto* yp, auto* rp) {
          using T = std::remove_pointer_t<decltype(yp)>;
          if constexpr (sizeof(T) == 2) {
            if (p.out_nhwc && rows_pay(nvalid, p.out_rows == 2)) {
              const bool cells = p.out_cells && nvalid == 32;
              if (rp != nullptr) {
                if (cells) staging_cells<true>(box, lane, rp, o.rows, uint32_t(chunk) * 4u);
                else if (p.out_rows == 2) staging_rows<true, true>(box, lane, rp, off, m_ok, nvalid);
                else staging_rows<false, true>(box, lane, rp, off, m_ok, nvalid);
              }
              __syncwarp();
              ptx::tmem_ld_wait();
              chunk_to_staging<T>(v, bias_w, box, lane, p.relu, rp != nullptr);
              __syncwarp();
              if (cells) staging_cells<false>(box, lane, yp, o.rows, uint32_t(chunk) * 4u);
              else if (p.out_rows == 2) staging_rows<true, false>(box, lane, yp, off, m_ok, nvalid);
              else staging_rows<false, false>(box, lane, yp, off, m_ok, nvalid);
              __syncwarp();
              return;
            }
          }
          __syncwarp();
          ptx::tmem_ld_wait();
          if (m_ok) store_chunk(v, bias_w, yp + off, rp != nullptr ? rp + off : nullptr, cstride, nvalid, p.relu);
        });
      }
      ptx::tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) {
        if constexpr (PAIR) ptx::mbar_arrive_cluster(acc_empty0 + uint32_t(buf) * 8u);
        else ptx::mbar_arrive(&acc_empty[buf]);
      }
    };

    int tcount = 0;
    for (int tile = tile_first; !cluster && tile < p.num_tiles; tile += tile_step, ++tcount) {
      const Tile t = decode(tile);
      const Out o = prepare_out(t);
      const int buf = tcount & 1;
      const bool ok = ptx::mbar_wait(&acc_full[buf], (tcount >> 1) & 1, p.status, kStatusEpilogueTimeout, p.wait_limit);
      if (!__all_sync(0xffffffffu, ok)) break;
      drain(t, buf, o);
    }
    if (cluster) {
      // Split-K inside a cluster (one tile per CTA): CTA `rank` owns the columns [rank * cpo, (rank + 1) * cpo) of the tile.
      // Every CTA writes its partial columns into the owner's idle operand stages through distributed shared memory, as
      // [sender][group of 4 columns][row][16 bytes]; the owner adds the senders in rank order (run-to-run identical).
      const Tile t = decode(tile_first);
      const bool ok = __all_sync(0xffffffffu, ptx::mbar_wait(&acc_full[0], 0, p.status, kStatusEpilogueTimeout, p.wait_limit));
      ptx::tc_fence_after_sync();
      const int rank = int(ptx::cluster_ctarank());
      const int gpo = BN / 4 / p.split;  // column groups per owner
      const int row = quad * 32 + lane;
      const uint32_t acc = tmem_base + (uint32_t(quad * 32) << 16);
      const uint32_t recv = ptx::smem_u32(a_base);
      ptx::cluster_sync_all();  // every CTA of the cluster has finished its MMAs: all stages are idle
      if (ok) {
        for (int chunk = par; chunk < BN / 32; chunk += EG) {
          if (t.n0 + chunk * 32 >= p.out_channels) break;
          uint32_t v[32];
          ptx::tmem_ld_32x32b_x32(acc + uint32_t(chunk * 32), v);
          ptx::tmem_ld_wait();
#pragma unroll
          for (int g = 0; g < 8; ++g) {
            const int grp = chunk * 8 + g, owner = p.fd_gpo.div(grp);
            const uint32_t dst = recv + uint32_t(((rank * gpo + (grp - owner * gpo)) * kTileM + row) * 16);
            ptx::st_cluster_v4(ptx::map_to_cta(dst, uint32_t(owner)), v[4 * g], v[4 * g + 1], v[4 * g + 2], v[4 * g + 3]);
          }
        }
      }
      ptx::cluster_sync_all();  // all partials have landed
      if (ok) {
        int img, pix;
        const bool m_ok = out_pixel(t.m0 + row, img, pix);
        const int64_t base = p.out_nhwc ? (int64_t(img) * p.pq + pix) * p.out_channels + t.n0
                                        : (int64_t(img) * p.out_channels + t.n0) * p.pq + pix;
        for (int g = par; g < gpo; g += EG) {
          const int col = (rank * gpo + g) * 4;
          if (t.n0 + col >= p.out_channels) break;
          float b4[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) b4[e] = bias_at(t.n0 + col + e);
          float4 part[8];
#pragma unroll
          for (int s = 0; s < 8; ++s)
            if (s < p.split) part[s] = *reinterpret_cast<const float4*>(a_base + size_t((s * gpo + g) * kTileM + row) * 16);
          float4 sum = part[0];
#pragma unroll
          for (int s = 1; s < 8; ++s)
            if (s < p.split) { sum.x += part[s].x; sum.y += part[s].y; sum.z += part[s].z; sum.w += part[s].w; }
          if (!m_ok) continue;
          const float a4[4] = {sum.x, sum.y, sum.z, sum.w};
          with_type([&](auto* yp, auto* rp) {
            using T = std::remove_pointer_t<decltype(yp)>;
            float r4[4] = {0.f, 0.f, 0.f, 0.f};
            if (rp != nullptr) {
#pragma unroll
              for (int e = 0; e < 4; ++e)
                if (t.n0 + col + e < p.out_channels) r4[e] = load_as_float(rp + base + int64_t(col + e) * cstride);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              float f = a4[e] + b4[e] + r4[e];
              if (p.relu) f = fmaxf(f, 0.f);
              if (t.n0 + col + e < p.out_channels) yp[base + int64_t(col + e) * cstride] = round_to<T>(f);
            }
          });
        }
      }
      ptx::tc_fence_before_sync();
    }
  }

  ptx::tc_fence_before_sync();
  if constexpr (PAIR) {
    // Neither CTA of a pair may leave (or free tensor memory) while the other can still signal its barriers or while the
    // leader's MMAs can still read its shared memory: both meet here once all their roles have finished.
    ptx::cluster_sync_all();
    if (warp == kProducerWarps) {
      ptx::tc_fence_after_sync();
      ptx::tmem_dealloc_pair(tmem_base, TMEM_COLS);
    }
  } else {
    __syncthreads();
    if (warp == kProducerWarps) {
      ptx::tc_fence_after_sync();
      ptx::tmem_dealloc(tmem_base, TMEM_COLS);
    }
  }
}

template <int BN, int NW, bool PAIR>
cudaError_t halo_prepare_one(size_t smem) {
  return cudaFuncSetAttribute(conv_halo_kernel<BN, NW, PAIR>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
}
template <int BN, int NW, bool PAIR>
cudaError_t halo_launch_one(const CUtensorMap& ta, const CUtensorMap& tw, const ConvHaloParams& p, dim3 grid, size_t smem, cudaStream_t st) {
  return launch_pdl_cluster(conv_halo_kernel<BN, NW, PAIR>, grid, dim3(32 * (kProducerWarps + 1 + NW)), smem, st,
                            PAIR ? 2u : unsigned(p.split), ta, tw, p);
}

#define GIEB_HALO_DISPATCH(FN, ...)                                      \
  switch ((pair ? 100000 : 0) + tile_n * 100 + workers) {                \
    case 32 * 100 + 8: return FN<32, 8, false>(__VA_ARGS__);             \
    case 64 * 100 + 8: return FN<64, 8, false>(__VA_ARGS__);             \
    case 128 * 100 + 8: return FN<128, 8, false>(__VA_ARGS__);           \
    case 256 * 100 + 16: return FN<256, 16, false>(__VA_ARGS__);         \
    case 100000 + 128 * 100 + 16: return FN<128, 16, true>(__VA_ARGS__); \
    case 100000 + 256 * 100 + 16: return FN<256, 16, true>(__VA_ARGS__); \
    default: return cudaErrorInvalidValue;                               \
  }

}  // namespace

size_t conv_halo_smem_bytes(int tile_n, bool pair, int workers, int taps_per_load, int a_stages, size_t a_stage_bytes, int b_stages, bool staging) {
  return 1024 /* for the alignment */ + kHaloCtrl + size_t(a_stages) * a_stage_bytes + size_t(b_stages) * taps_per_load * (pair ? tile_n / 2 : tile_n) * 128 +
         (staging ? size_t(workers) * 2048 : 0);
}

cudaError_t conv_halo_prepare(int tile_n, int workers, bool pair, size_t smem) { GIEB_HALO_DISPATCH(halo_prepare_one, smem) }

cudaError_t conv_halo_launch(int tile_n, int workers, bool pair, const CUtensorMap& tm_act, const CUtensorMap& tm_wgt,
                             const ConvHaloParams& p, dim3 grid, size_t smem, cudaStream_t stream) {
  GIEB_HALO_DISPATCH(halo_launch_one, tm_act, tm_wgt, p, grid, smem, stream)
}

}  // namespace gieb
