// Strict-FP32 convolution (no tensor cores, no TF32): register-blocked SIMT implicit GEMM straight from NCHW with
// the bias + ReLU epilogue fused.  Stands in for implicit_gemm_kernel (src/kernels/implicit_gemm.cu:47-189).
//
// GEMM view: rows = output pixels (b, oh, ow), columns = output channels, k = (c, r, s) in OIHW order so a weight
// row is contiguous in k.  Per CTA of 128 threads: a TP x TO output tile (64 x 64, or 128 x 32 for few channels), 8 pixels x
// 4 channels per thread, BK = 16 reduction slabs in a ring of shared-memory buffers (pixels contiguous in the X slab, so the
// gather from NCHW is coalesced along ow; 128-bit copies of W along k).  Accumulation is fmaf in k order.
//
// What bounds it: with enough CTAs per SM, ~1030 cycles per 64 x 64 x 16 slab against 512 of FMA issue -- a thread reads 12
// words of shared memory per 32 FMAs, and the SM delivers 128 bytes per cycle (8 x 8 tiles read less but leave 12 warps per SM,
// too few to hide their latencies: 1120).  The packed FMA (fma.rn.f32x2, two adjacent pixels against a duplicated weight; each
// half rounds as fmaf does) halves the FMA instructions.  Gathered elements pass through registers: a 4-byte asynchronous
// copy per element keeps the load/store unit busy several times as long.  Problems with few tiles split the reduction over
// the CTAs of a thread-block cluster, which exchange their partial tiles through distributed shared memory and add them in
// slice order, so that results are run-to-run identical.  Measured against scalar FMAs on 32 x 32 tiles: 11 x 212 -> 560
// channels, 17 x 17, 5x5 1004 -> 540 us; 512 -> 512, 7 x 7, 3x3 137 -> 31 us; 64 -> 64, 56 x 56, 3x3 18.4 -> 15.9 us.
#include <stdint.h>

#include <cmath>
#include <mutex>
#include <set>
#include <type_traits>
#include <utility>

#include "conv_fp32_device.cuh"
#include "conv_fp32_table.h"
#include "internal.h"
#include "ptx.cuh"

namespace gieb {
namespace {

constexpr int kBK = kFp32Slab;
constexpr int kMaxSmem = 96 * 1024;

struct Fp32Args {
  const float* x;
  const float* w;
  const float* bias;
  float* y;
  int batch, c, h, wd, o, r, s, stride_h, stride_w, pad_h, pad_w, out_h, out_w, relu;
  int pixels;  // batch * out_h * out_w
  int k;       // c * r * s
  int slices;  // CTAs of a cluster that share one output tile, each reducing slabs_per_slice slabs
  int slabs_per_slice;
  FastDiv fd_rs, fd_s, fd_pq, fd_out_w;  // multiply-high reciprocals of r*s, s, out_h*out_w, out_w
};

// 4-byte asynchronous copy global -> shared; `valid` false writes zero (nothing is read: the source size is 0).
__device__ __forceinline__ void cp_async4(void* dst, const float* src, bool valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(ptx::smem_u32(dst)), "l"(src), "r"(valid ? 4 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

constexpr int kWPitch = kBK + 4;  // floats per weight row in shared memory: 16-byte aligned rows, conflict-free 128-bit reads
constexpr int kThreads = 128;
constexpr int kRing = 4;          // slabs in shared memory

// X slab [kBK][TP]: gathered from NCHW element by element with zeros for padding (pixels contiguous), or, for unpadded 1x1
//   kernels of stride 1 whose planes are multiples of 4 pixels (XVEC), 16-byte asynchronous copies along the pixels;
// W slab [TO][kBK]: asynchronous copies, 16 bytes along k (OIHW rows are contiguous in k) when W16, else 4 bytes.
// LUT: k -> (offset of (c, r, s) inside one image, r, s) comes from a table built once per CTA (the analogue of
// build_conv_lut, src/kernels/conv_common.cu:25-37) instead of two divisions per gathered element.
// A cluster of `slices` CTAs (blockIdx.x = pixel tile * slices + slice) shares one output tile.
template <int TP, int TO, bool LUT, bool W16, bool XVEC>
__global__ void __launch_bounds__(kThreads)
conv_fp32_kernel(const Fp32Args a) {
  static_assert(TP / 8 * (TO / 4) == kThreads, "8 pixels x 4 channels per thread");
  constexpr int GP = TP / 8, GO = TO / 4;          // thread grid over pixels and channels
  constexpr int XE = kBK * TP / kThreads;          // X-slab elements loaded per thread
  constexpr int XS = kBK * TP, WS = TO * kWPitch;  // floats per X / W slab
  extern __shared__ __align__(16) float tiles[];    // [kRing] X slabs, [kRing] W slabs, the table; reused for the exchange of partial tiles
  float* xs_base = tiles;
  float* ws_base = tiles + kRing * XS;
  int2* lut = reinterpret_cast<int2*>(tiles + kRing * (XS + WS));

  const int t = threadIdx.x;
  const int tx = t % GP, ty = t / GP;  // pixels tx*4 .. +3 and TP/2 + tx*4 .. +3; channels ty + GO*j
  const int slice = a.slices > 1 ? int(blockIdx.x % unsigned(a.slices)) : 0;
  const int pix0 = int(blockIdx.x / unsigned(a.slices)) * TP, oc0 = blockIdx.y * TO;
  const int rs = a.r * a.s;
  const int pq = a.out_h * a.out_w;
  const int slabs_all = fp32_slabs(a.k);
  const int slab0 = slice * a.slabs_per_slice;
  const int slabs = max(0, min(a.slabs_per_slice, slabs_all - slab0));
  const int kbase = slab0 * kBK;

  // Loader role for X: thread owns pixel (t % TP) and slab rows (t / TP) + i * (kThreads / TP).
  const int lp = t % TP;
  const int lpix = pix0 + lp;
  const bool lp_ok = lpix < a.pixels;
  int ih0 = 0, iw0 = 0;
  const float* xb = a.x;
  if (!XVEC && lp_ok) {
    const int b = a.fd_pq.div(lpix), rem = lpix - b * pq;
    const int oh = a.fd_out_w.div(rem), ow = rem - oh * a.out_w;
    ih0 = oh * a.stride_h - a.pad_h;
    iw0 = ow * a.stride_w - a.pad_w;
    xb = a.x + size_t(b) * a.c * a.h * a.wd;
  }
  const int xoff0 = ih0 * a.wd + iw0;  // offset of tap (0, 0) of this pixel inside a channel plane (may be negative)
  // XVEC: thread owns pixel group (t % (TP/4)) and slab rows (t / (TP/4)) + i * (kThreads / (TP/4)); a group of four pixels
  // lies in one image because planes are multiples of four
  const int vg = t % (TP / 4), vpix = pix0 + vg * 4;
  const bool v_ok = XVEC && vpix < a.pixels;
  if (v_ok) {
    const int b = a.fd_pq.div(vpix);
    xb = a.x + size_t(b) * a.c * pq + (vpix - b * pq);
  }
  ptx::grid_dep_wait();
  if (LUT) {
    for (int i = t; i < slabs * kBK; i += kThreads) {
      const int k = kbase + i;
      int2 e = make_int2(0, kNoRow << 16);  // a row outside the image: never loaded
      if (k < a.k) {
        const int c = a.fd_rs.div(k), q = k - c * rs;
        const int r = a.fd_s.div(q), sx = q - r * a.s;
        e = make_int2((c * a.h + r) * a.wd + sx, (r << 16) | sx);
      }
      lut[i] = e;
    }
    __syncthreads();
  }

  // gathered elements of a slab: loaded into registers one slab ahead of their store into the ring
  float xreg[XVEC ? 1 : XE];
  auto load_x = [&](int sl) {
    const int k0 = kbase + sl * kBK;
#pragma unroll
    for (int i = 0; i < XE; ++i) {
      const int kk = t / TP + i * (kThreads / TP);
      const int k = k0 + kk;
      float v = 0.f;
      if (LUT) {
        const int2 e = lut[sl * kBK + kk];
        const int ih = ih0 + (e.y >> 16), iw = iw0 + (e.y & 0xffff);
        if (lp_ok && unsigned(ih) < unsigned(a.h) && unsigned(iw) < unsigned(a.wd)) v = xb[e.x + xoff0];
      } else if (lp_ok && k < a.k) {
        const int c = a.fd_rs.div(k), q = k - c * rs;
        const int r = a.fd_s.div(q), sx = q - r * a.s;
        const int ih = ih0 + r, iw = iw0 + sx;
        if (ih >= 0 && ih < a.h && iw >= 0 && iw < a.wd) v = xb[(size_t(c) * a.h + ih) * a.wd + iw];
      }
      xreg[i] = v;
    }
  };
  auto store_x = [&](int slot) {
    float* xs = xs_base + slot * XS;
#pragma unroll
    for (int i = 0; i < XE; ++i) xs[(t / TP + i * (kThreads / TP)) * TP + lp] = xreg[i];
  };
  // issue the asynchronous copies of slab `sl` of this slice into ring slot `slot`
  auto fetch = [&](int sl, int slot) {
    float* xs = xs_base + slot * XS;
    float* ws = ws_base + slot * WS;
    const int k0 = kbase + sl * kBK;
    if (XVEC) {
#pragma unroll
      for (int i = 0; i < kBK * TP / 4 / kThreads; ++i) {
        const int kk = t / (TP / 4) + i * (kThreads / (TP / 4));
        const bool ok = v_ok && k0 + kk < a.k;
        cp_async16(xs + kk * TP + vg * 4, ok ? xb + size_t(k0 + kk) * pq : a.x, ok ? 16 : 0);
      }
    }
    if (W16) {  // TO rows x 4 vectors of 4 k-values
#pragma unroll
      for (int i = 0; i < TO * 4 / kThreads; ++i) {
        const int v = t + i * kThreads;
        const int row = v >> 2, kq = (v & 3) * 4;
        const int oc = oc0 + row, k = k0 + kq;
        const int left = (oc < a.o && k < a.k) ? min(4, a.k - k) * 4 : 0;
        cp_async16(ws + row * kWPitch + kq, left ? a.w + size_t(oc) * a.k + k : a.w, left);
      }
    } else {
      const int wk = t % kBK;
#pragma unroll
      for (int i = 0; i < kBK * TO / kThreads; ++i) {
        const int row = t / kBK + i * (kThreads / kBK);
        const int oc = oc0 + row, k = k0 + wk;
        const bool ok = oc < a.o && k < a.k;
        cp_async4(ws + row * kWPitch + wk, ok ? a.w + size_t(oc) * a.k + k : a.w, ok);
      }
    }
  };

  uint64_t acc[4][4];  // [pixel pair][channel]
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0;

#pragma unroll
  for (int s = 0; s < kRing - 1; ++s) {  // prologue: kRing - 1 slabs in flight
    if (s < slabs) fetch(s, s);
    cp_async_commit();
  }
  if (!XVEC && slabs > 0) {
    load_x(0);
    store_x(0);
    if (slabs > 1) load_x(1);
  }
  for (int sl = 0; sl < slabs; ++sl) {
    cp_async_wait<kRing - 2>();  // this thread's copies of slab sl have landed
    __syncthreads();             // everyone's have; and everyone has finished reading the slots refilled below
    if (sl + kRing - 1 < slabs) fetch(sl + kRing - 1, (sl + kRing - 1) % kRing);
    cp_async_commit();
    if (!XVEC && sl + 1 < slabs) {
      store_x((sl + 1) % kRing);
      if (sl + 2 < slabs) load_x(sl + 2);
    }
    const float* xs = xs_base + (sl % kRing) * XS + tx * 4;
    const float* ws = ws_base + (sl % kRing) * WS + ty * kWPitch;
#pragma unroll
    for (int q = 0; q < kBK / 4; ++q) {
      float4 wv[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) wv[j] = *reinterpret_cast<const float4*>(ws + j * GO * kWPitch + q * 4);
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {  // k order: the accumulation order of the strict-FP32 contract
        const ulonglong2 xl = *reinterpret_cast<const ulonglong2*>(xs + (q * 4 + kk) * TP);
        const ulonglong2 xh = *reinterpret_cast<const ulonglong2*>(xs + (q * 4 + kk) * TP + TP / 2);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float wk = kk == 0 ? wv[j].x : (kk == 1 ? wv[j].y : (kk == 2 ? wv[j].z : wv[j].w));
          const uint64_t w2 = pack2(wk, wk);
          fma2(acc[0][j], xl.x, w2);
          fma2(acc[1][j], xl.y, w2);
          fma2(acc[2][j], xh.x, w2);
          fma2(acc[3][j], xh.y, w2);
        }
      }
    }
  }
  cp_async_wait<0>();
  ptx::grid_dep_launch();  // late: CTAs of the next launch that became resident earlier would crowd onto the SMs of this one

  float out[4][8];  // [channel][pixel]
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 v = unpack2(acc[i][j]);
      out[j][2 * i] = v.x;
      out[j][2 * i + 1] = v.y;
    }

  if (a.slices > 1) {
    // Partial tiles meet through distributed shared memory: every CTA lays its own out as [vector][thread] (16-byte vector
    // v = 2 j + half), then thread t of CTA s sums the vectors v with v % slices == s over all slices, in slice order.
    __syncthreads();  // all slabs consumed: the tiles may be overwritten
    float4* mine = reinterpret_cast<float4*>(tiles);
#pragma unroll
    for (int v = 0; v < 8; ++v) mine[v * kThreads + t] = make_float4(out[v >> 1][(v & 1) * 4], out[v >> 1][(v & 1) * 4 + 1], out[v >> 1][(v & 1) * 4 + 2], out[v >> 1][(v & 1) * 4 + 3]);
    ptx::cluster_sync_all();
    const uint32_t base = ptx::smem_u32(mine) + uint32_t(t) * 16u;
#pragma unroll
    for (int v = 0; v < 8; ++v) {
      if (v % a.slices != slice) continue;
      float4 part[8];
#pragma unroll
      for (int s = 0; s < 8; ++s)  // all loads in flight, then the adds
        if (s < a.slices) part[s] = ptx::ld_cluster_v4(ptx::map_to_cta(base + uint32_t(v * kThreads) * 16u, uint32_t(s)));
      float4 sum = part[0];
#pragma unroll
      for (int s = 1; s < 8; ++s)
        if (s < a.slices) { sum.x += part[s].x; sum.y += part[s].y; sum.z += part[s].z; sum.w += part[s].w; }
      out[v >> 1][(v & 1) * 4] = sum.x; out[v >> 1][(v & 1) * 4 + 1] = sum.y; out[v >> 1][(v & 1) * 4 + 2] = sum.z; out[v >> 1][(v & 1) * 4 + 3] = sum.w;
    }
    ptx::cluster_sync_all();  // nobody leaves while a peer still reads its tile
  }

  // Epilogue (fused_epilogue.cuh:11-16 order): + bias, ReLU, store.  Pixels are the fast index of NCHW: a run of four
  // pixels leaves as one 128-bit store when it lies in one image and the address is 16-byte aligned.
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const int pixq = pix0 + half * (TP / 2) + tx * 4;
    const int bq = pixq < a.pixels ? a.fd_pq.div(pixq) : 0, remq = pixq - bq * pq;
    const bool quad_ok = pixq + 3 < a.pixels && remq + 3 < pq;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int oc = oc0 + ty + j * GO;
      if (oc >= a.o || (a.slices > 1 && (2 * j + half) % a.slices != slice)) continue;
      const float bv = a.bias ? __ldg(a.bias + oc) : 0.f;
      float v[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        v[i] = out[j][half * 4 + i] + bv;
        if (a.relu) v[i] = fmaxf(v[i], 0.f);
      }
      float* dst = a.y + (size_t(bq) * a.o + oc) * pq + remq;
      if (quad_ok && (reinterpret_cast<uintptr_t>(dst) & 15u) == 0) {
        *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int pix = pixq + i;
          if (pix >= a.pixels) continue;
          const int b = a.fd_pq.div(pix), rem = pix - b * pq;
          a.y[(size_t(b) * a.o + oc) * pq + rem] = v[i];
        }
      }
    }
  }
}

// Tile shape: 64 channels wide unless at most 32 are there to be computed.
int tile_o(int o) { return o <= 32 ? 32 : 64; }
int tile_p(int o) { return o <= 32 ? 128 : 64; }

constexpr int kMaxWideTaps = 31;  // filter taps in a pixel's bit mask (conv_fp32_wide.cu)

}  // namespace

// Clusters of 1 to 8 CTAs that the machine holds at a time, with at most 1 to 5 CTAs per SM (cudaOccupancyMaxActiveClusters).
constexpr int kClusters[5][8] = {{148, 74, 45, 33, 26, 22, 15, 15}, {296, 148, 93, 71, 56, 45, 37, 33}, {444, 222, 142, 104, 82, 71, 56, 48},
                                 {592, 296, 187, 142, 112, 93, 78, 71}, {740, 370, 235, 175, 142, 116, 97, 86}};
// As many clusters are spread with one CTA per SM although two would fit.  (Wide tiles of clusters of eight: 15 take the time of CTAs
// alone on their SMs, 16 that of pairs; of five 21 and 25; of six 14, with 16 to 19 between the two; three and four not measured.)
constexpr int kSpread[8] = {148, 74, 41, 30, 22, 15, 15, 15};

// The choice by SM cycles.
// This kernel: the CTAs that an SM holds together hide each other's latencies: a slab costs ~1600 cycles of a CTA alone on its SM,
// ~1100 per CTA of two and ~1030 of more; a CTA's prologue and epilogue cost ~1500 cycles, a cluster's exchange ~2000 more, and up to
// five CTAs share an SM.  Without the decode table (reductions of more than kLutMax terms per slice) everything takes twice as long.
// The wide tiles (fitted to 230 timings of 18 layers, 7 % off on average): 16 terms of a CTA's tiles are 2048 cycles of FMA issue and
// cost 3510 cycles of a CTA alone on its SM, 3075 each of two; ~6900 per wave of CTAs, and ~12,100 to exchange partial tiles.
// Both run in waves of what kClusters says: a wave of more clusters than that, as of more CTAs than SMs, takes as long as two.
// So they are taken for long reductions and many tiles: 17 x 64 -> 109 at 69 x 38, 5x5 474 -> 402 us; 2 x 762 -> 256 at 18 x 18,
// 3x3/2 48.3 -> 40.6; 2 x 976 -> 80 at 37 x 37, 5x5 885 -> 433; not for 64 -> 64 at 56 x 56, 3x3, one image (16.1 us; 19.9 wide).
Fp32Choice conv_fp32_choose(const Fp32Shape& g) {
  const int o = g.o;
  const int64_t pixels = int64_t(g.batch) * g.out_h * g.out_w;
  const int slabs = fp32_slabs(g.c * g.r * g.s);
  Fp32Choice best{0, tile_p(o), tile_o(o), 1};
  const int64_t tiles = ((pixels + best.tile_p - 1) / best.tile_p) * ((o + best.tile_o - 1) / best.tile_o);
  auto narrow = [&](int sl, double load) {
    const double slab = load <= 1 ? 1600.0 : (load <= 2 ? 1100.0 : 1030.0);
    return load * ((slabs + sl - 1) / sl) * slab + std::ceil(load / 5.0) * (1500.0 + (sl > 1 ? 2000.0 : 0.0));
  };
  double best_t = 1e300;
  for (int sl = 1; sl <= 8 && sl <= slabs; ++sl) {
    const int per = (slabs + sl - 1) / sl;
    if ((slabs + per - 1) / per != sl) continue;  // (an empty slice)
    const double t = narrow(sl, double((tiles * sl + kNumSms - 1) / kNumSms));
    if (t < best_t * 0.98) { best_t = t; best.slices = sl; }
  }
  if (g.r * g.s > kMaxWideTaps || !conv_fp32_wide_offsets_fit(g.c, g.h, g.w, g.r, g.s)) return best;
  const int64_t five = kClusters[4][best.slices - 1], left = tiles % five;
  int level = 0;
  while (level < 5 && left > (level ? kClusters[level - 1][best.slices - 1] : 0)) ++level;
  const bool table = int64_t((slabs + best.slices - 1) / best.slices) * kBK <= kLutMax;
  const double other = narrow(best.slices, double(5 * (tiles / five) + level)) * (table ? 1.0 : 2.0) + 7600.0;
  double limit = 1e300;
  for (int tp = 128; tp >= 64; tp /= 2) {
    const int groups = 256 / tp;
    const int64_t clusters = ((pixels + tp - 1) / tp) * ((o + 63) / 64);
    for (int sl = 1; sl <= 8 && sl * groups <= slabs; ++sl) {
      const int members = sl * groups, per = (slabs + members - 1) / members;
      if (clusters * (sl - 1) > 6 * kNumSms) break;  // (clusters of many waves of CTAs: not measured, and splitting gains nothing)
      const int64_t wave = kClusters[1][sl - 1], rest = clusters % wave;
      const double pair = 2.0 * per * 3075.0 + 6900.0;
      double t = double(clusters / wave) * pair + (rest == 0 ? 0.0 : (rest <= kSpread[sl - 1] ? per * 3510.0 + 6900.0 : pair));
      if (members > 1) t += 12100.0 * double((clusters + wave - 1) / wave);
      // (margins: with them none of 134 layers is more than 1 % slower than on narrow tiles)
      if (t < limit && t < (tp == 128 ? 0.88 : 0.85) * other - 3200.0) { limit = t; best = Fp32Choice{1, tp, 64, sl}; }
    }
  }
  return best;
}

namespace {

// How conv_fp32_kernel is launched for a choice: the instance, the slabs of a CTA and its shared memory.
struct Form {
  bool xvec, lut;
  int slabs_per_slice;
  size_t smem;
};
Form form_of(const Fp32Choice& ch, const Fp32Shape& g, bool x_aligned) {
  Form f;
  const int slabs = fp32_slabs(g.c * g.r * g.s);
  f.slabs_per_slice = (slabs + ch.slices - 1) / ch.slices;
  f.xvec = x_aligned && g.r == 1 && g.s == 1 && g.stride_h == 1 && g.stride_w == 1 && g.pad_h == 0 && g.pad_w == 0 && (g.out_h * g.out_w) % 4 == 0;
  f.lut = !f.xvec && conv_fp32_table_fits(int64_t(f.slabs_per_slice) * kBK, g.c, g.h, g.w, g.r, g.s, g.pad_h);
  f.smem = size_t(kRing) * (kBK * ch.tile_p + ch.tile_o * kWPitch) * sizeof(float) + (f.lut ? size_t(f.slabs_per_slice) * kBK * sizeof(int2) : 0);
  return f;
}

}  // namespace

size_t conv_fp32_smem_bytes(const Fp32Choice& ch, const Fp32Shape& g) {
  return ch.wide ? conv_fp32_wide_smem_bytes(ch.tile_p) : form_of(ch, g, true).smem;
}

cudaError_t conv_fp32_launch(const Fp32Choice& ch, const Fp32Shape& g, const void* x, const void* w, const void* bias, void* y, int relu,
                             cudaStream_t stream) {
  if (ch.wide) return conv_fp32_wide_launch(ch, g, x, w, bias, y, relu, stream);
  Fp32Args a;
  a.x = static_cast<const float*>(x);
  a.w = static_cast<const float*>(w);
  a.bias = static_cast<const float*>(bias);
  a.y = static_cast<float*>(y);
  a.batch = g.batch; a.c = g.c; a.h = g.h; a.wd = g.w; a.o = g.o; a.r = g.r; a.s = g.s;
  a.stride_h = g.stride_h; a.stride_w = g.stride_w; a.pad_h = g.pad_h; a.pad_w = g.pad_w;
  a.out_h = g.out_h; a.out_w = g.out_w; a.relu = relu;
  a.pixels = g.batch * g.out_h * g.out_w;
  a.k = g.c * g.r * g.s;
  a.fd_rs = FastDiv::make(g.r * g.s);
  a.fd_s = FastDiv::make(g.s);
  a.fd_pq = FastDiv::make(g.out_h * g.out_w);
  a.fd_out_w = FastDiv::make(g.out_w);
  const int tp = ch.tile_p, to = ch.tile_o;
  const int64_t tiles_p = (int64_t(a.pixels) + tp - 1) / tp, tiles_o = (g.o + to - 1) / to;
  const Form f = form_of(ch, g, (reinterpret_cast<uintptr_t>(x) & 15u) == 0);
  a.slices = ch.slices;
  a.slabs_per_slice = f.slabs_per_slice;
  const bool w16 = a.k % 4 == 0 && (reinterpret_cast<uintptr_t>(w) & 15u) == 0;  // 128-bit copies along k
  const size_t smem = f.smem;
  const dim3 grid(unsigned(tiles_p * a.slices), unsigned(tiles_o));
  auto go = [&](auto kernel) -> cudaError_t {
    // the opt-in to more than 48 KiB of dynamic shared memory is per function and device: done once each, under a mutex
    // (set_max_dynamic_smem of the reference, src/kernels/conv_common.cu:9-21)
    if (smem > 48 * 1024) {
      static std::mutex mu;
      static std::set<std::pair<const void*, int>> done;
      int dev = 0;
      cudaError_t e = cudaGetDevice(&dev);
      if (e != cudaSuccess) return e;
      std::lock_guard<std::mutex> lock(mu);
      const auto key = std::make_pair(reinterpret_cast<const void*>(kernel), dev);
      if (done.find(key) == done.end()) {
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem);
        if (e != cudaSuccess) return e;
        done.insert(key);
      }
    }
    return launch_pdl_cluster(kernel, grid, dim3(kThreads), smem, stream, unsigned(a.slices), a);
  };
  auto pick = [&](auto tpc, auto toc) {
    constexpr int TP = decltype(tpc)::value, TO = decltype(toc)::value;
    if (f.xvec) return w16 ? go(conv_fp32_kernel<TP, TO, false, true, true>) : go(conv_fp32_kernel<TP, TO, false, false, true>);
    if (f.lut) return w16 ? go(conv_fp32_kernel<TP, TO, true, true, false>) : go(conv_fp32_kernel<TP, TO, true, false, false>);
    return w16 ? go(conv_fp32_kernel<TP, TO, false, true, false>) : go(conv_fp32_kernel<TP, TO, false, false, false>);
  };
  return to == 32 ? pick(std::integral_constant<int, 128>{}, std::integral_constant<int, 32>{})
                  : pick(std::integral_constant<int, 64>{}, std::integral_constant<int, 64>{});
}

}  // namespace gieb
