// Strict-FP32 convolution for layers with enough work to fill the machine with larger thread tiles than conv_fp32.cu's: 16 pixels x
// 8 channels per thread on packed FMAs (fma.rn.f32x2, two adjacent pixels against a duplicated weight; each half rounds as fmaf).
//
// A 128-bit shared-memory read returns 512 bytes to a warp, four cycles at the SM's 128 bytes per cycle, whatever its lanes share.
// Per term of the reduction a thread tile of 8 x 4 takes 3 such reads for 32 FMAs (12 cycles for 8 of FMA issue), 8 x 8 takes 4
// for 64 (16 for 16), 16 x 8 takes 6 for 128 (24 for 32): only then do the FMAs bound the loop.  Everything else a slab needs is
// kept below what is left: a gathered element costs a predicate out of the pixel's bit mask of valid filter taps, an addition, a
// load and a store, and a decoded (c, r, s) entry serves two pixels; weights are stored [k][channel], so eight of them are two reads.
// In the end the loop takes 1.5 times its FMA issue (3075 cycles per 2048, two CTAs per SM; 8 x 4 tiles take 2.0 times), and a CTA's
// first loads and last stores ~6900 cycles: see conv_fp32_choose() for where it is taken and what it gains.
// A CTA has 128 threads in KG groups, which compute the same TP x 64 tile over slices of the reduction of their own (KG * TP = 256: two
// groups and 128 pixels, or four and 64); a cluster of `slices` CTAs splits it further.  The partial tiles are added in slice order: results are run-to-run identical.
#include <stdint.h>

#include <type_traits>

#include "conv_fp32_device.cuh"
#include "conv_fp32_table.h"
#include "internal.h"

namespace gieb {
namespace {

constexpr int kBK = kFp32Slab;         // terms of a slab
constexpr int kHalf = kBK / 2;  // gathered elements pass through registers half a slab at a time
constexpr int kThreads = 128;
constexpr int kTO = 64;
constexpr int kWRow = kTO + 4;  // floats per term of a weight slab
constexpr int kXRing = 3;

struct Fp32WideArgs {
  const float* x;
  const float* w;
  const float* bias;
  float* y;
  int c, h, wd, o, s, taps;
  int stride_h, stride_w, pad_h, pad_w, out_w, pq, relu;
  int pixels, k;
  int slices, slabs_per_group;
  FastDiv fd_rs, fd_s, fd_pq, fd_out_w, fd_slices;
};

// XVEC: unpadded 1x1 of stride 1 whose planes are multiples of 4 pixels, x 16-byte aligned: 16-byte copies along the pixels.
// W16: rows of w are multiples of 4 terms and 16-byte aligned.
template <int TP, bool XVEC, bool W16>
__global__ void __launch_bounds__(kThreads, 2) conv_fp32_wide_kernel(const __grid_constant__ Fp32WideArgs a) {
  constexpr int G = TP / 2, KG = kThreads / G;  // threads of a group, groups
  constexpr int GP = TP / 16;                   // threads along the pixels; kTO / 8 along the channels
  constexpr int XS = kBK * TP, WS = kBK * kWRow;
  constexpr int GROUP_FLOATS = kXRing * XS + 2 * WS + 2 * 3 * kBK;
  static_assert(G * KG == kThreads && G >= 32, "whole warps per group");
  extern __shared__ __align__(16) float tiles[];

  const int grp = threadIdx.x / G, t = threadIdx.x % G;
  const int tx = t % GP, ty = t / GP;  // pixels tx * 4 + i * TP / 4 + (0..3), channels ty * 4 + i * 32 + (0..3)
  float* xs_base = tiles + grp * GROUP_FLOATS;
  float* ws_base = xs_base + kXRing * XS;
  int2* table = reinterpret_cast<int2*>(ws_base + 2 * WS);  // [3 slabs][kBK] offset of (c, r, s) inside an image, tap

  const int tile = a.fd_slices.div(int(blockIdx.x)), slice = int(blockIdx.x) - tile * a.slices;
  const int pix0 = tile * TP, oc0 = int(blockIdx.y) * kTO;
  const int slabs_all = fp32_slabs(a.k);
  const int slab0 = (slice * KG + grp) * a.slabs_per_group;
  const int slabs = max(0, min(a.slabs_per_group, slabs_all - slab0));
  const int kbase = slab0 * kBK;
  auto group_sync = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(grp + 1), "n"(G) : "memory"); };

  // ---- loaders' roles ----
  // gathered: pixels t and t + G of the tile, every term; mask bit q: filter tap q lies inside the image
  const float* xb[2] = {a.x, a.x};
  uint32_t mask[2] = {0u, 0u};
  const float* vb = a.x;  // XVEC: four pixels of an image (planes are multiples of four)
  bool v_ok = false;
  constexpr int VG = TP / 4, VROWS = XVEC ? (G > VG ? G / VG : 1) : 1;  // groups of four pixels; terms taken at a time
  if (XVEC) {
    const int p = pix0 + t % VG * 4;
    v_ok = p < a.pixels;
    if (v_ok) {
      const int b = a.fd_pq.div(p);
      vb = a.x + size_t(b) * a.c * a.pq + (p - b * a.pq);
    }
  } else {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int p = pix0 + t + u * G;
      if (p < a.pixels) {
        const int b = a.fd_pq.div(p), rem = p - b * a.pq;
        const int oh = a.fd_out_w.div(rem), ow = rem - oh * a.out_w;
        const int ih = oh * a.stride_h - a.pad_h, iw = ow * a.stride_w - a.pad_w;
        for (int q = 0, r = 0, s = 0; q < a.taps; ++q) {
          if (unsigned(ih + r) < unsigned(a.h) && unsigned(iw + s) < unsigned(a.wd)) mask[u] |= 1u << q;
          if (++s == a.s) { s = 0; ++r; }
        }
        xb[u] = a.x + (int64_t(b) * a.c * a.h + ih) * a.wd + iw;
      }
    }
  }
  // weights: channel rows wr + i * (G / 4), terms wq .. wq + 3
  const int wq = (t & 3) * 4, wr = t >> 2;
  constexpr int WV = kTO * 4 / G;  // four-term vectors per thread and slab

  auto fill_table = [&](int sl) {
    if (!XVEC && t < kBK) {
      const int k = kbase + sl * kBK + t;
      int2 e = make_int2(0, 31);  // (a.taps <= 31: bit 31 of every mask is clear)
      if (sl < slabs && k < a.k) {
        const int c = a.fd_rs.div(k), q = k - c * a.taps;
        const int r = a.fd_s.div(q);
        e = make_int2((c * a.h + r) * a.wd + (q - r * a.s), q);
      }
      table[sl % 3 * kBK + t] = e;
    }
  };
  float xr[XVEC ? 1 : 2 * kHalf];
  auto load_x = [&](int sl, int half) {  // (reads nothing for a slab beyond the last: its table entries are empty)
    if constexpr (!XVEC) {
      const int2* e = table + sl % 3 * kBK + half * kHalf;
#pragma unroll
      for (int i = 0; i < kHalf; ++i) {
        const int2 en = e[i];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          float v = 0.f;
          if ((mask[u] >> en.y) & 1u) v = xb[u][en.x];
          xr[2 * i + u] = v;
        }
      }
    }
  };
  auto store_x = [&](int sl, int half) {
    if constexpr (!XVEC) {
      float* xs = xs_base + sl % kXRing * XS + half * kHalf * TP + t;
#pragma unroll
      for (int i = 0; i < kHalf; ++i) {
        xs[i * TP] = xr[2 * i];
        xs[i * TP + G] = xr[2 * i + 1];
      }
    }
  };
  auto copy_x = [&](int sl) {  // XVEC: asynchronous
    if constexpr (XVEC) {
      if (sl < slabs) {
        float* xs = xs_base + sl % kXRing * XS + t % VG * 4;
#pragma unroll
        for (int i = 0; i < kBK; i += VROWS) {
          const int kk = i + t / VG, k = kbase + sl * kBK + kk;
          const bool ok = v_ok && k < a.k;
          cp_async16(xs + kk * TP, ok ? vb + size_t(k) * a.pq : a.x, ok ? 16 : 0);
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
  };
  float4 wv[WV];
  auto load_w = [&](int sl) {
#pragma unroll
    for (int i = 0; i < WV; ++i) {
      const int oc = oc0 + wr + i * (G / 4), k = kbase + sl * kBK + wq;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (sl < slabs && oc < a.o) {
        const float* src = a.w + size_t(oc) * a.k + k;
        if (W16) {
          if (k < a.k) v = *reinterpret_cast<const float4*>(src);
        } else {
          if (k < a.k) v.x = src[0];
          if (k + 1 < a.k) v.y = src[1];
          if (k + 2 < a.k) v.z = src[2];
          if (k + 3 < a.k) v.w = src[3];
        }
      }
      wv[i] = v;
    }
  };
  auto store_w = [&](int sl) {
#pragma unroll
    for (int i = 0; i < WV; ++i) {
      float* ws = ws_base + (sl & 1) * WS + wq * kWRow + wr + i * (G / 4);
      ws[0] = wv[i].x;
      ws[kWRow] = wv[i].y;
      ws[2 * kWRow] = wv[i].z;
      ws[3 * kWRow] = wv[i].w;
    }
  };

  uint64_t acc[8][8];  // [pixel pair][channel]
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0;

  ptx::grid_dep_wait();
  fill_table(0);
  fill_table(1);
  load_w(0);
  copy_x(0);
  copy_x(1);
  group_sync();
  store_w(0);
  load_w(1);
  if (slabs > 0) {
    load_x(0, 0);
    store_x(0, 0);
    load_x(0, 1);
    store_x(0, 1);
  }
  for (int sl = 0; sl < slabs; ++sl) {
    if (XVEC) asm volatile("cp.async.wait_group 1;" ::: "memory");  // this thread's copies of slab sl have landed
    group_sync();  // everyone's have, and everyone has finished with the slots refilled below
    fill_table(sl + 2);
    copy_x(sl + 2);
    store_w(sl + 1);
    load_w(sl + 2);
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
      load_x(sl + 1, half);
      const float* xs = xs_base + sl % kXRing * XS + half * kHalf * TP + tx * 4;
      const float* ws = ws_base + (sl & 1) * WS + half * kHalf * kWRow + ty * 4;
#pragma unroll
      for (int kk = 0; kk < kHalf; ++kk) {
        ulonglong2 xv[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) xv[i] = *reinterpret_cast<const ulonglong2*>(xs + kk * TP + i * (TP / 4));
#pragma unroll
        for (int jh = 0; jh < 2; ++jh) {
          const float4 wf = *reinterpret_cast<const float4*>(ws + kk * kWRow + jh * 32);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float w1 = j == 0 ? wf.x : (j == 1 ? wf.y : (j == 2 ? wf.z : wf.w));
            const uint64_t w2 = pack2(w1, w1);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              fma2(acc[2 * i][jh * 4 + j], xv[i].x, w2);
              fma2(acc[2 * i + 1][jh * 4 + j], xv[i].y, w2);
            }
          }
        }
      }
      store_x(sl + 1, half);
    }
  }
  if (XVEC) asm volatile("cp.async.wait_group 0;" ::: "memory");
  ptx::grid_dep_launch();  // late: see conv_fp32.cu

  // Vector v = 4 j + i of a thread: four pixels (group i) of channel j.  Partial tiles are laid out as [vector][thread] in every CTA;
  // of the slices * KG partial sums of a tile, member m (slice and group) adds those of the vectors v % (slices * KG) == m.
  const int members = a.slices * KG, member = slice * KG + grp;
  float4* part = reinterpret_cast<float4*>(tiles);
  if (members > 1) {
    __syncthreads();  // all slabs consumed: the tiles may be overwritten
#pragma unroll
    for (int v = 0; v < 32; ++v) {
      const float2 lo = unpack2(acc[2 * (v & 3)][v >> 2]), hi = unpack2(acc[2 * (v & 3) + 1][v >> 2]);
      part[v * kThreads + threadIdx.x] = make_float4(lo.x, lo.y, hi.x, hi.y);
    }
    if (a.slices > 1) ptx::cluster_sync_all();
    else __syncthreads();
  }
  int pixq[4], bq[4], remq[4];
  bool quad_ok[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    pixq[i] = pix0 + i * (TP / 4) + tx * 4;
    bq[i] = pixq[i] < a.pixels ? a.fd_pq.div(pixq[i]) : 0;
    remq[i] = pixq[i] - bq[i] * a.pq;
    quad_ok[i] = pixq[i] + 3 < a.pixels && remq[i] + 3 < a.pq;
  }
  auto finish = [&](int i, int oc, float4 v) {
    const float bv = a.bias ? __ldg(a.bias + oc) : 0.f;
    float f[4] = {v.x + bv, v.y + bv, v.z + bv, v.w + bv};
    if (a.relu) {
#pragma unroll
      for (int e = 0; e < 4; ++e) f[e] = fmaxf(f[e], 0.f);
    }
    float* dst = a.y + (size_t(bq[i]) * a.o + oc) * a.pq + remq[i];
    if (quad_ok[i] && (reinterpret_cast<uintptr_t>(dst) & 15u) == 0) {
      *reinterpret_cast<float4*>(dst) = make_float4(f[0], f[1], f[2], f[3]);
      return;
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int pix = pixq[i] + e;
      if (pix >= a.pixels) continue;
      const int b = a.fd_pq.div(pix);
      a.y[(size_t(b) * a.o + oc) * a.pq + (pix - b * a.pq)] = f[e];
    }
  };
  if (members == 1) {
#pragma unroll
    for (int v = 0; v < 32; ++v) {
      const int j = v >> 2, oc = oc0 + ty * 4 + (j >> 2) * 32 + (j & 3);
      const float2 lo = unpack2(acc[2 * (v & 3)][j]), hi = unpack2(acc[2 * (v & 3) + 1][j]);
      if (oc < a.o) finish(v & 3, oc, make_float4(lo.x, lo.y, hi.x, hi.y));
    }
    return;
  }
  const uint32_t base = ptx::smem_u32(part) + uint32_t(t) * 16u;
  // (pixel groups are compile-time indexes: the vectors of one in turn)
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    for (int j = 0; j < 8; ++j) {
      const int v = j * 4 + i;
      if (v % members != member) continue;
      float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int s0 = 0; s0 < a.slices; s0 += 2) {
        float4 q[2 * KG];
#pragma unroll
        for (int m = 0; m < 2 * KG; ++m) {
          const int s = s0 + m / KG;
          if (s < a.slices) {
            const uint32_t at = base + uint32_t(v * kThreads + (m % KG) * G) * 16u;
            q[m] = ptx::ld_cluster_v4(a.slices > 1 ? ptx::map_to_cta(at, uint32_t(s)) : at);
          }
        }
#pragma unroll
        for (int m = 0; m < 2 * KG; ++m) {
          if (s0 + m / KG >= a.slices) break;
          if (s0 == 0 && m == 0) sum = q[0];
          else { sum.x += q[m].x; sum.y += q[m].y; sum.z += q[m].z; sum.w += q[m].w; }
        }
      }
      const int oc = oc0 + ty * 4 + (j >> 2) * 32 + (j & 3);
      if (oc < a.o) finish(i, oc, sum);
    }
  }
  if (a.slices > 1) ptx::cluster_sync_all();  // nobody leaves while a peer still reads its tile
}

}  // namespace

size_t conv_fp32_wide_smem_bytes(int tile_p) {
  const size_t group = size_t(kXRing) * kBK * tile_p + 2 * kBK * kWRow + 2 * 3 * kBK;
  const size_t loop = group * (256 / tile_p) * sizeof(float), exchange = size_t(32) * kThreads * 16;
  return loop > exchange ? loop : exchange;
}

namespace {

// 16-byte copies along the pixels, and of rows of w, for tensors on 16-byte boundaries.
bool copies_x(const Fp32Shape& g) {
  return g.r == 1 && g.s == 1 && g.stride_h == 1 && g.stride_w == 1 && g.pad_h == 0 && g.pad_w == 0 && g.out_h * g.out_w % 4 == 0;
}
bool copies_w(const Fp32Shape& g) { return g.c * g.r * g.s % 4 == 0; }

// (which instance a call takes depends on its pointers: all that the layer can take)
template <int TP>
cudaError_t prepare(const Fp32Shape& g) {
  cudaError_t e = cudaSuccess;
  auto set = [&](bool reached, auto kernel) {
    if (reached && e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(conv_fp32_wide_smem_bytes(TP)));
  };
  set(copies_x(g) && copies_w(g), conv_fp32_wide_kernel<TP, true, true>);
  set(copies_x(g), conv_fp32_wide_kernel<TP, true, false>);
  set(copies_w(g), conv_fp32_wide_kernel<TP, false, true>);
  set(true, conv_fp32_wide_kernel<TP, false, false>);
  return e;
}

template <int TP, bool XVEC, bool W16>
cudaError_t go(const Fp32WideArgs& a, dim3 grid, cudaStream_t st) {
  return launch_pdl_cluster(conv_fp32_wide_kernel<TP, XVEC, W16>, grid, dim3(kThreads), conv_fp32_wide_smem_bytes(TP), st, unsigned(a.slices), a);
}

}  // namespace

cudaError_t conv_fp32_wide_prepare(const Fp32Choice& ch, const Fp32Shape& g) { return ch.tile_p == 128 ? prepare<128>(g) : prepare<64>(g); }

cudaError_t conv_fp32_wide_launch(const Fp32Choice& ch, const Fp32Shape& g, const void* x, const void* w, const void* bias, void* y, int relu,
                                  cudaStream_t stream) {
  Fp32WideArgs a;
  a.x = static_cast<const float*>(x);
  a.w = static_cast<const float*>(w);
  a.bias = static_cast<const float*>(bias);
  a.y = static_cast<float*>(y);
  a.c = g.c; a.h = g.h; a.wd = g.w; a.o = g.o; a.s = g.s; a.taps = g.r * g.s;
  a.stride_h = g.stride_h; a.stride_w = g.stride_w; a.pad_h = g.pad_h; a.pad_w = g.pad_w;
  a.out_w = g.out_w; a.pq = g.out_h * g.out_w; a.relu = relu;
  a.pixels = g.batch * g.out_h * g.out_w;
  a.k = g.c * g.r * g.s;
  a.slices = ch.slices;
  const int slabs = fp32_slabs(a.k), members = ch.slices * (256 / ch.tile_p);
  a.slabs_per_group = (slabs + members - 1) / members;
  a.fd_rs = FastDiv::make(a.taps);
  a.fd_s = FastDiv::make(g.s);
  a.fd_pq = FastDiv::make(a.pq);
  a.fd_out_w = FastDiv::make(g.out_w);
  a.fd_slices = FastDiv::make(a.slices);
  const bool xvec = copies_x(g) && (reinterpret_cast<uintptr_t>(x) & 15u) == 0;
  const bool w16 = copies_w(g) && (reinterpret_cast<uintptr_t>(w) & 15u) == 0;
  const dim3 grid(unsigned((int64_t(a.pixels) + ch.tile_p - 1) / ch.tile_p * ch.slices), unsigned((g.o + kTO - 1) / kTO));
  auto pick = [&](auto tp) {
    constexpr int TP = decltype(tp)::value;
    if (xvec) return w16 ? go<TP, true, true>(a, grid, stream) : go<TP, true, false>(a, grid, stream);
    return w16 ? go<TP, false, true>(a, grid, stream) : go<TP, false, false>(a, grid, stream);
  };
  if (ch.tile_p == 128) return pick(std::integral_constant<int, 128>{});
  return pick(std::integral_constant<int, 64>{});
}

}  // namespace gieb
