// The layout repack of repack.cu ([B][C][HW] -> [B][HW][Cp], 16-bit, bit-exact) for small tensors, where what counts is how long ONE
// block takes: a load round trip, the instructions of a warp one behind the other, a store.  repack.cu's tiles and slabs pass through
// shared memory element by element and find their way by the job's mode; here a thread turns eight channels of V pixels, or of a whole
// filter, in its registers.  512 -> 512, 3x3, 7 x 7, one image: the launch 4.57 -> 2.3 us, with its convolution 11.9 -> 9.6; 256 -> 256,
// 14 x 14, 32 images 14.6 -> 13.7; 184 -> 64, 31 x 31, 3 images, weights converted beforehand 10.1 -> 9.3; 256 -> 1024, 1x1, 14 x 14,
// 4 images 7.8 -> 6.35.  Spread over the SMs by launch_pdl_spread (without: 16.1 us instead of 13.6 for 32 x 256 x 14 x 14 and its
// convolution, although the launch by itself takes 2.9).
#include <string.h>

#include "internal.h"
#include "ptx.cuh"
#include "repack_grid.h"

namespace gieb {
namespace {

struct DirectJob {
  const uint16_t* src;
  uint16_t* dst;
  int C, HW, Cp, hw_tiles, c_tiles;
  FastDiv fd_hw_tiles, fd_c_tiles;
  unsigned blocks;
  int prefetch;  // L2 prefetch of the source lines before the dependency wait
};
struct FilterJob {
  const uint4* src;
  uint4* dst;
  int src_groups, groups, units;  // vectors of eight channels per filter before and after padding, units in all
  int per;                        // units of a block
  FastDiv fd_groups;
  unsigned blocks;
  int prefetch;
};

// A block takes 64 channels by 128, 64 or 32 pixels (V = 4, 2, 1).  A warp covers 8 channel groups x 4 runs of V pixels, so that a store
// instruction writes whole 128-byte lines; with V = 1 (odd planes, or a source off its alignment) 2 groups x 16 pixels, so that rows
// are read by 32 bytes as well.
template <int V>
__device__ __forceinline__ void direct_tile(const DirectJob& j, unsigned id) {
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int row = j.fd_hw_tiles.div(int(id)), hw_tile = int(id) - row * j.hw_tiles;
  const int bi = j.fd_c_tiles.div(row), c_tile = row - bi * j.c_tiles;
  const int group = V == 1 ? (warp & 3) * 2 + (lane & 1) : lane & 7;
  const int px = hw_tile * (32 * V) + (V == 1 ? (warp >> 2) * 16 + (lane >> 1) : (warp * 4 + (lane >> 3)) * V);
  const int c0 = c_tile * 64 + group * 8;
  const bool ok = px < j.HW && c0 < j.Cp;
  const uint16_t* s = j.src + (size_t(bi) * j.C + c0) * j.HW + px;
  uint16_t* d = j.dst + (size_t(bi) * j.HW + px) * j.Cp + c0;
  // (an L2 fill, legal before the wait: see repack_jobs_kernel; one lane for each row of a warp)
  if (j.prefetch && ok && (V == 1 ? (lane >> 1) == 0 : (lane >> 3) == 0))
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (c0 + k < j.C) ptx::prefetch_l2(s + size_t(k) * j.HW);
  ptx::grid_dep_wait();
  ptx::grid_dep_launch();
  if (!ok) return;
  uint32_t lo[8], hi[8];  // pixels 0, 1 and 2, 3 of channel k
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    lo[k] = hi[k] = 0;
    if (c0 + k < j.C) {
      const uint16_t* at = s + size_t(k) * j.HW;
      if (V == 4) {
        const uint2 q = *reinterpret_cast<const uint2*>(at);
        lo[k] = q.x;
        hi[k] = q.y;
      } else if (V == 2) lo[k] = *reinterpret_cast<const uint32_t*>(at);
      else lo[k] = *at;
    }
  }
#pragma unroll
  for (int p = 0; p < V; ++p) {
    const uint32_t(&w)[8] = p < 2 ? lo : hi;
    const uint32_t sel = p & 1 ? 0x7632 : 0x5410;
    *reinterpret_cast<uint4*>(d + size_t(p) * j.Cp) =
        make_uint4(__byte_perm(w[0], w[1], sel), __byte_perm(w[2], w[3], sel), __byte_perm(w[4], w[5], sel), __byte_perm(w[6], w[7], sel));
  }
}

// Filters of 9 taps or 1: eight channels of a filter are TAPS whole vectors, element (channel k, tap t) at TAPS * k + t, and become TAPS
// vectors of eight channels.  Nine come through shared memory, only to be read in the order in which they lie (144 bytes from thread
// to thread: no bank conflicts); where channels are padded, filters do not follow each other and each thread fetches its own.
template <int TAPS>
__device__ __forceinline__ void filter_units(uint4* slab, const FilterJob& j, unsigned id) {
  const int t = threadIdx.x, unit = int(id) * j.per + t;
  const bool mine = t < j.per && unit < j.units;
  const int o = j.fd_groups.div(unit), g = unit - o * j.groups;
  uint4* d = j.dst + size_t(o) * TAPS * j.groups + g;
  uint4 v[TAPS];
  if (TAPS > 1 && j.src_groups == j.groups) {
    const uint4* s = j.src + size_t(id) * j.per * TAPS;
    const int n = min(j.per, j.units - int(id) * j.per) * TAPS;
    if (j.prefetch)
      for (int i = t * 8; i < n; i += 256 * 8) ptx::prefetch_l2(s + i);
    ptx::grid_dep_wait();
    ptx::grid_dep_launch();
#pragma unroll
    for (int k = 0; k < TAPS; ++k)
      if (t + k * 256 < n) v[k] = s[t + k * 256];
#pragma unroll
    for (int k = 0; k < TAPS; ++k)
      if (t + k * 256 < n) slab[t + k * 256] = v[k];
    __syncthreads();
    if (mine)
#pragma unroll
      for (int k = 0; k < TAPS; ++k) v[k] = slab[t * TAPS + k];
  } else {
    ptx::grid_dep_wait();
    ptx::grid_dep_launch();
#pragma unroll
    for (int k = 0; k < TAPS; ++k)
      v[k] = mine && g < j.src_groups ? j.src[(size_t(o) * j.src_groups + g) * TAPS + k] : make_uint4(0, 0, 0, 0);
  }
  if (!mine) return;
  uint32_t w[4 * TAPS];  // element (channel k, tap t) at TAPS * k + t
#pragma unroll
  for (int k = 0; k < TAPS; ++k) {
    w[4 * k] = v[k].x; w[4 * k + 1] = v[k].y; w[4 * k + 2] = v[k].z; w[4 * k + 3] = v[k].w;
  }
  auto pair = [&](int a, int b) { return __byte_perm(w[a >> 1], w[b >> 1], (a & 1 ? 0x32 : 0x10) | ((b & 1 ? 0x76 : 0x54) << 8)); };
#pragma unroll
  for (int tap = 0; tap < TAPS; ++tap)
    d[size_t(tap) * j.groups] = make_uint4(pair(tap, TAPS + tap), pair(2 * TAPS + tap, 3 * TAPS + tap), pair(4 * TAPS + tap, 5 * TAPS + tap),
                                           pair(6 * TAPS + tap, 7 * TAPS + tap));
}

template <int V, int TAPS>
__global__ void __launch_bounds__(256) repack_direct_kernel(const __grid_constant__ DirectJob a, const __grid_constant__ FilterJob b) {
  extern __shared__ uint4 slab[];
  if (TAPS && (V == 0 || blockIdx.x < b.blocks)) filter_units<TAPS ? TAPS : 1>(slab, b, blockIdx.x);  // (first: their way is the longest)
  else direct_tile<V ? V : 1>(a, blockIdx.x - b.blocks);
}

template <int V, int TAPS>
cudaError_t direct_launch(const DirectJob& a, const FilterJob& b, cudaStream_t stream) {
  return launch_pdl_spread(repack_direct_kernel<V, TAPS>, a.blocks + b.blocks, 0, TAPS > 1 ? size_t(b.per) * TAPS * sizeof(uint4) : 0, stream, a, b);
}

}  // namespace

bool repack_direct_launch(const void* src_a, void* dst_a, int batch_a, int ch_a, int hw_a, int cp_a, const void* src_b, void* dst_b, int batch_b,
                          int ch_b, int hw_b, int cp_b, cudaStream_t stream, cudaError_t* status) {
  DirectJob a;
  memset(&a, 0, sizeof(a));
  FilterJob b;
  memset(&b, 0, sizeof(b));
  a.prefetch = b.prefetch = prefetch_enabled() ? 1 : 0;
  int v = direct_pixels(hw_a, reinterpret_cast<uintptr_t>(src_a));
  if (src_a != nullptr) {
    a.src = static_cast<const uint16_t*>(src_a);
    a.dst = static_cast<uint16_t*>(dst_a);
    a.C = ch_a; a.HW = hw_a; a.Cp = cp_a;
    a.hw_tiles = tiles_of(hw_a, 32 * v);
    a.c_tiles = tiles_of(cp_a, 64);
    const int64_t n = direct_blocks(v, hw_a, cp_a, batch_a);
    // Above these sizes repack.cu's wider rows count for more than its way is long (with the convolution, here and there): V 4 with
    // rows of whole vectors, 100 blocks 7.17 and 7.24 us, 192 13.8 and 13.6, 896 21.1 and 19.2; other rows of V 4, 256 blocks 13.6 and
    // 14.0, 512 21.3 and 21.0; V 2, 384 13.3 and 13.6, 960 15.6 and 14.4; V 1, 768 13.9 and 14.2, 1984 15.5 and 15.7, 3120 27.2 and
    // 26.9, beside filters of nine taps 768 14.2 and 14.6, 2048 23.9 and 23.4.  140 layers of 40 to 2800 blocks: below these sizes 0.93 of
    // the time (0.79 to 1.02), above them, to twice the size, 1.01 (0.92 to 1.11; V 1 with one tap, 0.965 up to 2800 blocks, and other rows
    // of V 4, 0.99 up to 520, would bear a little more).
    if (n > (v == 4 ? (hw_a % 8 == 0 ? kNumSms : 2 * kNumSms) : (v == 2 ? 3 * kNumSms : (src_b != nullptr && hw_b == 9 ? 1024 : 2048)))) return false;
    a.fd_hw_tiles = FastDiv::make(a.hw_tiles);
    a.fd_c_tiles = FastDiv::make(a.c_tiles);
    a.blocks = unsigned(n);
  }
  if (src_b != nullptr) {
    if ((hw_b != 1 && hw_b != 9) || ch_b % 8 != 0 || reinterpret_cast<uintptr_t>(src_b) % 16 != 0) return false;
    const int64_t units = int64_t(batch_b) * (cp_b / 8);
    if (units > (1 << 30)) return false;
    b.src = static_cast<const uint4*>(src_b);
    b.dst = static_cast<uint4*>(dst_b);
    b.src_groups = ch_b / 8;
    b.groups = cp_b / 8;
    b.units = int(units);
    b.fd_groups = FastDiv::make(b.groups);
    // Few filters of nine taps in blocks of 64 units, whose loads all threads share: as one block or a few of 256 they take one or a few
    // SMs for 36 KB each (64 -> 64 at 56 x 56 7.14 and 6.92 us, 256 -> 16 at 10 x 10, 4 images 7.98 and 7.48, 160 -> 17 at 17 x 17, 6
    // images 7.99 and 7.20, 128 -> 256 at 28 x 28 8.14 and 7.90).  From 8192 units on 256 are as fast or faster (256 -> 256 at 14 x 14,
    // 32 images 14.55 and 14.82, 1024 -> 512 at 7 x 7 18.1 and 18.5; 320 -> 320 at 15 x 15, 12800 units, 9.61 and 9.30).  One tap: 512 ->
    // 2048 at 7 x 7 7.95 and 9.59.
    b.per = hw_b == 9 && units <= 4096 ? 64 : 256;
    b.blocks = unsigned((units + b.per - 1) / b.per);
  }
  const int taps = src_b == nullptr ? 0 : hw_b;
  if (src_a == nullptr) v = 0;
#define GO(V) *status = taps == 9 ? direct_launch<V, 9>(a, b, stream) : (taps == 1 ? direct_launch<V, 1>(a, b, stream) : direct_launch<V, 0>(a, b, stream))
  if (v == 4) GO(4);
  else if (v == 2) GO(2);
  else if (v == 1) GO(1);
  else GO(0);
  return true;
}

}  // namespace gieb
