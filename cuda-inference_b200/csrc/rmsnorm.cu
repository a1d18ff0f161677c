// Fused RMSNorm and residual-add + RMSNorm.  Stands in for rmsnorm_kernel (src/transformer/rmsnorm.cu:39-98):
//   s = x                       (plain)      or   s = round_T(x + residual_in), residual_out = s   (fused)
//   y = round_T( s * rsqrt(mean(s^2) + eps) * gamma )
// FP32 arithmetic, one rounding per stored value; the residual stream is rounded to T BEFORE the square sum, as in
// the reference (rmsnorm.cu:57-66).
//
// Vector path (tensor pointers 16-byte aligned, rows of up to 8 vectors x 1024 threads): 128-bit loads issued up front, the
// row stays in registers (in storage form: rounded values need no more) across the reduction, so every byte crosses HBM
// exactly once (x, residual in; residual, y out).  Rows of at most 64 vectors are one warp's work, eight rows to a CTA, with
// no barrier at all; longer rows are one CTA's.  A hidden size that is no multiple of the vector shifts every row by
// another amount, but all the tensors of a row by the same one: its vectors start `lead` elements before the row and the
// first and the last are taken element by element (RAGGED).  Anything else (tensors on differing alignments, longer rows)
// takes the element-wise path.
// Launched with programmatic stream serialization: a launch follows the one before it without the drain-and-refill gap, and
// costs the host 0.45 us less.  Calls in a stream, residual form, before and after: 8192 x 4096 BF16 43.4 -> 41.7 us (6.4
// TB/s), 4741 x 12224 BF16 110 -> 72 us (the row held as floats spilled), 4000 x 3185 BF16 64 -> 25 us (element-wise before),
// 4775 x 128 FP32 6.1 -> 3.2 us, 16 x 4096 BF16 4.8 -> 3.1 us (bound by the launch: most of it the host's, see
// python_calls.cpp).
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include <type_traits>

#include "internal.h"
#include "ptx.cuh"

namespace gieb {
namespace {

// Storage type <-> FP32 (one rounding on the way back).
template <typename T> struct Num;
template <> struct Num<float> {
  static __device__ __forceinline__ float up(float v) { return v; }
  static __device__ __forceinline__ float down(float v) { return v; }
};
template <> struct Num<__half> {
  static __device__ __forceinline__ float up(__half v) { return __half2float(v); }
  static __device__ __forceinline__ __half down(float v) { return __float2half_rn(v); }
};
template <> struct Num<__nv_bfloat16> {
  static __device__ __forceinline__ float up(__nv_bfloat16 v) { return __bfloat162float(v); }
  static __device__ __forceinline__ __nv_bfloat16 down(float v) { return __float2bfloat16_rn(v); }
};

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// Sum over the CTA, the same bits in every thread: each warp reduces its own values, warp leaders publish one partial
// each, and after ONE barrier every warp reduces the (at most 32) partials itself.
__device__ __forceinline__ float cta_sum(float v, float* partial) {
  v = warp_sum(v);
  const int warps = (blockDim.x + 31) >> 5, lane = threadIdx.x & 31;
  if (warps == 1) return v;
  if (lane == 0) partial[threadIdx.x >> 5] = v;
  __syncthreads();
  return warp_sum(lane < warps ? partial[lane] : 0.f);
}

template <typename T> struct Vec { static constexpr int N = 16 / sizeof(T); };

// gamma vector i (VEC elements) as floats, from either T or float storage.
template <typename T, bool GAMMA_F32>
__device__ __forceinline__ void load_gamma(const void* gamma, int i, float (&g)[Vec<T>::N]) {
  constexpr int VEC = Vec<T>::N;
  if (GAMMA_F32) {
    const float4* gp = reinterpret_cast<const float4*>(gamma) + size_t(i) * (VEC / 4);
#pragma unroll
    for (int q = 0; q < VEC / 4; ++q) {
      const float4 f = __ldg(gp + q);
      g[q * 4 + 0] = f.x; g[q * 4 + 1] = f.y; g[q * 4 + 2] = f.z; g[q * 4 + 3] = f.w;
    }
  } else {
    const uint4 raw = __ldg(reinterpret_cast<const uint4*>(gamma) + i);
    T tv[VEC];
    memcpy(tv, &raw, 16);
#pragma unroll
    for (int j = 0; j < VEC; ++j) g[j] = Num<T>::up(tv[j]);
  }
}

// NV vectors per thread; WARP: a row per warp (blockDim.x / 32 rows per CTA), else a row per CTA.
template <typename T, bool FUSED, bool GAMMA_F32, int NV, bool WARP, bool RAGGED>
__global__ void __launch_bounds__(WARP ? 256 : (NV <= 2 ? 512 : 1024))
rmsnorm_row_kernel(const T* x, const void* __restrict__ gamma, T* __restrict__ y, const T* res_in,
                   T* res_out, int rows, int hidden, float eps) {
  constexpr int VEC = Vec<T>::N;
  __shared__ float red[32];
  ptx::grid_dep_launch();
  const int row = WARP ? int(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) : int(blockIdx.x);
  const int t = WARP ? int(threadIdx.x & 31) : int(threadIdx.x), step = WARP ? 32 : int(blockDim.x);
  ptx::grid_dep_wait();
  if (WARP && row >= rows) return;
  const size_t base = size_t(row) * hidden;
  const int lead = RAGGED ? int(base % VEC) : 0;  // elements of the first vector that belong to the row before
  const int nvec = (lead + hidden + VEC - 1) / VEC;
  const T* xr = x + base - lead;
  const T* rr = FUSED ? res_in + base - lead : nullptr;
  // whether vector i, or element j of it, belongs to this row
  auto whole = [&](int i) { return !RAGGED || ((i > 0 || lead == 0) && (i + 1) * VEC <= lead + hidden); };
  auto mine = [&](int i, int j) { const int e = i * VEC + j - lead; return e >= 0 && e < hidden; };
  auto load = [&](const T* p, int i) {
    if (whole(i)) return reinterpret_cast<const uint4*>(p)[i];  // plain loads: res_out may alias x
    T v[VEC];
#pragma unroll
    for (int j = 0; j < VEC; ++j) v[j] = mine(i, j) ? p[i * VEC + j] : Num<T>::down(0.f);
    uint4 o;
    memcpy(&o, v, 16);
    return o;
  };
  auto store = [&](T* p, int i, const T (&v)[VEC]) {
    if (whole(i)) {
      uint4 o;
      memcpy(&o, v, 16);
      reinterpret_cast<uint4*>(p)[i] = o;
    } else {
#pragma unroll
      for (int j = 0; j < VEC; ++j)
        if (mine(i, j)) p[i * VEC + j] = v[j];
    }
  };

  uint4 s[NV];  // the stream that is normalised, in storage form
  float ss = 0.f;
  constexpr int BATCH = NV < 4 ? NV : 4;  // vectors whose loads are in flight together
#pragma unroll
  for (int k0 = 0; k0 < NV; k0 += BATCH) {
    uint4 rv[BATCH];
#pragma unroll
    for (int k = 0; k < BATCH; ++k) {
      const int i = t + (k0 + k) * step;
      s[k0 + k] = rv[k] = make_uint4(0u, 0u, 0u, 0u);
      if (i < nvec) {
        s[k0 + k] = load(xr, i);
        if (FUSED) rv[k] = load(rr, i);
      }
    }
#pragma unroll
    for (int k = 0; k < BATCH; ++k) {
      const int i = t + (k0 + k) * step;
      if (i >= nvec) continue;
      T a[VEC];
      memcpy(a, &s[k0 + k], 16);
      if (FUSED) {
        T b[VEC];
        memcpy(b, &rv[k], 16);
#pragma unroll
        for (int j = 0; j < VEC; ++j) a[j] = Num<T>::down(Num<T>::up(a[j]) + Num<T>::up(b[j]));
        memcpy(&s[k0 + k], a, 16);
        store(res_out + base - lead, i, a);
      }
#pragma unroll
      for (int j = 0; j < VEC; ++j) ss = fmaf(Num<T>::up(a[j]), Num<T>::up(a[j]), ss);
    }
  }
  ss = WARP ? warp_sum(ss) : cta_sum(ss, red);
  const float inv = rsqrtf(ss / float(hidden) + eps);
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const int i = t + k * step;
    if (i >= nvec) continue;
    float g[VEC];
    if constexpr (RAGGED) {  // gamma is not shifted with the rows: element by element
      auto at = [&](int e) { return GAMMA_F32 ? __ldg(static_cast<const float*>(gamma) + e) : Num<T>::up(static_cast<const T*>(gamma)[e]); };
      if (whole(i)) {
#pragma unroll
        for (int j = 0; j < VEC; ++j) g[j] = at(i * VEC - lead + j);
      } else {
#pragma unroll
        for (int j = 0; j < VEC; ++j) g[j] = mine(i, j) ? at(i * VEC - lead + j) : 0.f;
      }
    } else {
      load_gamma<T, GAMMA_F32>(gamma, i, g);
    }
    T a[VEC], o[VEC];
    memcpy(a, &s[k], 16);
#pragma unroll
    for (int j = 0; j < VEC; ++j) o[j] = Num<T>::down(Num<T>::up(a[j]) * inv * g[j]);
    store(y + base - lead, i, o);
  }
}

// Element-wise path for tensors on differing alignments and very long rows.  The normalised stream (x, or the rounded
// x + residual) is kept as FP32 in shared memory between the square sum and the scaling when the row fits (`staged` floats
// of dynamic shared memory, 0 = it does not): global memory is then read once here as well; longer rows are read again.
template <typename T, bool FUSED, bool GAMMA_F32>
__global__ void __launch_bounds__(1024)
rmsnorm_generic_kernel(const T* x, const void* __restrict__ gamma, T* __restrict__ y, const T* res_in,
                       T* res_out, int hidden, float eps, int staged) {
  extern __shared__ float row_f32[];
  __shared__ float red[32];
  ptx::grid_dep_launch();
  ptx::grid_dep_wait();
  const size_t base = size_t(blockIdx.x) * hidden;
  auto stream_value = [&](int i) {   // element i of the stream that is normalised (stores the residual stream when fused)
    float f = Num<T>::up(x[base + i]);
    if (FUSED) {
      const T sv = Num<T>::down(f + Num<T>::up(res_in[base + i]));
      res_out[base + i] = sv;
      f = Num<T>::up(sv);
    }
    return f;
  };
  float ss = 0.f;
  for (int i = threadIdx.x; i < hidden; i += blockDim.x) {
    const float f = stream_value(i);
    if (i < staged) row_f32[i] = f;
    ss = fmaf(f, f, ss);
  }
  ss = cta_sum(ss, red);
  const float inv = rsqrtf(ss / float(hidden) + eps);
  for (int i = threadIdx.x; i < hidden; i += blockDim.x) {
    // beyond the staged part a thread reads back what it stored itself (res_out) or the input again
    const float f = i < staged ? row_f32[i] : Num<T>::up(FUSED ? res_out[base + i] : x[base + i]);
    const float g = GAMMA_F32 ? static_cast<const float*>(gamma)[i] : Num<T>::up(static_cast<const T*>(gamma)[i]);
    y[base + i] = Num<T>::down(f * inv * g);
  }
}

bool aligned16(const void* p) { return p == nullptr || (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

template <typename T, bool FUSED, bool GAMMA_F32>
cudaError_t run(int rows, int hidden, float eps, const void* x, const void* gamma, void* y, const void* rin, void* rout,
                cudaStream_t st) {
  constexpr int VEC = Vec<T>::N;
  const T* xp = static_cast<const T*>(x);
  T* yp = static_cast<T*>(y);
  const T* ri = static_cast<const T*>(rin);
  T* ro = static_cast<T*>(rout);
  // (gamma is read element by element when rows are shifted, so only unshifted rows need it aligned)
  const bool ragged = hidden % VEC != 0;
  const int nvec = (hidden + VEC - 1) / VEC + (ragged ? 1 : 0);
  const bool vectors = nvec <= 8 * 1024 && aligned16(x) && (ragged || aligned16(gamma)) && aligned16(y) && aligned16(rin) && aligned16(rout);
  if (vectors) {
    auto go = [&](auto nv, auto warp) {
      constexpr int NV = decltype(nv)::value;
      constexpr bool WARP = decltype(warp)::value;
      unsigned grid = unsigned(rows), threads = unsigned(((nvec + NV - 1) / NV + 31) & ~31);
      if (WARP) {  // eight rows to a CTA, fewer while that leaves SMs without one
        unsigned per = 8;
        while (per > 1 && unsigned(rows) < per * kNumSms) per >>= 1;
        grid = (unsigned(rows) + per - 1) / per;
        threads = per * 32;
      }
      return ragged ? launch_pdl(rmsnorm_row_kernel<T, FUSED, GAMMA_F32, NV, WARP, true>, dim3(grid), dim3(threads), 0, st, xp, gamma, yp, ri, ro, rows, hidden, eps)
                    : launch_pdl(rmsnorm_row_kernel<T, FUSED, GAMMA_F32, NV, WARP, false>, dim3(grid), dim3(threads), 0, st, xp, gamma, yp, ri, ro, rows, hidden, eps);
    };
    using std::integral_constant;
    if (nvec <= 32) return go(integral_constant<int, 1>{}, std::true_type{});
    if (nvec <= 64) return go(integral_constant<int, 2>{}, std::true_type{});
    // Enough rows for every SM: CTAs of up to 288 threads with two vectors each keep the most loads in flight (more
    // threads with four for long rows).  Few rows: latency decides, so a row is spread over up to 512 threads first.
    const bool few = rows < 2 * kNumSms;
    if (nvec <= (few ? 512 : 288)) return go(integral_constant<int, 1>{}, std::false_type{});
    if (nvec <= (few ? 1024 : 576)) return go(integral_constant<int, 2>{}, std::false_type{});
    if (nvec <= 4096) return go(integral_constant<int, 4>{}, std::false_type{});
    return go(integral_constant<int, 8>{}, std::false_type{});
  }
  int threads = 32;
  while (threads < hidden && threads < 1024) threads <<= 1;
  constexpr int kStagedMax = (48 * 1024 - 32 * int(sizeof(float))) / int(sizeof(float));  // 48 KiB need no opt-in, the kernel's own `red` included
  const int staged = hidden <= kStagedMax ? hidden : 0;
  return launch_pdl(rmsnorm_generic_kernel<T, FUSED, GAMMA_F32>, dim3(unsigned(rows)), dim3(unsigned(threads)), size_t(staged) * sizeof(float), st, xp,
                    gamma, yp, ri, ro, hidden, eps, staged);
}

template <typename T>
cudaError_t run_t(int rows, int hidden, float eps, int gamma_fp32, const void* x, const void* gamma, void* y, const void* rin,
                  void* rout, cudaStream_t st) {
  const bool fused = rin != nullptr && rout != nullptr;
  if (fused) return gamma_fp32 ? run<T, true, true>(rows, hidden, eps, x, gamma, y, rin, rout, st)
                               : run<T, true, false>(rows, hidden, eps, x, gamma, y, rin, rout, st);
  return gamma_fp32 ? run<T, false, true>(rows, hidden, eps, x, gamma, y, rin, rout, st)
                    : run<T, false, false>(rows, hidden, eps, x, gamma, y, rin, rout, st);
}

}  // namespace

cudaError_t rmsnorm_launch(int rows, int hidden, float eps, int dtype, int gamma_fp32, const void* x, const void* gamma,
                           void* y, const void* res_in, void* res_out, cudaStream_t stream) {
  switch (dtype) {
    case 0: return run_t<float>(rows, hidden, eps, 1, x, gamma, y, res_in, res_out, stream);
    case 1: return run_t<__half>(rows, hidden, eps, gamma_fp32, x, gamma, y, res_in, res_out, stream);
    case 2: return run_t<__nv_bfloat16>(rows, hidden, eps, gamma_fp32, x, gamma, y, res_in, res_out, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace gieb
