// When the strict-FP32 kernels may decode their reduction indices through tables (conv_fp32.cu, conv_fp32_wide.cu).  Host code only:
// the rules are compiled by themselves in the CPU tests.
#ifndef GIEB_CONV_FP32_TABLE_H_
#define GIEB_CONV_FP32_TABLE_H_

#include <cstdint>

namespace gieb {

constexpr int kLutMax = 4096;    // reduction length of a CTA up to which the (c, r, s) decode of k is tabulated in shared memory
constexpr int kNoRow = 0x7fff;   // filter row of a table entry beyond the reduction: no image has the row it leads to

constexpr int kFp32Slab = 16;
// Slabs that a reduction of k terms has, rounded up; k may be any positive 32-bit value.
#if defined(__CUDACC__)
__host__ __device__
#endif
constexpr int fp32_slabs(int k) { return (k - 1) / kFp32Slab + 1; }

// `terms`: table entries of a CTA.  An entry is the offset of (c, r, s) inside one image and (r << 16) | s, so offsets have 31
// bits, r 15 and s 16.  The kernel reads input row oh * stride - pad_h + r when that lies in [0, h): for r = kNoRow and the
// topmost output row it is kNoRow - pad_h, which lies below the image as long as h + pad_h <= kNoRow.
inline bool conv_fp32_table_fits(int64_t terms, int c, int h, int w, int r, int s, int pad_h) {
  return terms <= kLutMax && int64_t(c) * h * w < (int64_t(1) << 31) && r < kNoRow && s <= 0xffff && int64_t(h) + pad_h <= kNoRow;
}

// Whether the wide kernel (conv_fp32_wide.cu) may hold the offsets of its terms in 32 bits: an entry is the offset of (c, r, s) from
// the window's corner, which may lie in the padding, so the largest exceeds the image's own size by up to r rows and s columns.
inline bool conv_fp32_wide_offsets_fit(int c, int h, int w, int r, int s) {
  return ((int64_t(c) - 1) * h + r - 1) * w + s - 1 < (int64_t(1) << 31);
}

}  // namespace gieb

#endif  // GIEB_CONV_FP32_TABLE_H_
