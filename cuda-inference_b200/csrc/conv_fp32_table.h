// When the strict-FP32 kernel may decode its reduction indices through a table (conv_fp32.cu).  Host code only: the rule is
// compiled by itself in the CPU tests.
#ifndef GIEB_CONV_FP32_TABLE_H_
#define GIEB_CONV_FP32_TABLE_H_

#include <cstdint>

namespace gieb {

constexpr int kLutMax = 4096;    // reduction length of a CTA up to which the (c, r, s) decode of k is tabulated in shared memory
constexpr int kNoRow = 0x7fff;   // filter row of a table entry beyond the reduction: no image has the row it leads to

// `terms`: table entries of a CTA.  An entry is the offset of (c, r, s) inside one image and (r << 16) | s, so offsets have 31
// bits, r 15 and s 16.  The kernel reads input row oh * stride - pad_h + r when that lies in [0, h): for r = kNoRow and the
// topmost output row it is kNoRow - pad_h, which lies below the image as long as h + pad_h <= kNoRow.
inline bool conv_fp32_table_fits(int64_t terms, int c, int h, int w, int r, int s, int pad_h) {
  return terms <= kLutMax && int64_t(c) * h * w < (int64_t(1) << 31) && r < kNoRow && s <= 0xffff && int64_t(h) + pad_h <= kNoRow;
}

}  // namespace gieb

#endif  // GIEB_CONV_FP32_TABLE_H_
