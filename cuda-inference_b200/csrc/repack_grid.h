// Sizes of the repack kernels' grids (repack.cu, repack_direct.cu).  Host code only: compiled by itself in the CPU tests.
#ifndef GIEB_REPACK_GRID_H_
#define GIEB_REPACK_GRID_H_

#include <cstdint>

namespace gieb {

// Tiles that n elements take; n may be any positive 32-bit value (planes of nearly 2^31 pixels: the sum is a 64-bit one).
inline int tiles_of(int n, int tile) { return int((int64_t(n) + tile - 1) / tile); }

// Pixels that a thread of the register repack takes from each of its eight channels: as many as every row of the planes allows to load
// at once.
inline int direct_pixels(int hw, uintptr_t src) { return hw % 4 == 0 && src % 8 == 0 ? 4 : (hw % 2 == 0 && src % 4 == 0 ? 2 : 1); }

// Blocks of the register repack: 64 channels by 32 such runs.
inline int64_t direct_blocks(int pixels, int hw, int c_padded, int batch) {
  return int64_t(tiles_of(hw, 32 * pixels)) * tiles_of(c_padded, 64) * batch;
}

}  // namespace gieb

#endif  // GIEB_REPACK_GRID_H_
