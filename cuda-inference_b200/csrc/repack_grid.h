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

// Whether a launch of both tensors begins with the activations although the weights' blocks take longest: few of them behind eight times
// as many of the weights are the ones that everything waits for.  64 -> 704 at 45 x 45, 5x5, 2 images, 64 and 704 blocks: 17.8 us weights
// first, 16.5 so; 458 -> 496 at 4 x 4, 5x5, 8 and 1984: 25.2 and 23.7; TF32 128 -> 496 at 4 x 4, 3x3, 15 images, 15 and 496: 11.1 and 9.8.
// Of 27 such layers 13 gain 1 to 12 % and five lose 1 to 1.7 %; with fewer weights it goes either way (TF32 96 -> 192 at 27 x 27, 5x5, 16
// images, 576 and 192: 32.5 and 34.1; 192 -> 64 at 41 x 41, 5x5, 16 images, 2592 and 128: 61.4 and 59.0).
inline bool activations_first(int64_t activation_blocks, int64_t weight_blocks) { return weight_blocks >= 8 * activation_blocks; }

}  // namespace gieb

#endif  // GIEB_REPACK_GRID_H_
