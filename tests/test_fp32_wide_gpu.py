"""The strict-FP32 kernel of 16 x 8 thread tiles at the sizes where it can go wrong: every tile width, reductions split over groups and
clusters with a short last slice, 16-byte pixel copies of 1x1 layers and gathered ones, reduction lengths that are no multiple of four
or of a slab, channel and pixel tails, strides, 25 taps, and pointers off their alignment."""
import numpy as np
import pytest

import gpu_util as gu

pytestmark = pytest.mark.gpu

CASES = [
    # shape, output pixels of a tile (64: the long reductions over few pixels), offset of the pointers in elements
    ((3, 97, 40, 25, 70, 5, 5, 1, 1, 2, 2), 128, 0),        # 25 taps, 2425 terms: weights read one by one; clusters; a channel tail
    ((10, 108, 30, 30, 70, 3, 3, 1, 1, 1, 1), 128, 1),       # pointers off by one element
    ((10, 97, 31, 29, 70, 3, 3, 1, 1, 1, 1), 128, 0),       # odd planes, tiles over two images
    ((3, 97, 100, 80, 130, 3, 3, 2, 2, 1, 1), 128, 0),      # stride
    ((5, 762, 60, 30, 70, 1, 1, 1, 1, 0, 0), 128, 0),       # 1x1, planes of 1800 pixels: 16-byte copies; 762 terms
    ((5, 762, 60, 30, 70, 1, 1, 1, 1, 0, 0), 128, 1),       # the same off its alignment: gathered
    ((2, 762, 18, 18, 256, 3, 3, 2, 2, 1, 1), 64, 0),       # 429 slabs over few pixels
    ((1, 1030, 12, 12, 40, 3, 3, 1, 1, 1, 1), 64, 1),
    ((1, 4090, 16, 16, 70, 1, 1, 1, 1, 0, 0), 64, 0),       # 1x1 in four groups: 16-byte copies, 4090 terms, a channel tail
    ((1, 4094, 12, 17, 40, 1, 1, 1, 1, 0, 0), 64, 1),       # the same off its alignment, a last tile of 12 pixels
]
SHARED_MEMORY = {128: 67328, 64: 85504}  # of this kernel's CTAs (the other kernel has tiles of 64 pixels too)


@pytest.mark.parametrize("case", range(len(CASES)))
def test_fp32_wide_tiles(pkg, orc, oracle, case):
    args, tile, off = CASES[case]
    p = orc.Problem.P(*args, precision=orc.FP32, bias=(case % 2 == 0), relu=(case % 3 == 0))
    x, w, b = oracle.make_conv_data(p, 600 + case, case % 4)
    ref, scale = oracle.conv2d(p, x, w, b if p.has_bias else None)
    got, plan, out = gu.run_conv(pkg, oracle, p, x, w, b if p.has_bias else None, offsets=(off, off, off))
    assert plan.info.cfg.tile_m == tile and plan.info.dynamic_smem_bytes == SHARED_MEMORY[tile]
    m = oracle.compare(p, got, ref, scale)   # the reference's FP32 policy: the rounding of FP32 sums of this length
    assert m.passed(), f"fp32 case {case}: {m.summary()}"
    again, _, out2 = gu.run_conv(pkg, oracle, p, x, w, b if p.has_bias else None, plan=plan, offsets=(off, off, off))
    assert np.array_equal(out.raw_bits(), out2.raw_bits())
