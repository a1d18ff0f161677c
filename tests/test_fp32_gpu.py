"""The strict-FP32 convolution at the sizes where its tiling can go wrong: reductions split over clusters (with a short last
slice), tiles with many CTAs per SM, channel counts around the narrow tile, the 16-byte pixel copies of 1x1 layers, reduction
lengths that are no multiple of four, and the form without the decode table."""
import numpy as np
import pytest

import gpu_util as gu

pytestmark = pytest.mark.gpu

CASES = [
    ((1, 64, 56, 56, 64, 3, 3, 1, 1, 1, 1), 0),      # 49 tiles: the reduction is split over a cluster
    ((1, 70, 9, 9, 130, 3, 3, 1, 1, 1, 1), 0),       # 40 slabs, channel tail of 2
    ((8, 32, 40, 40, 96, 3, 3, 1, 1, 1, 1), 0),      # 400 tiles, no split
    ((2, 40, 9, 11, 33, 3, 3, 2, 2, 1, 1), 1),       # stride, odd extents, pointers off by one element
    ((3, 5, 13, 17, 32, 7, 5, 1, 2, 3, 2), 0),       # 32 channels: the narrow tile; 175 terms
    ((2, 12, 8, 12, 20, 1, 1, 1, 1, 0, 0), 0),       # 1x1, planes of 96 pixels: 16-byte copies; 12 terms, one slab
    ((2, 13, 5, 4, 70, 1, 1, 1, 1, 0, 0), 0),        # the same with 13 terms (4-byte weight copies)
    ((2, 816, 13, 31, 80, 1, 1, 1, 1, 0, 0), 0),     # 1x1, planes of 403 pixels
    ((1, 4, 33000, 1, 8, 3, 1, 1, 1, 1, 0), 0),      # taller than the decode table's fields
    ((1, 1, 1, 1, 1, 1, 1, 1, 1, 0, 0), 0),
    ((1, 1, 32760, 3, 8, 3, 1, 1, 1, 20, 0), 0),     # image and padding together are taller than the decode table's fields; 3 terms
    ((1, 2, 32700, 1, 4, 3, 1, 1, 1, 67, 0), 0),     # exactly as tall
]


@pytest.mark.parametrize("case", range(len(CASES)))
def test_fp32_tiles(pkg, orc, oracle, case):
    args, off = CASES[case]
    p = orc.Problem.P(*args, precision=orc.FP32, bias=(case % 2 == 0), relu=(case % 3 == 0))
    x, w, b = oracle.make_conv_data(p, 500 + case, case % 4)
    ref, scale = oracle.conv2d(p, x, w, b if p.has_bias else None)
    got, plan, out = gu.run_conv(pkg, oracle, p, x, w, b if p.has_bias else None, offsets=(off, off, off))
    m = oracle.compare(p, got, ref, scale)   # the reference's FP32 policy: the rounding of FP32 sums of this length
    assert m.passed(), f"fp32 case {case}: {m.summary()}"
    again, _, out2 = gu.run_conv(pkg, oracle, p, x, w, b if p.has_bias else None, plan=plan, offsets=(off, off, off))
    assert np.array_equal(out.raw_bits(), out2.raw_bits())
