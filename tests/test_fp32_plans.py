"""CPU test of what a query says about strict-FP32 plans: the CTAs of the launch and the shared memory each asks for, which also tells
the two kernels apart (conv_fp32.cu: a ring of four slabs and the decode table; conv_fp32_wide.cu: two or four groups of threads)."""
import pytest

WIDE = {128: 2 * 4 * (3 * 16 * 128 + 2 * 16 * 68 + 96), 64: 4 * 4 * (3 * 16 * 64 + 2 * 16 * 68 + 96)}


def query(pkg, *args):
    return pkg.query(pkg.ConvProblem(*args, precision=pkg.FP32, has_bias=True, relu=True))


@pytest.mark.parametrize("args,tile", [((3, 97, 40, 25, 70, 5, 5, 1, 1, 2, 2), 128), ((2, 762, 18, 18, 256, 3, 3, 2, 2, 1, 1), 64)])
def test_wide_tiles(pkg, args, tile):
    i = query(pkg, *args)
    tiles = -(-(args[0] * (args[2] // args[7]) * (args[3] // args[8])) // tile) * -(-args[4] // 64)
    assert (i.cfg.tile_m, i.cfg.tile_n, i.dynamic_smem_bytes, i.threads_per_block) == (tile, 64, WIDE[tile], 128)
    assert i.num_blocks % tiles == 0 and 1 <= i.num_blocks // tiles <= 8


@pytest.mark.parametrize("args,tiles,terms", [((1, 64, 56, 56, 64, 3, 3, 1, 1, 1, 1), 49, 576), ((4, 32, 10, 10, 20, 3, 3, 1, 1, 1, 1), 4, 288)])
def test_narrow_tiles(pkg, args, tiles, terms):
    i = query(pkg, *args)
    to = 64 if args[4] > 32 else 32
    slices = i.num_blocks // tiles
    assert i.num_blocks == tiles * slices and 1 <= slices <= 8
    slabs = -(-(-(-terms // 16)) // slices)   # of a slice
    assert i.dynamic_smem_bytes == 4 * 4 * (16 * i.cfg.tile_m + 20 * to) + 8 * 16 * slabs
    # 16-byte copies along the pixels need no table
    one = query(pkg, 64, 256, 28, 28, 64, 1, 1)
    assert one.dynamic_smem_bytes == 4 * 4 * (16 * 64 + 20 * 64)
