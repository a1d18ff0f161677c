"""CPU test of what a query says about first layers over images (few channels, horizontal stride 2, even width): the kernel that reads
the image in place, its shared memory, threads and CTAs; and that whatever it is not gets the form that gathers first when asked for."""
import pytest

SIZES = [  # layer, channel-contiguous output, dynamic shared memory, CTAs
    ((1, 3, 64, 64, 64, 7, 7, 2, 2, 3, 3), False, 40704, 32),
    ((4, 3, 224, 224, 64, 7, 7, 2, 2, 3, 3), False, 59136, 296),
    ((32, 3, 224, 224, 64, 7, 7, 2, 2, 3, 3), True, 99328, 296),
    ((128, 3, 224, 224, 64, 7, 7, 2, 2, 3, 3), False, 103424, 296),
    ((1, 3, 23, 600, 40, 7, 7, 2, 2, 3, 3), False, 107264, 12),
    ((1, 3, 9, 1200, 160, 7, 7, 2, 2, 3, 3), False, 184064, 15),   # one CTA per SM, three tiles of channels
]


def query(pkg, args, flags=0, **cfg):
    return pkg.query(pkg.ConvProblem(*args, precision=pkg.FP16, has_bias=True, relu=True, flags=flags), pkg.make_cfg(**cfg) if cfg else None)


@pytest.mark.parametrize("args,nhwc,smem,ctas", SIZES)
def test_the_kernel_that_runs(pkg, args, nhwc, smem, ctas):
    flags = pkg.FLAG_OUTPUT_NHWC if nhwc else 0
    i = query(pkg, args, flags)
    c = i.cfg
    assert (i.variant, i.launches, i.workspace_bytes, i.padded_channels) == (5, 1, 0, 32)
    assert (i.dynamic_smem_bytes, i.threads_per_block, i.num_blocks) == (smem, 416, ctas)
    assert (c.tile_m, c.tile_n, c.tile_k, c.stages, c.split_k, c.variant, c.reduce, c.cta_pair) == (128, 64, 32, 2, 1, 5, 0, 1)
    # what it is may be asked for, in part or in full
    for asked in (dict(tile_m=128), dict(tile_n=64), dict(tile_k=32), dict(stages=2), dict(split_k=1), dict(variant=5), dict(cta_pair=1),
                  {f: getattr(c, f) for f, _ in c._fields_}):
        j = query(pkg, args, flags, **asked)
        assert (j.launches, j.dynamic_smem_bytes, j.num_blocks) == (1, smem, ctas), asked


@pytest.mark.parametrize("args,nhwc,smem,ctas", SIZES)
def test_what_is_asked_for_runs(pkg, args, nhwc, smem, ctas):
    gathered = None
    for asked in (dict(tile_n=32), dict(tile_n=128), dict(tile_n=256), dict(tile_m=256), dict(stages=3), dict(stages=4, tile_n=64), dict(tile_k=16),
                  dict(split_k=2), dict(split_k=3, reduce=1), dict(cta_pair=2, tile_n=64)):
        i = query(pkg, args, pkg.FLAG_OUTPUT_NHWC if nhwc else 0, **asked)
        assert i.supported and i.variant == 5 and i.launches >= 2, asked
        assert all(getattr(i.cfg, k) == v for k, v in asked.items()), asked
        if i.cfg.reduce != 1:
            assert gathered in (None, i.workspace_bytes) and i.workspace_bytes > 0
            gathered = i.workspace_bytes


def test_more_channels_than_the_grid_takes(pkg):
    """Tiles of channels are the grid's second dimension: 65535 of 64.  Beyond, the form that gathers first takes the layer."""
    for filters, launches in ((65535 * 64, 1), (65535 * 64 + 1, 2)):
        i = query(pkg, (1, 1, 4, 4, filters, 3, 3, 2, 2, 1, 1))
        assert i.supported and i.variant == 5 and i.launches == launches, filters
