"""CPU test of the tiles that the direct-NCHW route takes when they are left to the library: the narrowest of 32, 64 and 128 channels
with at most one tile per SM; where there is none, 128 (64 or 32 where a layer has no more channels), or 256 for reductions of more
than two slabs whose tiles of 128 channels take an SM more than 7/8 of the time that those of 256 do, and for up to 192 channels of
shorter ones.  What is asked for stays."""
SMS = 148


def test_direct_tiles_by_the_number_of_tiles(pkg):
    seen = set()
    for b in (1, 2, 4, 8, 16, 64):
        for c in (16, 64, 191, 512):
            for h, w in ((8, 8), (24, 13), (28, 28), (56, 56)):
                for o in (21, 37, 64, 128, 160, 200, 256, 768):
                    def query(**kw):
                        return pkg.query(pkg.ConvProblem(b, c, h, w, o, 1, 1, precision=pkg.BF16, has_bias=True, relu=True), pkg.make_cfg(**kw) if kw else None)
                    auto = query()
                    assert auto.variant == 2 and auto.cfg.cta_pair == 1
                    tiles_m = -(-(b * -(-(h * w) // 64)) // 2)   # 128 rows: two boxes of 64 pixels of an image
                    widths = [n for n in (32, 64, 128) if n == 32 or n // 2 < o]
                    walks = {n: -(-tiles_m * -(-o // n) // SMS) for n in (32, 64, 128, 256)}
                    fitting = [n for n in widths if walks[n] == 1]
                    want = fitting[0] if fitting else widths[-1]
                    if not fitting and o > 128 and (walks[256] > 1 and 8 * walks[128] > 7 * 2 * walks[256] if c > 128 else o <= 192):
                        want = 256
                    assert auto.cfg.tile_n == want, (b, c, h, w, o)
                    seen.add(want)
                    for n in (32, 64, 128, 256):
                        asked = query(tile_n=n)
                        assert asked.supported and asked.cfg.tile_n == n
                    if c == 512 and o >= 64:   # (a split in clusters needs tiles of 64 channels or more: its search keeps every width)
                        assert query(split_k=2, reduce=2).supported
    assert seen == {32, 64, 128, 256}


def test_direct_tiles_and_rings_with_a_residual(pkg):
    """More tiles of 128 channels than SMs: a residual takes 256 channels for three to seven slabs; without one, tiles of 128 have six
    stages from four slabs on."""
    seen = set()
    for residual in (False, True):
        for c, slabs in ((191, 3), (256, 4), (320, 5), (512, 8)):
            for b in (1, 16, 32, 64):
                for o in (128, 200, 256, 768):
                    p = pkg.ConvProblem(b, c, 28, 28, o, 1, 1, precision=pkg.BF16, has_bias=True, relu=True, flags=pkg.FLAG_RESIDUAL if residual else 0)
                    cfg = pkg.query(p).cfg
                    tiles_m = -(-(b * -(-784 // 64)) // 2)
                    walks = {n: -(-tiles_m * -(-o // n) // SMS) for n in (32, 64, 128, 256)}
                    fitting = [n for n in (32, 64, 128) if walks[n] == 1]
                    want = fitting[0] if fitting else 128
                    if not fitting and o > 128 and ((residual and slabs < 8) or (walks[256] > 1 and 8 * walks[128] > 7 * 2 * walks[256])):
                        want = 256
                    assert cfg.tile_n == want, (residual, c, b, o)
                    if want == 128 and cfg.tile_m == 128:
                        six = slabs >= 8 or (slabs >= 4 and not residual)
                        assert (cfg.stages == 6) == six, (residual, c, b, o, cfg.stages)
                    seen.add((residual, slabs, want))
    assert {(True, 4, 256), (False, 4, 128), (False, 3, 128), (True, 3, 256), (True, 5, 128), (True, 8, 128)} <= seen, seen


def test_short_pointwise_tiles(pkg):
    """1x1 layers of one or two slabs over channel-contiguous tensors: no tiles of 32 channels beyond two of them per SM, none of 256
    pixels and 128 channels; what is asked for stays."""
    seen = set()
    for b in (1, 3, 9, 30, 58, 128):
        for c in (16, 64, 128):
            for h, w in ((7, 7), (10, 19), (33, 33), (61, 61)):
                for o in (24, 64, 192, 640, 896):
                    def query(**kw):
                        return pkg.query(pkg.ConvProblem(b, c, h, w, o, 1, 1, precision=pkg.FP16, has_bias=True, relu=True, flags=pkg.FLAG_INPUT_NHWC | pkg.FLAG_OUTPUT_NHWC),
                                         pkg.make_cfg(**kw) if kw else None)
                    cfg = query().cfg
                    if cfg.cta_pair == 2:
                        continue
                    if o > 32 and -(-(b * h * w) // 128) * -(-o // 32) > 2 * SMS:
                        assert cfg.tile_n != 32, (b, c, h, w, o)
                    assert (cfg.tile_m, cfg.tile_n) != (256, 128), (b, c, h, w, o)
                    assert query(tile_n=32).cfg.tile_n == 32 and query(tile_m=256, tile_n=128).cfg.tile_m == 256
                    seen.add((cfg.tile_m, cfg.tile_n))
    assert {(128, 32), (128, 64), (128, 128)} <= seen
