"""CPU test of the strict-FP32 choice: a launch whose CTAs would fit the machine in one wave, but whose clusters would not, takes as long
as two waves and is not chosen.  (With two CTAs per SM the machine holds 296 CTAs, but 33 clusters of eight, 45 of six, 93 of three.)"""
import random

HELD = [296, 148, 93, 71, 56, 45, 37, 33]  # clusters of 1 .. 8 CTAs, two CTAs per SM
WIDE = {128: 2 * 4 * (3 * 16 * 128 + 2 * 16 * 68 + 96), 64: 4 * 4 * (3 * 16 * 64 + 2 * 16 * 68 + 96)}  # shared memory of a CTA


def choice(pkg, args):
    """(tile_m, clusters, slices), or None on the kernel of narrow tiles."""
    p = pkg.ConvProblem(*args, precision=pkg.FP32, has_bias=True, relu=True)
    i = pkg.query(p)
    if i.dynamic_smem_bytes != WIDE.get(i.cfg.tile_m):
        return None
    clusters = -(-args[0] * p.out_h * p.out_w // i.cfg.tile_m) * -(-args[4] // 64)
    return i.cfg.tile_m, clusters, i.num_blocks // clusters


def test_waves_of_clusters(pkg):
    # narrow tiles 44.8 us, wide ones in 26 clusters of five 50.7; 271 and 277 (77 of seven); 67.8 and 72.5 (37 of eight)
    for args in [(26, 448, 8, 31, 64, 3, 3, 2, 2, 1, 1), (3, 832, 57, 57, 48, 3, 3, 1, 1, 1, 1), (2, 331, 33, 33, 74, 3, 3, 1, 1, 1, 1)]:
        assert choice(pkg, args) is None, args
    # 128 pixels and three slices 445 us, narrow tiles 407, 64 pixels and five slices 360
    assert choice(pkg, (11, 360, 33, 33, 48, 5, 5, 1, 1, 2, 2)) == (64, 188, 5)
    rng = random.Random(3)
    seen = set()
    for _ in range(4000):
        k, stride = rng.choice([(1, 1), (3, 1), (3, 2), (5, 1)])
        args = (rng.randint(1, 32), rng.randint(16, 1024), rng.randint(7, 60), rng.randint(7, 60), rng.randint(16, 512), k, k, stride, stride, k // 2, k // 2)
        got = choice(pkg, args)
        if got is not None:
            _, clusters, slices = got
            assert clusters * slices > 296 or clusters <= HELD[slices - 1], (args, got)
            seen.add(slices)
    assert {1, 2, 3, 4, 5, 6, 8} <= seen, seen
