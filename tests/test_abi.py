"""CPU tests of the drop-in boundary: the shared library loads, exports every symbol include/gie_b200.h declares, and
its host-side logic (validation status codes, capability answers, workspace layout, configuration selection) behaves
as the reference's (tests/test_cpu_reference.cpp:158-171, tests/test_dispatcher.cpp, tests/test_validation.cpp).
No GPU is touched: nothing here launches or allocates on a device."""
import ctypes as C
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def declared_symbols():
    text = open(os.path.join(ROOT, "include", "gie_b200.h")).read()
    return sorted(set(re.findall(r"GIEB_API\s+[\w\s\*]+?\b(gieb_\w+)\s*\(", text)))


def test_library_exports_every_declared_symbol(pkg):
    names = declared_symbols()
    assert len(names) >= 17, names
    out = subprocess.check_output(["nm", "-D", "--defined-only", pkg.LIB_PATH], text=True)
    exported = set(re.findall(r"\b(gieb_\w+)\b", out))
    assert set(names) <= exported, sorted(set(names) - exported)
    lib = pkg.lib()
    for n in names:
        assert getattr(lib, n) is not None
    assert lib.gieb_version() >= 1


def P(pkg, *a, **k):
    return pkg.ConvProblem(*a, **k)


def test_validate_status_codes(pkg):
    ok = P(pkg, 1, 3, 8, 8, 4, 3, 3, 1, 1, 1, 1)
    pkg.validate_problem(ok)
    for bad in [P(pkg, 0, 1, 5, 5, 1, 3, 3), P(pkg, 1, 1, 2, 2, 1, 5, 5), P(pkg, 1, 1, 5, 5, 1, 3, 3, 0, 1),
                P(pkg, 1, 1, 5, 5, 1, 3, 3, 1, 1, -1, 0), P(pkg, 30000, 1, 512, 512, 1, 1, 1), P(pkg, 1, 1, 5, 5, 1, 3, 3, precision=9)]:
        with pytest.raises(pkg.GieError) as e:
            pkg.validate_problem(bad)
        assert e.value.code == pkg.INVALID_ARGUMENT, bad
    for uns in [P(pkg, 1, 1, 9, 9, 1, 3, 3, dilation_h=2), P(pkg, 1, 4, 9, 9, 4, 3, 3, groups=2)]:
        with pytest.raises(pkg.GieError) as e:
            pkg.validate_problem(uns)
        assert e.value.code == pkg.UNSUPPORTED
    assert "dilation" in pkg.last_error() or "grouped" in pkg.last_error()


def test_validation_matches_oracle_on_the_correctness_shapes(pkg, orc, oracle):
    for name, args in orc.CORRECTNESS_SHAPES.items():
        for prec in (orc.FP32, orc.FP16, orc.BF16):
            p = orc.Problem.P(*args, precision=prec)
            assert oracle.validate(p) == 0
            cp = P(pkg, *args, precision=prec)
            pkg.validate_problem(cp)
            assert (cp.out_h, cp.out_w, cp.flops) == (p.out_h, p.out_w, p.flops)
            info = pkg.query(cp)
            assert info.supported == 1, (name, prec, info.reason)   # no (shape, precision) cell may be left without a kernel


def test_epilogue_warp_count_follows_the_plan(pkg):
    """CTAs that own their SM run 16 epilogue warps (640 threads): every 256-column tile whose ring leaves no room for a
    second CTA, and 128-column tiles with one tile per CTA; everything else keeps 8 (384 threads)."""
    c2 = pkg.query(P(pkg, 32, 256, 14, 14, 256, 3, 3, 1, 1, 1, 1, precision=pkg.FP16))
    # a long reduction with enough pixels: 256-pixel tiles of CTA pairs, each CTA alone on its SM
    assert c2.supported and c2.threads_per_block == 640 and (c2.cfg.tile_m, c2.cfg.tile_n, c2.cfg.split_k, c2.cfg.cta_pair) == (256, 128, 1, 2)
    single = pkg.query(P(pkg, 32, 256, 14, 14, 256, 3, 3, 1, 1, 1, 1, precision=pkg.FP16), pkg.make_cfg(cta_pair=1))
    assert single.supported and single.threads_per_block == 640 and (single.cfg.tile_m, single.cfg.tile_n, single.cfg.cta_pair) == (128, 128, 1)
    c3 = pkg.query(P(pkg, 64, 512, 28, 28, 128, 1, 1, precision=pkg.FP16))
    assert c3.supported and c3.variant == 2 and c3.threads_per_block == 384 and c3.launches == 1   # 416 tiles on 148 CTAs; weights in place
    wide = pkg.query(P(pkg, 16, 128, 54, 54, 256, 3, 3, 2, 2, 1, 1, precision=pkg.FP16), pkg.make_cfg(tile_n=256, tile_k=64, stages=4))
    assert wide.supported and wide.threads_per_block == 640                                         # 27 x 27 output planes: pixel-lane kernel
    shallow = pkg.query(P(pkg, 16, 128, 54, 54, 256, 3, 3, 2, 2, 1, 1, precision=pkg.FP16), pkg.make_cfg(tile_n=128, tile_k=64, stages=2))
    assert shallow.supported and shallow.threads_per_block == 384                                   # two CTAs share an SM
    # NCHW output planes of 28 x 28 (16-byte multiples): transposed accumulator, a short epilogue on eight warps
    tr = pkg.query(P(pkg, 64, 512, 28, 28, 128, 1, 1, precision=pkg.FP16), pkg.make_cfg(tile_m=128, tile_n=128, tile_k=64, stages=6))
    assert tr.supported and tr.threads_per_block == 384 and tr.dynamic_smem_bytes == 1024 + 3072 + 6 * 32768 + 8 * 2048


def test_query_precision_routing_and_reasons(pkg):
    base = (2, 64, 14, 14, 64, 3, 3, 1, 1, 1, 1)
    i32 = pkg.query(P(pkg, *base, precision=pkg.FP32))
    assert i32.supported and i32.variant == 3 and i32.workspace_bytes == 0 and i32.launches == 1
    i16 = pkg.query(P(pkg, *base, precision=pkg.FP16))
    assert i16.supported and i16.variant == 1 and i16.threads_per_block == 384 and i16.padded_channels == 64
    ipw = pkg.query(P(pkg, 2, 64, 14, 14, 64, 1, 1, precision=pkg.BF16))
    assert ipw.supported and ipw.variant == 4                       # 1x1 / stride 1 / pad 0 -> tiled activation loads
    idr = pkg.query(P(pkg, 2, 64, 28, 28, 64, 1, 1, precision=pkg.BF16))
    assert idr.supported and idr.variant == 2                       # H*W % 8 == 0 -> straight from NCHW, no activation repack
    assert not pkg.query(P(pkg, 2, 64, 14, 14, 64, 1, 1, precision=pkg.FP16), pkg.make_cfg(variant=2)).supported
    tf = pkg.query(P(pkg, *base, precision=pkg.TF32))  # FP32 storage on the tensor cores (kind::tf32)
    assert tf.supported and tf.variant in (1, 4) and tf.cfg.tile_k in (8, 16, 32)
    assert not pkg.query(P(pkg, *base, precision=pkg.TF32, flags=pkg.FLAG_OUTPUT_NHWC)).supported
    big_stride = pkg.query(P(pkg, 1, 16, 64, 64, 16, 3, 3, 9, 9, 1, 1, precision=pkg.FP16))
    assert not big_stride.supported and b"stride" in big_stride.reason
    assert not pkg.query(P(pkg, *base, precision=pkg.FP16), pkg.make_cfg(variant=3)).supported
    assert not pkg.query(P(pkg, *base, precision=pkg.FP16), pkg.make_cfg(variant=4)).supported
    assert not pkg.query(P(pkg, *base, precision=pkg.FP32), pkg.make_cfg(variant=1)).supported


def test_query_rejects_impossible_configurations(pkg):
    p = P(pkg, 8, 64, 14, 14, 64, 3, 3, 1, 1, 1, 1, precision=pkg.FP16)
    too_much_smem = pkg.query(p, pkg.make_cfg(tile_n=128, tile_k=64, stages=8))
    assert not too_much_smem.supported and b"shared memory" in too_much_smem.reason
    assert not pkg.query(p, pkg.make_cfg(tile_n=48)).supported
    assert not pkg.query(p, pkg.make_cfg(tile_k=48)).supported
    assert not pkg.query(p, pkg.make_cfg(tile_m=64)).supported
    assert not pkg.query(p, pkg.make_cfg(stages=1)).supported
    short = pkg.query(P(pkg, 8, 64, 14, 14, 64, 1, 1, precision=pkg.FP16), pkg.make_cfg(split_k=4))
    assert not short.supported and b"split" in short.reason          # reduction too short (one slab)
    assert not pkg.query(p, pkg.make_cfg(tile_m=256, tile_n=256, tile_k=64, stages=4)).supported  # 4 x 64 KiB ring


def test_workspace_layout_and_padding(pkg):
    # C=130 -> padded channels; workspace = align256(B*H*W*Cp*2) + align256(O*R*S*Cp*2) (+ split * align4(|Y|) * 4)
    p = P(pkg, 2, 130, 9, 9, 130, 3, 3, 1, 1, 1, 1, precision=pkg.FP16)
    a256 = lambda v: (v + 255) // 256 * 256
    for tk, cp in ((16, 144), (32, 160), (64, 192)):
        i = pkg.query(p, pkg.make_cfg(tile_k=tk, split_k=1))
        assert i.padded_channels == cp
        assert i.workspace_bytes == a256(2 * 81 * cp * 2) + a256(130 * 9 * cp * 2)
    i = pkg.query(p, pkg.make_cfg(tile_k=32, split_k=3))
    ys = 2 * 130 * 81
    assert i.cfg.split_k == 3 and i.workspace_bytes == a256(2 * 81 * 160 * 2) + a256(130 * 9 * 160 * 2) + a256(3 * ((ys + 3) // 4 * 4) * 4)
    assert i.launches == 3
    pre = P(pkg, 2, 130, 9, 9, 130, 3, 3, 1, 1, 1, 1, precision=pkg.FP16, flags=pkg.FLAG_WEIGHTS_PREPACKED)
    assert pkg.query(pre, pkg.make_cfg(tile_k=32, split_k=1)).workspace_bytes == a256(2 * 81 * 160 * 2)
    stem = P(pkg, 1, 3, 224, 224, 64, 7, 7, 2, 2, 3, 3, precision=pkg.FP16)
    assert pkg.query(stem, pkg.make_cfg(variant=1)).padded_channels == 16
    auto = pkg.query(stem)  # few channels: the 7 taps of a filter row become 7 * 3 -> 32 channels of a 7 x 1 convolution
    assert auto.variant == 5 and auto.padded_channels == 32
    # stride 2, 3 channels: the image is read in place, without scratch; where the layer is gathered first, column pairs are stored
    # once (115 positions of 16 bytes per input row: 2 of padding on the left, 112 pairs, 1 on the right) and adjacent windows overlap
    # in memory
    assert auto.workspace_bytes == 0
    assert pkg.query(stem, pkg.make_cfg(cta_pair=2)).workspace_bytes == a256(1 * 224 * 115 * 16) + a256(64 * 7 * 32 * 2)
    assert pkg.query(P(pkg, 1, 96, 27, 27, 192, 5, 5, 1, 1, 2, 2, precision=pkg.FP16)).padded_channels == 96


def test_selection_is_deterministic_and_fills_the_machine(pkg):
    """Ranking determinism (tests/test_dispatcher.cpp) and sanity of the choice: never more split-K than the
    reduction allows, every slice non-empty, grid within limits, shared memory within the per-CTA limit."""
    shapes = [(32, 256, 14, 14, 256, 3, 3, 1, 1, 1, 1), (64, 512, 28, 28, 128, 1, 1, 1, 1, 0, 0), (8, 512, 7, 7, 512, 3, 3, 1, 1, 1, 1),
              (16, 128, 56, 56, 256, 3, 3, 2, 2, 1, 1), (1, 512, 7, 7, 512, 3, 3, 1, 1, 1, 1), (256, 64, 56, 56, 256, 1, 1, 1, 1, 0, 0),
              (256, 3, 224, 224, 64, 7, 7, 2, 2, 3, 3), (1, 1, 1, 1, 1, 1, 1, 1, 1, 0, 0)]
    for a in shapes:
        p = P(pkg, *a, precision=pkg.FP16, has_bias=True, relu=True)
        i1, i2 = pkg.query(p), pkg.query(p)
        c = i1.cfg
        assert (c.tile_m, c.tile_n, c.tile_k, c.stages, c.split_k) == (i2.cfg.tile_m, i2.cfg.tile_n, i2.cfg.tile_k, i2.cfg.stages, i2.cfg.split_k)
        assert i1.supported and c.tile_m in (128, 256) and c.tile_n in (32, 64, 128, 256) and c.tile_k in (16, 32, 64)
        assert 2 <= c.stages <= 8 and i1.dynamic_smem_bytes <= 232448
        total_kb = a[5] * a[6] * (i1.padded_channels // c.tile_k)
        assert 1 <= c.split_k <= max(1, total_kb // 2)
        if i1.variant == 5:   # straight from the image: persistent CTAs, at most two per SM
            assert i1.launches == 1 and i1.num_blocks == 2 * 148
            continue
        pixels = a[0] * p.out_h * p.out_w
        rows = a[0] * -(-(a[2] * a[3]) // 64) * 64 if i1.variant == 2 else pixels   # direct NCHW route counts 64-pixel boxes
        if c.variant == 6:                # halo tiles cover the padded grid; at stride 1 neighbours share their padding
            assert (a[7], a[8]) == (1, 1)
            rows = a[0] * (a[2] + a[9]) * (a[3] + a[10])
        ctas_per_tile = 2 if c.cta_pair == 2 else 1   # a 256-pixel tile of a CTA pair is two CTAs
        assert i1.num_blocks == -(-rows // c.tile_m) * -(-a[4] // c.tile_n) * c.split_k * ctas_per_tile
    # the small deep layer gets split-K, the big ones do not
    assert pkg.query(P(pkg, 1, 512, 7, 7, 512, 3, 3, 1, 1, 1, 1, precision=pkg.FP16)).cfg.split_k > 1
    assert pkg.query(P(pkg, 256, 64, 56, 56, 256, 1, 1, precision=pkg.FP16)).cfg.split_k == 1


def test_static_scratch_size_check_needs_no_gpu(pkg):
    """The allocation-free entry point refuses oversized problems before touching the device."""
    big = P(pkg, 64, 512, 28, 28, 128, 1, 1, precision=pkg.FP16)
    with pytest.raises(pkg.GieError) as e:
        pkg.conv_forward_static(big, 256, 256, None, 256, 0)
    assert e.value.code == pkg.WORKSPACE_TOO_SMALL


def test_rmsnorm_argument_checks_need_no_gpu(pkg):
    for args in [(1, 4, 16, 32, 16, None, None), (1, 4, 16, 32, 48, 64, None), (1, 0, 16, 32, 48, None, None), (0, 4, 16, 32, 48, None, None),
                 (1, 4, None, 32, 48, None, None)]:
        rows, hidden, x, g, y, ri, ro = args
        with pytest.raises(pkg.GieError) as e:
            pkg.rmsnorm_forward(rows, hidden, 1e-6, 0, x, g, y, ri, ro, 0)
        assert e.value.code == pkg.INVALID_ARGUMENT


def test_dependents_start_behind_the_tensor_memory_allocation():
    """A kernel that allocates tensor memory lets the next kernel of the stream start only once it has its columns: the
    signal comes from the allocating warp, after the allocation, and from nowhere else."""
    csrc = os.path.join(ROOT, "cuda-inference_b200", "csrc")
    seen = 0
    for f in sorted(os.listdir(csrc)):
        text = re.sub(r"//[^\n]*", "", open(os.path.join(csrc, f)).read())
        if f == "ptx.cuh" or not re.search(r"ptx::tmem_alloc\(", text):
            continue
        seen += 1
        signals = [m.start() for m in re.finditer(r"ptx::grid_dep_launch\(\)", text)]
        allocs = [m.start() for m in re.finditer(r"ptx::tmem_alloc(?:_pair)?\(", text)]
        assert len(signals) == 1, f
        assert max(allocs) < signals[0] < text.index("ptx::tc_fence_before_sync()"), f
        block = text[text.rindex("if (warp == kProducerWarps) {", 0, signals[0]):signals[0]]
        assert block.count("{") > block.count("}") and "tmem_alloc" in block, f  # still inside the allocating warp's block
    assert seen == 2


def test_shared_memory_keeps_tensor_memory_from_running_out(pkg):
    """An allocation of tensor memory waits for another CTA of the SM to end.  CTAs of all 512 columns ask for more than half of
    an SM's shared memory, so that two never share one; CTAs that wait for one another (pairs, split-K clusters) ask for at
    least their columns' share of it, so that no set of them that fits an SM wants more than its 512 columns."""
    sm = 228 * 1024
    seen = {"full": 0, "pair": 0, "cluster": 0}
    shapes = [(237, 64, 81, 81, 320, 1, 1, 2, 2, 0, 0), (237, 64, 41, 41, 320, 1, 1, 1, 1, 0, 0), (8, 512, 7, 7, 512, 3, 3, 1, 1, 1, 1),
              (1, 512, 7, 7, 512, 3, 3, 1, 1, 1, 1), (32, 256, 14, 14, 256, 3, 3, 1, 1, 1, 1), (64, 512, 28, 28, 512, 3, 3, 1, 1, 1, 1),
              (1, 1024, 7, 7, 512, 1, 1, 1, 1, 0, 0), (2, 320, 8, 8, 40, 5, 5, 1, 1, 2, 2), (8, 64, 31, 31, 512, 3, 3, 1, 1, 1, 1),
              (2, 256, 67, 67, 512, 1, 3, 1, 1, 0, 1), (1, 2048, 9, 9, 256, 3, 3, 1, 1, 1, 1), (4, 64, 12, 12, 256, 1, 1, 1, 1, 0, 0)]
    cfgs = [None] + [dict(tile_m=m, tile_n=n, stages=2, cta_pair=1) for m in (128, 256) for n in (32, 64, 128, 256)]
    cfgs += [dict(tile_n=n, stages=2, cta_pair=2) for n in (64, 128, 256)] + [dict(tile_n=n, split_k=2, reduce=2) for n in (64, 128, 256)]
    for a in shapes:
        for prec in (pkg.FP16, pkg.BF16, pkg.FP8_E4M3):
            for kw in cfgs:
                info = pkg.query(P(pkg, *a, precision=prec, has_bias=True, relu=True), pkg.make_cfg(**kw) if kw else None)
                if not info.supported:
                    continue
                c = info.cfg
                one = c.tile_n * (1 if c.cta_pair == 2 else c.tile_m // 128)   # columns of one accumulator; two when they fit
                cols = max(32, 2 * one if one <= 256 else one)
                smem = info.dynamic_smem_bytes
                assert smem <= 227 * 1024
                if cols == 512:
                    seen["full"] += 1
                    assert 2 * (smem + 1024) > sm, (a, prec, kw, smem)
                waits = "pair" if c.cta_pair == 2 else ("cluster" if c.reduce == 2 else None)
                if waits:
                    seen[waits] += 1
                    assert (smem + 1024) * 512 >= sm * cols, (a, prec, kw, smem, cols)
    assert min(seen.values()) > 10, seen


def _random_problems(pkg, n, seed):
    """Convolutions over the sizes, layouts and types that networks have, ragged ones among them."""
    import random
    rng = random.Random(seed)
    made = 0
    while made < n:
        k = rng.choice([(1, 1), (3, 3), (3, 3), (5, 5), (7, 7), (1, 3), (3, 2)])
        stride = rng.choice([1, 1, 1, 2])
        h = rng.choice([7, 8, 9, 13, 14, 17, 28, 31, 35, 56, 67])
        w = rng.choice([h, h, rng.randint(5, 80)])
        c = rng.choice([3, 16, 33, 48, 64, 72, 80, 96, 112, 128, 130, 144, 160, 192, 200, 256, 320, 512, 816])
        o = rng.choice([8, 17, 32, 40, 64, 70, 96, 128, 131, 144, 192, 200, 256, 320, 512])
        b = rng.choice([1, 1, 2, 3, 4, 8, 16, 32, 64, 128])
        prec = rng.choice([pkg.FP16, pkg.FP16, pkg.BF16, pkg.TF32, pkg.FP8_E4M3, pkg.FP32])
        flags = 0
        if prec in (pkg.FP16, pkg.BF16):
            flags = (rng.choice([0, pkg.FLAG_INPUT_NHWC if c % 16 == 0 else 0]) | rng.choice([0, pkg.FLAG_OUTPUT_NHWC]) |
                     rng.choice([0, pkg.FLAG_RESIDUAL]) | rng.choice([0, pkg.FLAG_WEIGHTS_PREPACKED]))
        p = P(pkg, b, c, h, w, o, k[0], k[1], stride, stride, k[0] // 2, k[1] // 2, precision=prec, has_bias=True, relu=True, flags=flags)
        if pkg.query(p).supported:
            made += 1
            yield p


def _reported(info):
    return (tuple(getattr(info.cfg, f) for f, _ in info.cfg._fields_), info.variant, info.workspace_bytes, info.dynamic_smem_bytes, info.threads_per_block,
            info.num_blocks, info.launches, info.padded_channels)


def test_reported_configuration_gives_the_same_plan(pkg):
    """What a query reports as its configuration can be handed back, and then stands for the same plan: tiles, workspace,
    weight layout and grid (the halo kernel's plans and partial last slabs among them)."""
    seen = {}
    for p in _random_problems(pkg, 3000, 5):
        auto = pkg.query(p)
        c = auto.cfg
        again = pkg.query(p, pkg.make_cfg(**{f: getattr(c, f) for f, _ in c._fields_}))
        assert again.supported, (p, again.reason)
        assert _reported(again) == _reported(auto), (p, _reported(auto), _reported(again))
        kind = (c.variant, c.cta_pair, c.split_k > 1, auto.padded_channels % max(1, c.tile_k) != 0)
        seen[kind] = seen.get(kind, 0) + 1
    for kind in [(6, 1, False, False), (6, 1, True, False), (6, 2, False, False), (6, 1, False, True), (1, 1, True, False), (1, 1, False, True),
                 (1, 2, False, False), (4, 1, False, True), (2, 1, False, False), (5, 1, False, False), (3, 0, False, False)]:
        assert seen.get(kind, 0) >= 3, (kind, seen)


def test_reported_configuration_of_gathered_rows(pkg):
    """The same for layers of few channels and wide kernels, whose slab width is that of a gathered row: split and unsplit, with the
    slices summed in clusters (shares of 8 columns and up) or in the workspace."""
    import random
    rng = random.Random(11)
    seen = {}
    for _ in range(2500):
        k = rng.choice([5, 7, 9, 11, 13])
        c, o = rng.randint(1, 7), rng.choice([8, 16, 24, 32, 48, 64, 96, 128, 200, 256])
        h, w, s = rng.randint(5, 40), rng.randint(5, 40), rng.choice([1, 1, 2])
        flags = rng.choice([0, pkg.FLAG_OUTPUT_NHWC]) | rng.choice([0, pkg.FLAG_RESIDUAL]) | rng.choice([0, pkg.FLAG_WEIGHTS_PREPACKED])
        p = P(pkg, rng.choice([1, 1, 2, 3, 8]), c, h, w, o, k, k, s, s, k // 2, k // 2, precision=rng.choice([pkg.FP16, pkg.BF16]), has_bias=True, relu=True, flags=flags)
        auto = pkg.query(p)
        assert auto.supported
        again = pkg.query(p, pkg.make_cfg(**{f: getattr(auto.cfg, f) for f, _ in auto.cfg._fields_}))
        assert again.supported, (p, again.reason)
        assert _reported(again) == _reported(auto), (p, _reported(auto), _reported(again))
        kind = (auto.cfg.variant, auto.cfg.split_k > 1, auto.cfg.reduce)
        seen[kind] = seen.get(kind, 0) + 1
        if auto.cfg.variant == 5 and auto.cfg.reduce == 2 and auto.cfg.tile_n // auto.cfg.split_k < 32:
            seen["narrow"] = seen.get("narrow", 0) + 1
    assert all(seen.get(kind, 0) >= 50 for kind in [(5, False, 0), (5, True, 2), "narrow"]), seen


def test_tiles_and_splits_asked_for_leave_the_rest_as_it_was(pkg):
    """What is left open beside a tile, a split or a reduction that is asked for does not follow the choices for layers that ask for
    nothing: shares of 32 columns and up, and their cost.  (route, tile_n, split_k, reduce) of layers where it makes a difference."""
    for args, prec, flags, kw, want in [
            ((11, 64, 85, 85, 232, 5, 5, 1, 1, 2, 2), pkg.FP16, 12, dict(reduce=2), (1, 256, 1, 0)),
            ((22, 1024, 53, 53, 80, 1, 1, 1, 1, 0, 0), pkg.BF16, 2, dict(reduce=2), (4, 128, 1, 0)),
            ((5, 835, 18, 18, 288, 1, 1, 2, 2, 0, 0), pkg.BF16, 16, dict(reduce=2), (4, 32, 1, 0)),
            ((2, 576, 5, 4, 399, 5, 5, 2, 2, 2, 2), pkg.BF16, 12, dict(split_k=4), (1, 32, 4, 1)),
            ((1, 1024, 17, 17, 128, 3, 3, 2, 2, 1, 1), pkg.BF16, 12, dict(split_k=4), (1, 32, 4, 1)),
            ((9, 768, 6, 6, 400, 3, 3, 1, 1, 1, 1), pkg.FP16, 0, dict(split_k=8), (1, 128, 8, 1)),
            ((2, 112, 33, 33, 32, 5, 5, 1, 1, 2, 2), pkg.FP16, 0, dict(tile_n=64), (1, 64, 8, 1)),
            ((4, 704, 18, 12, 192, 1, 1, 1, 1, 0, 0), pkg.BF16, 14, dict(tile_n=64), (4, 64, 1, 0)),
            ((2, 384, 31, 4, 192, 3, 3, 2, 2, 1, 1), pkg.BF16, 2, dict(tile_n=128), (1, 128, 14, 1)),
            ((13, 64, 19, 19, 864, 5, 5, 1, 1, 2, 2), pkg.FP16, 12, dict(tile_n=64, reduce=2), (1, 64, 1, 0))]:
        i = pkg.query(P(pkg, *args, precision=prec, has_bias=True, relu=True, flags=flags), pkg.make_cfg(**kw))
        assert i.supported and (i.cfg.variant, i.cfg.tile_n, i.cfg.split_k, i.cfg.reduce) == want, (args, kw)
    # shares of less than 32 columns: in a configuration whose fields are all set, not otherwise
    p = P(pkg, 2, 256, 9, 7, 64, 3, 3, 1, 1, 1, 1, precision=pkg.FP16)
    narrow = dict(tile_n=64, split_k=4, reduce=2)
    assert not pkg.query(p, pkg.make_cfg(**narrow)).supported
    assert pkg.query(p, pkg.make_cfg(tile_m=128, tile_k=64, stages=4, variant=1, cta_pair=1, **narrow)).supported


def test_split_asked_for_with_its_reduction_left_open(pkg):
    """A split with every field set but the reduction: no query reports that (it names the reduction of its slices), so how they are summed
    is chosen as for any split that is asked for.  (tile_n, split_k) of layers where shares of less than 32 columns would be narrow ones."""
    for args, prec, flags, tile_n, split, tile_k, want in [
            ((1, 512, 26, 33, 83, 1, 1, 1, 1, 0, 0), pkg.FP16, 0, 64, 4, 64, 2103040), ((1, 512, 47, 37, 32, 5, 5, 1, 1, 2, 2), pkg.FP16, 12, 32, 4, 64, 1709568),
            ((16, 32, 14, 24, 32, 5, 5, 2, 2, 2, 2), pkg.TF32, 0, 64, 4, 32, 1478656), ((2, 1024, 23, 23, 32, 1, 1, 1, 1, 0, 0), pkg.FP16, 14, 128, 8, 64, 1083392),
            ((16, 768, 14, 14, 32, 1, 1, 1, 1, 0, 0), pkg.FP16, 28, 64, 4, 64, 1654784), ((2, 144, 51, 51, 64, 3, 3, 2, 2, 1, 1), pkg.FP8_E4M3, 0, 64, 4, 128, 2309120)]:
        variant = 4 if args[5] == 1 else 1
        cfg = dict(tile_m=128, tile_n=tile_n, tile_k=tile_k, stages=4, split_k=split, variant=variant, cta_pair=1)
        p = P(pkg, *args, precision=prec, has_bias=True, relu=True, flags=flags)
        i = pkg.query(p, pkg.make_cfg(**cfg))
        assert i.supported and (i.cfg.reduce, i.workspace_bytes) == (1, want), (args, i.cfg.reduce, i.workspace_bytes)
        assert pkg.query(p, pkg.make_cfg(reduce=2, **cfg)).supported


def test_shares_of_a_cluster_are_named_in_the_refusal(pkg):
    """Which columns per CTA a cluster reduction takes depends on what else is set and on the output's size; a refusal says so, in full."""
    full = dict(tile_m=128, tile_k=64, stages=4, variant=1, cta_pair=1, reduce=2)
    large, small = [P(pkg, 1, 512, s, s, 256, 3, 3, 1, 1, 1, 1, precision=pkg.FP16) for s in (4, 3)]   # 16 output pixels, and nine
    for p, kw, takes, says in [(large, dict(full, tile_n=32, split_k=4), True, None), (large, dict(full, tile_n=128, split_k=8), True, None),
                               (large, dict(full, tile_n=32, split_k=8), False, "dividing tile_n / 8,"), (large, dict(tile_n=32, split_k=4, reduce=2), False, "(tile_n / 8 where"),
                               (large, dict(tile_n=128, split_k=4, reduce=2), True, None), (small, dict(full, tile_n=32, split_k=4), False, "16 pixels or more"),
                               (small, dict(full, tile_n=128, split_k=4), True, None)]:
        i = pkg.query(p, pkg.make_cfg(**kw))
        assert bool(i.supported) == takes, (kw, i.reason)
        if not takes:
            reason = i.reason.decode() if isinstance(i.reason, bytes) else i.reason
            assert says in reason and reason.endswith("received slices"), reason


def test_halo_variant_takes_and_refuses(pkg):
    """The halo-tile kernel by name: what it can run it runs with the fields given, what it cannot is refused with a reason."""
    p = P(pkg, 4, 144, 14, 14, 200, 3, 3, 1, 1, 1, 1, precision=pkg.FP16)
    for kw in (dict(), dict(tile_n=256), dict(tile_n=64, split_k=2), dict(tile_n=128, split_k=2, reduce=2), dict(cta_pair=2), dict(cta_pair=2, tile_n=256),
               dict(tile_n=32, stages=3), dict(tile_m=128, tile_k=64)):
        i = pkg.query(p, pkg.make_cfg(variant=6, **kw))
        assert i.supported and i.cfg.variant == 6 and i.variant == 1, (kw, i.reason)
        assert i.padded_channels == 144 and all(getattr(i.cfg, k) == v for k, v in kw.items()), kw
    for kw in (dict(tile_n=48), dict(split_k=3), dict(cta_pair=2, split_k=2), dict(cta_pair=2, tile_n=64), dict(cta_pair=2, tile_m=128), dict(reduce=1),
               dict(reduce=2, split_k=1), dict(tile_k=32), dict(stages=1), dict(stages=9), dict(cta_pair=3), dict(tile_m=64)):
        i = pkg.query(p, pkg.make_cfg(variant=6, **kw))
        assert not i.supported and i.reason, kw
    for a in [(2, 64, 14, 14, 64, 1, 1, 1, 1, 0, 0), (2, 64, 40, 40, 64, 3, 3, 3, 3, 1, 1), (2, 64, 14, 14, 64, 3, 3, 1, 1, 3, 1), (2, 64, 3, 3, 64, 3, 3, 1, 1, 1, 1),
              (2, 64, 30, 30, 64, 9, 9, 1, 1, 4, 4)]:
        assert not pkg.query(P(pkg, *a, precision=pkg.FP16), pkg.make_cfg(variant=6)).supported, a
    assert not pkg.query(P(pkg, 1, 64, 14, 14, 64, 3, 3, 1, 1, 1, 1, precision=pkg.TF32), pkg.make_cfg(variant=6, cta_pair=2)).supported
    assert not pkg.query(P(pkg, 1, 64, 14, 14, 64, 3, 3, 1, 1, 1, 1, precision=pkg.FP32), pkg.make_cfg(variant=6)).supported


def test_halo_variant_leaves_outputs_beyond_its_row_offsets(pkg):
    """Rows of a channel-contiguous output are addressed by 32-bit counts of 16-byte cells: 64 GiB and no more."""
    flags = pkg.FLAG_INPUT_NHWC | pkg.FLAG_OUTPUT_NHWC | pkg.FLAG_WEIGHTS_PREPACKED
    for o, flag, fits in [(16, flags, True), (24, flags, True), (32, flags, False), (64, flags, False), (64, pkg.FLAG_INPUT_NHWC | pkg.FLAG_WEIGHTS_PREPACKED, True)]:
        p = P(pkg, 65536, 16, 128, 128, o, 3, 3, 1, 1, 1, 1, precision=pkg.FP16, has_bias=True, relu=True, flags=flag)
        i = pkg.query(p, pkg.make_cfg(variant=6))
        assert bool(i.supported) == fits, o
        auto = pkg.query(p)
        assert auto.supported and (fits or auto.cfg.variant != 6)


def test_channels_of_a_copy_are_padded_to_whole_slabs_where_that_is_cheap(pkg):
    """At most a third (15 % for more than nine taps): whole slabs of 64.  More, or a tensor that is read in place: multiples of 16."""
    cases = [((3, 605, 29, 29, 256, 1, 1, 1, 1, 0, 0), 0, 640), ((2, 288, 11, 86, 64, 1, 1, 2, 2, 0, 0), 0, 320), ((4, 240, 14, 14, 64, 3, 3, 3, 3, 1, 1), 0, 256),
             ((4, 144, 14, 14, 64, 3, 3, 3, 3, 1, 1), 0, 192), ((4, 80, 14, 14, 64, 3, 3, 3, 3, 1, 1), 0, 80), ((4, 48, 14, 14, 64, 3, 3, 3, 3, 1, 1), 0, 64),
             ((4, 144, 14, 14, 64, 5, 5, 3, 3, 2, 2), 0, 144), ((4, 240, 14, 14, 64, 5, 5, 3, 3, 2, 2), 0, 256),
             ((4, 240, 14, 14, 64, 3, 3, 3, 3, 1, 1), pkg.FLAG_INPUT_NHWC, 240),
             ((9, 240, 54, 8, 64, 1, 1, 1, 1, 0, 0), 0, 240), ((9, 240, 54, 8, 64, 1, 1, 1, 1, 0, 0), pkg.FLAG_WEIGHTS_PREPACKED, 256),
             ((9, 245, 54, 8, 64, 1, 1, 1, 1, 0, 0), 0, 256)]
    for args, flags, padded in cases:
        p = P(pkg, *args, precision=pkg.FP16, has_bias=True, relu=True, flags=flags)
        i = pkg.query(p)
        assert i.supported and i.padded_channels == padded, (args, flags, i.padded_channels)
    # the halo kernel, whose steps cost more, pads its blocks by up to 15 %
    for c, padded in ((240, 256), (144, 144)):
        assert pkg.query(P(pkg, 4, c, 14, 14, 64, 3, 3, 1, 1, 1, 1, precision=pkg.FP16), pkg.make_cfg(variant=6)).padded_channels == padded
    # FP8 values count half, TF32 values twice
    assert pkg.query(P(pkg, 4, 480, 14, 14, 64, 3, 3, 3, 3, 1, 1, precision=pkg.FP8_E4M3)).padded_channels == 512
    assert pkg.query(P(pkg, 4, 120, 14, 14, 64, 3, 3, 3, 3, 1, 1, precision=pkg.TF32)).padded_channels == 128
    # read in place: one launch
    assert pkg.query(P(pkg, 9, 240, 54, 8, 64, 1, 1, precision=pkg.FP16)).launches == 1
