"""The halo-tile convolution kernel at the sizes where the padded grid, the phases of a stride, the channel tails, the split of
the reduction, the CTA pairs and the row-wise output can go wrong.  Every plan asks for it by its variant, which is refused where
it cannot run, and the plan's own report says which tiles, pairs and splits were taken."""
import numpy as np
import pytest

import gpu_util as gu

pytestmark = pytest.mark.gpu

HALO = 6  # cfg.variant of the kernel

# shape (batch, channels, h, w, filters, r, s, stride_h, stride_w, pad_h, pad_w), input nhwc, output nhwc, residual [, fields asked for]
CASES = [
    ((2, 64, 14, 14, 64, 3, 3, 1, 1, 1, 1), False, False, False),     # neighbouring images share their padding rows
    ((3, 144, 9, 11, 200, 3, 3, 1, 1, 1, 1), True, True, True),       # 64 + 64 + 16 channels; two channel tiles, 16-byte output cells
    ((2, 130, 9, 9, 131, 3, 3, 1, 1, 1, 1), False, True, True),       # odd output channel count: single-channel row stores
    ((1, 80, 21, 7, 70, 5, 5, 1, 1, 2, 2), True, True, False),        # 5x5; output rows of 140 bytes: channel pairs
    ((2, 64, 17, 23, 96, 3, 5, 2, 1, 1, 2), False, False, True),      # two phases (rows only)
    ((2, 96, 28, 28, 128, 3, 3, 2, 2, 1, 1), True, True, True),       # four phases
    ((1, 64, 12, 12, 32, 4, 2, 1, 1, 0, 1), False, False, False),     # even extents, no vertical padding
    ((1, 512, 7, 7, 512, 3, 3, 1, 1, 1, 1), False, False, True),      # few pixels: the reduction is split over a cluster
    ((1, 320, 8, 8, 40, 5, 5, 1, 1, 2, 2), True, True, False),        # the same with a channel tail
    ((12, 64, 56, 56, 64, 3, 3, 1, 1, 1, 1), True, True, False),      # several tiles per CTA, weights kept in shared memory
    ((32, 128, 28, 28, 256, 3, 3, 1, 1, 1, 1), True, True, True),     # many tiles per CTA
    ((40, 192, 14, 14, 136, 3, 3, 1, 1, 1, 1), False, False, False),  # pairs with a channel tail
    ((2, 32, 100, 6, 24, 3, 3, 1, 1, 1, 1), False, False, False),     # narrow rows: many small boxes
    ((1, 16, 5, 120, 16, 3, 3, 1, 1, 1, 1), True, True, False),       # wide rows
    # 256 columns (all of tensor memory, two chunks per worker warp): single CTAs ..
    ((3, 80, 19, 21, 300, 3, 3, 1, 1, 1, 1), True, True, True, dict(tile_n=256, cta_pair=1)),     # 64 + 16 channels, 256 + 44 columns, 16-byte cells
    ((8, 64, 31, 31, 512, 3, 3, 1, 1, 1, 1), False, False, False, dict(tile_n=256, cta_pair=1)),
    ((2, 64, 17, 23, 290, 3, 3, 2, 2, 1, 1), False, False, True, dict(tile_n=256, cta_pair=1)),
    # .. pairs ..
    ((3, 144, 20, 22, 328, 3, 3, 1, 1, 1, 1), False, False, True, dict(tile_n=256, cta_pair=2)),
    ((3, 128, 21, 19, 264, 3, 3, 1, 1, 1, 1), True, True, True, dict(tile_n=256, cta_pair=2)),
    ((2, 96, 40, 40, 256, 1, 3, 1, 1, 0, 1), False, True, False, dict(tile_n=256, cta_pair=2)),
    # .. and a cluster
    ((1, 256, 14, 14, 512, 3, 3, 1, 1, 1, 1), False, False, False, dict(tile_n=256, split_k=4)),
    # 128 columns: single CTAs, pairs whose last tile has a peer without pixels, clusters
    ((4, 64, 30, 30, 136, 3, 3, 1, 1, 1, 1), True, True, False, dict(tile_n=128, cta_pair=1)),
    ((9, 64, 7, 7, 130, 3, 3, 1, 1, 1, 1), True, True, True, dict(tile_n=128, cta_pair=2)),       # 576 padded rows: 2 x 256 + 64
    ((1, 256, 14, 14, 200, 3, 3, 1, 1, 1, 1), False, False, True, dict(tile_n=128, split_k=4)),
    ((1, 144, 9, 9, 100, 3, 3, 1, 1, 1, 1), True, True, True, dict(tile_n=128, split_k=2)),
    # 64 and 32 columns in clusters of two, four and eight
    ((1, 128, 10, 10, 60, 3, 3, 1, 1, 1, 1), True, True, False, dict(tile_n=64, split_k=2)),
    ((1, 512, 7, 7, 70, 3, 3, 1, 1, 1, 1), False, False, True, dict(tile_n=64, split_k=4)),
    ((1, 512, 8, 8, 64, 3, 3, 2, 2, 1, 1), True, True, True, dict(tile_n=64, split_k=8)),
    ((2, 192, 9, 9, 33, 5, 5, 1, 1, 2, 2), False, True, False, dict(tile_n=32, split_k=2, stages=3)),
]


@pytest.mark.parametrize("case", range(len(CASES)))
def test_halo_tiles(pkg, orc, oracle, case):
    import torch
    args, in_nhwc, out_nhwc, with_res, *asked = CASES[case]
    asked = asked[0] if asked else {}
    prec = orc.FP16 if case % 2 == 0 else orc.BF16
    relu = case % 3 != 0
    p_lin = orc.Problem.P(*args, precision=prec, bias=True, relu=False)
    p = orc.Problem.P(*args, precision=prec, bias=True, relu=relu)
    x, w, b = oracle.make_conv_data(p, 9100 + case, case % 4)
    lin, scale = oracle.conv2d(p_lin, x, w, b)
    res = oracle.quantize(prec, oracle.rng(9200 + case).uniform(-1, 1, lin.size)).reshape(lin.shape)
    ref = lin.astype(np.float64) + (res if with_res else 0.0)
    ref = (np.maximum(ref, 0.0) if relu else ref).astype(np.float32)
    if with_res:
        scale = (scale.astype(np.float64) + np.abs(res)).astype(np.float32)
    nhwc = lambda a: np.ascontiguousarray(a.transpose(0, 2, 3, 1))
    flags = (pkg.FLAG_INPUT_NHWC if in_nhwc else 0) | (pkg.FLAG_OUTPUT_NHWC if out_nhwc else 0) | (pkg.FLAG_RESIDUAL if with_res else 0)
    plan = pkg.ConvPlan(gu.pkg_problem(pkg, p, flags), pkg.make_cfg(variant=HALO, **asked))
    assert plan.info.cfg.variant == HALO and all(getattr(plan.info.cfg, k) == v for k, v in asked.items())
    stream = torch.cuda.current_stream().cuda_stream
    yoff = 1 if case % 4 == 1 else 0            # (row stores instead of 16-byte cells)
    tx, px = gu.to_device_storage(oracle, prec, nhwc(x) if in_nhwc else x)
    tw, pw = gu.to_device_storage(oracle, prec, w)
    tb, pb = gu.to_device_storage(oracle, prec, b)
    tr, pr = gu.to_device_storage(oracle, prec, nhwc(res) if out_nhwc else res)
    out = gu.OutBuf(prec, int(np.prod(p.y_shape)), yoff)
    ws = gu.Workspace(plan.workspace_bytes)
    for _ in range(2):
        if with_res:
            plan.launch_fused(px, pw, pb, pr, out.ptr, ws.ptr if plan.workspace_bytes else None, plan.workspace_bytes, stream)
        else:
            plan.launch(px, pw, pb, out.ptr, ws.ptr if plan.workspace_bytes else None, plan.workspace_bytes, stream)
    torch.cuda.synchronize()
    assert plan.device_status() == 0
    ws.check_guard()
    got = out.read(oracle)
    B, O, P, Q = p.y_shape
    got = np.ascontiguousarray(got.reshape(B, P, Q, O).transpose(0, 3, 1, 2)) if out_nhwc else got.reshape(p.y_shape)
    m = oracle.compare(p, got, ref, scale)   # the reference's scale-aware policy: rounding of sums of this length
    assert m.passed(), f"halo case {case}: {m.summary()}"


@pytest.mark.parametrize("prec_name", ["tf32", "fp8"])
def test_halo_tiles_of_other_widths(pkg, orc, oracle, prec_name):
    """4-byte and 1-byte operands through the same tiles (32 and 128 values per row), channel tails included."""
    import torch
    from oracle import oracle as orc_mod
    cfg = pkg.make_cfg(variant=HALO)
    for k, args in enumerate([(2, 72, 13, 9, 100, 3, 3, 1, 1, 1, 1), (3, 200, 14, 14, 64, 5, 5, 2, 2, 2, 2), (24, 96, 28, 28, 128, 3, 3, 1, 1, 1, 1)]):
        if prec_name == "tf32":
            p = orc.Problem.P(*args, precision=orc.TF32, bias=True, relu=True)
            x, w, b = oracle.make_conv_data(p, 9300 + k, k)
            ref, scale = oracle.conv2d(p, x, w, b)
            got, plan, _ = gu.run_conv(pkg, oracle, p, x, w, b, cfg=cfg)
        else:
            p = orc.Problem.P(*args, precision=orc.FP16, bias=True, relu=True)
            x, w, b = oracle.make_conv_data(p, 9300 + k, k)
            x, w = orc_mod.e4m3_quantize(x), orc_mod.e4m3_quantize(w)
            ref, scale = oracle.conv2d(p, x, w, b)
            plan = pkg.ConvPlan(pkg.ConvProblem(*args, 1, 1, 1, pkg.FP8_E4M3, True, True, 0), cfg)
            tx = torch.from_numpy(orc_mod.e4m3_bits(x).ravel()).cuda()
            tw = torch.from_numpy(orc_mod.e4m3_bits(w).ravel()).cuda()
            tb = torch.from_numpy(np.ascontiguousarray(b, dtype=np.float32)).cuda()
            out = gu.OutBuf(orc.FP16, int(np.prod(p.y_shape)))
            ws = gu.Workspace(plan.workspace_bytes)
            plan.launch(tx.data_ptr(), tw.data_ptr(), tb.data_ptr(), out.ptr, ws.ptr, plan.workspace_bytes, torch.cuda.current_stream().cuda_stream)
            torch.cuda.synchronize()
            assert plan.device_status() == 0
            ws.check_guard()
            got = out.read(oracle).reshape(p.y_shape)
        assert plan.info.cfg.variant == HALO
        m = oracle.compare(p, got, ref, scale)
        assert m.passed(), f"{prec_name} {args}: {m.summary()}"


def test_halo_waits_run_out_and_report(pkg, orc, oracle):
    """The injected stall of test_conv_gpu.py on this kernel: every wait gives up, the kernel ends by itself and reports."""
    import torch
    cfg = pkg.make_cfg(variant=HALO)
    p = orc.Problem.P(4, 64, 14, 14, 64, 3, 3, 1, 1, 1, 1, precision=orc.FP16, bias=True, relu=True)
    x, w, b = oracle.make_conv_data(p, 31, 1)
    ref, scale = oracle.conv2d(p, x, w, b)
    for roles, expect in ((1, 2), (2, 4)):
        plan = pkg.ConvPlan(gu.pkg_problem(pkg, p), cfg)
        assert plan.info.cfg.variant == HALO
        plan.inject_stall(roles, 2_000_000)
        tx, px = gu.to_device_storage(oracle, p.precision, x)
        tw, pw = gu.to_device_storage(oracle, p.precision, w)
        tb, pb = gu.to_device_storage(oracle, p.precision, b)
        out = gu.OutBuf(p.precision, int(np.prod(p.y_shape)))
        ws = gu.Workspace(plan.workspace_bytes)
        plan.launch(px, pw, pb, out.ptr, ws.ptr, plan.workspace_bytes, torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        assert plan.device_status() & expect == expect
        out.read(oracle)
        plan.close()
    got, _, _ = gu.run_conv(pkg, oracle, p, x, w, b, cfg=cfg)
    assert oracle.compare(p, got, ref, scale).passed()
