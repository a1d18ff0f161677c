"""First layers over images (few channels, horizontal stride 2), which one kernel reads straight from the NCHW tensor: every channel
count, windows of two, four and eight positions, groups whose last rows or columns fill no tile, outputs wider than a tile, several
tiles of output channels, vertical strides of 1 to 3, both output layouts with their alignments, a residual, and converted weights."""
import numpy as np
import pytest

import gpu_util as gu

pytestmark = pytest.mark.gpu

CASES = [
    # shape, channel-contiguous output, residual, prepacked weights, offsets of x and of y / residual in elements
    ((2, 3, 64, 64, 64, 7, 7, 2, 2, 3, 3), False, False, False, 0, 0),
    ((2, 3, 64, 64, 64, 7, 7, 2, 2, 3, 3), True, True, True, 0, 0),
    ((3, 3, 37, 254, 64, 7, 7, 2, 2, 3, 3), False, True, False, 1, 1),     # 127 columns: one tile and its windows beyond it
    ((2, 3, 41, 256, 64, 7, 7, 2, 2, 3, 3), True, False, False, 0, 0),     # 128 columns
    ((1, 3, 30, 258, 72, 7, 7, 2, 2, 3, 3), True, False, True, 0, 0),      # 129 columns, a second tile of channels with 8
    ((1, 3, 23, 600, 40, 7, 7, 2, 2, 3, 3), False, False, False, 0, 0),    # 300 columns
    ((1, 4, 50, 46, 30, 5, 7, 2, 2, 2, 3), True, True, False, 0, 0),       # channels no multiple of 8: stored one pixel per lane
    ((1, 4, 50, 46, 136, 5, 7, 1, 2, 2, 3), True, True, False, 1, 4),      # stride 1 down, y off its alignment
    ((2, 2, 40, 18, 33, 7, 7, 3, 2, 3, 3), False, True, True, 0, 1),       # stride 3 down, 9 columns
    ((2, 1, 19, 34, 16, 3, 3, 2, 2, 1, 1), False, False, False, 0, 0),     # windows of two positions
    ((2, 1, 19, 34, 64, 1, 15, 2, 2, 0, 7), True, False, True, 0, 0),     # windows of eight positions, one filter row
    ((40, 3, 128, 128, 64, 7, 7, 2, 2, 3, 3), True, False, False, 0, 0),   # several groups per CTA
    ((1, 3, 7, 6, 64, 7, 7, 2, 2, 0, 2), False, False, False, 0, 0),       # one output row
]


@pytest.mark.parametrize("case", range(len(CASES)))
@pytest.mark.parametrize("prec_name", ["fp16", "bf16"])
def test_image_layers(pkg, orc, oracle, case, prec_name):
    import torch
    args, out_nhwc, with_res, prepacked, xoff, yoff = CASES[case]
    prec = orc.FP16 if prec_name == "fp16" else orc.BF16
    relu = case % 3 != 1
    p_lin = orc.Problem.P(*args, precision=prec, bias=True, relu=False)
    p = orc.Problem.P(*args, precision=prec, bias=True, relu=relu)
    x, w, b = oracle.make_conv_data(p, 7000 + case, case % 4)
    lin, scale = oracle.conv2d(p_lin, x, w, b)
    res = oracle.quantize(prec, oracle.rng(7100 + case).uniform(-1, 1, lin.size)).reshape(lin.shape) if with_res else np.zeros_like(lin)
    ref = lin.astype(np.float64) + res
    ref = (np.maximum(ref, 0.0) if relu else ref).astype(np.float32)
    scale = (scale.astype(np.float64) + np.abs(res)).astype(np.float32)
    nhwc = (lambda a: np.ascontiguousarray(a.transpose(0, 2, 3, 1))) if out_nhwc else (lambda a: a)
    flags = (pkg.FLAG_OUTPUT_NHWC if out_nhwc else 0) | (pkg.FLAG_RESIDUAL if with_res else 0) | (pkg.FLAG_WEIGHTS_PREPACKED if prepacked else 0)
    plan = pkg.ConvPlan(gu.pkg_problem(pkg, p, flags))
    assert plan.info.variant == 5 and plan.info.launches == 1
    stream = torch.cuda.current_stream().cuda_stream
    tx, px = gu.to_device_storage(oracle, prec, x, xoff)
    tw, pw = gu.to_device_storage(oracle, prec, w)
    tb, pb = gu.to_device_storage(oracle, prec, b)
    if prepacked:
        packed = torch.empty(plan.prepacked_weight_bytes, dtype=torch.uint8, device="cuda")
        plan.prepack_weights(pw, packed.data_ptr(), stream)
        pw = packed.data_ptr()
    tr, pr = gu.to_device_storage(oracle, prec, nhwc(res), yoff)
    ws = gu.Workspace(plan.workspace_bytes)
    out = gu.OutBuf(prec, int(np.prod(p.y_shape)), yoff)
    if with_res:
        plan.launch_fused(px, pw, pb, pr, out.ptr, ws.ptr, plan.workspace_bytes, stream)
    else:
        plan.launch(px, pw, pb, out.ptr, ws.ptr, plan.workspace_bytes, stream)
    torch.cuda.synchronize()
    assert plan.device_status() == 0
    ws.check_guard()
    got = out.read(oracle)
    B, O, P, Q = p.y_shape
    got = np.ascontiguousarray(got.reshape(B, P, Q, O).transpose(0, 3, 1, 2)) if out_nhwc else got.reshape(p.y_shape)
    m = oracle.compare(p, got, ref, scale)   # the reference's scale-aware policy: rounding of sums of this length
    assert m.passed(), f"case {case} {prec_name}: {m.summary()}"


@pytest.mark.parametrize("roles", [1, 2, 3])
def test_expired_waits_are_reported(pkg, orc, oracle, roles):
    p = orc.Problem.P(2, 3, 40, 40, 64, 7, 7, 2, 2, 3, 3, precision=orc.FP16, bias=True, relu=True)
    x, w, b = oracle.make_conv_data(p, 7200, 1)
    plan = pkg.ConvPlan(gu.pkg_problem(pkg, p))
    plan.inject_stall(roles, 2_000_000)  # about a millisecond per wait
    with pytest.raises(AssertionError, match="bounded device-side wait"):
        gu.run_conv(pkg, oracle, p, x, w, b, plan=plan)
    plan.inject_stall(0, 0)
    ref, scale = oracle.conv2d(p, x, w, b)
    got, _, _ = gu.run_conv(pkg, oracle, p, x, w, b, plan=pkg.ConvPlan(gu.pkg_problem(pkg, p)))
    m = oracle.compare(p, got, ref, scale)
    assert m.passed(), m.summary()


def test_plans_of_other_sizes_leave_a_plan_alone(pkg, orc, oracle):
    """A plan keeps working when plans and allocation-free calls of the same window width that ask for less shared memory come after it
    (600 columns: 107,264 bytes; 64: 40,704)."""
    def problem(args, seed):
        p = orc.Problem.P(*args, precision=orc.FP16, bias=True, relu=True)
        x, w, b = oracle.make_conv_data(p, seed, 1)
        return p, x, w, b, oracle.conv2d(p, x, w, b)
    large = problem((1, 3, 23, 600, 40, 7, 7, 2, 2, 3, 3), 7300)
    small = problem((1, 3, 64, 64, 64, 7, 7, 2, 2, 3, 3), 7301)
    plans = [pkg.ConvPlan(gu.pkg_problem(pkg, large[0])), pkg.ConvPlan(gu.pkg_problem(pkg, small[0]))]

    def check(plan, data):
        p, x, w, b, (ref, scale) = data
        got, _, _ = gu.run_conv(pkg, oracle, p, x, w, b, plan=plan)
        m = oracle.compare(p, got, ref, scale)
        assert m.passed(), m.summary()
    check(plans[0], large)
    check(plans[1], small)
    check(plans[0], large)
    p, x, w, b, _ = small
    bufs = [gu.to_device_storage(oracle, p.precision, a) for a in (x, w, b)]
    out = gu.OutBuf(p.precision, int(np.prod(p.y_shape)))
    pkg.conv_forward_static(gu.pkg_problem(pkg, p), bufs[0][1], bufs[1][1], bufs[2][1], out.ptr, 0)
    assert pkg.conv_static_status(0) == 0
    check(plans[0], large)


@pytest.mark.parametrize("static", [False, True])
def test_no_workspace(pkg, orc, oracle, static):
    """The image is read in place: no scratch, so the allocation-free call takes layers whose gathered copy (32 MB here) would not fit
    its own."""
    import torch
    p = orc.Problem.P(1, 1, 4000, 1000, 2, 3, 3, 2, 2, 1, 1, precision=orc.FP16, bias=True, relu=True)
    x, w, b = oracle.make_conv_data(p, 7400, 1)
    ref, scale = oracle.conv2d(p, x, w, b)
    plan = pkg.ConvPlan(gu.pkg_problem(pkg, p))
    assert plan.workspace_bytes == 0
    bufs = [gu.to_device_storage(oracle, p.precision, a) for a in (x, w, b)]
    out = gu.OutBuf(p.precision, int(np.prod(p.y_shape)))
    if static:
        pkg.conv_forward_static(gu.pkg_problem(pkg, p), bufs[0][1], bufs[1][1], bufs[2][1], out.ptr, 0)
        assert pkg.conv_static_status(0) == 0
    else:
        plan.launch(bufs[0][1], bufs[1][1], bufs[2][1], out.ptr, None, 0, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert plan.device_status() == 0
    m = oracle.compare(p, out.read(oracle).reshape(p.y_shape), ref, scale)
    assert m.passed(), m.summary()


@pytest.mark.parametrize("cfg", [dict(tile_n=32), dict(tile_n=128), dict(tile_n=256), dict(tile_m=256, tile_n=64), dict(tile_n=64, stages=4), dict(tile_k=16)])
@pytest.mark.parametrize("args", [(2, 3, 64, 64, 64, 7, 7, 2, 2, 3, 3), (1, 3, 30, 258, 72, 7, 7, 2, 2, 3, 3)])
@pytest.mark.parametrize("nhwc", [False, True])
def test_forms_that_gather_first(pkg, orc, oracle, cfg, args, nhwc):
    """Tiles, stages and slabs other than the image kernel's, asked for: overlapping windows read from the copy of the image."""
    p = orc.Problem.P(*args, precision=orc.BF16, bias=True, relu=True)
    x, w, b = oracle.make_conv_data(p, 7500, 2)
    ref, scale = oracle.conv2d(p, x, w, b)
    flags = pkg.FLAG_OUTPUT_NHWC if nhwc else 0
    plan = pkg.ConvPlan(gu.pkg_problem(pkg, p, flags), pkg.make_cfg(**cfg))
    assert plan.info.launches == 2 and all(getattr(plan.info.cfg, k) == v for k, v in cfg.items())
    got, _, _ = gu.run_conv(pkg, oracle, p, x, w, b, flags=flags, plan=plan)
    if nhwc:
        B, O, P, Q = p.y_shape
        got = np.ascontiguousarray(got.reshape(B, P, Q, O).transpose(0, 3, 1, 2))
    m = oracle.compare(p, got, ref, scale)
    assert m.passed(), m.summary()
