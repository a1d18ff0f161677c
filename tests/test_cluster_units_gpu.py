"""Split-K inside clusters where a CTA finishes 8 or 16 columns of a tile instead of whole chunks of 32: every pair of tile and split,
channel tails inside a unit of eight, both layouts with and without a residual, outputs off their alignment."""
import numpy as np
import pytest

import gpu_util as gu

pytestmark = pytest.mark.gpu

# tile_n, split: units of 8 columns that a CTA finishes: 1, 2, 1, 2, 4
POINTS = [(32, 4), (32, 2), (64, 8), (64, 4), (128, 4)]


def _cfg(pkg, p, tile_n, split, flags=0):
    """The point with every field set, as a query reports it (left to the library, narrow shares are its own choice)."""
    auto = pkg.query(gu.pkg_problem(pkg, p, flags)).cfg
    return pkg.make_cfg(tile_m=128, tile_n=tile_n, tile_k=auto.tile_k, stages=4, split_k=split, variant=1, reduce=2, cta_pair=1)


@pytest.mark.parametrize("tile_n,split", POINTS)
@pytest.mark.parametrize("filters,off", [(64, 0), (70, 0), (61, 1), (129, 3)])
@pytest.mark.parametrize("prec_name", ["fp16", "bf16", "tf32"])
def test_nchw(pkg, orc, oracle, tile_n, split, filters, off, prec_name):
    prec = {"fp16": orc.FP16, "bf16": orc.BF16, "tf32": orc.TF32}[prec_name]
    p = orc.Problem.P(2, 256, 9, 7, filters, 3, 3, 1, 1, 1, 1, precision=prec, bias=filters != 70, relu=filters % 2 == 0)
    x, w, b = oracle.make_conv_data(p, 40 + tile_n + split, filters % 4)
    ref, scale = oracle.conv2d(p, x, w, b if p.has_bias else None)
    got, plan, out = gu.run_conv(pkg, oracle, p, x, w, b if p.has_bias else None, cfg=_cfg(pkg, p, tile_n, split), offsets=(0, 0, off))
    c = plan.info.cfg
    assert (c.tile_n, c.split_k, c.reduce) == (tile_n, split, 2)
    m = oracle.compare(p, got, ref, scale)   # the reference's policy: rounding of sums of this length
    assert m.passed(), m.summary()
    again, _, out2 = gu.run_conv(pkg, oracle, p, x, w, b if p.has_bias else None, plan=plan, offsets=(0, 0, off))
    assert np.array_equal(out.raw_bits(), out2.raw_bits())


# channels 80 at tile_k 64: the last slab of a tap is partial (kernels of their own)
@pytest.mark.parametrize("tile_k,channels,stages", [(16, 16, 8), (32, 32, 4), (64, 128, 4), (64, 80, 4)])
@pytest.mark.parametrize("tile_n", [32, 64, 128, 256])
@pytest.mark.parametrize("split", [2, 4])
def test_every_kernel(pkg, orc, oracle, tile_k, channels, stages, tile_n, split):
    p = orc.Problem.P(2, channels, 9, 8, 150, 4, 4, 1, 1, 0, 0, precision=orc.FP16, bias=True, relu=True)
    x, w, b = oracle.make_conv_data(p, 7 + tile_n + split, 1)
    ref, scale = oracle.conv2d(p, x, w, b)
    cfg = pkg.make_cfg(tile_m=128, tile_n=tile_n, tile_k=tile_k, stages=stages, split_k=split, variant=1, reduce=2, cta_pair=1)
    got, plan, _ = gu.run_conv(pkg, oracle, p, x, w, b, cfg=cfg)
    c = plan.info.cfg
    assert (c.tile_n, c.tile_k, c.split_k, c.reduce) == (tile_n, tile_k, split, 2)
    m = oracle.compare(p, got, ref, scale)
    assert m.passed(), m.summary()


@pytest.mark.parametrize("tile_n,split", POINTS)
@pytest.mark.parametrize("filters,off", [(64, 0), (72, 0), (72, 1), (61, 0)])
@pytest.mark.parametrize("with_res", [False, True])
@pytest.mark.parametrize("nhwc", [False, True])
def test_layouts_and_residual(pkg, orc, oracle, tile_n, split, filters, off, with_res, nhwc):
    import torch
    prec = orc.FP16 if (tile_n + split) % 8 else orc.BF16
    args = (3, 208, 6, 11, filters, 3, 3, 1, 1, 1, 1)
    p_lin = orc.Problem.P(*args, precision=prec, bias=True, relu=False)
    p = orc.Problem.P(*args, precision=prec, bias=True, relu=True)
    x, w, b = oracle.make_conv_data(p, 90 + tile_n, split % 4)
    lin, scale = oracle.conv2d(p_lin, x, w, b)
    res = oracle.quantize(prec, oracle.rng(71).uniform(-1, 1, lin.size)).reshape(lin.shape) if with_res else np.zeros_like(lin)
    ref = np.maximum(lin.astype(np.float64) + res, 0.0).astype(np.float32)
    scale = (scale.astype(np.float64) + np.abs(res)).astype(np.float32)
    swap = (lambda a: np.ascontiguousarray(a.transpose(0, 2, 3, 1))) if nhwc else (lambda a: a)
    flags = (pkg.FLAG_INPUT_NHWC | pkg.FLAG_OUTPUT_NHWC if nhwc else 0) | (pkg.FLAG_RESIDUAL if with_res else 0)
    plan = pkg.ConvPlan(gu.pkg_problem(pkg, p, flags), _cfg(pkg, p, tile_n, split, flags))
    assert (plan.info.cfg.tile_n, plan.info.cfg.split_k, plan.info.cfg.reduce) == (tile_n, split, 2)
    stream = torch.cuda.current_stream().cuda_stream
    tx, px = gu.to_device_storage(oracle, prec, swap(x))
    tw, pw = gu.to_device_storage(oracle, prec, w)
    tb, pb = gu.to_device_storage(oracle, prec, b)
    tr, pr = gu.to_device_storage(oracle, prec, swap(res), off)
    ws = gu.Workspace(plan.workspace_bytes)
    out = gu.OutBuf(prec, int(np.prod(p.y_shape)), off)
    if with_res:
        plan.launch_fused(px, pw, pb, pr, out.ptr, ws.ptr, plan.workspace_bytes, stream)
    else:
        plan.launch(px, pw, pb, out.ptr, ws.ptr, plan.workspace_bytes, stream)
    torch.cuda.synchronize()
    assert plan.device_status() == 0
    ws.check_guard()
    B, O, P, Q = p.y_shape
    got = out.read(oracle)
    got = np.ascontiguousarray(got.reshape(B, P, Q, O).transpose(0, 3, 1, 2)) if nhwc else got.reshape(p.y_shape)
    m = oracle.compare(p, got, ref, scale)
    assert m.passed(), m.summary()


# Planes of 200 pixels in boxes of 64: the last box of an image has eight, so warps hold lanes with a pixel and lanes without one while
# they go from unit to unit (tile_n / split / 8 units of the CTA, two or four warps of a lane quarter).
@pytest.mark.parametrize("tile_n,split", [(64, 2), (64, 4), (128, 2), (128, 8), (256, 2), (256, 4), (256, 8)])
@pytest.mark.parametrize("variant,nhwc_out", [(2, False), (2, True), (4, False)])
@pytest.mark.parametrize("with_res", [False, True])
def test_lanes_without_a_pixel(pkg, orc, oracle, tile_n, split, variant, nhwc_out, with_res):
    import torch
    prec = orc.BF16 if split == 4 else orc.FP16
    args = (3, 1024, 10, 20, 139, 1, 1, 1, 1, 0, 0)
    p_lin = orc.Problem.P(*args, precision=prec, bias=True, relu=False)
    p = orc.Problem.P(*args, precision=prec, bias=True, relu=True)
    x, w, b = oracle.make_conv_data(p, 17 + tile_n + split, variant % 4)
    lin, scale = oracle.conv2d(p_lin, x, w, b)
    res = oracle.quantize(prec, oracle.rng(5).uniform(-1, 1, lin.size)).reshape(lin.shape) if with_res else np.zeros_like(lin)
    ref = np.maximum(lin.astype(np.float64) + res, 0.0).astype(np.float32)
    scale = (scale.astype(np.float64) + np.abs(res)).astype(np.float32)
    swap = (lambda a: np.ascontiguousarray(a.transpose(0, 2, 3, 1))) if nhwc_out else (lambda a: a)
    flags = (pkg.FLAG_OUTPUT_NHWC if nhwc_out else 0) | (pkg.FLAG_RESIDUAL if with_res else 0)
    cfg = pkg.make_cfg(tile_m=128, tile_n=tile_n, tile_k=64, stages=4, split_k=split, variant=variant, reduce=2, cta_pair=1)
    plan = pkg.ConvPlan(gu.pkg_problem(pkg, p, flags), cfg)
    c = plan.info.cfg
    assert (c.variant, c.tile_n, c.split_k, c.reduce) == (variant, tile_n, split, 2)
    stream = torch.cuda.current_stream().cuda_stream
    tx, px = gu.to_device_storage(oracle, prec, x)
    tw, pw = gu.to_device_storage(oracle, prec, w)
    tb, pb = gu.to_device_storage(oracle, prec, b)
    tr, pr = gu.to_device_storage(oracle, prec, swap(res))
    ws = gu.Workspace(plan.workspace_bytes)
    out = gu.OutBuf(prec, int(np.prod(p.y_shape)))
    if with_res:
        plan.launch_fused(px, pw, pb, pr, out.ptr, ws.ptr, plan.workspace_bytes, stream)
    else:
        plan.launch(px, pw, pb, out.ptr, ws.ptr, plan.workspace_bytes, stream)
    torch.cuda.synchronize()
    assert plan.device_status() == 0
    ws.check_guard()
    B, O, P, Q = p.y_shape
    got = out.read(oracle)
    got = np.ascontiguousarray(got.reshape(B, P, Q, O).transpose(0, 3, 1, 2)) if nhwc_out else got.reshape(p.y_shape)
    m = oracle.compare(p, got, ref, scale)   # one rounding to the stored type of an FP32 sum of 1024 products, bias and residual
    assert m.passed(), m.summary()


@pytest.mark.parametrize("tile_n,split", [(32, 4), (64, 4), (64, 8), (128, 8)])   # what plans of FP8 layers take by themselves
@pytest.mark.parametrize("kernel", [3, 1])
@pytest.mark.parametrize("filters", [64, 77])
def test_fp8(pkg, orc, oracle, tile_n, split, kernel, filters):
    import torch
    from oracle import oracle as orc_mod
    args = (2, 2048 if kernel == 1 else 512, 9, 7, filters, kernel, kernel, 1, 1, kernel // 2, kernel // 2)
    p = orc.Problem.P(*args, precision=orc.FP16, bias=True, relu=True)   # every E4M3 value is an FP16 value
    x, w, b = oracle.make_conv_data(p, 60 + tile_n + split, kernel)
    x, w = orc_mod.e4m3_quantize(x), orc_mod.e4m3_quantize(w)
    ref, scale = oracle.conv2d(p, x, w, b)
    cfg = pkg.make_cfg(tile_m=128, tile_n=tile_n, tile_k=128, stages=4, split_k=split, variant=4 if kernel == 1 else 1, reduce=2, cta_pair=1)
    plan = pkg.ConvPlan(pkg.ConvProblem(*args, precision=pkg.FP8_E4M3, has_bias=True, relu=True), cfg)
    c = plan.info.cfg
    assert (c.tile_n, c.split_k, c.reduce) == (tile_n, split, 2)
    tx, tw, tb = [torch.from_numpy(a).cuda() for a in (orc_mod.e4m3_bits(x).ravel(), orc_mod.e4m3_bits(w).ravel(), np.ascontiguousarray(b, np.float32))]
    ws = gu.Workspace(plan.workspace_bytes)
    out = gu.OutBuf(orc.FP16, int(np.prod(p.y_shape)))
    plan.launch(tx.data_ptr(), tw.data_ptr(), tb.data_ptr(), out.ptr, ws.ptr, plan.workspace_bytes, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert plan.device_status() == 0
    ws.check_guard()
    m = oracle.compare(p, out.read(oracle).reshape(p.y_shape), ref, scale)
    assert m.passed(), m.summary()


@pytest.mark.parametrize("relu", [False, True])
@pytest.mark.parametrize("nhwc", [False, True])
@pytest.mark.parametrize("prec_name", ["fp16", "bf16"])
def test_infinities_and_nan(pkg, orc, oracle, relu, nhwc, prec_name):
    """NaN, both infinities and infinities that meet, in different slices of the reduction: the classes of the outputs follow from the
    inputs alone, whatever the order of the sums.  The ReLU of a NaN is zero here, as in every kernel of the library."""
    import torch
    prec = {"fp16": orc.FP16, "bf16": orc.BF16}[prec_name]
    p = orc.Problem.P(1, 256, 9, 7, 72, 3, 3, 1, 1, 1, 1, precision=prec, bias=True, relu=relu)
    x, w, b = oracle.make_conv_data(p, 3, 1)
    x, w, b = x.reshape(1, 256, 9, 7).copy(), w.reshape(72, 256, 3, 3), b.reshape(72)
    x[0, 5, 0, 0], x[0, 70, 4, 0], x[0, 130, 8, 6], x[0, 200, 8, 5], x[0, 255, 0, 6] = np.nan, np.inf, np.inf, -np.inf, -np.inf
    want = torch.nn.functional.conv2d(torch.from_numpy(x).double(), torch.from_numpy(w).double(), torch.from_numpy(b).double(), padding=1).numpy()
    if relu:
        want = np.where(want > 0, want, 0.0)
    flags = pkg.FLAG_OUTPUT_NHWC if nhwc else 0
    got, plan, _ = gu.run_conv(pkg, oracle, p, x, w, b, cfg=_cfg(pkg, p, 64, 4, flags), flags=flags)
    assert (plan.info.cfg.tile_n, plan.info.cfg.split_k, plan.info.cfg.reduce) == (64, 4, 2)
    got = got.reshape(9, 7, 72).transpose(2, 0, 1)[None] if nhwc else got
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isposinf(got), np.isposinf(want)) and np.array_equal(np.isneginf(got), np.isneginf(want))
    fin = np.isfinite(want)
    # one rounding to the stored type (2^-11 or 2^-8 of the value), and the FP32 rounding of 2304 terms near zero
    tol = {"fp16": 2.0 ** -11, "bf16": 2.0 ** -8}[prec_name] * np.abs(want[fin]) * 1.01 + 2304 * 2.0 ** -23 * np.abs(want[fin]).max()
    assert np.all(np.abs(got[fin] - want[fin]) <= tol)
    assert fin.sum() > 0.5 * fin.size and (relu or np.isnan(want).sum() >= 72)
