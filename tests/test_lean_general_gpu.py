"""The two forms of every slab kernel: the lean one, and the general one that a partial last slab or a row-wise output (odd channel
counts, or an output off its 16-byte alignment, decided per launch) calls for.  Both forms of a plan in turn, against the oracle."""
import numpy as np
import pytest

import gpu_util as gu

pytestmark = pytest.mark.gpu

POINTS = [dict(tile_m=128, tile_n=32, cta_pair=1), dict(tile_m=128, tile_n=64, cta_pair=1), dict(tile_m=256, tile_n=64, cta_pair=1),
          dict(tile_m=128, tile_n=128, cta_pair=1), dict(tile_m=256, tile_n=128, cta_pair=1), dict(tile_m=128, tile_n=256, cta_pair=1),
          dict(tile_m=256, tile_n=64, cta_pair=2), dict(tile_m=256, tile_n=128, cta_pair=2), dict(tile_m=256, tile_n=256, cta_pair=2)]


@pytest.mark.parametrize("point", range(len(POINTS)))
@pytest.mark.parametrize("channels,filters", [(128, 264), (144, 264), (128, 131), (80, 70)])   # lean / partial slab / odd rows / both
def test_both_forms(pkg, orc, oracle, point, channels, filters):
    import torch
    kw = POINTS[point]
    prec = orc.FP16 if (point + channels) % 2 == 0 else orc.BF16
    with_res = point % 2 == 1
    args = (3, channels, 13, 11, filters, 3, 3, 1, 1, 1, 1)
    p_lin = orc.Problem.P(*args, precision=prec, bias=True, relu=False)
    p = orc.Problem.P(*args, precision=prec, bias=True, relu=True)
    x, w, b = oracle.make_conv_data(p, 60 + point, point % 4)
    lin, scale = oracle.conv2d(p_lin, x, w, b)
    res = oracle.quantize(prec, oracle.rng(70 + point).uniform(-1, 1, lin.size)).reshape(lin.shape) if with_res else np.zeros_like(lin)
    ref = np.maximum(lin.astype(np.float64) + res, 0.0).astype(np.float32)
    scale = (scale.astype(np.float64) + np.abs(res)).astype(np.float32)
    nhwc = lambda a: np.ascontiguousarray(a.transpose(0, 2, 3, 1))
    flags = pkg.FLAG_INPUT_NHWC | pkg.FLAG_OUTPUT_NHWC | (pkg.FLAG_RESIDUAL if with_res else 0)
    plan = pkg.ConvPlan(gu.pkg_problem(pkg, p, flags), pkg.make_cfg(variant=1, tile_k=64, stages=2, split_k=1, **kw))
    assert plan.info.padded_channels == channels and all(getattr(plan.info.cfg, k) == v for k, v in kw.items())
    stream = torch.cuda.current_stream().cuda_stream
    tx, px = gu.to_device_storage(oracle, prec, nhwc(x))
    tw, pw = gu.to_device_storage(oracle, prec, w)
    tb, pb = gu.to_device_storage(oracle, prec, b)
    ws = gu.Workspace(plan.workspace_bytes)
    for off in (0, 1, 4, 0):   # TMA stores where rows allow them, single channels, channel pairs, and back
        tr, pr = gu.to_device_storage(oracle, prec, nhwc(res), off)
        out = gu.OutBuf(prec, int(np.prod(p.y_shape)), off)
        if with_res:
            plan.launch_fused(px, pw, pb, pr, out.ptr, ws.ptr, plan.workspace_bytes, stream)
        else:
            plan.launch(px, pw, pb, out.ptr, ws.ptr, plan.workspace_bytes, stream)
        torch.cuda.synchronize()
        assert plan.device_status() == 0
        ws.check_guard()
        B, O, P, Q = p.y_shape
        got = np.ascontiguousarray(out.read(oracle).reshape(B, P, Q, O).transpose(0, 3, 1, 2))
        m = oracle.compare(p, got, ref, scale)   # the reference's scale-aware policy: rounding of sums of this length
        assert m.passed(), f"{kw} {channels}->{filters} offset {off}: {m.summary()}"


@pytest.mark.parametrize("kw", [dict(tile_m=128, tile_n=128), dict(tile_m=256, tile_n=128), dict(tile_m=128, tile_n=256)])
@pytest.mark.parametrize("channels", [80, 192])
def test_transposed_accumulator_with_partial_slab(pkg, orc, oracle, channels, kw, monkeypatch):
    monkeypatch.setenv("GIEB_TRANSPOSED_ACC", "2")
    p = orc.Problem.P(2, channels, 12, 14, 200, 3, 3, 1, 1, 1, 1, precision=orc.FP16, bias=True, relu=True)
    x, w, b = oracle.make_conv_data(p, 90, 2)
    ref, scale = oracle.conv2d(p, x, w, b)
    cfg = pkg.make_cfg(variant=1, tile_k=64, stages=2, split_k=1, cta_pair=1, **kw)
    got, plan, _ = gu.run_conv(pkg, oracle, p, x, w, b, cfg=cfg)
    assert plan.info.padded_channels == channels
    m = oracle.compare(p, got, ref, scale)
    assert m.passed(), f"{kw} {channels}: {m.summary()}"
