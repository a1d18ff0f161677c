"""The residual of NCHW outputs where a tile's last 32 channels are a partial chunk: one valid channel, a group of eight and one more,
31, in every kernel that adds it to the pixel-lane accumulator, on odd planes and off their alignment, and the halo kernel's clusters on
channel-contiguous outputs (which take no staging)."""
import numpy as np
import pytest

import gpu_util as gu

pytestmark = pytest.mark.gpu

POINTS = [dict(variant=1, cta_pair=1, tile_n=64), dict(variant=1, cta_pair=1, tile_n=64, tile_m=256), dict(variant=1, cta_pair=2, tile_n=64),
          dict(variant=1, cta_pair=1, tile_n=32, split_k=3, reduce=1), dict(variant=1, cta_pair=1, tile_n=64, split_k=2, reduce=2),
          dict(variant=6, cta_pair=1, tile_n=64), dict(variant=6, cta_pair=2, tile_n=128), dict(variant=6, tile_n=64, split_k=2)]


def _run(pkg, orc, oracle, args, prec, kw, flags, seed, yoff):
    import torch
    nhwc = (flags & pkg.FLAG_OUTPUT_NHWC) != 0
    p_lin = orc.Problem.P(*args, precision=prec, bias=True, relu=False)
    p = orc.Problem.P(*args, precision=prec, bias=True, relu=True)
    x, w, b = oracle.make_conv_data(p, seed, seed % 4)
    lin, scale = oracle.conv2d(p_lin, x, w, b)
    res = oracle.quantize(prec, oracle.rng(seed + 1).uniform(-1, 1, lin.size)).reshape(lin.shape)
    ref = np.maximum(lin.astype(np.float64) + res, 0.0).astype(np.float32)
    scale = (scale.astype(np.float64) + np.abs(res)).astype(np.float32)
    to_layout = (lambda a: np.ascontiguousarray(a.transpose(0, 2, 3, 1))) if nhwc else (lambda a: a)
    plan = pkg.ConvPlan(gu.pkg_problem(pkg, p, flags | pkg.FLAG_RESIDUAL), pkg.make_cfg(**kw))
    tx, px = gu.to_device_storage(oracle, prec, x)
    tw, pw = gu.to_device_storage(oracle, prec, w)
    tb, pb = gu.to_device_storage(oracle, prec, b)
    tr, pr = gu.to_device_storage(oracle, prec, to_layout(res), yoff)
    ws = gu.Workspace(plan.workspace_bytes)
    out = gu.OutBuf(prec, int(np.prod(p.y_shape)), yoff)
    plan.launch_fused(px, pw, pb, pr, out.ptr, ws.ptr, plan.workspace_bytes, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert plan.device_status() == 0
    ws.check_guard()
    got = out.read(oracle)
    B, O, P, Q = p.y_shape
    got = np.ascontiguousarray(got.reshape(B, P, Q, O).transpose(0, 3, 1, 2)) if nhwc else got.reshape(p.y_shape)
    m = oracle.compare(p, got, ref, scale)   # the reference's scale-aware policy: rounding of sums of this length
    assert m.passed(), f"{args} {kw}: {m.summary()}"
    return plan


@pytest.mark.parametrize("point", range(len(POINTS)))
@pytest.mark.parametrize("filters", [33, 41, 63, 64])
def test_partial_chunk(pkg, orc, oracle, point, filters):
    prec = orc.FP16 if (point + filters) % 2 == 0 else orc.BF16
    plan = _run(pkg, orc, oracle, (3, 128, 9, 11, filters, 3, 3, 1, 1, 1, 1), prec, POINTS[point], 0, 7600 + point, filters % 3)
    assert all(getattr(plan.info.cfg, k) == v for k, v in POINTS[point].items())


@pytest.mark.parametrize("filters", [40, 37, 96])
@pytest.mark.parametrize("split", [2, 4, 8])
def test_halo_clusters_channel_contiguous(pkg, orc, oracle, filters, split):
    _run(pkg, orc, oracle, (1, 512, 7, 9, filters, 3, 3, 1, 1, 1, 1), orc.FP16, dict(variant=6, tile_n=32, split_k=split), pkg.FLAG_OUTPUT_NHWC, 7700 + split, filters % 2)
