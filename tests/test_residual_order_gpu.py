"""Sum, bias and residual are added in one order, (sum + bias) + residual, whether a chunk of 32 channels is whole or partial: with a sum
of 2^24, a bias of 1 and a residual of -2^24 that gives 0 (2^24 + 1 rounds to 2^24 in FP32), any other order 1."""
import numpy as np
import pytest

import gpu_util as gu

pytestmark = pytest.mark.gpu

POINTS = [dict(variant=1, cta_pair=1, tile_n=64, split_k=1), dict(variant=1, cta_pair=1, tile_n=64, tile_m=256, split_k=1), dict(variant=1, cta_pair=2, tile_n=64),
          dict(variant=1, cta_pair=1, tile_n=64, split_k=2, reduce=2), dict(variant=6, cta_pair=1, tile_n=64), dict(variant=6, cta_pair=2, tile_n=128),
          dict(variant=6, tile_n=64, split_k=2)]


def run(pkg, orc, oracle, args, cfg):
    import torch
    p = orc.Problem.P(*args, precision=orc.BF16, bias=True, relu=False)
    B, O, P, Q = p.y_shape
    # one product of 4096 x 4096 per output: the middle tap of channel 0 (every pixel is 4096)
    x = np.zeros((args[0], args[1], args[2], args[3]), np.float32)
    x[:, 0] = 4096.0
    w = np.zeros((O, args[1], args[5], args[6]), np.float32)
    w[:, 0, args[9], args[10]] = 4096.0
    plan = pkg.ConvPlan(gu.pkg_problem(pkg, p, pkg.FLAG_RESIDUAL), cfg)
    bufs = [gu.to_device_storage(oracle, orc.BF16, a) for a in (x, w, np.ones(O, np.float32), np.full(B * O * P * Q, -float(1 << 24), np.float32))]
    ws, out = gu.Workspace(plan.workspace_bytes), gu.OutBuf(orc.BF16, B * O * P * Q)
    plan.launch_fused(bufs[0][1], bufs[1][1], bufs[2][1], bufs[3][1], out.ptr, ws.ptr, plan.workspace_bytes, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert plan.device_status() == 0
    got = out.read(oracle).reshape(p.y_shape)
    assert not got.any(), np.unique(np.argwhere(got)[:, 1])


@pytest.mark.parametrize("point", range(len(POINTS)))
def test_partial_chunks(pkg, orc, oracle, point):
    run(pkg, orc, oracle, (3, 128, 9, 11, 53, 3, 3, 1, 1, 1, 1), pkg.make_cfg(**POINTS[point]))


def test_partial_chunks_over_images(pkg, orc, oracle):
    run(pkg, orc, oracle, (1, 3, 30, 34, 53, 7, 7, 2, 2, 3, 3), None)
