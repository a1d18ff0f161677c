"""Convolutions that follow one another in a stream with nothing between them (channel-contiguous tensors, prepacked weights),
with rings short enough for CTAs of three launches to lie on one SM: their tensor memory does not fit it side by side, so a
later launch may take columns only when every CTA of the launch before it has its own.  Same bits as one launch at a time."""
import itertools

import numpy as np
import pytest

import gpu_util as gu

pytestmark = pytest.mark.gpu

# 512, 256, 128 and 64 columns a CTA; two, one and half a wave of CTAs
CFGS = [dict(tile_m=128, tile_n=256, stages=2, cta_pair=1, split_k=1), dict(tile_m=128, tile_n=128, stages=2, cta_pair=1, split_k=1),
        dict(tile_m=128, tile_n=64, stages=2, cta_pair=1, split_k=1), dict(tile_m=128, tile_n=32, stages=2, cta_pair=1, split_k=1), None]


@pytest.mark.parametrize("batch", [1, 3, 12])
def test_launches_back_to_back(pkg, orc, oracle, batch):
    import torch
    c, hw = 256, 24
    p = orc.Problem.P(batch, c, hw, hw, c, 3, 3, 1, 1, 1, 1, precision=orc.FP16, bias=True, relu=True)
    x, w, b = oracle.make_conv_data(p, 77, 1)
    flags = pkg.FLAG_INPUT_NHWC | pkg.FLAG_OUTPUT_NHWC | pkg.FLAG_WEIGHTS_PREPACKED
    stream = torch.cuda.current_stream().cuda_stream
    tw, pw = gu.to_device_storage(oracle, p.precision, w)
    tb, pb = gu.to_device_storage(oracle, p.precision, b)
    plans = []
    for kw in CFGS:
        plan = pkg.ConvPlan(gu.pkg_problem(pkg, p, flags), pkg.make_cfg(**kw) if kw else None)
        packed = torch.empty(plan.prepacked_weight_bytes, dtype=torch.uint8, device="cuda")
        plan.prepack_weights(pw, packed.data_ptr(), stream)
        assert plan.workspace_bytes == 0 and plan.info.launches == 1
        plans.append((plan, packed))
    n = int(np.prod(p.y_shape))
    start = torch.from_numpy(oracle.to_storage(p.precision, np.ascontiguousarray(x.transpose(0, 2, 3, 1)).ravel()).view(np.int16)).cuda()

    def run(order, wait):
        bufs = [start.clone(), torch.full_like(start, -1)]
        assert bufs[0].numel() == n
        for k, i in enumerate(order):
            plan, packed = plans[i]
            plan.launch(bufs[k & 1].data_ptr(), packed.data_ptr(), pb, bufs[(k + 1) & 1].data_ptr(), None, 0, stream)
            if wait:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return bufs[len(order) & 1]

    order = [i for pair in itertools.permutations(range(len(CFGS)), 2) for i in pair] * 2
    want = run(order, True)
    for _ in range(3):
        got = run(order, False)
        assert torch.equal(want, got)
    assert all(plan.device_status() == 0 for plan, _ in plans)
