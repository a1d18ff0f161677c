"""The allocation-free call where a plan would sum its split-K slices in a workspace that the built-in scratch does not hold: the slices
are clusters then, more of them than the machine holds at once."""
import numpy as np
import pytest

import gpu_util as gu


def _layers(pkg):
    nhwc = pkg.FLAG_INPUT_NHWC | pkg.FLAG_OUTPUT_NHWC
    pre = pkg.FLAG_WEIGHTS_PREPACKED
    for args, flags, cfg in [((6, 624, 55, 55, 96, 5, 5, 2, 2, 2, 2), nhwc, (128, 4, 6)), ((33, 768, 10, 10, 576, 5, 5, 2, 2, 2, 2), pre, (128, 4, 6)),
                             ((6, 672, 46, 17, 96, 5, 5, 1, 1, 2, 2), pre, (128, 4, 6)), ((7, 704, 18, 18, 144, 5, 5, 1, 1, 2, 2), 0, (256, 8, 4))]:
        clusters = pkg.make_cfg(tile_m=128, tile_n=cfg[0], tile_k=64, stages=cfg[2], split_k=cfg[1], variant=1, reduce=2, cta_pair=1)
        yield pkg.ConvProblem(*args, precision=pkg.BF16, has_bias=True, relu=True, flags=flags), clusters


def test_partials_beyond_the_scratch_are_no_refusal(pkg):
    import torch
    if torch.cuda.is_available():
        pytest.skip("the addresses below are none: the call must not reach a device")
    for p, _ in _layers(pkg):
        info = pkg.query(p)
        assert info.cfg.reduce == 1 and info.workspace_bytes > 8 << 20
        with pytest.raises(pkg.GieError) as e:
            pkg.conv_forward_static(p, 256, 256, 256, 256, 0)
        assert e.value.code == pkg.CUDA_ERROR, e.value     # past the checks: no device to run on
        with pytest.raises(pkg.GieError) as e:             # asked for, the workspace stays
            pkg.conv_forward_static(p, 256, 256, 256, 256, 0, pkg.make_cfg(reduce=1, split_k=info.cfg.split_k, tile_n=info.cfg.tile_n))
        assert e.value.code == pkg.WORKSPACE_TOO_SMALL


@pytest.mark.gpu
def test_rounds_of_clusters_give_the_bits_of_their_plan(pkg):
    import torch
    stream = torch.cuda.current_stream().cuda_stream
    for n, (p, cfg) in enumerate(_layers(pkg)):
        plan = pkg.ConvPlan(p, cfg)
        assert plan.info.cfg.reduce == 2 and plan.workspace_bytes <= 8 << 20
        g = torch.Generator(device="cuda")
        g.manual_seed(n)
        x = torch.randn(p.batch * p.in_channels * p.in_h * p.in_w, device="cuda", generator=g).to(torch.bfloat16)
        fan = p.in_channels * p.kernel_h * p.kernel_w
        w = (torch.randn(p.out_channels * fan, device="cuda", generator=g) / fan ** 0.5).to(torch.bfloat16)
        b = torch.randn(p.out_channels, device="cuda", generator=g).to(torch.bfloat16)
        wp = w
        if p.flags & pkg.FLAG_WEIGHTS_PREPACKED:
            wp = torch.empty(plan.prepacked_weight_bytes // 2, dtype=torch.bfloat16, device="cuda")
            plan.prepack_weights(w.data_ptr(), wp.data_ptr(), stream)
        y = torch.zeros(2, p.batch * p.out_channels * p.out_h * p.out_w, dtype=torch.bfloat16, device="cuda")
        ws = gu.Workspace(plan.workspace_bytes)
        plan.launch(x.data_ptr(), wp.data_ptr(), b.data_ptr(), y[0].data_ptr(), ws.ptr, plan.workspace_bytes, stream)
        pkg.conv_forward_static(p, x.data_ptr(), wp.data_ptr(), b.data_ptr(), y[1].data_ptr(), stream)
        assert pkg.conv_static_status(stream) == 0 and plan.device_status() == 0
        assert torch.equal(y[0].view(torch.int16), y[1].view(torch.int16)), p
        # the plan with its partials in the workspace: FP32 sums in another order, so at most one BF16 step (2^-7 of the value) apart,
        # or the sums' own rounding near zero (2^-24 times the square root of their length, a few standard deviations of it)
        other = pkg.ConvPlan(p)
        z = torch.zeros_like(y[0])
        ws = gu.Workspace(other.workspace_bytes)
        other.launch(x.data_ptr(), wp.data_ptr(), b.data_ptr(), z.data_ptr(), ws.ptr, other.workspace_bytes, stream)
        torch.cuda.synchronize()
        a, c = y[0].float(), z.float()
        assert bool(((a - c).abs() <= 2.0 ** -7 * torch.maximum(a.abs(), c.abs()) + 2.0 ** -21 * fan ** 0.5).all()), p
        assert float(a.abs().max()) > 1
