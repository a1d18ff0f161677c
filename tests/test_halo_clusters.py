"""Clusters of the halo kernel on channel-contiguous outputs.  Where they all fit the machine with one CTA per SM (15 of eight, 33 of
four) a CTA asks for the staging of its layout as well, which it does not use: two would share an SM without it.  Where they do not
fit, the CTAs ask for what they use."""
import pytest

STAGING = 8 * 2048  # eight worker warps


@pytest.mark.parametrize("split,fits", [(2, 74), (4, 33), (8, 15)])
def test_shared_memory_of_clusters(pkg, split, fits):
    for tiles in (1, fits // 2, fits, fits + 1):
        if tiles * split > 148:
            continue
        smem = []
        for flags in (pkg.FLAG_INPUT_NHWC, pkg.FLAG_INPUT_NHWC | pkg.FLAG_OUTPUT_NHWC):
            p = pkg.ConvProblem(1, 512, 7, 7, 32 * tiles, 3, 3, 1, 1, 1, 1, precision=pkg.FP16, has_bias=True, relu=True, flags=flags)
            i = pkg.query(p, pkg.make_cfg(variant=6, tile_n=32, split_k=split, stages=3))
            assert i.supported and i.num_blocks == tiles * split
            smem.append(i.dynamic_smem_bytes)
        assert smem[1] - smem[0] == (0 if tiles > fits else STAGING), tiles


@pytest.mark.gpu
@pytest.mark.parametrize("filters,split", [(480, 8), (512, 8), (1056, 4), (1088, 4)])
def test_clusters_with_and_without_staging(pkg, orc, oracle, filters, split):
    import numpy as np
    import torch
    import gpu_util as gu
    p = orc.Problem.P(1, 512, 7, 7, filters, 3, 3, 1, 1, 1, 1, precision=orc.FP16, bias=True, relu=True)
    x, w, b = oracle.make_conv_data(p, 7800 + filters, filters % 4)
    ref, scale = oracle.conv2d(p, x, w, b)
    plan = pkg.ConvPlan(gu.pkg_problem(pkg, p, pkg.FLAG_OUTPUT_NHWC), pkg.make_cfg(variant=6, tile_n=32, split_k=split))
    tx, px = gu.to_device_storage(oracle, orc.FP16, x)
    tw, pw = gu.to_device_storage(oracle, orc.FP16, w)
    tb, pb = gu.to_device_storage(oracle, orc.FP16, b)
    ws, out = gu.Workspace(plan.workspace_bytes), gu.OutBuf(orc.FP16, int(np.prod(p.y_shape)))
    for _ in range(3):  # in a row: CTAs of two launches on one SM
        plan.launch(px, pw, pb, out.ptr, ws.ptr, plan.workspace_bytes, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert plan.device_status() == 0
    ws.check_guard()
    got = np.ascontiguousarray(out.read(oracle).reshape(1, 7, 7, filters).transpose(0, 3, 1, 2))
    m = oracle.compare(p, got, ref, scale)   # the reference's scale-aware policy: rounding of sums of this length
    assert m.passed(), m.summary()
