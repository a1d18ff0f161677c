"""The repack of small tensors through registers (csrc/repack_direct.cu) at the sizes where its blocks end, its rules change and it
hands over: bit-exact against a permutation by torch (NaN patterns among the values), with guard values around every destination."""
import pytest

pytestmark = pytest.mark.gpu

GUARD = 64


def _values(n, seed):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.randint(-32768, 32768, (n,), device="cuda", generator=g, dtype=torch.int32).to(torch.int16)


# batch, channels, pixels, padded channels
ACTIVATIONS = [(2, 64, 196, 64), (1, 8, 4, 8), (3, 70, 132, 80), (2, 130, 128, 192),      # runs of four pixels (the last two: 128-byte rows)
               (1, 64, 50, 64), (2, 33, 66, 48), (5, 72, 2, 80),                           # of two
               (2, 64, 49, 64), (3, 40, 33, 64), (1, 200, 31, 208), (4, 9, 65, 16),        # single pixels
               (148, 64, 124, 64), (149, 64, 128, 64), (297, 64, 124, 64),                 # the last sizes of runs of four, and beyond
               (444, 64, 62, 64), (445, 64, 62, 64), (2048, 8, 31, 8), (2049, 8, 31, 8)]


@pytest.mark.parametrize("off", [0, 1, 2, 4, 7])
@pytest.mark.parametrize("shape", ACTIVATIONS)
def test_small_planes(pkg, shape, off):
    import torch
    b, c, hw, cp = shape
    n = b * c * hw
    src = _values(n + 8, 100 * off + c)[off:off + n]
    dst = torch.full((b * hw * cp + 2 * GUARD,), 0x5a5a, dtype=torch.int16, device="cuda")
    pkg.repack_nchw_to_nhwc(src.data_ptr(), dst.data_ptr() + 2 * GUARD, b, c, hw, cp, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    got = dst[GUARD:GUARD + b * hw * cp].view(b, hw, cp)
    assert torch.equal(got[:, :, :c], src.view(b, c, hw).transpose(1, 2)) and not got[:, :, c:].any()
    assert torch.all(dst[:GUARD] == 0x5a5a) and torch.all(dst[GUARD + b * hw * cp:] == 0x5a5a)


# filters, channels, taps, padded channels: shares of a block, exactly one, one more; padding; channels that are no whole groups
FILTERS = [(8, 64, 9, 64), (9, 56, 9, 64), (512, 64, 9, 64), (513, 64, 9, 64), (4097, 8, 9, 8),   # blocks of 64 units, and the first of 256
           (31, 64, 9, 64), (32, 64, 9, 64), (33, 64, 9, 64), (257, 8, 9, 8), (70, 48, 9, 64), (3, 144, 9, 192), (5, 20, 9, 32), (512, 512, 9, 512),
           (31, 64, 1, 64), (257, 8, 1, 8), (70, 48, 1, 64), (1, 8, 1, 8), (9, 12, 1, 16)]


@pytest.mark.parametrize("off", [0, 3, 8])
@pytest.mark.parametrize("shape", FILTERS)
def test_filters(pkg, shape, off):
    import torch
    o, c, rs, cp = shape
    n = o * c * rs
    src = _values(n + 8, 10 * off + c)[off:off + n]
    dst = torch.full((o * rs * cp + 2 * GUARD,), 0x5a5a, dtype=torch.int16, device="cuda")
    pkg.prepack_weights(src.data_ptr(), dst.data_ptr() + 2 * GUARD, o, c, rs, cp, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    got = dst[GUARD:GUARD + o * rs * cp].view(o, rs, cp)
    assert torch.equal(got[:, :, :c], src.view(o, c, rs).transpose(1, 2)) and not got[:, :, c:].any()
    assert torch.all(dst[:GUARD] == 0x5a5a) and torch.all(dst[GUARD + o * rs * cp:] == 0x5a5a)


@pytest.mark.parametrize("xoff,woff", [(0, 0), (1, 0), (2, 8), (0, 1)])
@pytest.mark.parametrize("shape", [(2, 64, 14, 14, 70, 3), (3, 128, 7, 7, 33, 3), (2, 72, 10, 9, 64, 3), (2, 144, 9, 11, 40, 3), (5, 64, 7, 7, 96, 1), (2, 96, 10, 5, 65, 1),
                                   (2, 64, 9, 9, 40, 5), (3, 20, 7, 7, 24, 3), (12, 77, 9, 9, 752, 1), (1, 20, 6, 6, 300, 3),
                                   (41, 130, 19, 21, 40, 3), (43, 130, 19, 21, 40, 5)])  # the last four: activations first (odd planes: from 740 blocks)
def test_both_tensors_of_a_layer(pkg, shape, xoff, woff):
    """One launch for the activations and the weights, as a forward call leaves them in the workspace."""
    import torch
    b, c, h, w, o, k = shape
    plan = pkg.ConvPlan(pkg.ConvProblem(b, c, h, w, o, k, k, 1, 1, k // 2, k // 2, precision=pkg.FP16, has_bias=False, relu=True))
    cp, hw, rs = plan.info.padded_channels, h * w, k * k
    x = _values(b * c * hw + 8, 1)[xoff:xoff + b * c * hw]
    wt = _values(o * c * rs + 8, 2)[woff:woff + o * c * rs]
    y = torch.empty(b * o * hw, dtype=torch.float16, device="cuda")
    ws = torch.full((plan.workspace_bytes // 2 + 128,), 0x5a5a, dtype=torch.int16, device="cuda")
    plan.launch_stages(1, x.data_ptr(), wt.data_ptr(), None, y.data_ptr(), ws.data_ptr(), plan.workspace_bytes, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    nx, nw = b * hw * cp, o * rs * cp
    at_w = (2 * nx + 255) // 256 * 128
    got_x, got_w = ws[:nx].view(b, hw, cp), ws[at_w:at_w + nw].view(o, rs, cp)
    assert torch.equal(got_x[:, :, :c], x.view(b, c, hw).transpose(1, 2)) and not got_x[:, :, c:].any()
    assert torch.equal(got_w[:, :, :c], wt.view(o, c, rs).transpose(1, 2)) and not got_w[:, :, c:].any()
    assert torch.all(ws[nx:at_w] == 0x5a5a) and torch.all(ws[at_w + nw:] == 0x5a5a)
    plan.close()


@pytest.mark.parametrize("shape", [(2, 64, 9, 9, 40, 3), (3, 20, 7, 7, 24, 5), (1, 64, 5, 5, 400, 3), (1, 40, 11, 13, 64, 1)])  # weights first, and few activations first
def test_both_tensors_of_a_tf32_layer(pkg, shape):
    """Values that TF32 holds exactly (13 low bits zero), so a permutation once more."""
    import torch
    b, c, h, w, o, k = shape
    plan = pkg.ConvPlan(pkg.ConvProblem(b, c, h, w, o, k, k, 1, 1, k // 2, k // 2, precision=pkg.TF32, has_bias=False, relu=True))
    cp, hw, rs = plan.info.padded_channels, h * w, k * k
    g = torch.Generator(device="cuda")
    g.manual_seed(c)
    x, wt = [torch.randint(-1000, 1000, (n,), device="cuda", generator=g).float() for n in (b * c * hw, o * c * rs)]
    y = torch.empty(b * o * hw, device="cuda")
    ws = torch.full((plan.workspace_bytes // 4 + 64,), 0.5, device="cuda")
    plan.launch_stages(1, x.data_ptr(), wt.data_ptr(), None, y.data_ptr(), ws.data_ptr(), plan.workspace_bytes, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    nx, nw = b * hw * cp, o * rs * cp
    at_w = (4 * nx + 255) // 256 * 64
    got_x, got_w = ws[:nx].view(b, hw, cp), ws[at_w:at_w + nw].view(o, rs, cp)
    assert torch.equal(got_x[:, :, :c], x.view(b, c, hw).transpose(1, 2)) and not got_x[:, :, c:].any()
    assert torch.equal(got_w[:, :, :c], wt.view(o, c, rs).transpose(1, 2)) and not got_w[:, :, c:].any()
    assert torch.all(ws[nx:at_w] == 0.5) and torch.all(ws[at_w + nw:] == 0.5)
    plan.close()


def test_without_prefetch():
    """The same with the prefetches switched off (an environment variable that a process reads once)."""
    import os
    import subprocess
    import sys
    r = subprocess.run([sys.executable, "-m", "pytest", "-q", "-x", "-m", "gpu", "-k", "test_both_tensors_of_a_layer", os.path.abspath(__file__)],
                       env=dict(os.environ, GIEB_DISABLE_PREFETCH="1"), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
