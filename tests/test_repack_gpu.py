"""The data-movement kernels that are chosen by the size of the job alone, above the sizes at which they are chosen: bit-exact
against a permutation by torch, with guard values around every destination."""
import pytest

pytestmark = pytest.mark.gpu

SMS = 148


def _blocks(batch, hw, cp, px=64):
    return batch * -(-hw // px) * -(-cp // 64)


# batch, channels, pixels, padded channels
LARGE = [(16, 130, 57 * 57, 136),    # odd planes, a channel tail: nine vectors per row, shifted by the row
         (40, 70, 33 * 33, 72),      # a last pixel tile of one pixel
         (20, 64, 67 * 67, 64),      # 4489 = 70 tiles and 9 pixels
         (16, 130, 58 * 57, 144),    # even planes: 4-byte words (nine vectors when the pointer is odd)
         (16, 72, 64 * 58, 80)]      # planes of whole vectors (nine vectors when the pointer is off)


@pytest.mark.parametrize("off", range(8))
@pytest.mark.parametrize("shape", LARGE)
def test_large_repack_is_bit_exact(pkg, shape, off):
    import torch
    b, c, hw, cp = shape
    assert _blocks(b, hw, cp) > 8 * SMS
    n = b * c * hw
    g = torch.Generator(device="cuda")
    g.manual_seed(100 * off + c)
    buf = torch.randint(-32768, 32768, (n + 16,), device="cuda", generator=g, dtype=torch.int32).to(torch.int16)   # NaN patterns among them
    src = buf[off:off + n]
    guard = 64
    dst = torch.full((b * hw * cp + 2 * guard,), 0x5a5a, dtype=torch.int16, device="cuda")
    pkg.repack_nchw_to_nhwc(src.data_ptr(), dst.data_ptr() + 2 * guard, b, c, hw, cp, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    got = dst[guard:guard + b * hw * cp].view(b, hw, cp)
    assert torch.equal(got[:, :, :c], src.view(b, c, hw).transpose(1, 2))
    assert not got[:, :, c:].any()
    assert torch.all(dst[:guard] == 0x5a5a) and torch.all(dst[guard + b * hw * cp:] == 0x5a5a)


def test_large_filter_repack_is_bit_exact(pkg):
    """The slab form (few taps) in the same kernel: more filters than fit one wave."""
    import torch
    for o, c, rs, cp, off in [(3000, 70, 9, 80, 0), (2500, 33, 25, 40, 1), (1500, 500, 9, 512, 3)]:
        buf = torch.randint(-32768, 32768, (o * c * rs + 8,), device="cuda", dtype=torch.int32).to(torch.int16)
        src = buf[off:off + o * c * rs]
        dst = torch.full((o * rs * cp + 64,), 0x5a5a, dtype=torch.int16, device="cuda")
        pkg.prepack_weights(src.data_ptr(), dst.data_ptr(), o, c, rs, cp, torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        got = dst[:o * rs * cp].view(o, rs, cp)
        assert torch.equal(got[:, :, :c], src.view(o, c, rs).transpose(1, 2)) and not got[:, :, c:].any()
        assert torch.all(dst[o * rs * cp:] == 0x5a5a)


@pytest.mark.parametrize("off", range(5))
@pytest.mark.parametrize("shape", [(32, 70, 57, 57, 40), (24, 130, 58, 57, 24), (70, 64, 36, 64, 64), (52, 33, 67, 43, 17), (3, 70, 13, 9, 20), (2, 128, 20, 20, 32)])
def test_fp8_repack_is_bit_exact(pkg, shape, off):
    """Both tensors of an FP8 layer as its repack launch leaves them in the workspace: [B][HW][Cp], then [O][9][Cp].  The last two
    shapes are small jobs (tiles of 64 pixels), the others take tiles of 128."""
    import torch
    b, c, h, w, o = shape
    plan = pkg.ConvPlan(pkg.ConvProblem(b, c, h, w, o, 3, 3, 1, 1, 1, 1, precision=pkg.FP8_E4M3, has_bias=False, relu=True))
    cp, hw = plan.info.padded_channels, h * w
    assert (_blocks(b, hw, cp, 128) > 8 * SMS) == (b > 3)
    g = torch.Generator(device="cuda")
    g.manual_seed(10 * off + c)
    xbuf = torch.randint(0, 256, (b * c * hw + 16,), device="cuda", generator=g, dtype=torch.int32).to(torch.uint8)
    wbuf = torch.randint(0, 256, (o * c * 9 + 16,), device="cuda", generator=g, dtype=torch.int32).to(torch.uint8)
    x, wt = xbuf[off:off + b * c * hw], wbuf[(off * 3) % 5:(off * 3) % 5 + o * c * 9]
    y = torch.empty(b * o * hw, dtype=torch.float16, device="cuda")
    ws = torch.full((plan.workspace_bytes + 256,), 0x5a, dtype=torch.uint8, device="cuda")
    plan.launch_stages(1, x.data_ptr(), wt.data_ptr(), None, y.data_ptr(), ws.data_ptr(), plan.workspace_bytes, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    nx, nw = b * hw * cp, o * 9 * cp
    at_w = (nx + 255) // 256 * 256
    got_x, got_w = ws[:nx].view(b, hw, cp), ws[at_w:at_w + nw].view(o, 9, cp)
    assert torch.equal(got_x[:, :, :c], x.view(b, c, hw).transpose(1, 2)) and not got_x[:, :, c:].any()
    assert torch.equal(got_w[:, :, :c], wt.view(o, c, 9).transpose(1, 2)) and not got_w[:, :, c:].any()
    assert torch.all(ws[nx:at_w] == 0x5a) and torch.all(ws[at_w + nw:] == 0x5a)
    plan.close()


# batch, channels, h, w; bands of output rows: 148 * 1024 threads or 8 rows a thread, whichever is more bands
POOLS = [(64, 64, 112, 112, 8), (16, 64, 112, 112, 3), (40, 72, 57, 61, 3), (40, 72, 58, 61, 3), (24, 128, 35, 34, 1), (96, 64, 23, 57, 2), (200, 64, 31, 57, 4), (2, 8, 9, 4, 1), (3, 8, 2, 2, 1)]


@pytest.mark.parametrize("case", POOLS)
@pytest.mark.parametrize("dt", ["float16", "bfloat16"])
def test_channel_contiguous_pool_bands(pkg, case, dt):
    """3x3 / 2 / 1: the row that a thread carries from one output row to the next, infinities and NaNs (a number beats a NaN, a
    window of NaNs stays NaN)."""
    import torch
    b, c, h, w, rows = case
    oh, ow = (h - 1) // 2 + 1, (w - 1) // 2 + 1
    columns = b * ow * c // 8
    bands = min(oh, max(-(-SMS * 1024 // columns), -(-oh // 8)))
    assert -(-oh // bands) == rows
    dtype = getattr(torch, dt)
    g = torch.Generator(device="cuda")
    g.manual_seed(h * w)
    x = torch.randn(b, h, w, c, device="cuda", generator=g)
    r = torch.rand(b, h, w, c, device="cuda", generator=g)
    x = torch.where(r < 0.1, torch.tensor(float("nan"), device="cuda"), torch.where(r < 0.2, torch.tensor(float("-inf"), device="cuda"), x))
    x[:, : min(h, 5), : min(w, 4), 0] = float("nan")     # whole windows
    x[:, -3:, -3:, 1] = float("-inf")
    x = x.to(dtype)
    y = torch.full((b * oh * ow * c + 64,), 7, dtype=dtype, device="cuda")
    pkg.maxpool2d_nhwc(pkg.FP16 if dt == "float16" else pkg.BF16, b, c, h, w, 3, 2, 1, x.data_ptr(), y.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    planar = x.float().permute(0, 3, 1, 2)
    want = torch.nn.functional.max_pool2d(planar.nan_to_num(nan=float("-inf"), posinf=float("inf"), neginf=float("-inf")), 3, 2, 1)
    numbers = torch.nn.functional.max_pool2d((~planar.isnan()).float(), 3, 2, 1)
    want = torch.where(numbers > 0, want, torch.tensor(float("nan"), device="cuda")).permute(0, 2, 3, 1)
    got = y[:b * oh * ow * c].view(b, oh, ow, c).float()
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.nan_to_num(nan=5.0), want.nan_to_num(nan=5.0))
    assert want.isnan().any() and torch.all(y[b * oh * ow * c:] == 7)
