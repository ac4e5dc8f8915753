"""Filter gradient of strided channels-last convolutions in the halo form: every stride / dilation / padding that gives up to four
phases of input pixels, odd images, tiles that end inside an image, taps shared out among groups of CTAs. Integer-valued operands: the sums
are exact in f32, so the result is the 64-bit one rounded once. An explicit variant (bit 26) keeps the im2col form, which must agree."""
import pytest

pytestmark = pytest.mark.gpu

# n, h, w, c, k, (y, x), stride, dilation, padding
SHAPES = [(3, 28, 28, 128, 128, (3, 3), (2, 2), (1, 1), (1, 1)), (2, 33, 29, 64, 64, (3, 3), (2, 2), (1, 1), (1, 1)),
          (1, 14, 15, 64, 64, (1, 1), (2, 2), (1, 1), (0, 0)), (2, 17, 19, 128, 64, (5, 5), (2, 2), (1, 1), (2, 2)),
          (2, 21, 13, 64, 128, (7, 7), (2, 2), (1, 1), (3, 3)), (1, 20, 23, 64, 192, (3, 2), (2, 1), (1, 1), (0, 1)),
          (2, 19, 20, 64, 64, (2, 3), (1, 2), (1, 1), (1, 0)), (2, 24, 25, 64, 64, (3, 3), (2, 2), (2, 2), (2, 2)),
          (1, 31, 30, 64, 64, (3, 3), (2, 2), (3, 1), (3, 0)), (5, 8, 8, 256, 256, (3, 3), (2, 2), (1, 1), (1, 1)),
          (40, 9, 9, 64, 64, (3, 3), (2, 2), (1, 1), (1, 1)), (1, 3, 3, 64, 64, (3, 3), (2, 2), (1, 1), (0, 0)),
          (4, 28, 28, 128, 128, (3, 3), (1, 1), (1, 1), (1, 1))]


@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
@pytest.mark.parametrize("n,h,w,c,k,fil,stride,dil,pad", SHAPES)
def test_filter_gradient(cuda_device, dtype, n, h, w, c, k, fil, stride, dil, pad):
    import torch
    from rocmlir_b200 import _lib as L
    from rocmlir_b200 import conv as rb_conv
    cfg = rb_conv.ConvConfig(n, c, k, h, w, fil[0], fil[1], stride_h=stride[0], stride_w=stride[1], dil_h=dil[0], dil_w=dil[1],
                             pad_h=pad[0], pad_w=pad[1], fil_layout="gkyxc", in_layout="nhwgc", out_layout="nhwgk")
    gen = torch.Generator(device="cuda").manual_seed(3)
    dt = getattr(torch, dtype)
    x = torch.randint(-2, 3, (n, h, w, c), device="cuda", generator=gen).to(dt)
    dy = torch.randint(-1, 2, (n, cfg.ho, cfg.wo, k), device="cuda", generator=gen).to(dt)
    op = rb_conv.OPERATIONS["conv_bwd_weight"]
    got = []
    for variant in (0, 1 << 26):
        fil_grad = torch.full((k, fil[0], fil[1], c), 7.0, device="cuda", dtype=dt)
        L.lib().rbSetGemmVariant(variant)
        try:
            ws = torch.empty(max(16, rb_conv.workspace_size(cfg, dt, op)), dtype=torch.uint8, device="cuda")
            rb_conv.conv(cfg, op, fil_grad.view(-1), x.view(-1), dy.view(-1), workspace=ws)
        finally:
            L.lib().rbSetGemmVariant(0)
        torch.cuda.synchronize()
        got.append(fil_grad)
    assert L.kernel_status() == 0
    with torch.backends.cudnn.flags(enabled=False):
        want = torch.nn.grad.conv2d_weight(x.double().permute(0, 3, 1, 2).contiguous(), (k, c, fil[0], fil[1]),
                                           dy.double().permute(0, 3, 1, 2).contiguous(), stride=stride, padding=pad, dilation=dil)
    want = want.permute(0, 2, 3, 1).to(dt)
    assert torch.equal(got[0], want) and torch.equal(got[1], want)


@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
@pytest.mark.parametrize("where", ["x_corner", "x_column", "x_all", "dy"])
@pytest.mark.parametrize("n,h,w,c,k,fil,stride,dil,pad", [s for s in SHAPES if s[6] != (1, 1)])
def test_values_that_are_not_finite_reach_the_taps_that_meet_them(cuda_device, dtype, where, n, h, w, c, k, fil, stride, dil, pad):
    """With a stride. An Inf or NaN pixel lies in the padded raster of taps that never meet it; the im2col form multiplies no others."""
    import math
    import torch
    from rocmlir_b200 import _lib as L
    from rocmlir_b200 import conv as rb_conv
    cfg = rb_conv.ConvConfig(n, c, k, h, w, fil[0], fil[1], stride_h=stride[0], stride_w=stride[1], dil_h=dil[0], dil_w=dil[1],
                             pad_h=pad[0], pad_w=pad[1], fil_layout="gkyxc", in_layout="nhwgc", out_layout="nhwgk")
    gen = torch.Generator(device="cuda").manual_seed(3)
    dt = getattr(torch, dtype)
    x = torch.randint(-2, 3, (n, h, w, c), device="cuda", generator=gen).to(dt)
    dy = torch.randint(1, 3, (n, cfg.ho, cfg.wo, k), device="cuda", generator=gen).to(dt)
    if where == "x_corner":
        x[n // 2, h - 1, w - 1, 5] = math.inf
        x[0, 0, 0, 40] = math.nan
    if where == "x_column":
        x[:, h // 2, w - 1] = -math.inf
    if where == "x_all":
        x.fill_(math.nan)
    if where == "dy":
        dy[n // 2, cfg.ho - 1, 0, 7] = math.inf
        dy[0, 0, cfg.wo - 1, 9] = math.nan
    op = rb_conv.OPERATIONS["conv_bwd_weight"]
    got = []
    for variant in (0, 1 << 26):
        fil_grad = torch.full((k, fil[0], fil[1], c), 7.0, device="cuda", dtype=dt)
        L.lib().rbSetGemmVariant(variant)
        try:
            ws = torch.empty(max(16, rb_conv.workspace_size(cfg, dt, op)), dtype=torch.uint8, device="cuda")
            rb_conv.conv(cfg, op, fil_grad.view(-1), x.view(-1), dy.view(-1), workspace=ws)
        finally:
            L.lib().rbSetGemmVariant(0)
        torch.cuda.synchronize()
        got.append(fil_grad)
    assert L.kernel_status() == 0
    assert torch.equal(got[0].isnan(), got[1].isnan())
    assert torch.equal(got[0].nan_to_num(nan=0.5), got[1].nan_to_num(nan=0.5))
