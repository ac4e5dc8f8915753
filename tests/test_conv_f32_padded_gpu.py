"""f32 convolutions whose channels are no multiple of a 128-byte run: planes padded with zeros against the im2col matrix (variant bit 26), every
layout, and images too small to gain from it."""
import pytest

pytestmark = pytest.mark.gpu
MATRIX = 1 << 26


@pytest.mark.parametrize("lay", [("gkcyx", "ngchw", "ngkhw"), ("gkyxc", "nhwgc", "nhwgk"), ("gkcyx", "nhwgc", "ngkhw"), ("gkyxc", "ngchw", "nhwgk")])
@pytest.mark.parametrize("n,c,k,hw,fil,stride,dil,pad", [(9, 16, 64, 40, 3, 1, 1, 1), (20, 16, 65, 41, 3, 2, 1, 0), (3, 24, 33, 50, 5, 1, 2, 4),
                                                         (30, 40, 128, 31, 1, 1, 1, 0), (2, 48, 130, 60, 3, 1, 1, 1), (40, 16, 64, 29, 1, 2, 1, 0),
                                                         (1, 16, 64, 9, 3, 1, 1, 1)])
def test_padded_channels(cuda_device, lay, n, c, k, hw, fil, stride, dil, pad):
    import torch
    from rocmlir_b200 import _lib as L
    from rocmlir_b200 import conv as rb_conv
    cfg = rb_conv.ConvConfig(n, c, k, hw, hw, fil, fil, stride_h=stride, stride_w=stride, dil_h=dil, dil_w=dil, pad_h=pad, pad_w=pad,
                             fil_layout=lay[0], in_layout=lay[1], out_layout=lay[2])
    gen = torch.Generator(device="cuda").manual_seed(1)
    x, w = (torch.randn(s, device="cuda", generator=gen) for s in ((n, c, hw, hw), (k, c, fil, fil)))
    xs = (x.permute(0, 2, 3, 1) if lay[1] == "nhwgc" else x).contiguous()
    fs = (w.permute(0, 2, 3, 1) if lay[0] == "gkyxc" else w).contiguous()
    got = []
    for variant in (0, MATRIX):
        out = torch.full((cfg.numel("out"),), 5.0, device="cuda")
        L.lib().rbSetGemmVariant(variant)
        try:
            ws = torch.full((max(16, rb_conv.workspace_size(cfg, torch.float32, rb_conv.OPERATIONS["conv"])),), 255, dtype=torch.uint8, device="cuda")
            rb_conv.conv(cfg, rb_conv.OPERATIONS["conv"], fs.view(-1), xs.view(-1), out, workspace=ws)
        finally:
            L.lib().rbSetGemmVariant(0)
        torch.cuda.synchronize()
        got.append((out.view(n, cfg.ho, cfg.wo, k).permute(0, 3, 1, 2) if lay[2] == "nhwgk" else out.view(n, k, cfg.ho, cfg.wo)).double())
    assert L.kernel_status() == 0
    with torch.backends.cudnn.flags(enabled=False):
        want = torch.nn.functional.conv2d(x.double(), w.double(), stride=stride, padding=pad, dilation=dil)
    err = [((g - want).norm() / want.norm()).item() for g in got]
    assert err[0] <= 1.001 * err[1], err
