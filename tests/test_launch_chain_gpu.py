"""Kernels are set up while their predecessor in the stream still runs and wait for its end before they touch memory. Chains in which
every call reads what the one before wrote, or overwrites what it read, give the bits of the same calls with a synchronisation after each."""
import math

import pytest

pytestmark = pytest.mark.gpu


def steps():
    import torch
    from rocmlir_b200 import conv as rb_conv
    from rocmlir_b200.attention import attention
    from rocmlir_b200.gemm import Epilogue, gemm, problem, workspace_size
    gen = torch.Generator(device="cuda").manual_seed(2)
    t = lambda *s, dt=torch.float16: (torch.randn(s, device="cuda", generator=gen) * 0.1).to(dt)
    n, h, c = 8, 28, 64
    x, dy = t(n, h, h, c), torch.empty((n, h, h, c), dtype=torch.float16, device="cuda")
    fil, fil_s, stem = t(c, 3, 3, c), t(c, 3, 3, c), t(c, 7, 7, 3)
    unit = rb_conv.ConvConfig(n, c, c, h, h, 3, 3, pad_h=1, pad_w=1, fil_layout="gkyxc", in_layout="nhwgc", out_layout="nhwgk")
    half = rb_conv.ConvConfig(n, c, c, h, h, 3, 3, stride_h=2, stride_w=2, pad_h=1, pad_w=1, fil_layout="gkyxc", in_layout="nhwgc", out_layout="nhwgk")
    image = rb_conv.ConvConfig(n, 3, c, h, h, 7, 7, stride_h=2, stride_w=2, pad_h=3, pad_w=3, fil_layout="gkyxc", in_layout="nhwgc", out_layout="nhwgk")
    small = torch.empty((n, half.ho, half.wo, c), dtype=torch.float16, device="cuda")
    ws = torch.empty(64 << 20, dtype=torch.uint8, device="cuda")   # one workspace for every call
    op = rb_conv.OPERATIONS

    def conv(cfg, which, f, i, o):
        rb_conv.conv(cfg, op[which], f.view(-1), i.view(-1), o.view(-1), workspace=ws)

    def mm(a, b, out, **kw):
        gemm(a, b, out=out, workspace=ws, out_dtype=out.dtype, **kw)

    att, w = torch.empty((n, 784, c), dtype=torch.float16, device="cuda"), t(1, 512, 64)
    few, deep, odd = (torch.empty(s, dtype=torch.float16, device="cuda") for s in ((1, 16, 512), (1, 64, 64), (1, 61, 61)))
    single = torch.empty((1, 64, 64), dtype=torch.float32, device="cuda")
    bias = t(64)
    return [x, dy, small, fil, fil_s, att, few, deep, odd, single], [
        lambda: conv(unit, "conv", fil, x, dy),
        lambda: attention(dy.view(n, 784, c), dy.view(n, 784, c), x.view(n, 784, c), trans_k=True, scale=0.125, causal=True, out=att),
        lambda: conv(half, "conv", fil_s, att, small),
        lambda: conv(half, "conv_bwd_data", fil_s, x, small),            # x again, which the calls above read
        lambda: conv(half, "conv_bwd_weight", fil, x, small),            # the filter of the first call
        lambda: mm(x.view(1, -1, 64)[:, :16], w, few, trans_b=True),
        lambda: attention(few.view(64, 1, 128), few.view(64, 1, 128), few.view(64, 1, 128), trans_k=True, scale=0.1, out=few.view(64, 1, 128)),
        lambda: mm(dy.view(1, -1, 64), x.view(1, -1, 64), deep, trans_a=True),   # K in ranges and their sum
        lambda: mm(deep[:, :61, :61].contiguous(), deep[:, :61, :61].contiguous(), odd),   # operands and rows off 16 bytes
        lambda: mm(deep.float(), deep.float(), single, trans_b=True),
        lambda: small.view(-1)[:3721].copy_(odd.view(-1)),
        lambda: conv(image, "conv", stem, dy.view(-1)[:n * h * h * 3], small),
        lambda: x.add_(small.repeat_interleave(2, 1).repeat_interleave(2, 2), alpha=1e-3),
    ]


def test_chain_of_calls(cuda_device):
    import torch
    from rocmlir_b200 import _lib as L
    seen = []
    for wait in (True, False):
        tensors, calls = steps()
        for _ in range(6):
            for call in calls:
                call()
                if wait:
                    torch.cuda.synchronize()
        torch.cuda.synchronize()
        assert L.kernel_status() == 0
        seen.append([x.clone() for x in tensors])
    for a, b in zip(*seen):
        assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))   # bits: a NaN equals itself
