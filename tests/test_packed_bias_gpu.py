"""[round] -> [+ bias, round] -> [ReLU] on packed 16-bit pairs (bias, declared type and result of one 16-bit type) against the steps in f32
that a bias of another type, holding the same values, takes: bit for bit, for GEMM tiles of every width, rows off 16 bytes and the
convolution kernel with its filter in shared memory; values over the whole range of the type."""
import pytest

pytestmark = pytest.mark.gpu


def spread(shape, dtype, gen):
    """Values of all magnitudes, both signs, with zeros, infinities and NaN among them."""
    import torch
    x = torch.randn(shape, device="cuda", generator=gen) * torch.exp2(torch.randint(-26, 17, shape, device="cuda", generator=gen).float())
    x.view(-1)[::97] = 0.0
    x.view(-1)[5::1009] = float("inf")
    x.view(-1)[7::1013] = float("nan")
    return x.to(dtype)


@pytest.mark.parametrize("relu", [False, True])
@pytest.mark.parametrize("dt", ["float16", "bfloat16"])
@pytest.mark.parametrize("m,n,k,variant", [(70, 64, 64, 0x1001), (129, 200, 128, 0x2001), (300, 512, 64, 0x3002), (65, 131, 64, 1), (256, 1024, 96, 0x3001)])
def test_gemm(cuda_device, m, n, k, variant, dt, relu):
    import torch
    from rocmlir_b200 import _lib as L
    from rocmlir_b200.gemm import Epilogue, gemm, rb_dtype
    dtype = getattr(torch, dt)
    gen = torch.Generator(device="cuda").manual_seed(3)
    a, b = spread((m, k), dtype, gen), torch.zeros((k, n), dtype=dtype, device="cuda")
    b[torch.arange(n, device="cuda") % k, torch.arange(n, device="cuda")] = 1.0   # every column of the product is a column of A
    a = torch.nan_to_num(a, nan=1.5, posinf=2.0, neginf=-3.0)                      # (a zero times an infinity would spread)
    bias = spread((n,), dtype, gen)
    got = [gemm(a, b, epilogue=Epilogue(bias=v, relu=relu, mid_type=rb_dtype(dtype)), variant=variant) for v in (bias, bias.float())]
    torch.cuda.synchronize()
    assert torch.equal(got[0].isnan(), got[1].isnan()) and torch.equal(got[0].nan_to_num(7.0), got[1].nan_to_num(7.0))
    assert L.kernel_status() == 0


@pytest.mark.parametrize("relu", [False, True])
@pytest.mark.parametrize("dt", ["float16", "bfloat16"])
@pytest.mark.parametrize("n,k,hw,f", [(3, 64, 13, 3), (2, 32, 30, 1), (1, 96, 8, 3)])
def test_convolution(cuda_device, n, k, hw, f, dt, relu):
    import torch
    from rocmlir_b200 import _lib as L
    from rocmlir_b200.conv import ConvConfig, conv_fused
    from rocmlir_b200.gemm import Epilogue, rb_dtype
    dtype = getattr(torch, dt)
    gen = torch.Generator(device="cuda").manual_seed(4)
    cfg = ConvConfig(n, 64, k, hw, hw, f, f, pad_h=f // 2, pad_w=f // 2, fil_layout="gkyxc", in_layout="nhwgc", out_layout="nhwgk")
    fil, inp = (torch.randn(cfg.numel(w), device="cuda", generator=gen).to(dtype) for w in ("fil", "in"))
    bias = spread((k,), dtype, gen)
    got = []
    for v in (bias, bias.float()):
        out = torch.empty(cfg.numel("out"), dtype=dtype, device="cuda")
        conv_fused(cfg, fil, inp, out, Epilogue(bias=v, relu=relu, mid_type=rb_dtype(dtype)))
        got.append(out)
    torch.cuda.synchronize()
    assert torch.equal(got[0].isnan(), got[1].isnan()) and torch.equal(got[0].nan_to_num(7.0), got[1].nan_to_num(7.0))
    assert L.kernel_status() == 0
