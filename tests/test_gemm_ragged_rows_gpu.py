"""Results whose rows do not start on 16-byte boundaries (staged in shared memory, copied out by the warps): integer-valued
operands, so they equal the 64-bit product exactly; with a fused tail they equal the element-wise stores of an explicit variant.
What lies before and behind the result stays as it was."""
import pytest

pytestmark = pytest.mark.gpu
PLAIN = 1 << 8   # variant word: element-wise stores

# (g, m, n, k): one row and one column; around the warp's 32 rows and the 64 / 32 columns of a staging row; ragged tiles of
# 64, 128 and 256 columns; a K split (its planes have the same rows)
SHAPES = [(1, 1, 1, 64), (2, 33, 63, 64), (1, 65, 65, 128), (1, 128, 127, 64), (3, 257, 259, 96), (1, 130, 1663, 512),
          (1, 70, 515, 2048), (2, 300, 31, 80)]
TYPES = [("float16", "float16"), ("bfloat16", "bfloat16"), ("float16", "float32"), ("float32", "float32"), ("int8", "int32"),
         ("float8_e4m3fn", "bfloat16")]


def run(a, b, out_dtype, off, epilogue=None, **kw):
    import torch
    from rocmlir_b200.gemm import gemm
    g, m, n = a.shape[0], a.shape[1], b.shape[1]
    buf = torch.full((g * m * n + 128,), 77, device="cuda").to(out_dtype)
    out = buf[off:off + g * m * n].view(g, m, n)
    gemm(a, b, trans_b=True, out_dtype=out_dtype, out=out, epilogue=epilogue, **kw)
    torch.cuda.synchronize()
    guard = torch.full((1,), 77, device="cuda").to(out_dtype).float()
    assert (buf[:off].float() == guard).all() and (buf[off + g * m * n:].float() == guard).all()
    return out


@pytest.mark.parametrize("off", [0, 1, 2])
@pytest.mark.parametrize("g,m,n,k", SHAPES)
@pytest.mark.parametrize("dt,out", TYPES)
def test_rows_anywhere(cuda_device, dt, out, g, m, n, k, off):
    import torch
    from rocmlir_b200 import _lib as L
    gen = torch.Generator(device="cuda").manual_seed(7)
    a, b = (torch.randint(-2, 3, s, device="cuda", generator=gen).float() for s in ((g, m, k), (g, n, k)))
    ref = (a.double() @ b.double().transpose(1, 2)).to(getattr(torch, out))
    got = run(a.to(getattr(torch, dt)), b.to(getattr(torch, dt)), getattr(torch, out), off)
    assert torch.equal(got, ref) and L.kernel_status() == 0


@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("g,m,n,k", SHAPES[:6])
def test_fused_tails_equal_element_stores(cuda_device, g, m, n, k, off):
    import torch
    from rocmlir_b200 import _lib as L
    from rocmlir_b200.gemm import Epilogue
    gen = torch.Generator(device="cuda").manual_seed(8)
    ints = lambda s, dt: torch.randint(-4, 5, s, device="cuda", generator=gen).to(dt)
    bias, scale = torch.randn(n, device="cuda", generator=gen), torch.rand(n, device="cuda", generator=gen)
    cases = [(torch.float16, torch.float16, dict(bias=bias.half(), relu=True, mid_type=L.F16)),
             (torch.float16, torch.float32, dict(alpha=0.3, bias=bias, unary="tanh")),
             (torch.bfloat16, torch.bfloat16, dict(bias=bias[:1].contiguous(), bias_mode="scalar", clip=(-1.0, 2.0))),
             (torch.int8, torch.int8, dict(col_scale=scale, requant_scale=3.0, out_zero=2))]
    for dt, out, kw in cases:
        a, b = ints((g, m, k), dt), ints((g, n, k), dt)
        got = [run(a, b, out, off, epilogue=Epilogue(**kw), variant=v) for v in (1, 1 | PLAIN)]
        assert torch.equal(got[0], got[1]), (dt, out, kw.keys())
    assert L.kernel_status() == 0


@pytest.mark.parametrize("m,n", [(64, 128), (33, 192), (200, 80), (130, 1344), (128, 65)])
@pytest.mark.parametrize("off", [0, 1])
def test_eight_bit_results_in_narrow_tiles(cuda_device, m, n, off):
    """Tiles of 64 columns are half of a staged row of bytes: they do not touch the columns of their neighbours."""
    import torch
    from rocmlir_b200 import _lib as L
    from rocmlir_b200.gemm import Epilogue
    gen = torch.Generator(device="cuda").manual_seed(8)
    a, b = (torch.randint(-9, 10, (1, r, 256), device="cuda", generator=gen).to(torch.int8) for r in (m, n))
    epi = Epilogue(col_scale=torch.rand(n, device="cuda", generator=gen), requant_scale=3.0)
    got = [run(a, b, torch.int8, off, epilogue=epi, variant=v) for v in (0x1001, 0x2001 | PLAIN)]   # 64 columns, 128
    assert torch.equal(got[0], got[1]) and L.kernel_status() == 0


@pytest.mark.parametrize("dt,g,m,n,k", [("float16", 1, 64, 1023, 256), ("bfloat16", 1, 63, 567, 64), ("float16", 1, 36, 1030, 256), ("float16", 1, 37, 1030, 256),
                                        ("float16", 1, 35, 10245, 64), ("float16", 1, 64, 1023, 4096), ("bfloat16", 3, 64, 515, 2048)])
def test_few_rows_take_the_faster_kernel(cuda_device, dt, g, m, n, k):
    """At most 64 rows against weights stored N x K: the library's choice against the general kernel in its own configuration."""
    import ctypes as C
    import torch
    from rocmlir_b200 import _lib as L
    from rocmlir_b200.gemm import gemm, problem, workspace_size
    from test_dispatch_lines_gpu import under
    t = getattr(torch, dt)
    a, b, c = (torch.randn(s, device="cuda").to(t) for s in ((g, m, k), (g, n, k), (g, m, n)))
    p, general = problem(a, b, False, True, False, t), L.RbGemmConfigInfo()
    ws = torch.empty(max(16, workspace_size(p)), dtype=torch.uint8, device="cuda")
    L.check(L.lib().rbGemmGetConfig(C.byref(p), C.byref(general)))
    run = lambda: gemm(a, b, trans_b=True, out=c, workspace=ws)
    assert under(0, run) <= 1.25 * under(general.variant, run)
