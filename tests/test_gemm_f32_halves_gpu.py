"""f32 operands as two f16 planes (large products): no further from the 64-bit result than the TF32 planes that a call without room for their state
takes, and bit for bit those wherever an operand does not fit f16's range - seen in the sample or only by the pass itself."""
import math

import pytest

pytestmark = pytest.mark.gpu
RULE = 1 << 27   # an explicit variant word: TF32 planes


def both(a, b, out=None, **kw):
    """The product with all of its workspace and with 256 bytes less."""
    import torch
    from rocmlir_b200 import _lib as L
    from rocmlir_b200.gemm import gemm, problem, workspace_size
    p = problem(a, b, kw.get("trans_a", False), kw.get("trans_b", False), False, torch.float32)
    res = []
    for room in (0, 256):
        ws = torch.empty(workspace_size(p) - room, dtype=torch.uint8, device="cuda")
        res.append(gemm(a, b, out_dtype=torch.float32, workspace=ws, **kw).clone())
        torch.cuda.synchronize()
    assert L.kernel_status() == 0
    return res


def normal(*shape, seed=0):
    import torch
    return torch.randn(shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed))


def error(got, want):
    return ((got.double() - want).norm() / want.norm()).item()


@pytest.mark.parametrize("g,m,n,k,ta,tb", [(1, 2048, 2048, 1024, False, False), (1, 1999, 2001, 1003, False, True), (1, 1024, 1024, 4160, True, False),
                                           (1, 2300, 900, 2049, True, True), (3, 1100, 1300, 1000, False, True), (1, 64, 8192, 8192, False, True),
                                           (1, 8200, 4100, 130, False, False)])
def test_error_is_no_larger(cuda_device, g, m, n, k, ta, tb):
    import torch
    for scale in (1.0, 1e-25, 1e15):
        a, b = normal(*((g, k, m) if ta else (g, m, k)), seed=1) * scale, normal(*((g, n, k) if tb else (g, k, n)), seed=2)
        half, tf32 = both(a, b, trans_a=ta, trans_b=tb)
        want = (a.double().transpose(1, 2) if ta else a.double()) @ (b.double().transpose(1, 2) if tb else b.double())
        assert not torch.equal(half, tf32)   # the f16 planes were taken
        assert error(half, want) <= 1.001 * error(tf32, want)


@pytest.mark.parametrize("kind", ["relu", "uniform", "rows", "sparse", "integers"])
def test_other_distributions(cuda_device, kind):
    import torch
    a, b = normal(1, 2048, 2048, seed=3), normal(1, 2048, 2048, seed=4)
    if kind == "relu":
        a = a.relu()
    if kind == "uniform":
        a, b = torch.rand_like(a), torch.rand_like(b) * 2 - 1
    if kind == "rows":      # three decades, row by row and column by column
        a = a * torch.logspace(-1.5, 1.5, 2048, device="cuda")[None, :, None]
        b = b * torch.logspace(-1.5, 1.5, 2048, device="cuda")[None, None, :]
    if kind == "sparse":
        a = a * (torch.rand_like(a) < 0.01)
    if kind == "integers":  # exact in both
        a, b = a.mul(3).round(), b.mul(3).round()
    half, tf32 = both(a, b)
    want = a.double() @ b.double()
    assert error(half, want) <= 1.001 * error(tf32, want)
    if kind == "integers":
        assert torch.equal(half.double(), want)


@pytest.mark.parametrize("kind", ["huge", "huge_unsampled", "rows", "row_unsampled", "k", "inf", "nan", "subnormal", "largest", "alternate"])
@pytest.mark.parametrize("which", [0, 1])
def test_operands_that_do_not_fit_take_tf32_planes(cuda_device, kind, which):
    import torch
    x, y = normal(1, 2048, 2048, seed=5), normal(1, 2048, 2048, seed=6)
    if which:   # the other operand, whose K runs down the rows
        x = x.transpose(1, 2).contiguous()
    rows, cols = ((2, 1) if which else (1, 2))
    if kind == "huge":
        x.select(rows, 17).mul_(1e9)
    if kind == "huge_unsampled":
        x[0, 1031, 77] = 1e7
    if kind == "rows":
        x = x * torch.logspace(-9, 9, 2048, device="cuda").view((1, 2048, 1) if rows == 1 else (1, 1, 2048))
    if kind == "row_unsampled":
        x.select(rows, 1033).mul_(1e-9)
    if kind == "k":
        x = x * torch.logspace(-6, 6, 2048, device="cuda").view((1, 1, 2048) if cols == 2 else (1, 2048, 1))
    if kind == "inf":
        x[0, 3, 1999] = math.inf
    if kind == "nan":
        x[0, 1500, 2] = math.nan
    if kind == "subnormal":
        x = x * 1e-41
    if kind == "largest":
        x[0, 5, 6] = 3.4e38
    if kind == "alternate":
        mask = (torch.arange(2048, device="cuda") % 2 == 0).view((1, 1, 2048) if cols == 2 else (1, 2048, 1))
        x = torch.where(mask, x * 1e-7, x)
    half, tf32 = both(y, x) if which else both(x, y)
    assert torch.equal(half.view(torch.int32), tf32.view(torch.int32))


def test_zeros_epilogue_and_result_over_an_operand(cuda_device):
    import torch
    from rocmlir_b200.gemm import Epilogue, gemm, problem, workspace_size
    a, b, bias = normal(1, 2048, 2048, seed=7), normal(1, 2048, 2048, seed=8), normal(2048, seed=9)
    for x in both(torch.zeros_like(a), b):
        assert not x.any()
    plain, fused = both(a, b)[0], both(a, b, epilogue=Epilogue(bias=bias, relu=True))[0]
    assert torch.equal(fused, (plain + bias).relu())
    ws = torch.empty(workspace_size(problem(a, b, False, False, False, torch.float32)), dtype=torch.uint8, device="cuda")
    over = a.clone()
    gemm(over, b, out=over, workspace=ws)
    assert torch.equal(over, plain)


@pytest.mark.parametrize("layout", ["nchw", "nhwc"])
@pytest.mark.parametrize("n,c,k,hw,fil,stride,fits", [(24, 128, 128, 28, 3, 1, True), (20, 256, 64, 28, 3, 1, True), (20, 192, 130, 33, 3, 2, True),
                                                      (24, 128, 128, 28, 3, 1, False)])
def test_convolution(cuda_device, layout, n, c, k, hw, fil, stride, fits):
    import torch
    from rocmlir_b200 import _lib as L
    from rocmlir_b200 import conv as rb_conv
    last = layout == "nhwc"
    lay = ("gkyxc", "nhwgc", "nhwgk") if last else ("gkcyx", "ngchw", "ngkhw")
    cfg = rb_conv.ConvConfig(n, c, k, hw, hw, fil, fil, stride_h=stride, stride_w=stride, pad_h=1, pad_w=1, fil_layout=lay[0], in_layout=lay[1],
                             out_layout=lay[2])
    x, w = normal(n, c, hw, hw, seed=10), normal(k, c, fil, fil, seed=11)
    if not fits:
        x[n // 2] *= 1e8
    order = (0, 2, 3, 1) if last else (0, 1, 2, 3)
    xs, wsrc = x.permute(order).contiguous(), w.permute(order).contiguous()
    got = []
    for variant in (0, RULE):
        out = torch.empty(cfg.numel("out"), device="cuda")
        L.lib().rbSetGemmVariant(variant)
        try:
            ws = torch.empty(max(16, rb_conv.workspace_size(cfg, torch.float32, rb_conv.OPERATIONS["conv"])), dtype=torch.uint8, device="cuda")
            rb_conv.conv(cfg, rb_conv.OPERATIONS["conv"], wsrc.view(-1), xs.view(-1), out, workspace=ws)
        finally:
            L.lib().rbSetGemmVariant(0)
        torch.cuda.synchronize()
        o = out.view(n, cfg.ho, cfg.wo, k).permute(0, 3, 1, 2) if last else out.view(n, k, cfg.ho, cfg.wo)
        got.append(o.contiguous())
    assert L.kernel_status() == 0
    if not fits:
        assert torch.equal(got[0], got[1])
        return
    with torch.backends.cudnn.flags(enabled=False):
        want = torch.nn.functional.conv2d(x.double(), w.double(), stride=stride, padding=1)
    assert not torch.equal(got[0], got[1]) and error(got[0], want) <= 1.001 * error(got[1], want)


@pytest.mark.parametrize("m,n,k", [(128, 1152, 50176), (128, 1100, 49920), (100, 2048, 20544), (300, 384, 40000)])
def test_every_range_of_k_has_blocks(cuda_device, m, n, k):
    """Ranges counted in blocks of 32, of which a range of blocks of 64 may have none left: every plane that is summed has been written. The
    workspace starts as NaN; sums of small whole numbers are exact."""
    import torch
    from rocmlir_b200.gemm import gemm, problem, workspace_size
    g = torch.Generator(device="cuda").manual_seed(k)
    a, b = (torch.randint(-2, 3, (1, r, k), generator=g, device="cuda").float() for r in (m, n))
    ws = torch.full((workspace_size(problem(a, b, False, True, False, torch.float32)) // 4 + 64,), float("nan"), device="cuda").view(torch.uint8)
    c = torch.empty(1, m, n, device="cuda")
    gemm(a, b, trans_b=True, out=c, workspace=ws)
    assert torch.equal(c.double(), torch.bmm(a.double(), b.double().transpose(1, 2)))


def worst(got, want, size, dim):
    """Largest error along `dim` in units of the sum of the magnitudes that were added (|A||B|)."""
    return ((got.double() - want).abs() / size.clamp(min=1e-300)).amax(dim)


def no_worse(half, tf32, a, b):
    """Row by row and column by column, no further from the 64-bit result than the TF32 form, apart from what both may leave of each single
    product: lo.lo, 2^-22 of it, and 2^-23 of it for the rounding of each lo, 2^-21 together."""
    want, size = a.double() @ b.double(), a.double().abs() @ b.double().abs()
    for dim in (1, 2):
        assert (worst(half, want, size, dim) <= 2 * worst(tf32, want, size, dim) + 2.0 ** -21).all()


def uneven(kind, shape, seed):
    """Operands most of which are zero, or some of whose values are far below the others, rows first."""
    import torch
    x = normal(*shape, seed=seed)
    rows, cols = shape[1], shape[2]
    r, c = torch.arange(rows, device="cuda")[:, None], torch.arange(cols, device="cuda")[None, :]
    gen = torch.Generator(device="cuda").manual_seed(seed + 1)
    some = torch.rand(shape, device="cuda", generator=gen)
    fall = lambda lo, n: torch.logspace(0, lo, n, device="cuda", dtype=torch.float64).float()
    if kind.startswith("superdiagonal"):
        x = torch.where(c == r + 64, 1 + some, 0) * float(kind[13:])
    if kind == "diagonal":
        x = torch.where(c == r, 1 + some, 0) * fall(-9, rows)[None, :, None]
    if kind == "few":
        x = x * (some < 0.05) * 1e-4 * (c >= 32)
    if kind == "few_by_rows":
        x = x * (some < 0.05) * fall(-8, rows)[None, :, None]
    if kind == "sparse_row":
        x = torch.where(r == 1033, x * (some < 0.2) * 1e-9, x)
    if kind == "relu_row":
        x = torch.where(r == 1033, x.relu() * (c % 4 == 0) * 1e-12, x)
    if kind == "dense_row_underflows":
        x = torch.where(r == 1033, x * 1e-25, x * 1e30)
    if kind == "low_columns":
        x = torch.where(c % 64 < 12, x * 1e-9, x)
    if kind == "one_low_column":
        x = torch.where(c == 77, x * 1e-8, x)
    if kind == "scattered":
        x = torch.where(some < 1e-3, x * 1e-10, x)
    if kind == "one_value":
        x[0, 1033, 77] = 1e-9
    return x.contiguous()


UNEVEN = ["superdiagonal1.1e-3", "superdiagonal1e-4", "superdiagonal1e-9", "diagonal", "few", "few_by_rows", "sparse_row", "relu_row",
          "dense_row_underflows", "low_columns", "one_low_column", "scattered", "one_value"]


@pytest.mark.parametrize("kind", UNEVEN)
@pytest.mark.parametrize("other", ["normal", "identity"])
@pytest.mark.parametrize("which", [0, 1])
def test_small_values_keep_their_digits(cuda_device, kind, other, which):
    import torch
    x = uneven(kind, (1, 2048, 2048), 21)
    y = torch.eye(2048, device="cuda")[None].contiguous() if other == "identity" else normal(1, 2048, 2048, seed=23)
    if which:
        x = x.transpose(1, 2).contiguous()
    a, b = (y, x) if which else (x, y)
    no_worse(*both(a, b), a, b)


@pytest.mark.parametrize("which", [0, 1])
def test_short_sums_keep_the_digits_of_small_rows(cuda_device, which):
    import torch
    x, y = normal(1, 16384, 16, seed=31), normal(1, 16384, 16, seed=32)
    x[:, 1::2] *= 1e-9
    a, b = (y, x) if which else (x, y)
    half, tf32 = both(a, b, trans_b=True)
    no_worse(half, tf32, a, b.transpose(1, 2))


@pytest.mark.parametrize("seed", range(4))
def test_ordinary_operands_take_f16_planes(cuda_device, seed):
    """4096 x 4096 normal values: now and then a single one lies below what f16 planes hold in full (none of these four below 2^-18)."""
    import torch
    a, b = normal(1, 4096, 4096, seed=100 + seed), normal(1, 4096, 4096, seed=200 + seed)
    half, tf32 = both(a, b)
    assert not torch.equal(half, tf32)
    no_worse(half, tf32, a, b)


@pytest.mark.parametrize("layout", ["nchw", "nhwc"])
@pytest.mark.parametrize("c", [40, 128])
@pytest.mark.parametrize("kind", ["dim_image", "few", "dim_filter"])
def test_convolution_keeps_the_digits_of_small_values(cuda_device, layout, c, kind):
    import torch
    from rocmlir_b200 import _lib as L
    from rocmlir_b200 import conv as rb_conv
    n, k, hw, last = 48, 128, 28, layout == "nhwc"
    lay = ("gkyxc", "nhwgc", "nhwgk") if last else ("gkcyx", "ngchw", "ngkhw")
    cfg = rb_conv.ConvConfig(n, c, k, hw, hw, 3, 3, pad_h=1, pad_w=1, fil_layout=lay[0], in_layout=lay[1], out_layout=lay[2])
    x, w = normal(n, c, hw, hw, seed=41), normal(k, c, 3, 3, seed=42)
    if kind == "dim_image":
        x[n // 2] *= (normal(c, hw, hw, seed=43) > 1.0) * 1e-9
    if kind == "few":
        x = x * (normal(n, c, hw, hw, seed=43) > 2.0) * 1e-4
        x[:, :32] = 0
        x[0, 0, 0, 0] = 1.0
    if kind == "dim_filter":
        w[17] *= (normal(c, 3, 3, seed=43) > 1.0) * 1e-9
    order = (0, 2, 3, 1) if last else (0, 1, 2, 3)
    xs, wsrc = x.permute(order).contiguous(), w.permute(order).contiguous()
    got = []
    for variant in (0, RULE):
        out = torch.empty(cfg.numel("out"), device="cuda")
        L.lib().rbSetGemmVariant(variant)
        try:
            ws = torch.empty(max(16, rb_conv.workspace_size(cfg, torch.float32, rb_conv.OPERATIONS["conv"])), dtype=torch.uint8, device="cuda")
            rb_conv.conv(cfg, rb_conv.OPERATIONS["conv"], wsrc.view(-1), xs.view(-1), out, workspace=ws)
        finally:
            L.lib().rbSetGemmVariant(0)
        torch.cuda.synchronize()
        got.append((out.view(n, cfg.ho, cfg.wo, k).permute(0, 3, 1, 2) if last else out.view(n, k, cfg.ho, cfg.wo)).reshape(n * k, -1))
    assert L.kernel_status() == 0
    with torch.backends.cudnn.flags(enabled=False):
        want, size = (torch.nn.functional.conv2d(p.double(), q.double(), padding=1).reshape(n * k, -1) for p, q in ((x, w), (x.abs(), w.abs())))
    for dim in (0, 1):   # (per image and filter, per filter and pixel over the images)
        assert (worst(got[0], want, size, dim) <= 2 * worst(got[1], want, size, dim) + 2.0 ** -21).all()
