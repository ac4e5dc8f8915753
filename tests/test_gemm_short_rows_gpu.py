"""Products of fewer rows than a tile: only the rows that exist (rounded up to eight) are loaded. Small whole numbers, so every sum is exact."""
import pytest
import torch

from rocmlir_b200.gemm import gemm

pytestmark = pytest.mark.gpu


def whole(shape, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randint(-2, 3, shape, generator=g, device="cuda").to(dtype)


@pytest.mark.parametrize("m", [1, 7, 8, 9, 63, 65, 119, 120, 121, 127, 128])
@pytest.mark.parametrize("dtype,out", [("float16", "float16"), ("bfloat16", "float32"), ("int8", "int32"), ("float32", "float32")])
@pytest.mark.parametrize("g,n,k,trans_b", [(1, 200, 72, False), (3, 320, 432, True), (1, 64, 2064, True)])
def test_rows(m, dtype, out, g, n, k, trans_b):
    dt, ct = getattr(torch, dtype), getattr(torch, out)
    a = whole((g, m, k), dt, m)
    b = whole((g, n, k) if trans_b else (g, k, n), dt, m + 1)
    want = torch.bmm(a.float(), (b.transpose(1, 2) if trans_b else b).float())
    c = torch.full((g, m + 1, n), 77, device="cuda").to(ct)[:, :m].contiguous()
    gemm(a, b, trans_b=trans_b, out=c, out_dtype=ct)
    assert torch.equal(c.float(), want.to(ct).float())


def test_rows_of_f16_planes():
    """100 x 8192 x 8192 f32: enough work for f16 planes."""
    a, b = whole((1, 100, 8192), torch.float32, 1), whole((1, 8192, 8192), torch.float32, 2)
    c = torch.empty(1, 100, 8192, device="cuda")
    gemm(a, b, trans_b=True, out=c)
    assert torch.equal(c.double(), torch.bmm(a.double(), b.double().transpose(1, 2)))
