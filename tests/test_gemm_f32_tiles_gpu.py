"""f32 products on both sides of the line between tiles of 256 and of 128 columns (K up to 256 with more tiles than CTA pairs):
whole and ragged tiles, rows of C on and off 16 bytes, the smallest K, the last K on either side."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("trans_b", [False, True])
@pytest.mark.parametrize("g,m,n,k", [(1, 2560, 2304, 256), (1, 2560, 2304, 257), (1, 2561, 2053, 100), (1, 2304, 2304, 8), (19, 256, 1024, 31),
                                     (19, 300, 700, 128), (1, 2048, 2048, 64)])
def test_short_k(cuda_device, g, m, n, k, trans_b):
    import torch
    from rocmlir_b200 import _lib as L
    from rocmlir_b200.gemm import gemm
    gen = torch.Generator(device="cuda").manual_seed(11)
    a = torch.randn((g, m, k), device="cuda", generator=gen)
    b = torch.randn((g, n, k) if trans_b else (g, k, n), device="cuda", generator=gen)
    got = gemm(a, b, trans_b=trans_b)
    torch.cuda.synchronize()
    assert L.kernel_status() == 0
    bd = (b.transpose(1, 2) if trans_b else b).double()
    # per product: hi + lo of each operand is exact to 2^-23, lo . lo (2^-24) is left out; every eight products are added with a
    # truncation of 2^-24 of the sum so far, 33 times at most
    bound = (a.double().abs() @ bd.abs()) * (2.0 ** -21 + 34 * 2.0 ** -24)
    assert ((got.double() - a.double() @ bd).abs() <= bound).all()
