"""Tiles beyond the last row of C store nothing; the staging rows of the tile before them are still being read. Short sums of many tiles in groups,
small whole numbers, so every result is exact; many runs, since what it shows is a matter of timing."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,out,k", [("float32", "float32", 51), ("float16", "float16", 72), ("int8", "int32", 80)])
@pytest.mark.parametrize("m,n", [(2056, 1976), (1631, 2104), (1626, 2176)])
def test_rows_beyond_the_last_leave_the_staged_ones_alone(cuda_device, dtype, out, k, m, n):
    import torch
    from rocmlir_b200.gemm import gemm
    dt, ct = getattr(torch, dtype), getattr(torch, out)
    g = torch.Generator(device="cuda").manual_seed(m)
    a, b = (torch.randint(-2, 3, (3, r, k), generator=g, device="cuda").to(dt) for r in (m, n))
    want = torch.bmm(a.float(), b.float().transpose(1, 2)).to(ct)
    c, wrong = torch.empty_like(want), torch.zeros((), dtype=torch.int64, device="cuda")
    for _ in range(300):
        c.fill_(77)
        gemm(a, b, trans_b=True, out=c, out_dtype=ct)
        wrong += (c != want).sum()
    assert wrong.item() == 0
