"""f32 products whose K is cut into ranges of at most 2048 elements: operands of small whole numbers (times a power of two), so that
every partial sum is exact and the result must equal the 64-bit product bit for bit."""
import pytest

pytestmark = pytest.mark.gpu

# (g, m, n, k, ranges): from the shortest K that needs two on; ragged tiles, several groups, rows off 16 bytes; a short K that few tiles cut in two
SHAPES = [(1, 1100, 2308, 2048, 1), (1, 1100, 2308, 2049, 2), (3, 1029, 1028, 4096, 2), (2, 769, 1539, 2600, 2), (1, 1100, 2308, 4097, 3),
          (1, 684, 64, 576, 2), (1, 130, 260, 2304, 9)]


def operands(g, m, n, k, scale=1.0):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(5)
    a, b = (torch.randint(-3, 4, s, device="cuda", generator=gen).float() for s in ((g, m, k), (g, k, n)))
    return a * scale, b * scale, a.double() @ b.double()


def ranges(a, b, f32_mode=0):
    import ctypes as C
    import torch
    from rocmlir_b200 import _lib as L
    from rocmlir_b200.gemm import problem
    p, info = problem(a, b, False, False, False, torch.float32, f32_mode), L.RbGemmConfigInfo()
    L.check(L.lib().rbGemmGetConfig(C.byref(p), C.byref(info)))
    return info.splits


@pytest.mark.parametrize("g,m,n,k,cut", SHAPES)
def test_ranges_add_up(cuda_device, g, m, n, k, cut):
    """Whatever the result held before, call after call, and replayed from a graph."""
    import torch
    from rocmlir_b200 import _lib as L
    from rocmlir_b200.gemm import gemm, problem, workspace_size
    a, b, ref = operands(g, m, n, k)
    assert ranges(a, b) == cut
    out = torch.full((g, m, n), float("nan"), device="cuda")
    ws = torch.empty(max(16, workspace_size(problem(a, b, False, False, False, torch.float32))), dtype=torch.uint8, device="cuda")
    for _ in range(3):
        gemm(a, b, out=out, workspace=ws)
        assert torch.equal(out, ref.float())
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.stream(side), torch.cuda.graph(graph, stream=side):
        gemm(a, b, out=out, workspace=ws)
    for _ in range(2):
        out.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, ref.float())
    assert L.kernel_status() == 0


@pytest.mark.parametrize("k,cut,f32_mode", [(2048, 1, 0), (2052, 2, 0), (3000, 2, 0), (4096, 2, 0), (4100, 3, 0), (1536, 2, 1)])
@pytest.mark.parametrize("over", ["a", "b"])
def test_the_result_may_lie_over_an_operand(cuda_device, over, k, cut, f32_mode):
    """The operands have been read before the result is written (a single TF32 pass: before the sum of the ranges is)."""
    import torch
    from rocmlir_b200.gemm import gemm
    g, m, n = (1, 1100, k) if over == "a" else (1, k, 1100)
    a, b, ref = operands(g, m, n, k)
    assert ranges(a, b, f32_mode) == cut
    out = gemm(a, b, out=a if over == "a" else b, f32_mode=f32_mode)
    assert torch.equal(out, ref.float())


@pytest.mark.parametrize("exponent", [-70, -67])
@pytest.mark.parametrize("k,cut", [(2048, 1), (2304, 2), (4096, 2), (4100, 3)])
def test_subnormal_sums_are_kept(cuda_device, k, cut, exponent):
    """Products of 2^-140: every sum is a subnormal number, exact in f32. Of 2^-134: some partial sums are normal numbers, some results not."""
    import torch
    from rocmlir_b200.gemm import gemm
    a, b, ref = operands(1, 1100, 2308, k, scale=2.0 ** exponent)
    assert ranges(a, b) == cut
    out = gemm(a, b).cpu()
    ref = (ref.cpu() * 2.0 ** (2 * exponent)).float()
    assert ((ref.abs() < 2.0 ** -126) & (ref != 0)).sum() > 0.5 * ref.numel()
    assert torch.equal(out, ref)
