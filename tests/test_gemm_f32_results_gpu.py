"""f32 results of 16- and 8-bit operands whose K is cut so that no accumulator sums too many elements, although one range would be faster: with the
workspace that the library asks for, without it, without any, and as the one kernel that a client launches itself."""
import ctypes as C

import pytest

from test_cubin_gpu import driver_launch

pytestmark = pytest.mark.gpu

# the last one's planes do not fit the built-in scratch
SHAPES = [("float16", 1024, 1024, 1024), ("bfloat16", 384, 4288, 1472), ("float8_e4m3fn", 1984, 256, 4160), ("float16", 2304, 1024, 1024)]


def setup(dt, m, n, k, real):
    import torch
    from rocmlir_b200.gemm import problem, workspace_size
    gen = torch.Generator(device="cuda").manual_seed(2)
    t = getattr(torch, dt)
    a, b = (torch.randn(s, device="cuda", generator=gen).to(t) if real else torch.randint(-3, 4, s, device="cuda", generator=gen).to(t) for s in ((m, k), (n, k)))
    p = problem(a, b, False, True, False, torch.float32)
    return a, b, p, workspace_size(p), a.double() @ b.double().T


@pytest.mark.parametrize("dt,m,n,k", SHAPES)
def test_every_way_of_launching(cuda_device, dt, m, n, k):
    """Operands of small whole numbers: every sum is exact."""
    import torch
    from rocmlir_b200 import _lib as L
    lib = L.lib()
    a, b, p, need, ref = setup(dt, m, n, k, False)
    assert need >= 2 * m * n * 4
    ws, out, stream = torch.empty(need, dtype=torch.uint8, device="cuda"), torch.empty((m, n), device="cuda"), torch.cuda.current_stream().cuda_stream
    operands = (a.data_ptr(), b.data_ptr(), out.data_ptr())
    launch = L.RbKernelLaunch()
    image, size = C.c_void_p(), C.c_size_t()
    L.check(lib.rbGetKernelBinary(C.byref(image), C.byref(size)))

    def client():
        L.check(lib.rbGemmEncodeLaunch(C.byref(p), None, *operands, C.byref(launch)))
        driver_launch(C.string_at(image.value, size.value), launch, stream)

    for run in (lambda: L.check(lib.rbGemm(C.byref(p), None, *operands, ws.data_ptr(), need, stream)),
                lambda: L.check(lib.rbGemm(C.byref(p), None, *operands, ws.data_ptr(), need - 1, stream)),
                lambda: L.check(lib.rbGemm(C.byref(p), None, *operands, None, 0, stream)),
                lambda: L.check(lib.rbGemmNoAlloc(C.byref(p), None, *operands, stream)), client):
        out.fill_(float("nan"))
        run()
        torch.cuda.synchronize()
        assert torch.equal(out.double(), ref)
    assert L.kernel_status() == 0


@pytest.mark.parametrize("dt,m,n,k", SHAPES)
def test_shorter_sums_are_nearer(cuda_device, dt, m, n, k):
    """The tensor core truncates what it adds: the error against 64 bits grows with the elements that one accumulator sums."""
    from rocmlir_b200.gemm import gemm
    import torch
    from rocmlir_b200 import _lib as L
    a, b, p, need, ref = setup(dt, m, n, k, True)
    got = gemm(a, b, trans_b=True, out_dtype=torch.float32)
    whole = torch.empty_like(got)
    L.check(L.lib().rbGemm(C.byref(p), None, a.data_ptr(), b.data_ptr(), whole.data_ptr(), None, 0, torch.cuda.current_stream().cuda_stream))
    errors = [float((x.double() - ref).norm() / ref.norm()) for x in (got, whole)]
    assert errors[0] < 0.75 * errors[1]
