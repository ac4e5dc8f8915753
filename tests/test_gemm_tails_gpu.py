"""The three instantiations of the GEMM kernel by what a launch does between accumulator and result: nothing, fused elementwise work, rows
that are copied out. Each launch takes the smallest one that has its work, and the code object handed to clients holds all three."""
import ctypes as C

import pytest

from test_cubin_gpu import driver_launch

pytestmark = pytest.mark.gpu

# (type, result, m, n, k, epilogue, instantiation): n off 16 bytes is copied out with and without a tail
CASES = [("float16", "float16", 256, 512, 128, None, 0), ("float16", "float16", 256, 512, 128, "bias_relu", 1), ("float16", "float16", 300, 515, 128, None, 2),
         ("float16", "float16", 300, 515, 128, "bias_relu", 2), ("int8", "int8", 256, 512, 128, "requant", 1), ("int8", "int8", 300, 515, 128, "requant", 2),
         ("int8", "int32", 300, 512, 128, None, 0), ("int8", "int32", 300, 514, 128, None, 2), ("float8_e4m3fn", "bfloat16", 130, 260, 96, "tanh", 2),
         ("float8_e4m3fn", "bfloat16", 130, 264, 96, "tanh", 1)]


@pytest.mark.parametrize("dt,out,m,n,k,tail,instantiation", CASES)
def test_instantiation_and_result(cuda_device, dt, out, m, n, k, tail, instantiation):
    import torch
    from rocmlir_b200 import _lib as L
    from rocmlir_b200.gemm import Epilogue, gemm, problem
    L.lib().rbSetGemmVariant(0x2001)   # tiles of 128 columns (of 64, an 8-bit row is half of a staged one, which is copied out)
    gen = torch.Generator(device="cuda").manual_seed(3)
    a, b = (torch.randint(-4, 5, s, device="cuda", generator=gen).to(getattr(torch, dt)) for s in ((m, k), (n, k)))
    vec = torch.rand(n, device="cuda", generator=gen)
    epilogue = {None: None, "bias_relu": Epilogue(bias=vec.half(), relu=True, mid_type=L.F16), "requant": Epilogue(col_scale=vec, requant_scale=3.0),
                "tanh": Epilogue(alpha=0.1, unary="tanh")}[tail]
    want = gemm(a, b, trans_b=True, out_dtype=getattr(torch, out), epilogue=epilogue)
    got = torch.zeros_like(want)
    p, launch = problem(a, b, False, True, False, got.dtype), L.RbKernelLaunch()
    e = C.byref(epilogue.to_c()) if epilogue is not None else None
    L.check(L.lib().rbGemmEncodeLaunch(C.byref(p), e, a.data_ptr(), b.data_ptr(), got.data_ptr(), C.byref(launch)))
    assert launch.symbol.decode().split("EEEvNS_")[0].endswith(f"Li{instantiation}")
    image, size = C.c_void_p(), C.c_size_t()
    L.check(L.lib().rbGetKernelBinary(C.byref(image), C.byref(size)))
    driver_launch(C.string_at(image.value, size.value), launch, torch.cuda.current_stream().cuda_stream)
    assert torch.equal(got, want) and want.any() and L.kernel_status() == 0
