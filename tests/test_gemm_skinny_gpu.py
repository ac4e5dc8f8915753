"""GPU parity of the kernel for at most 64 rows against weights stored N x K (csrc/gemm_skinny_sm100.cu): integer-valued data,
so the result must equal the oracle's, and the general kernel's (an explicit variant), bit for bit."""
import numpy as np
import pytest

import oracle
from helpers import reference_random, uniform_int8
from test_gemm_gpu import run_gemm

pytestmark = pytest.mark.gpu

# (g, m, n, k): token counts around the padded sizes 16 / 32 / 64; one column, ragged and whole tiles of 128 columns; one K
# block, a ragged last one, parts of uneven length; one to eight parts of K
SHAPES = [(1, 1, 1, 64), (1, 8, 4096, 4096), (2, 7, 130, 520), (1, 16, 100, 2048), (1, 17, 1000, 1096), (3, 32, 257, 384),
          (1, 33, 640, 4160), (1, 64, 11008, 320), (1, 64, 576, 8192), (40, 5, 512, 640)]


@pytest.mark.parametrize("code", [oracle.F16, oracle.BF16, oracle.F8E4M3, oracle.F8E5M2])
@pytest.mark.parametrize("g,m,n,k", SHAPES)
def test_few_rows_float_exact(cuda_device, g, m, n, k, code):
    k = k // 16 * 16 if code in (oracle.F8E4M3, oracle.F8E5M2) else k
    (af, araw), (bf, braw) = reference_random([(g, m, k), (g, n, k)], code, seed=1)
    out_code = oracle.F32 if code in (oracle.F8E4M3, oracle.F8E5M2) else code
    ref = oracle.from_f32(oracle.gemm_f32(af, bf, g, m, n, k, tb=True, threads=oracle.max_threads()), out_code)
    got = run_gemm(araw, braw, code, out_code, tb=True)
    np.testing.assert_array_equal(got.reshape(ref.shape), ref)


@pytest.mark.parametrize("g,m,n,k", [(g, m, n, max(16, k // 16 * 16)) for g, m, n, k in SHAPES])
def test_few_rows_int8_exact(cuda_device, g, m, n, k):
    a, b = uniform_int8((g, m, k), seed=3), uniform_int8((g, n, k), seed=4)
    ref = oracle.gemm_i8(a, b, g, m, n, k, tb=True, threads=oracle.max_threads())
    got = run_gemm(a, b, oracle.I8, oracle.I32, tb=True)
    assert oracle.verify_int(got, ref)[0] == [1, 1, 1]


@pytest.mark.parametrize("m,n,k", [(1, 300, 4096), (20, 1001, 512), (64, 128, 192)])
def test_few_rows_epilogues_equal_the_general_kernel(cuda_device, m, n, k):
    import torch
    from rocmlir_b200 import _lib as L
    from rocmlir_b200.gemm import Epilogue, gemm
    gen = torch.Generator(device="cuda").manual_seed(5)
    ints = lambda shape, dt: torch.randint(-4, 5, shape, device="cuda", generator=gen).to(dt)
    bias = torch.randn(n, device="cuda", generator=gen)
    scale = torch.rand(n, device="cuda", generator=gen)
    rows = torch.randn(m, device="cuda", generator=gen).half()
    res = torch.randn((m, n), device="cuda", generator=gen).half()
    cases = [(torch.float16, torch.float16, dict(bias=bias.half(), relu=True, mid_type=L.F16)),
             (torch.float16, torch.float32, dict(alpha=0.3, bias=rows, bias_mode="row", residual=res, unary="tanh")),
             (torch.bfloat16, torch.bfloat16, dict(bias=bias[:1].contiguous(), bias_mode="scalar", clip=(-1.0, 2.0))),
             (torch.int8, torch.int8, dict(col_scale=scale, requant_scale=3.0, out_zero=2))]
    for dt, out, kw in cases:
        a, b = ints((m, k), dt), ints((n, k), dt)
        got = [gemm(a, b, trans_b=True, out_dtype=out, epilogue=Epilogue(**kw), variant=v) for v in (None, 1)]
        torch.cuda.synchronize()
        assert torch.equal(got[0], got[1]), (dt, out, kw.keys())
    a, b = ints((m, k), torch.float16), ints((n, k), torch.float16)
    c = [res.clone() for _ in range(2)]
    for v, t in zip((None, 1), c):
        gemm(a, b, trans_b=True, out=t, accumulate=True, variant=v)
    assert torch.equal(c[0], c[1]) and L.kernel_status() == 0
