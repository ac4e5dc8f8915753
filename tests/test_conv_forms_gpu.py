"""Fused tails of the two kernels for few-channel images (csrc/conv_window_sm100.cu, csrc/conv_patch_sm100.cu), each by a variant word of its own and for
every way in which it reads the image: equal, bit for bit, to the GEMM epilogue of the im2col form on the same exact sums. The gathering
kernel against the oracle, which the window kernel's tests leave to it."""
import ctypes as C

import numpy as np
import pytest

import oracle
from helpers import to_device, torch_dtype
from test_conv_gpu import LAYOUTS, make_cfgs, run_conv
from test_conv_patch_gpu import IM2COL, MIXED, SHAPES as PATCH_SHAPES, data
from test_conv_window_gpu import GATHER, WINDOW

pytestmark = pytest.mark.gpu

# entries of the window / runs of the gather: shifted words / single elements and padded runs; words of two channels; of four; whole groups of
# eight straight from the image; channel planes; columns further apart than one
READS = [("nhwc", dict(c=3, h=30, w=17, y=7, x=7, stride_h=2, stride_w=2, pad_h=3, pad_w=3)),
         ("nhwc", dict(c=7, h=12, w=13, y=3, x=3, pad_h=1, pad_w=1)),
         ("nhwc", dict(c=2, h=20, w=17, y=5, x=5, pad_h=2, pad_w=2)),
         ("nhwc", dict(c=6, h=14, w=18, y=3, x=3, stride_h=2, stride_w=1, pad_h=1, pad_w=1)),
         ("nhwc", dict(c=4, h=19, w=18, y=3, x=3, pad_h=1, pad_w=1)),
         ("nhwc", dict(c=12, h=13, w=10, y=3, x=3, pad_h=1, pad_w=1)),
         ("nhwc", dict(c=8, h=15, w=18, y=5, x=5, stride_h=2, stride_w=2, pad_h=2, pad_w=2)),
         ("nhwc", dict(c=16, h=10, w=40, y=3, x=3, pad_h=1, pad_w=1)),
         ("nchw", dict(c=3, h=30, w=18, y=7, x=7, stride_h=2, stride_w=2, pad_h=3, pad_w=3)),
         ("nchw", dict(c=5, h=11, w=16, y=3, x=3, pad_h=1, pad_w=1)),
         ("nhwc", dict(c=3, h=15, w=16, y=3, x=3, dil_h=2, dil_w=2, pad_h=2, pad_w=2))]


def patch_kernel(cfg, code):
    from rocmlir_b200 import _lib as L
    return L.lib().rbConvPatchKernel(C.byref(cfg.to_c(torch_dtype(code), 0)))


@pytest.mark.parametrize("k,out_dtype", [(64, "same"), (40, "same"), (40, "float32"), (64, "int8")])
@pytest.mark.parametrize("code", [oracle.F16, oracle.BF16])
@pytest.mark.parametrize("layout,shape", READS, ids=lambda s: s if isinstance(s, str) else "x".join(str(v) for v in s.values()))
def test_fused_tails_equal_the_im2col_form(cuda_device, layout, shape, code, k, out_dtype):
    import torch
    from rocmlir_b200 import _lib as L
    from rocmlir_b200.conv import conv_fused
    from rocmlir_b200.gemm import Epilogue
    cfg, ocfg = make_cfgs(n=2, k=k, **shape, **LAYOUTS[layout])
    (_, fraw), (_, iraw), _ = data(ocfg, code)
    gen = torch.Generator(device="cuda").manual_seed(3)
    t = torch_dtype(code)
    bias = torch.randn(k, device="cuda", generator=gen).to(t)
    epi = Epilogue(bias=bias, relu=True, mid_type=L.F16 if code == oracle.F16 else L.BF16)
    if out_dtype == "int8":
        epi = Epilogue(col_scale=torch.rand(k, device="cuda", generator=gen), bias=bias, requant_scale=3.0)
    elif layout == "nhwc":
        epi.residual = torch.randn(ocfg.numel("out"), device="cuda", generator=gen).to(t)
    res = []
    for variant, kernel in ((WINDOW, 2), (GATHER, 1), (IM2COL, 0)):
        out = torch.zeros(ocfg.numel("out"), dtype=t if out_dtype == "same" else getattr(torch, out_dtype), device="cuda")
        L.lib().rbSetGemmVariant(variant)
        assert patch_kernel(cfg, code) == kernel
        conv_fused(cfg, to_device(fraw, code), to_device(iraw, code), out, epi)
        res.append(out)
    torch.cuda.synchronize()
    assert L.kernel_status() == 0 and res[2].any()
    assert torch.equal(res[0], res[2]) and torch.equal(res[1], res[2])


@pytest.mark.parametrize("layout", ["nhwc", "nchw", "mixed"])
@pytest.mark.parametrize("code", [oracle.F16, oracle.BF16])
@pytest.mark.parametrize("shape", PATCH_SHAPES[:-1], ids=lambda s: "x".join(str(v) for v in s.values()))
def test_gathering_kernel_exact(cuda_device, shape, code, layout):
    from rocmlir_b200 import _lib as L
    cfg, ocfg = make_cfgs(**shape, **(MIXED if layout == "mixed" else LAYOUTS[layout]))
    (ff, fraw), (inf, iraw), (of, oraw) = data(ocfg, code)
    ref = oracle.from_f32(oracle.conv_f32(ocfg, 0, ff, inf, of, threads=oracle.max_threads()), code)
    L.lib().rbSetGemmVariant(GATHER)
    assert patch_kernel(cfg, code) == 1
    got = run_conv(cfg, 0, code, {"fil": fraw, "in": iraw, "out": oraw})
    np.testing.assert_array_equal(got.ravel(), ref.ravel())
    assert L.kernel_status() == 0
