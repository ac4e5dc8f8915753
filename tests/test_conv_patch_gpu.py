"""GPU parity of the patch kernel (csrc/conv_patch_sm100.cu): 16-bit forward convolutions of one group whose channels are
not whole 128-byte runs. Integer-valued data, so every partial sum is exact in f32 and the result must equal the oracle's
bit for bit, and the result of the im2col form of the same library (variant bit 26). Variant bit 30 takes the kernel wherever
it fits, also where the library itself would choose the im2col form as the faster one."""
import numpy as np
import pytest

import oracle
from helpers import from_device, reference_random, to_device
from test_conv_gpu import LAYOUTS, make_cfgs, run_conv

pytestmark = pytest.mark.gpu

IM2COL, PATCH = 1 << 26, 1 << 30
MIXED = dict(fil_layout="gyxck", in_layout="hngwc", out_layout="ngkwh")
# runs of 1 / 2 / 4 / 8 channels; image rows that start on 16-, 8-, 4- and 2-byte boundaries; output rows wider than a tile,
# several rows per tile with a ragged last one; k extents of one MMA step, of exactly one 64-element block, of more blocks than the operand area
# holds; one and several passes over the output channels; strides beyond the filter, dilation, asymmetric padding
SHAPES = [
    dict(n=2, c=3, k=64, h=32, w=32, y=7, x=7, stride_h=2, stride_w=2, pad_h=3, pad_w=3),
    dict(n=1, c=3, k=33, h=9, w=301, y=3, x=3, pad_h=1, pad_w=1),
    dict(n=3, c=1, k=8, h=5, w=4, y=2, x=2),
    dict(n=2, c=4, k=160, h=13, w=11, y=4, x=4, pad_h=1, pad_w=2),
    dict(n=2, c=2, k=32, h=20, w=21, y=3, x=5, stride_h=3, stride_w=2, pad_h=2, pad_w=0),
    dict(n=1, c=16, k=128, h=18, w=18, y=7, x=7, pad_h=3, pad_w=3),
    dict(n=2, c=24, k=300, h=10, w=7, y=3, x=3, dil_h=2, dil_w=2, pad_h=2, pad_w=2),
    dict(n=1, c=7, k=40, h=130, w=6, y=5, x=1, stride_h=4, stride_w=4, pad_h=0, pad_w=1, pad_h_r=3, pad_w_r=0),
    dict(n=1, c=96, k=64, h=6, w=6, y=3, x=3, pad_h=1, pad_w=1),
    dict(n=2, c=5, k=16, h=1, w=1, y=1, x=1),
]


@pytest.fixture(autouse=True)
def _patch_kernel(_default_gemm_variant):
    from rocmlir_b200 import _lib as L
    L.lib().rbSetGemmVariant(PATCH)


def data(ocfg, code):
    return reference_random([(ocfg.numel("fil"),), (ocfg.numel("in"),), (ocfg.numel("out"),)], code, seed=1)


def patch_route(cfg, code):
    import ctypes as C
    from helpers import torch_dtype
    from rocmlir_b200 import _lib as L
    p = cfg.to_c(torch_dtype(code), 0)
    return int(L.lib().rbConvWorkspaceSize(C.byref(p))) == 0 and int(L.lib().rbConvKernelCount(C.byref(p))) == 1


@pytest.mark.parametrize("layout", ["nhwc", "nchw", "mixed"])
@pytest.mark.parametrize("code", [oracle.F16, oracle.BF16])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(str(v) for v in s.values()))
def test_patch_kernel_exact(cuda_device, shape, code, layout):
    from rocmlir_b200 import _lib as L
    cfg, ocfg = make_cfgs(**shape, **(MIXED if layout == "mixed" else LAYOUTS[layout]))
    # (a pointwise convolution of a single pixel is a plain matrix product in every layout)
    pointwise = shape["y"] * shape["x"] * shape["h"] * shape["w"] == 1
    assert patch_route(cfg, code) or pointwise
    (ff, fraw), (inf, iraw), (of, oraw) = data(ocfg, code)
    ref_raw = oracle.from_f32(oracle.conv_f32(ocfg, 0, ff, inf, of, threads=oracle.max_threads()), code)
    raws = {"fil": fraw, "in": iraw, "out": oraw}
    got = run_conv(cfg, 0, code, raws)
    np.testing.assert_array_equal(got.ravel(), ref_raw.ravel())
    L.lib().rbSetGemmVariant(IM2COL)
    try:
        assert not patch_route(cfg, code) or pointwise
        form = run_conv(cfg, 0, code, raws)
    finally:
        L.lib().rbSetGemmVariant(0)
    np.testing.assert_array_equal(form.ravel(), got.ravel())


@pytest.mark.parametrize("offset", [0, 1, 2, 4])
def test_patch_kernel_image_and_result_addresses(cuda_device, offset):
    """Buffers that start 0, 2, 4 and 8 bytes past a 16-byte boundary: narrower window copies and result stores."""
    import torch
    from rocmlir_b200.conv import conv
    cfg, ocfg = make_cfgs(n=2, c=4, k=32, h=12, w=16, y=3, x=3, pad_h=1, pad_w=1, **LAYOUTS["nhwc"])
    (ff, fraw), (inf, iraw), (of, oraw) = data(ocfg, oracle.F16)
    ref = oracle.from_f32(oracle.conv_f32(ocfg, 0, ff, inf, of, threads=oracle.max_threads()), oracle.F16)
    inp = torch.zeros(iraw.size + 8, dtype=torch.float16, device="cuda")[offset:offset + iraw.size]
    out = torch.zeros(oraw.size + 8, dtype=torch.float16, device="cuda")
    inp.copy_(to_device(iraw, oracle.F16).view(-1))
    conv(cfg, 0, to_device(fraw, oracle.F16), inp, out[offset:offset + oraw.size])
    np.testing.assert_array_equal(from_device(out[offset:offset + oraw.size], oracle.F16).ravel(), ref.ravel())
    assert not out[:offset].any() and not out[offset + oraw.size:].any()


@pytest.mark.parametrize("layout", ["nhwc", "nchw"])
@pytest.mark.parametrize("k,out_dtype", [(64, "float16"), (40, "float32"), (64, "float32"), (64, "int8")])
def test_patch_kernel_epilogue_equals_im2col_form(cuda_device, k, out_dtype, layout):
    """Fused tails: the same steps on the same exact sums as the im2col form's GEMM epilogue, bit for bit."""
    import torch
    from rocmlir_b200 import _lib as L
    from rocmlir_b200.conv import conv_fused
    from rocmlir_b200.gemm import Epilogue
    cfg, ocfg = make_cfgs(n=2, c=3, k=k, h=30, w=18, y=7, x=7, stride_h=2, stride_w=2, pad_h=3, pad_w=3, **LAYOUTS[layout])
    (_, fraw), (_, iraw), _ = data(ocfg, oracle.F16)
    gen = torch.Generator(device="cuda").manual_seed(3)
    bias = torch.randn(k, device="cuda", generator=gen).half()
    dt = getattr(torch, out_dtype)
    epi = Epilogue(bias=bias, relu=True, mid_type=L.F16)
    if out_dtype == "int8":
        epi = Epilogue(col_scale=torch.rand(k, device="cuda", generator=gen), bias=bias, requant_scale=3.0)
    elif out_dtype == "float16" and layout == "nhwc":
        epi.residual = torch.randn(ocfg.numel("out"), device="cuda", generator=gen).half()
    res = []
    for variant in (PATCH, IM2COL):
        out = torch.zeros(ocfg.numel("out"), dtype=dt, device="cuda")
        L.lib().rbSetGemmVariant(variant)
        try:
            conv_fused(cfg, to_device(fraw, oracle.F16), to_device(iraw, oracle.F16), out, epi)
        finally:
            L.lib().rbSetGemmVariant(0)
        torch.cuda.synchronize()
        res.append(out)
    assert L.kernel_status() == 0
    assert res[0].any() and torch.equal(res[0], res[1])
