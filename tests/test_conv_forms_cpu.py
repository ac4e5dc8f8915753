"""The few-channel test shapes reach the kernel that their tests are about (no GPU needed: rbConvPatchKernel)."""
import ctypes as C

import pytest
import torch

from rocmlir_b200 import _lib as L
from test_conv_gpu import LAYOUTS, make_cfgs
from test_conv_forms_gpu import READS
from test_conv_window_gpu import GATHER, SHAPES, WINDOW


def kernel(variant, layout, **shape):
    cfg, _ = make_cfgs(**shape, **LAYOUTS[layout])
    L.lib().rbSetGemmVariant(variant)
    return L.lib().rbConvPatchKernel(C.byref(cfg.to_c(torch.float16, 0)))


@pytest.mark.parametrize("layout", ["nhwc", "nchw"])
def test_window_shapes(layout):
    address = [dict(n=2, c=c, k=32, h=12, w=16, y=3, x=3, pad_h=1, pad_w=1) for c in (3, 4, 6, 8, 16)]
    for shape in SHAPES + address:
        assert kernel(WINDOW, layout, **shape) == 2 and kernel(GATHER, layout, **shape) == 1 and kernel(1 << 26, layout, **shape) == 0, shape


def test_shapes_of_the_fused_tails():
    for layout, shape in READS:
        assert kernel(WINDOW, layout, n=2, k=64, **shape) == 2 and kernel(GATHER, layout, n=2, k=64, **shape) == 1, shape


def test_other_problems():
    stem = dict(n=64, c=3, k=64, h=224, w=224, y=7, x=7, stride_h=2, stride_w=2, pad_h=3, pad_w=3)
    assert kernel(0, "nhwc", **stem) == 2
    assert kernel(0, "nhwc", **dict(stem, c=64)) == 0
    cfg, _ = make_cfgs(**stem, **LAYOUTS["nhwc"])
    assert L.lib().rbConvPatchKernel(C.byref(cfg.to_c(torch.float16, 2))) == 0 and L.lib().rbConvPatchKernel(C.byref(cfg.to_c(torch.float32, 0))) == 0
    assert L.lib().rbConvPatchKernel(None) == -1
