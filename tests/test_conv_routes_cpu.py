"""Which kernels the convolution plan chooses (no GPU needed: kernel counts and workspace sizes)."""
import ctypes as C

import pytest
import torch

from rocmlir_b200 import _lib as L
from rocmlir_b200.conv import ConvConfig

NHWC = dict(fil_layout="kyxc", in_layout="nhwc", out_layout="nhwk")
NCHW = dict(fil_layout="kcyx", in_layout="nchw", out_layout="nkhw")


def plan(dtype, direction=0, **kw):
    p = ConvConfig(**kw).to_c(dtype, direction)
    return int(L.lib().rbConvKernelCount(C.byref(p))), int(L.lib().rbConvWorkspaceSize(C.byref(p)))


@pytest.mark.parametrize("layout", [NHWC, NCHW], ids=["nhwc", "nchw"])
def test_few_channel_images_run_as_one_kernel_without_workspace(layout):
    stem = dict(n=64, c=3, k=64, h=224, w=224, y=7, x=7, stride_h=2, stride_w=2, pad_h=3, pad_w=3, **layout)
    assert plan(torch.float16, **stem) == (1, 0) and plan(torch.bfloat16, **stem) == (1, 0)
    # other types, directions and groups keep the matrix form
    assert plan(torch.float32, **stem)[1] > 0 and plan(torch.float16, 2, **stem)[1] > 0
    assert plan(torch.float16, **dict(stem, g=2))[1] > 0
    # a reduction whose filter does not fit beside the operand, even a quarter of the output channels at a time
    assert plan(torch.float16, **dict(stem, c=72, k=512))[1] > 0


# (layout, n, c, k, h = w, filter, stride): measured on a B200 in both forms, the patch kernel first
PAYS = [(NHWC, 32, 3, 64, 112, 7, 2), (NHWC, 32, 16, 32, 32, 3, 1), (NCHW, 32, 24, 64, 28, 3, 1), (NCHW, 16, 48, 96, 28, 3, 1), (NHWC, 8, 1, 32, 28, 5, 1)]
DOES_NOT = [(NCHW, 64, 512, 512, 7, 1, 1),    # 497 us against 32
            (NHWC, 16, 96, 192, 14, 3, 1),    # 64 / 16
            (NCHW, 32, 128, 128, 28, 3, 2),   # 299 / 75
            (NHWC, 125, 160, 48, 35, 3, 1),   # 1084 / 294
            (NHWC, 18, 32, 192, 224, 3, 2),   # 261 / 123
            (NCHW, 10, 160, 48, 7, 3, 1),     # 99 / 24
            (NHWC, 32, 32, 64, 28, 3, 2)]     # 13.9 / 10.7


@pytest.mark.parametrize("case", PAYS + DOES_NOT, ids=lambda c: "-".join(map(str, c[1:])))
def test_the_patch_kernel_is_taken_where_it_is_faster(case):
    layout, n, c, k, hw, f, s = case
    got = plan(torch.float16, n=n, c=c, k=k, h=hw, w=hw, y=f, x=f, stride_h=s, stride_w=s, pad_h=f // 2, pad_w=f // 2, **layout)
    assert (got == (1, 0)) == (case in PAYS)


def test_f32_convolutions_of_one_tap_stay_on_the_gemm_kernel():
    wide = dict(n=16, c=64, k=64, h=56, w=56, **NCHW)
    assert plan(torch.float32, y=3, x=3, pad_h=1, pad_w=1, **wide)[0] == 3      # image planes, filter planes, streamed filter
    assert plan(torch.float32, y=1, x=1, **wide)[0] == 1                        # one tap: no halo to share
