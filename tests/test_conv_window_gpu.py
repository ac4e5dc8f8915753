"""GPU parity of the window kernel (csrc/conv_window_sm100.cu) with the gathering form of the same convolution (variant bit 10) and the
oracle: integer-valued data, so every partial sum is exact and all results must be equal bit for bit."""
import numpy as np
import pytest

import oracle
from helpers import from_device, reference_random, to_device
from test_conv_gpu import LAYOUTS, make_cfgs, run_conv

pytestmark = pytest.mark.gpu
WINDOW, GATHER = 1 << 30, 1 << 30 | 1 << 10

# entries of runs (up to four channels) and of pixels; whole, half-empty and odd numbers of k columns; one raster tile to all of
# them; columns cut into several items; strides with used and unused phases; dilation; image rows that start on any even byte;
# one to three passes over the output channels; more items than SMs
SHAPES = [
    dict(n=2, c=3, k=64, h=61, w=63, y=7, x=7, stride_h=2, stride_w=2, pad_h=3, pad_w=3),
    dict(n=1, c=1, k=32, h=20, w=700, y=1, x=3, pad_w=1),
    dict(n=5, c=4, k=128, h=40, w=40, y=5, x=5, stride_h=1, stride_w=2, pad_h=2, pad_w=2),
    dict(n=3, c=2, k=40, h=17, w=23, y=3, x=4, stride_h=3, stride_w=4, pad_h=2, pad_w=1),
    dict(n=2, c=3, k=270, h=15, w=16, y=3, x=3, dil_h=2, dil_w=3, pad_h=2, pad_w=3),
    dict(n=2, c=5, k=64, h=33, w=30, y=3, x=3, stride_h=2, stride_w=2, pad_h=1, pad_w=1),
    dict(n=1, c=7, k=96, h=14, w=14, y=5, x=5, pad_h=2, pad_w=2),
    dict(n=2, c=8, k=64, h=28, w=29, y=7, x=7, stride_h=2, stride_w=2, pad_h=3, pad_w=3),
    dict(n=3, c=16, k=128, h=30, w=30, y=3, x=3, pad_h=1, pad_w=1),
    dict(n=1, c=16, k=32, h=19, w=65, y=3, x=5, stride_w=2, dil_h=2, dil_w=2, pad_h=0, pad_w=4),
    dict(n=1, c=24, k=64, h=12, w=12, y=3, x=3, stride_h=5, stride_w=5, pad_h=1, pad_w=1),
    dict(n=170, c=3, k=32, h=9, w=9, y=3, x=3, pad_h=1, pad_w=1),
    dict(n=1, c=8, k=16, h=1, w=1, y=3, x=3, pad_h=1, pad_w=1),
]


def data(ocfg, code):
    return reference_random([(ocfg.numel("fil"),), (ocfg.numel("in"),), (ocfg.numel("out"),)], code, seed=1)


@pytest.mark.parametrize("layout", ["nhwc", "nchw"])
@pytest.mark.parametrize("code", [oracle.F16, oracle.BF16])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(str(v) for v in s.values()))
def test_window_kernel_exact(cuda_device, shape, code, layout):
    from rocmlir_b200 import _lib as L
    cfg, ocfg = make_cfgs(**shape, **LAYOUTS[layout])
    (ff, fraw), (inf, iraw), (of, oraw) = data(ocfg, code)
    ref = oracle.from_f32(oracle.conv_f32(ocfg, 0, ff, inf, of, threads=oracle.max_threads()), code)
    for variant in (WINDOW, GATHER):
        L.lib().rbSetGemmVariant(variant)
        got = run_conv(cfg, 0, code, {"fil": fraw, "in": iraw, "out": oraw})
        np.testing.assert_array_equal(got.ravel(), ref.ravel())
    assert L.kernel_status() == 0


@pytest.mark.parametrize("layout", ["nhwc", "nchw"])
@pytest.mark.parametrize("c,offset", [(3, 1), (4, 1), (4, 2), (8, 0), (8, 1), (8, 4), (6, 2), (16, 2)])
def test_window_kernel_addresses(cuda_device, c, offset, layout):
    """Images and results that start 0, 2, 4 and 8 bytes past a 16-byte boundary; what lies around the result stays as it was."""
    import torch
    from rocmlir_b200 import _lib as L
    from rocmlir_b200.conv import conv
    cfg, ocfg = make_cfgs(n=2, c=c, k=32, h=12, w=16, y=3, x=3, pad_h=1, pad_w=1, **LAYOUTS[layout])
    (ff, fraw), (inf, iraw), (of, oraw) = data(ocfg, oracle.F16)
    ref = oracle.from_f32(oracle.conv_f32(ocfg, 0, ff, inf, of, threads=oracle.max_threads()), oracle.F16)
    for at in (0, offset):   # of the image: only the first takes the window kernel
        inp = torch.zeros(iraw.size + 8, dtype=torch.float16, device="cuda")[at:at + iraw.size]
        out = torch.zeros(oraw.size + 8, dtype=torch.float16, device="cuda")
        inp.copy_(to_device(iraw, oracle.F16).view(-1))
        L.lib().rbSetGemmVariant(WINDOW)
        conv(cfg, 0, to_device(fraw, oracle.F16), inp, out[offset:offset + oraw.size])
        np.testing.assert_array_equal(from_device(out[offset:offset + oraw.size], oracle.F16).ravel(), ref.ravel())
        assert not out[:offset].any() and not out[offset + oraw.size:].any()


@pytest.mark.parametrize("shape", SHAPES[:1] + SHAPES[4:8], ids=lambda s: "x".join(str(v) for v in s.values()))
def test_infinities_stay_where_the_filter_reaches(cuda_device, shape):
    """Padding of runs, pixels and odd k steps is zero whatever lies there: an infinity in the image reaches the outputs whose
    windows hold it and no others."""
    import torch
    from rocmlir_b200 import _lib as L
    from rocmlir_b200.conv import conv
    cfg, ocfg = make_cfgs(**shape, **LAYOUTS["nchw"])
    (_, fraw), (_, iraw), (_, oraw) = data(ocfg, oracle.F16)
    fil, inp = to_device(np.abs(fraw.view(np.float16)).view(np.uint16), oracle.F16).view(-1) + 1, to_device(iraw, oracle.F16).view(-1)
    inp[inp.numel() // 2] = float("inf")
    out = torch.empty(oraw.size, dtype=torch.float16, device="cuda")
    L.lib().rbSetGemmVariant(WINDOW)
    conv(cfg, 0, fil, inp, out)
    s = dict(dict(stride_h=1, stride_w=1, pad_h=0, pad_w=0, dil_h=1, dil_w=1), **shape)
    ref = torch.nn.functional.conv2d(inp.view(s["n"], s["c"], s["h"], s["w"]).double().isinf().double(),
                                     torch.ones((1, s["c"], s["y"], s["x"]), dtype=torch.float64, device="cuda"),
                                     stride=(s["stride_h"], s["stride_w"]), padding=(s["pad_h"], s["pad_w"]), dilation=(s["dil_h"], s["dil_w"]))
    got = out.view(s["n"], s["k"], ref.shape[2], ref.shape[3])
    assert torch.equal(got.isinf(), (ref > 0).expand_as(got)) and not got.isnan().any()
