"""Which form a few-channel convolution takes: the window kernel, the gathering one or an im2col matrix, by estimates of their times; and what
an image off 16 bytes, which the window kernel does not read, takes in its place."""
import ctypes as C

import numpy as np
import pytest

import oracle
from helpers import from_device, reference_random, to_device
from test_conv_gpu import LAYOUTS, make_cfgs
from test_dispatch_lines_gpu import IM2COL, PATCH, under

pytestmark = pytest.mark.gpu
GATHER = PATCH | 1 << 10

# (layout, n, c, k, h, w, filter, stride), each 1.6 to 4.2 times slower in the form that earlier estimates chose: results off 32 bytes, filters by
# channel planes, rows of single channels; and results off 16 bytes, which the product of a matrix copies out
CONVS = [("nchw", 2, 24, 100, 90, 32, 5, 1), ("nhwc", 2, 20, 96, 22, 256, 5, 1), ("nhwc", 6, 24, 200, 90, 90, 3, 1), ("nchw", 106, 12, 128, 42, 42, 5, 2),
         ("nhwc", 7, 8, 100, 196, 196, 3, 1), ("nhwc", 4, 1, 130, 136, 136, 3, 1), ("nhwc", 41, 24, 130, 31, 31, 7, 1), ("nhwc", 71, 3, 32, 141, 141, 3, 1)]


@pytest.mark.parametrize("layout,n,c,k,h,w,f,s", CONVS)
def test_the_faster_form(cuda_device, layout, n, c, k, h, w, f, s):
    import torch
    from rocmlir_b200 import conv as rc
    cfg, ocfg = make_cfgs(n=n, c=c, k=k, h=h, w=w, y=f, x=f, stride_h=s, stride_w=s, pad_h=f // 2, pad_w=f // 2, **LAYOUTS[layout])
    fil, inp, out = (torch.randn(ocfg.numel(t), device="cuda").half() for t in ("fil", "in", "out"))
    ws = torch.empty(1 << 30, dtype=torch.uint8, device="cuda")
    run = lambda: rc.conv(cfg, rc.FWD, fil, inp, out, workspace=ws)
    assert under(0, run) <= 1.35 * min(under(v, run) for v in (IM2COL, PATCH, GATHER))


# the window kernel pays, the gathering one does not
OFF16 = [dict(n=29, c=24, k=16, h=40, w=40, y=5, x=5, stride_h=2, stride_w=2, pad_h=2, pad_w=2),
         dict(n=43, c=24, k=64, h=55, w=55, y=3, x=3, stride_h=2, stride_w=2, pad_h=1, pad_w=1)]


@pytest.mark.parametrize("shape", OFF16, ids=lambda s: "x".join(str(v) for v in s.values()))
def test_images_off_16_bytes_take_the_matrix(cuda_device, shape):
    import torch
    from rocmlir_b200 import _lib as L
    from rocmlir_b200.conv import conv, workspace_size
    cfg, ocfg = make_cfgs(**shape, **LAYOUTS["nhwc"])
    (ff, fraw), (inf, iraw), (of, oraw) = reference_random([(ocfg.numel(w),) for w in ("fil", "in", "out")], oracle.F16, seed=1)
    ref = oracle.from_f32(oracle.conv_f32(ocfg, 0, ff, inf, of, threads=oracle.max_threads()), oracle.F16)
    lib, p = L.lib(), cfg.to_c(torch.float16, 0)
    size = workspace_size(cfg, torch.float16, 0)
    assert size > 0 and lib.rbConvKernelCount(C.byref(p)) == 1
    fil, ws = to_device(fraw, oracle.F16), torch.empty(size, dtype=torch.uint8, device="cuda")
    out = torch.empty(oraw.size, dtype=torch.float16, device="cuda")
    for off in (0, 1, 4):
        inp = torch.zeros(iraw.size + 8, dtype=torch.float16, device="cuda")[off:off + iraw.size]
        inp.copy_(to_device(iraw, oracle.F16).view(-1))
        for space in (ws, None, ws[:16]):   # (the package's call brings a workspace of its own where it is given none; the library's does not)
            out.zero_()
            before = L.launch_count()
            if space is ws:
                conv(cfg, 0, fil, inp, out, workspace=ws)
            else:
                address, length = (space.data_ptr(), space.nbytes) if space is not None else (None, 0)
                L.check(lib.rbConv(C.byref(p), fil.data_ptr(), inp.data_ptr(), out.data_ptr(), address, length, torch.cuda.current_stream().cuda_stream))
            launches = L.launch_count() - before
            np.testing.assert_array_equal(from_device(out, oracle.F16).ravel(), ref.ravel())
            assert (launches > 1) == (off != 0 and space is ws)
    assert L.kernel_status() == 0
