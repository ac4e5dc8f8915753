"""Calls on both sides of the lines between two kernels that compute the same: the library's own choice is not slower than the form
an explicit variant word selects. Device times of graph replays, the lowest of several; 1.5 leaves room for clocks and for what
the lines leave on the table (at most 13 % where they were fitted); most choices that this guards against were 1.7 to 16
times slower."""
import pytest

from test_conv_gpu import LAYOUTS, make_cfgs

pytestmark = pytest.mark.gpu

GENERAL = 1 << 27        # any explicit variant word: the general GEMM kernel with its own choice of tiles
IM2COL, PATCH = 1 << 26, 1 << 30
SLACK = 1.5


def device_us(run):
    import torch
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        run()
        s.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            for _ in range(10):
                run()
        times = []
        for _ in range(7):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(s)
            g.replay()
            b.record(s)
            b.synchronize()
            times.append(a.elapsed_time(b) * 100)
    return min(times[1:])


def under(variant, run):
    from rocmlir_b200 import _lib as L
    L.lib().rbSetGemmVariant(variant)
    try:
        return device_us(run)
    finally:
        L.lib().rbSetGemmVariant(0)


# (type, g, m, n, k), weights stored N x K: many groups with short K; rows that one part of K carries alone; few tiles and a long K;
# clusters that do not pack; and products that belong to the kernel for few rows
FEW_ROWS = [("float16", 512, 64, 2048, 128), ("float16", 64, 33, 4096, 128), ("float16", 2048, 64, 128, 64), ("float16", 1, 64, 4096, 128),
            ("bfloat16", 1, 64, 1024, 256), ("float16", 1, 16, 128, 32768), ("float16", 3, 64, 4096, 4096), ("int8", 512, 64, 2048, 128),
            ("float16", 1, 8, 4096, 4096), ("float16", 1, 64, 4096, 4096), ("float16", 1, 16, 11008, 4096), ("int8", 1, 16, 4096, 4096),
            ("float16", 1, 40, 16711, 80)]


@pytest.mark.parametrize("dtype,g,m,n,k", FEW_ROWS)
def test_few_rows(cuda_device, dtype, g, m, n, k):
    import torch
    from rocmlir_b200.gemm import gemm, problem, workspace_size
    dt = getattr(torch, dtype)
    out = torch.int32 if dt == torch.int8 else dt
    make = (lambda s: torch.randint(-9, 10, s, device="cuda").to(dt))
    a, b, c = make((g, m, k)), make((g, n, k)), torch.empty((g, m, n), dtype=out, device="cuda")
    ws = torch.empty(max(16, workspace_size(problem(a, b, False, True, False, out))), dtype=torch.uint8, device="cuda")
    run = lambda: gemm(a, b, trans_b=True, out_dtype=out, out=c, workspace=ws)
    assert under(0, run) <= SLACK * under(GENERAL, run)


# (layout, n, c, k, h = w, filter, stride): many channels, planes of many channels, several passes over the output channels, channel
# counts whose pixels fall into the same banks; and the few-channel layers that the patch kernel is for
CONVS = [("nchw", 64, 512, 512, 7, 1, 1), ("nhwc", 16, 96, 192, 14, 3, 1), ("nchw", 32, 128, 128, 28, 3, 2), ("nhwc", 18, 32, 192, 224, 3, 2),
         ("nhwc", 125, 160, 48, 35, 3, 1), ("nchw", 42, 64, 512, 7, 3, 1), ("nhwc", 64, 3, 64, 112, 7, 2), ("nchw", 64, 3, 64, 56, 3, 1),
         ("nhwc", 64, 16, 32, 56, 3, 1), ("nchw", 16, 48, 96, 28, 3, 1), ("nhwc", 32, 24, 33, 56, 3, 1)]


@pytest.mark.parametrize("layout,n,c,k,hw,f,s", CONVS)
def test_few_channels(cuda_device, layout, n, c, k, hw, f, s):
    import torch
    from rocmlir_b200 import conv as rc
    cfg, ocfg = make_cfgs(n=n, c=c, k=k, h=hw, w=hw, y=f, x=f, stride_h=s, stride_w=s, pad_h=f // 2, pad_w=f // 2, **LAYOUTS[layout])
    fil, inp, out = (torch.randn(ocfg.numel(w), device="cuda").half() for w in ("fil", "in", "out"))
    ws = torch.empty(1 << 30, dtype=torch.uint8, device="cuda")
    run = lambda: rc.conv(cfg, rc.FWD, fil, inp, out, workspace=ws)
    assert under(0, run) <= SLACK * min(under(IM2COL, run), under(PATCH, run))
