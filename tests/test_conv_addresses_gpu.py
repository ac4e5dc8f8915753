"""Buffers of convolutions that start off the boundaries the kernels load and store on: taken by a form that looks at the
address, or refused before anything is launched, as a wide access at such an address would fault."""
import numpy as np
import pytest

import oracle
from helpers import from_device, to_device
from test_conv_gpu import LAYOUTS, make_cfgs
from test_conv_patch_gpu import data

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", ["nhwc", "nchw"])
@pytest.mark.parametrize("y", [1, 3])
@pytest.mark.parametrize("offset", [4, 8])
def test_f32_planes_in_a_workspace_off_its_boundary(cuda_device, layout, y, offset):
    import ctypes as C
    import torch
    from rocmlir_b200 import _lib as L
    from rocmlir_b200 import conv as rc
    cfg, ocfg = make_cfgs(n=2, c=64, k=64, h=14, w=14, y=y, x=3, pad_h=y // 2, pad_w=1, **LAYOUTS[layout])
    p = cfg.to_c(torch.float32, rc.FWD)
    need = int(L.lib().rbConvWorkspaceSize(C.byref(p)))
    assert need > 0
    (_, fil), (_, inp), _ = data(ocfg, oracle.F32)
    fil, inp = to_device(fil, oracle.F32), to_device(inp, oracle.F32)
    out = torch.zeros(ocfg.numel("out"), device="cuda")
    space = torch.empty(need + 64, dtype=torch.uint8, device="cuda")
    launches = L.launch_count()
    with pytest.raises(L.RbError):
        rc.conv(cfg, rc.FWD, fil, inp, out, workspace=space[offset:])
    torch.cuda.synchronize()
    assert L.launch_count() == launches and not out.any()
    rc.conv(cfg, rc.FWD, fil, inp, out, workspace=space)
    torch.cuda.synchronize()
    assert L.launch_count() > launches and out.any() and L.kernel_status() == 0


@pytest.mark.parametrize("which", ["filter", "input", "output"])
def test_patch_kernel_tensors_off_their_elements(cuda_device, which):
    """An address between two elements: refused, as the general kernel refuses operands it cannot load."""
    import ctypes as C
    import torch
    from rocmlir_b200 import _lib as L
    cfg, ocfg = make_cfgs(n=1, c=3, k=32, h=12, w=12, y=3, x=3, pad_h=1, pad_w=1, **LAYOUTS["nhwc"])
    p = cfg.to_c(torch.float16, 0)
    assert int(L.lib().rbConvWorkspaceSize(C.byref(p))) == 0
    bufs = {n: torch.zeros(ocfg.numel(k) + 8, dtype=torch.float16, device="cuda") for n, k in (("filter", "fil"), ("input", "in"), ("output", "out"))}
    ptr = {n: t.data_ptr() + (1 if n == which else 0) for n, t in bufs.items()}
    launches = L.launch_count()
    st = L.lib().rbConv(C.byref(p), ptr["filter"], ptr["input"], ptr["output"], None, 0, torch.cuda.current_stream().cuda_stream)
    assert st == L.UNSUPPORTED and L.launch_count() == launches


# (direction, type, sizes): the halo kernel forward and backward, its streamed-filter forms, the weight-gradient kernel, and results
# that are not stored as they come out of the product
OFF = [("fwd", "f16", dict(c=64, k=64)), ("fwd", "f16", dict(c=256, k=64)), ("fwd", "f32", dict(c=64, k=64)),
       ("bwd_data", "f16", dict(c=64, k=64)), ("bwd_weight", "f16", dict(c=64, k=64)),
       ("bwd_data", "f16", dict(c=64, k=64, stride_h=2, stride_w=2))]


@pytest.mark.parametrize("layout", ["nhwc", "nchw"])
@pytest.mark.parametrize("direction,kind,sizes", OFF, ids=lambda v: str(v))
def test_results_off_their_boundary(cuda_device, direction, kind, sizes, layout):
    import torch
    from rocmlir_b200 import _lib as L
    from rocmlir_b200 import conv as rc
    code = oracle.F16 if kind == "f16" else oracle.F32
    cfg, ocfg = make_cfgs(n=2, h=14, w=14, y=3, x=3, pad_h=1, pad_w=1, **sizes, **LAYOUTS[layout])
    d = {"fwd": rc.FWD, "bwd_data": rc.BWD_DATA, "bwd_weight": rc.BWD_WEIGHT}[direction]
    which = {"fwd": 2, "bwd_data": 1, "bwd_weight": 0}[direction]
    raws = [raw for _, raw in data(ocfg, code)]
    results = []
    for skip in (0, 1):
        bufs = [to_device(raw, code).view(-1) for raw in raws]
        space = torch.zeros(bufs[which].numel() + 16, dtype=bufs[which].dtype, device="cuda")
        bufs[which] = space[skip:skip + bufs[which].numel()]
        try:
            rc.conv(cfg, d, *bufs)
        except L.RbError as e:
            assert e.status == L.UNSUPPORTED and skip
            return
        torch.cuda.synchronize()
        results.append(from_device(bufs[which], code))
        assert not space[:skip].any() and not space[skip + bufs[which].numel():].any() and L.kernel_status() == 0
    assert results[0].any()
    np.testing.assert_array_equal(results[0], results[1])
