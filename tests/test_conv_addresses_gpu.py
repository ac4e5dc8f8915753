"""Buffers of convolutions that start off the boundaries the kernels load and store on: refused before anything is launched, as
a wide access at such an address would fault."""
import pytest

import oracle
from helpers import to_device
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
