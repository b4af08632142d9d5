"""The helix step on interleaved vectors (gx_helix_dostep_xyz, the form that
DoStepArr calls) against the one on planes: the same kernel, the same bits."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [0, 1, 255, 256, 257, 4099])
def test_interleaved_equals_planes(n):
    import torch
    import geantexascalepilot_b200 as g
    from geantexascalepilot_b200._lib import check, lib
    gen = torch.Generator(device="cuda").manual_seed(3)
    pos, d = (torch.randn((n, 3), generator=gen, device="cuda", dtype=torch.float64) for _ in range(2))
    d = d / d.norm(dim=1, keepdim=True)
    q = torch.where(torch.arange(n, device="cuda") % 2 == 0, 1.0, -1.0).double()
    p, s = (torch.rand(n, generator=gen, device="cuda", dtype=torch.float64) + 0.01 for _ in range(2))
    B = [0.3, -0.2, 40.0]
    newpos, newdir = g.ConstFieldHelixStepper(B).DoStepArr(pos, d, q, p, s)
    planes = [x[:, k].contiguous() for x in (pos, d) for k in range(3)]
    out = [torch.empty(n, dtype=torch.float64, device="cuda") for _ in range(6)]
    ptr = [C.c_void_p(x.data_ptr()) for x in planes + [q, p, s] + out]
    check(lib.gx_helix_dostep((C.c_double * 3)(*B), -0.299792458e-3, n, *ptr,
                              C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    assert newpos.shape == newdir.shape == (n, 3)
    assert torch.equal(newpos, torch.stack(out[:3], 1)) and torch.equal(newdir, torch.stack(out[3:], 1))
