"""GPU check of the clearing near nodes with few and many bricks (a CTA per
brick, and per sixteen), odd brick counts, against the neighbourhoods."""
import ctypes as Ct

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,Dt,rate", [(1, 1, 4), (2, 3, 8), (1, 8, 8), (3, 7, 6), (1, 13, 4), (1, 14, 4), (5, 11, 2), (2, 17, 3)])
@pytest.mark.parametrize("C,shift", [(16, 0), (3, 0), (3, 1), (1, 1)])
def test_cleared_bricks(B, Dt, rate, C, shift):
    from sailor_gb300 import _native as N
    g = torch.Generator(device="cuda").manual_seed(Dt * 10 + rate)
    node = torch.where(torch.rand((B, Dt, Dt, Dt), generator=g, device="cuda") < 0.03, 5, -1).to(torch.int32)
    D = Dt * rate
    n = B * D ** 3 * C
    buf = torch.ones(n + 4, device="cuda")
    grid = buf[shift:shift + n]
    vb, vs = torch.zeros((B, 3, 2), device="cuda"), torch.zeros(B, device="cuda")
    t = N.SgTree(B, Dt, D, rate, 0, 0, 1, 1, N.ptr(node), None, None, None, None, None, None, N.ptr(vs), N.ptr(vb))
    N.check(N.lib.sg_zero_near_nodes(Ct.byref(t), N.ptr(grid), C, N.stream()), "zero_near_nodes")
    near = torch.nn.functional.max_pool3d((node >= 0).float()[:, None], 3, 1, 1)[:, 0] > 0
    fine = near.repeat_interleave(rate, 1).repeat_interleave(rate, 2).repeat_interleave(rate, 3)
    want = torch.where(fine, 0.0, 1.0)[..., None].expand(-1, -1, -1, -1, C).reshape(-1)
    assert torch.equal(grid, want)
    assert (buf[:shift] == 1).all() and (buf[shift + n:] == 1).all()
