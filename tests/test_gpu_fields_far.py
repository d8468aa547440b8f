"""GPU check of the grid gather and its adjoint at 2^31 samples and more, where
samples no longer divide by 32-bit multiplication: the last rays against a call
of their own, bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_more_than_2_31_samples():
    from sailor_gb300 import _native as N
    if torch.cuda.mem_get_info()[0] < 40 << 30:
        pytest.skip("not enough free memory")
    D, S, B = 16, 65, 3
    n = (2 ** 31 // S) // B + 1000  # rays a frame
    R = B * n
    assert R * S > 2 ** 31
    g = torch.Generator(device="cuda").manual_seed(1)
    ori = torch.rand((R, 3), generator=g, device="cuda") * 0.2 - 1.2
    dirs = torch.rand((R, 3), generator=g, device="cuda") + 0.2
    z = torch.rand((R, S), generator=g, device="cuda") * 2
    grid = torch.randn((B, D, D, D, 1), generator=g, device="cuda")
    bbox = torch.tensor([[[-1.0, 1.0]] * 3] * B, device="cuda")
    vs = torch.full((B,), 2.0 / (D - 1), device="cuda")
    out = torch.empty((R, S), device="cuda")
    N.check(N.lib.sg_grid_gather(N.ptr(ori), N.ptr(dirs), N.ptr(z), B, n, S, N.ptr(grid), D, 1, N.ptr(bbox), N.ptr(vs), 0,
                                 1.0, 1.0, N.ptr(out), N.stream()), "gather")
    for a in (0, n - 500, 2 * n - 500, R - 500):
        b, e = a // n, min(a + 500, R)
        part = torch.empty((e - a, S), device="cuda")
        e = min(e, (b + 1) * n)
        part = part[:e - a].contiguous()
        N.check(N.lib.sg_grid_gather(N.ptr(ori[a:e]), N.ptr(dirs[a:e]), N.ptr(z[a:e]), 1, e - a, S, N.ptr(grid[b]), D, 1,
                                     N.ptr(bbox[b]), N.ptr(vs[b:]), 0, 1.0, 1.0, N.ptr(part), N.stream()), "part")
        assert torch.equal(out[a:e], part) and part.abs().max().item() > 0
