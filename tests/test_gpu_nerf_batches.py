"""GPU checks of the occupancy network's sigma batches: the densities of a
large call, whose sigma tiles gather several feature tiles, against calls so
small that every feature tile is a batch of its own, bit for bit (a row of a
tile does not depend on the others)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V,N", [(1, 200001), (2, 70003), (3, 42 * 1600 + 1), (3, 42 * 2281), (5, 40007), (7, 30011),
                                 (40, 5003), (64, 3001), (100, 1777), (128, 1777)])
@pytest.mark.parametrize("B", [1, 2])
def test_batched_sigma_tiles_match_single_tiles(V, N, B):
    from sailor_gb300.nerf import infer_density
    g = torch.Generator(device="cuda").manual_seed(V + N)
    params = (torch.randn(22521, generator=g, device="cuda") * 0.2).half()
    z = torch.rand((B, V, N, 1), generator=g, device="cuda") * 2.5 + 0.5
    t = torch.rand((B, V, N, 1), generator=g, device="cuda") * 2.0 - 1.0
    f = torch.randn((B, V, N, 16), generator=g, device="cuda") * 0.5
    d = infer_density(z, t, f, params, B, N, V, 0)
    d2, geo = infer_density(z, t, f, params, B, N, V, 0, return_geo=True)
    assert torch.equal(d, d2)
    step = max(1, 128 // V) * 100  # at most 100 tiles: fewer than there are warpgroups
    for a in [0, step, (N // step) * step - step // 2, max(N - step, 0)]:
        a = max(0, min(a, N - 1))
        e = min(N, a + step)
        part, pg = infer_density(z[:1, :, a:e].contiguous(), t[:1, :, a:e].contiguous(), f[:1, :, a:e].contiguous(),
                                 params, 1, e - a, V, 0, return_geo=True)
        assert torch.equal(part[0, 0], d[0, 0, a:e])
        assert torch.equal(pg[0], geo[0, :, a:e])


def test_unaligned_parameters_and_extreme_inputs():
    """Parameters 2 bytes off a 16-byte boundary, and inputs that overflow
    float16 (infinities and NaN inside the layers: ReLU takes NaN to 0)."""
    from sailor_gb300.nerf import infer_density
    g = torch.Generator(device="cuda").manual_seed(1)
    V, N = 3, 500
    buf = (torch.randn(22522, generator=g, device="cuda") * 0.2).half()
    z = torch.rand((1, V, N, 1), generator=g, device="cuda")
    t = torch.rand((1, V, N, 1), generator=g, device="cuda")
    f = torch.randn((1, V, N, 16), generator=g, device="cuda")
    a = infer_density(z, t, f, buf[1:], 1, N, V, 0)
    b = infer_density(z, t, f, buf[1:].clone(), 1, N, V, 0)
    assert torch.equal(a, b)
    f[:, :, :7] = 1e30
    f[:, :, 7:9, ::2] = -1e30
    f[:, 0, 20] = float("nan")
    c = infer_density(z, t, f, buf[1:], 1, N, V, 0)
    keep = torch.ones(N, dtype=torch.bool, device="cuda")
    keep[:9] = False
    keep[20] = False
    assert torch.equal(c[0, 0, keep], b[0, 0, keep])
    assert not torch.isnan(c).any()
