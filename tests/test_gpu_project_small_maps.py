"""GPU checks of the feature gather on maps of a few pixels, read in lane
groups, with item counts that leave a warp's last lanes without an item."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,W", [(1, 1), (1, 3), (2, 2), (2, 3), (3, 2), (3, 3), (4, 4)])
@pytest.mark.parametrize("C", [5, 8, 32])
@pytest.mark.parametrize("n,n_pts", [(1, 1), (1, 17), (2, 33), (3, 21), (1, 32)])
def test_small_maps(H, W, C, n, n_pts):
    from sailor_gb300 import views
    g = torch.Generator(device="cuda").manual_seed(C + H * 8 + W + n_pts)
    geo = torch.randn((n, C, H, W), generator=g, device="cuda")
    rest = [torch.rand((n, c, H, W), generator=g, device="cuda") for c in (1, 6, 3)]
    xy = torch.rand((n, n_pts, 1, 2), generator=g, device="cuda") * 2 - 1  # every footprint inside the image
    z = torch.rand((n, 1, n_pts), generator=g, device="cuda") * 2 + 1
    got = views.forward_sample_feature(geo.contiguous(memory_format=torch.channels_last), *rest, xy, z)
    # the whole items' bits: a map of its own, in front of which lies what must not be read
    buf = torch.full((n * H * W * C + 64 * C,), float("nan"), device="cuda")
    at = buf[64 * C:].view(n, H, W, C).permute(0, 3, 1, 2)
    at.copy_(geo)
    again = views.forward_sample_feature(at, *rest, xy, z)
    for a, b in zip(got, again):
        assert torch.equal(a, b)
    want = torch.nn.functional.grid_sample(geo.double(), xy.double(), align_corners=True)[..., 0].transpose(1, 2)
    # five roundings of the pixel coordinate (edge at most 4), four of a weight, four of the sum
    assert (got[0].double() - want).abs().max().item() <= 64 * 2.0 ** -24 * geo.abs().max().item()
