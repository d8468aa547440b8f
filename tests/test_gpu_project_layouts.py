"""GPU checks of the feature gather's map layouts: every layout and channel
count gives the bits of the item-by-item gather of the NCHW map."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _layouts(m):
    """The same [n, C, H, W] values in other memory orders."""
    n, C, H, W = m.shape
    wide = torch.randn((n, H, W, C + 3), device="cuda")
    wide[..., 1:C + 1] = m.permute(0, 2, 3, 1)
    return dict(
        channels_last=m.contiguous(memory_format=torch.channels_last),
        sliced=wide[..., 1:C + 1].permute(0, 3, 1, 2),          # rows off 16 bytes, wider than C
        columns=m.permute(0, 3, 2, 1).contiguous().permute(0, 3, 2, 1),  # channels last, columns outer
        transposed=m.transpose(2, 3).contiguous().transpose(2, 3),       # NCWH
        nchw=m.contiguous())


@pytest.mark.parametrize("C", [1, 3, 4, 5, 6, 8, 12, 16, 30, 32, 36, 68])
@pytest.mark.parametrize("n_pts", [1, 31, 33, 700, 1500])
def test_layouts_give_the_same_bits(C, n_pts, monkeypatch):
    from sailor_gb300 import views
    g = torch.Generator(device="cuda").manual_seed(C * 7 + n_pts)
    n, H, W = 3, 65, 47
    geo = torch.randn((n, C, H, W), generator=g, device="cuda")
    rgbf = torch.randn((n, 9, 33, 70), generator=g, device="cuda")  # another size than the first map
    dep = torch.rand((n, 1, H, W), generator=g, device="cuda") * 2 + 1
    rgb = torch.rand((n, 3, H, W), generator=g, device="cuda")
    xy = torch.rand((n, n_pts, 1, 2), generator=g, device="cuda") * 2.4 - 1.2
    xy[:, :1] = -2.0
    if n_pts > 40:
        xy[:, 3] = float("nan")
        xy[:, 4] = 1.0
        xy[:, 5] = -1.0
        xy[:, 6] = 1e30
    z = torch.rand((n, 1, n_pts), generator=g, device="cuda") * 2 + 1
    with monkeypatch.context() as mp:
        mp.setattr(views, "CHANNELS_LAST_FROM", float("inf"))
        ref = views.forward_sample_feature(geo, dep, rgbf, rgb, xy, z)
    for name, m in _layouts(geo).items():
        for other in (rgbf, rgbf.contiguous(memory_format=torch.channels_last)):
            got = views.forward_sample_feature(m, dep, other, rgb, xy, z)
            for a, b in zip(got, ref):
                assert torch.equal(a, b), (name, a.shape)
    # a map shared by the images (stride 0)
    one = geo[:1].expand(n, -1, -1, -1)
    got = views.forward_sample_feature(one, dep, rgbf, rgb, xy, z)
    with monkeypatch.context() as mp:
        mp.setattr(views, "CHANNELS_LAST_FROM", float("inf"))
        ref = views.forward_sample_feature(one.contiguous(), dep, rgbf, rgb, xy, z)
    assert all(torch.equal(a, b) for a, b in zip(got, ref))


def test_infinite_texels_outside_the_footprint_stay_out():
    """Corners outside the image add nothing, whatever the nearest texel holds."""
    from sailor_gb300 import views
    m = torch.full((1, 8, 4, 4), float("inf"), device="cuda").contiguous(memory_format=torch.channels_last)
    rest = [torch.ones((1, c, 4, 4), device="cuda") for c in (1, 8, 3)]
    xy = torch.tensor([[[[-2.0, -2.0]], [[3.0, 0.0]]]], device="cuda")
    geo, _, _, _ = views.forward_sample_feature(m, *rest, xy, torch.ones((1, 1, 2), device="cuda"))
    assert torch.equal(geo, torch.zeros_like(geo))
