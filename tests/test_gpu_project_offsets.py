"""GPU checks of the feature gather on maps whose elements lie 2^31 and more
apart (channels or images outermost in a larger buffer): the bits of a
contiguous copy.  Buffers are allocated, not filled: only the map's own
elements are written and read."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _strided(m, stride):
    """The values of m [n, C, H, W] in a buffer of their own, at these strides."""
    span = 1 + sum((s - 1) * t for s, t in zip(m.shape, stride))
    if torch.cuda.mem_get_info()[0] < 4 * span + (8 << 30):
        pytest.skip("not enough free memory")
    out = torch.empty(span, device="cuda").as_strided(m.shape, stride)
    return out.copy_(m)


@pytest.mark.parametrize("C", [2, 5, 32])
@pytest.mark.parametrize("layout", ["channels", "images", "columns"])
@pytest.mark.parametrize("n_pts", [1, 33, 500])
def test_far_apart(C, layout, n_pts):
    from sailor_gb300 import views
    n, H, W = 3, 65, 47
    g = torch.Generator(device="cuda").manual_seed(C + n_pts)
    geo = torch.randn((n, C, H, W), generator=g, device="cuda")
    dep = torch.rand((n, 1, H, W), generator=g, device="cuda") * 2 + 1
    rgbf = torch.randn((n, 8, H, W), generator=g, device="cuda")
    rgb = torch.rand((n, 3, H, W), generator=g, device="cuda")
    xy = torch.rand((n, n_pts, 1, 2), generator=g, device="cuda") * 2.2 - 1.1
    z = torch.rand((n, 1, n_pts), generator=g, device="cuda") * 2 + 1
    far = 2 ** 31 // max(C - 1, 1) + 4  # the last channel begins behind 2^31 elements
    stride = dict(channels=(H * W, far, W, 1),                 # [C, n, H, W] transposed
                  images=(2 ** 30 + 4, 1, W * C, C),           # channels-last images in slots of 4 GB
                  columns=(H * C, 1, C, 2 ** 31 // (W - 1) + 4))[layout]  # channels contiguous, columns outermost
    ref = views.forward_sample_feature(geo, dep, rgbf, rgb, xy, z)
    got = views.forward_sample_feature(_strided(geo, stride), dep, rgbf, rgb, xy, z)
    for a, b in zip(got, ref):
        assert torch.equal(a, b)
