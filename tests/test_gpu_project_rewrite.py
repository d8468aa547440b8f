"""GPU checks of the feature gather where channel-first maps are rewritten
channels-last first: more images and channels than a grid dimension holds, and
no memory left for a copy.  Same bits as the gather through the strides."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _args(n, C, H, W, n_pts, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    maps = [torch.rand((n, c, H, W), generator=g, device="cuda") for c in (C, 1, 1, 3)]
    xy = torch.rand((n, n_pts, 1, 2), generator=g, device="cuda") * 2.2 - 1.1
    return maps + [xy, torch.rand((n, 1, n_pts), generator=g, device="cuda")]


def _direct(views, monkeypatch, args):
    with monkeypatch.context() as mp:
        mp.setattr(views, "CHANNELS_LAST_FROM", float("inf"))
        return views.forward_sample_feature(*args)


@pytest.mark.parametrize("n,C,H,W", [(70000, 32, 4, 4), (65535, 9, 3, 2), (1, 32 * 65535 + 40, 2, 2), (3, 33, 9, 8)])
def test_any_number_of_images_and_channels(n, C, H, W, monkeypatch):
    from sailor_gb300 import views
    args = _args(n, C, H, W, H * W, C)
    monkeypatch.setattr(views, "CHANNELS_LAST_FROM", 0.0)
    monkeypatch.setattr(views, "CHANNELS_LAST_WORK", 0)
    rows = views._channels_last(args[0])
    if C <= 32 * 65535:
        assert torch.equal(rows, args[0].permute(0, 2, 3, 1))
    else:
        assert rows is None  # gathered through its strides
    for a, b in zip(views.forward_sample_feature(*args), _direct(views, monkeypatch, args)):
        assert torch.equal(a, b)


def test_no_room_for_a_copy(monkeypatch):
    from sailor_gb300 import views
    n, C, H, W = 2, 64, 48, 40
    args = _args(n, C, H, W, H * W, 1)
    monkeypatch.setattr(views, "CHANNELS_LAST_FROM", 0.0)
    monkeypatch.setattr(views, "CHANNELS_LAST_WORK", 0)
    ref, real = views.forward_sample_feature(*args), torch.empty

    def full(shape, *a, **k):
        if shape == (n, H, W, C):
            raise torch.OutOfMemoryError("no room")
        return real(shape, *a, **k)
    with monkeypatch.context() as mp:
        mp.setattr(torch, "empty", full)
        assert views._channels_last(args[0]) is None
        got = views.forward_sample_feature(*args)
    for a, b in zip(got, ref):
        assert torch.equal(a, b)


def test_no_room_for_an_output_beside_the_copies(monkeypatch):
    """The third map's output has no room while the first map's copy is held."""
    from sailor_gb300 import views
    n, C, H, W = 2, 64, 48, 40
    args = _args(n, C, H, W, H * W, 1)
    monkeypatch.setattr(views, "CHANNELS_LAST_FROM", 0.0)
    monkeypatch.setattr(views, "CHANNELS_LAST_WORK", 0)
    ref, real, copies = views.forward_sample_feature(*args), torch.empty, []

    def full(shape, *a, **k):
        if shape == (n, H, W, C):
            copies.append(shape)
        if shape == (n, H * W, 3) and len(copies) == 1:
            copies.append("refused")
            raise torch.OutOfMemoryError("no room")
        return real(shape, *a, **k)
    with monkeypatch.context() as mp:
        mp.setattr(torch, "empty", full)
        got = views.forward_sample_feature(*args)
    assert copies == [(n, H, W, C), "refused"]  # and no copy the second time
    for a, b in zip(got, ref):
        assert torch.equal(a, b)
