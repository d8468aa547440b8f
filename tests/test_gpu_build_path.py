"""GPU checks of the drop-in build path: packed colours against the
expression, level totals, and the multi-level tables of a two-level tree."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,shift", [((1, 3, 1, 1), 0), ((2, 3, 5, 7), 0), ((3, 4, 8, 8), 0), ((2, 3, 64, 64), 0),
                                         ((2, 3, 64, 64), 1), ((1, 3, 333, 31), 2)])
def test_pack_colors(shape, shift):
    from sailor_gb300 import voxel_encoding as VE
    n = 1
    for d in shape:
        n *= d
    buf = torch.rand(n + 4, device="cuda") * 255.0
    buf[::7] = torch.floor(buf[::7])
    buf[::101] = float("nan")
    buf[::103] = float("inf")
    c = buf[shift:shift + n].view(shape)
    ref = torch.floor(c[:, 2] * 256.0 * 256.0 + c[:, 1] * 256.0 + c[:, 0])
    for x in (c, c.transpose(2, 3).contiguous().transpose(2, 3)):  # as given, and by the expression
        with torch.no_grad():
            assert torch.equal(VE.pack_colors(x).nan_to_num(-1.0, -2.0, -3.0), ref.nan_to_num(-1.0, -2.0, -3.0))
    leaf = c.clone().requires_grad_()
    assert VE.pack_colors(leaf).requires_grad
    with torch.no_grad():
        many = torch.vmap(VE.pack_colors)(torch.stack([c, c]))
    assert torch.equal(many[1].nan_to_num(-1.0, -2.0, -3.0), ref.nan_to_num(-1.0, -2.0, -3.0))
    assert torch.equal(VE.pack_colors(c.double()).float().nan_to_num(), torch.floor(
        c.double()[:, 2] * 256.0 * 256.0 + c.double()[:, 1] * 256.0 + c.double()[:, 0]).float().nan_to_num())


def test_level_totals():
    from sailor_gb300.voxel_encoding_helper import _totals
    a = torch.tensor([[3], [4]], dtype=torch.int32, device="cuda")
    b = torch.tensor([5], dtype=torch.int32, device="cuda")
    assert _totals([a, b]) == [7, 5] and _totals([]) == [] and _totals([a, b.cpu()]) == [7, 5]
    assert _totals([a.float(), b.long()]) == [7, 5] and _totals([a[:0], b]) == [0, 5]
    big = torch.full((3,), 2 ** 31 - 1, dtype=torch.int32, device="cuda")
    assert _totals([big]) == [3 * (2 ** 31 - 1)]
