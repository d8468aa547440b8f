"""GPU checks of the grid gather's adjoint with a ray's samples in parts (few
rays) and in one walk, at the parts' edges, against float64 sums."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _reference(o, d, z, g, D, lo, vs):
    """float64 gradient, the sum of |g| and the samples at each voxel and around it."""
    pt = o.double()[:, None] + d.double()[:, None] * z.double()[..., None]
    u = (pt - lo) / vs
    i0, C = torch.floor(u), g.shape[-1]
    f = u - i0
    grad = torch.zeros((D ** 3, C), dtype=torch.float64, device="cuda")
    mag, n = torch.zeros_like(grad), torch.zeros((D ** 3, 1), dtype=torch.float64, device="cuda")
    for k in range(8):
        b = torch.tensor([(k >> 2) & 1, (k >> 1) & 1, k & 1], device="cuda")
        i = i0.long() + b
        ok = ((i >= 0) & (i < D)).all(-1) & (z >= 0)
        w = torch.where(b.bool(), f, 1.0 - f).prod(-1)[ok][:, None]
        at = ((i[..., 0] * D + i[..., 1]) * D + i[..., 2])[ok]
        grad.index_add_(0, at, w * g[ok].double())
        mag.index_add_(0, at, g[ok].double().abs())
        n.index_add_(0, at, torch.ones_like(w))
    around = [torch.nn.functional.avg_pool3d(x.T.reshape(-1, 1, D, D, D), 3, 1, 1, divisor_override=1)[:, 0] for x in (mag, n)]
    return grad.reshape(D, D, D, C), around[0].permute(1, 2, 3, 0), around[1].permute(1, 2, 3, 0)


@pytest.mark.parametrize("C", [1, 3, 4, 8, 16])
@pytest.mark.parametrize("R,S", [(1, 1), (1, 9), (1, 640), (3, 7), (5, 8), (37, 17), (500, 64), (500, 100), (2000, 33),
                                 (19455, 16), (19456, 16), (30000, 9)])
def test_parts(C, R, S):
    from sailor_gb300 import fields
    D = 20
    g = torch.Generator(device="cuda").manual_seed(C * 1000 + R + S)
    o = torch.randn((R, 3), generator=g, device="cuda")
    o = o * (3.0 / o.norm(dim=-1, keepdim=True))
    d = (torch.rand((R, 3), generator=g, device="cuda") * 2.4 - 1.2) - o
    d = d / d.norm(dim=-1, keepdim=True)
    z = (torch.rand((R, S), generator=g, device="cuda") * 2.4 + 1.6).sort(-1).values
    z[torch.rand((R, S), generator=g, device="cuda") < 0.1] = -1.0
    go = torch.randn((R, S, C), generator=g, device="cuda")
    bbox = torch.tensor([[[-1.0, 1.0]] * 3], device="cuda")
    vs = torch.full((1, 1), 2.0 / (D - 1), device="cuda")
    grid = torch.zeros((1, D, D, D, C), device="cuda", requires_grad=True)
    out = fields.grid_gather(grid, o[None], d[None], z[None], bbox, vs)
    got, = torch.autograd.grad(out, grid, go[None])
    want, mag, n = _reference(o, d, z, go, D, -1.0, float(vs))
    # per term: the weight to 2^-20 (fractions to 2^-22 of a voxel: positions up to 4
    # of voxels of 0.1), and one rounding for each addition
    assert ((got[0].double() - want).abs() <= (2.0 ** -17 + n * 2.0 ** -24) * mag).all()
    assert want.abs().max().item() > 0
