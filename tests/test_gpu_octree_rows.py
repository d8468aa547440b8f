"""GPU checks of the multi-level traversal's two ways of descending a ray: the
coarse nodes of a ray over the lanes, and the ray walked again into its row
where a row or an entry list is too short.  Both give the same entries, bit
for bit, over depths, rates, ray counts off the warp, and two frames."""
import numpy as np
import pytest
import torch
from test_gpu_octree import _cuda, _scene, _trees

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[1, 2])
def scene(request):
    return _scene(64, 96, 3, 48, 11, batch=request.param)


@pytest.mark.parametrize("rate,L,start", [(2, 3, 0), (2, 4, 1), (2, 4, 0), (2, 6, 0), (4, 3, 0), (8, 2, 0)])
@pytest.mark.parametrize("n", [1, 5, 127, 2000])
def test_short_rows_hold_the_same_entries(scene, rate, L, start, n):
    o, _, _ = _trees(scene, rate, L)
    rng = np.random.default_rng(n + L)
    at = np.sort(rng.permutation(scene["ori"].shape[1])[:n])
    ori, dirs = _cuda(scene["ori"][:, at]), _cuda(scene["dirs"][:, at])

    def rows(Wc, Wf, th=-1, opt=-1):
        out = o.octree_traversal(ori, dirs, Wc, Wf, start, th, opt)
        return [x.clone() for x in out], o._ostatus.cpu().numpy().copy()

    full, st = rows(192, 1024)
    assert st[0] == 0
    idx, t0, t1, vl, ic, c0, c1 = full
    cc, fc = (ic >= 0).sum(-1), (idx >= 0).sum(-1)
    assert st[1] == cc.max().item() and st[2] == fc.max().item()
    # coarse rows too short: fine rows unchanged (the ray is walked again)
    half = max(int(cc.max().item()) // 2, 1)
    short, st = rows(half, 1024)
    assert bool(st[0]) == bool(cc.max().item() > half) and st[1] == cc.max().item()
    for a, b in zip(full[:4], short[:4]):
        assert torch.equal(a, b)
    for a, b in zip(full[4:], short[4:]):
        assert torch.equal(a[..., :half], b)
    # fine rows too short: the leading entries, the coarse rows unchanged
    W = max(int(fc.max().item()) // 2, 1)
    short, st = rows(192, W)
    assert bool(st[0]) == bool(fc.max().item() > W) and st[2] >= fc.max().item()
    fits = fc <= W
    for a, b in zip(full[:3], short[:3]):
        assert torch.equal(a[..., :W][fits], b[fits])
    assert torch.equal(vl[fits], short[3][fits])
    # an entry past the row's end can still take the place of one in it by a finer node: depths stay
    assert torch.equal(t0[..., :W], short[1]) and torch.equal(t1[..., :W], short[2])
    for a, b in zip(full[4:], short[4:]):
        assert torch.equal(a, b)
