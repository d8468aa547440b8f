"""GPU check of the traversal's rays that are walked again into rows which
other lanes of the warp have written just before: the same rows as rays that
were alone in their call, whatever their neighbours, run after run."""
import numpy as np
import pytest
import torch
from test_gpu_octree import _cuda, _scene, _trees

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rate,L,start", [(2, 4, 0), (4, 3, 0)])
def test_redone_rows_do_not_depend_on_neighbours(rate, L, start):
    scene = _scene(64, 96, 3, 48, 11, batch=1)
    o, _, _ = _trees(scene, rate, L)
    ori, dirs = _cuda(scene["ori"]), _cuda(scene["dirs"])
    idx = o.octree_traversal(ori, dirs, 192, 1024, start, -1, -1)[0]
    n = (idx[0] >= 0).sum(-1)
    at = torch.argsort(n, descending=True)[:256]
    ori, dirs = ori[:, at].contiguous(), dirs[:, at].contiguous()
    for W in (1, 2, max(int(n.max()) // 2, 3), int(n.max()) - 1):
        many = [x.clone() for x in o.octree_traversal(ori, dirs, 192, W, start, -1, -1)]
        for k in np.linspace(0, 255, 24).astype(int):
            one = o.octree_traversal(ori[:, k:k + 1].contiguous(), dirs[:, k:k + 1].contiguous(), 192, W, start, -1, -1)
            for a, b in zip(many, one):
                assert torch.equal(a[:, k:k + 1], b), (W, k)
        for _ in range(10):
            for a, b in zip(many, o.octree_traversal(ori, dirs, 192, W, start, -1, -1)):
                assert torch.equal(a, b), W
