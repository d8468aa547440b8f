"""GPU checks of the padded intersection where the padding changes kernels: ray
counts about the line, against the warp variant and against compact rows."""
import numpy as np
import pytest
import torch
from test_gpu_intersect_rows import _rays
from test_gpu_parity import _t, case  # noqa: F401  (case: fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 63, 127, 128, 129, 255, 256, 257])
@pytest.mark.parametrize("W", [1, 5, 64, 130, 1024])
def test_rows_about_the_line(case, n, W):  # noqa: F811
    from sailor_gb300 import autotune
    octree = case["g"]["octree"]
    o, d = _rays("random", case["ref"]["vol_bbox"].shape[0], n, case["ref"]["vol_bbox"], np.random.default_rng(n))
    saved, outs = autotune.current(), []
    try:
        for wv in (0, 1):
            autotune.set_knob("isect_warp", wv)
            rows = octree.voxel_traversal(_t(o), _t(d), W, 0, -1, False, -1)
            torch.cuda.synchronize()
            outs.append([x.clone() for x in rows] + [octree._status.clone()])
    finally:
        for k, v in saved.items():
            autotune.set_knob(k, v)
    for a, b in zip(*outs):
        assert torch.equal(a, b)
