"""GPU check of NaN gradients: the atomic scatter and the deterministic
reduction mark the same grid values."""
import pytest
import torch
from test_gpu_reduce_order import _pipeline

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C", [3, 16])
def test_nan_gradients_reach_every_touched_cell(C):
    """A target of NaN makes its ray's colour gradient NaN, and 0 x NaN is NaN:
    samples of weight 0 carry it as well, whichever way gradients are summed."""
    def target(bp):
        t = torch.full((bp.R, 3), 0.25, device="cuda")
        t[::97] = float("nan")
        return t
    d, a = (_pipeline((0, 1, 2), C, deterministic=q, sdf_s=0.0002, target=target) for q in (True, False))
    nd, na = torch.isnan(d.grad_feat), torch.isnan(a.grad_feat)
    assert nd.any() and torch.equal(nd, na), (nd.sum().item(), na.sum().item())
