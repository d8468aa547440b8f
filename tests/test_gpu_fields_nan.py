"""GPU check of the grid gather at samples without a corner inside the grid:
0, also where the sample's position is no number on one axis."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C", [1, 3, 4, 8, 16])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_nothing_inside(C, axis):
    from sailor_gb300 import fields
    D = 16
    grid = torch.ones((1, D, D, D, C), device="cuda")
    ori = torch.full((1, 40, 3), 50.0, device="cuda")  # far outside on every axis
    dirs = torch.ones((1, 40, 3), device="cuda")
    dirs[:, ::3, axis] = float("nan")
    dirs[:, 1::3, axis] = float("inf")
    z = torch.full((1, 40, 5), 1.0, device="cuda")
    bbox = torch.tensor([[[-1.0, 1.0]] * 3], device="cuda")
    vs = torch.full((1, 1), 2.0 / (D - 1), device="cuda")
    out = fields.grid_gather(grid, ori, dirs, z, bbox, vs)
    assert torch.equal(out, torch.zeros_like(out))
