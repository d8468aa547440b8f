"""GPU check of the coarse occupancy over row lengths and brick edges: short
rows shared by groups of threads (few and many CTAs), long rows, rows longer
than a CTA's threads, edges that are no power of two."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,D,rate", [(1, 4, 2), (2, 4, 4), (1, 8, 1), (3, 12, 3), (1, 32, 4), (2, 36, 6), (5, 64, 2),
                                      (1, 128, 8), (8, 128, 4), (2, 200, 5), (1, 252, 7), (1, 252, 14), (1, 256, 2),
                                      (2, 256, 8), (1, 260, 10), (1, 520, 4), (1, 1028, 4)])
@pytest.mark.parametrize("density", [0.0, 0.002, 0.5, 1.0])
def test_occupancy(B, D, rate, density):
    from sailor_gb300 import voxel_encoding as VE
    if D > 1000 and density not in (0.002,):
        pytest.skip("one density at this size")
    g = torch.Generator(device="cuda").manual_seed(D + rate)
    fine = torch.where(torch.rand((B, D, D, D), generator=g, device="cuda") < density, 0, -1).to(torch.int32)
    n = D // rate
    coarse = torch.full((B, n, n, n), 7, dtype=torch.int32, device="cuda")
    cnt = [torch.zeros((B, 1), dtype=torch.int32, device="cuda") for _ in range(2)]
    VE.build_multi_res_volumes([fine, coarse], cnt, 2, rate, 0)
    any_ = (fine > -1).view(B, n, rate, n, rate, n, rate).amax((2, 4, 6))
    ids = torch.arange(n ** 3, dtype=torch.int32, device="cuda").view(1, n, n, n)
    assert torch.equal(coarse, torch.where(any_, ids, -1))
    assert torch.equal(cnt[1].view(-1), any_.view(B, -1).sum(1).to(torch.int32))
