"""GPU checks of a BatchPipeline with and without packed fields: few samples
are not packed, none where there is no room, and the outputs are the same."""
import pytest
import torch
from test_gpu_batch import _pipeline, work  # noqa: F401  (work: fixture)

pytestmark = pytest.mark.gpu


def _run(bp):
    out = [t.clone() for t in bp.forward()]
    bp.backward(torch.ones((bp.R, 3), device="cuda"))
    out.append(bp.grad_feat.clone())
    bp.train_step()
    torch.cuda.synchronize()
    assert int(bp.status[0]) == 0
    return out + [t.clone() for t in (bp.out_rgb, bp.out_depth, bp.out_ws, bp.out_alpha, bp.out_loss, bp.grad_feat)]


@pytest.mark.parametrize("C", [3, 16])
@pytest.mark.parametrize("uses", [(True, True, True), (False, False, False), (True, False, False), (False, True, True)])
def test_routes_agree(work, C, uses):  # noqa: F811
    ref = _pipeline(work, C=C)
    ref.packed = None
    want = _run(ref)
    bp = _pipeline(work, C=C)
    bp.packed = torch.full((bp.B, bp.D, bp.D, bp.D, 4), float("nan"), device="cuda")
    bp._packs = dict(zip(("forward", "backward", "train"), uses))
    got = _run(bp)
    for k, (a, b) in enumerate(zip(got, want)):
        if k == 4:  # adjoint's atomics: the order of additions alone
            assert (a - b).abs().max().item() <= 1e-5 * b.abs().max().item()
        else:
            assert torch.equal(a, b), k


def test_few_rays_and_no_room():
    from sailor_gb300.batch import BatchPipeline
    few = BatchPipeline([[(16, 16)]], [(0, 64, 32)], D=64, rate=8, C=16, W_hits=32)
    assert few.packed is None
    torch.cuda.empty_cache()
    real = torch.empty

    def full(shape, *a, **k):
        if shape == (1, 64, 64, 64, 4):
            raise torch.OutOfMemoryError("no room")
        return real(shape, *a, **k)
    torch.empty = full
    try:
        bp = BatchPipeline([[(16, 16)]], [(0, 16384, 96)], D=64, rate=8, C=16, W_hits=32)
    finally:
        torch.empty = real
    assert bp._packs["train"] and bp.packed is None
    assert BatchPipeline([[(16, 16)]], [(0, 16384, 96)], D=64, rate=8, C=16, W_hits=32).packed is not None
