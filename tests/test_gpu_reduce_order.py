"""GPU checks of the deterministic reduction's sums: a frame's gradient does
not depend on the other frames of its batch, and gradients below the normal
range of float32 are kept."""
import numpy as np
import pytest
import torch
from test_gpu_batch import _t

from sailor_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu

D = 64


def _pipeline(frames, C, train_tsdf=False, deterministic=True, sdf_s=0.02, S=(32, 64, 128), feat=None, head=None, target=None):
    from sailor_gb300.batch import BatchPipeline
    w = syn.make_batch_workload(seed=5, n_frames=3, views=(2, 3), view_res=(64, 96), n_prims=8, D=D, trunc=0.06,
                                n_targets=3, target_res=(40, 41), target_S=S)
    assert sorted(t["frame"] for t in w["targets"]) == [0, 1, 2]
    fr = [w["frames"][f] for f in frames]
    tg = [(i, t) for i, f in enumerate(frames) for t in w["targets"] if t["frame"] == f]
    bp = BatchPipeline([[d.shape for d in x["depth"]] for x in fr], [(i, t["ori"].shape[0], t["S"]) for i, t in tg], D=D,
                       rate=4, C=C, W_hits=96, deterministic=deterministic)
    bp.load_views(fr, np.asarray(w["vol_bbox"])[:len(fr)], np.asarray(w["voxel_size"])[:len(fr)], w["trunc_weight"])
    bp.load_rays([(t["ori"], t["dir"]) for _, t in tg])
    rng = np.random.default_rng(3)
    full = _t(rng.normal(0, 0.5, (3, D, D, D, C))) if feat is None else feat
    bp.set_fields(feat=full[list(frames)], head=(_t(rng.normal(0, 0.5, (3, C))) if head is None else head) if C != 3 else None,
                  target_rgb=torch.full((bp.R, 3), 0.25, device="cuda") if target is None else target(bp))
    bp.render_args(float(w["voxel_size"][0]) * w["trunc_weight"], sdf_s=sdf_s, t_thres=1e-4)
    bp.train_tsdf = train_tsdf
    bp.train_step()
    torch.cuda.synchronize()
    assert int(bp.status[0]) == 0
    return bp


@pytest.mark.parametrize("train_tsdf", [False, True])
@pytest.mark.parametrize("C", [3, 16])
def test_other_frames_do_not_change_a_frame(C, train_tsdf):
    """The same three frames in another order: the loss and each frame's rays
    are the same, every frame's records lie elsewhere in the sorted list."""
    a, b = _pipeline((0, 1, 2), C, train_tsdf), _pipeline((1, 2, 0), C, train_tsdf)
    for x, y in ((0, 2), (1, 0), (2, 1)):
        assert torch.equal(a.grad_feat[x], b.grad_feat[y])
        if train_tsdf:
            assert torch.equal(a.grad_tsdf[x], b.grad_tsdf[y])
    assert a.grad_feat.abs().max().item() > 0


@pytest.mark.parametrize("C", [3, 16])
def test_subnormal_gradients_are_kept(C):
    """Features of zero and a gradient that scales with the head (C = 16) or the
    loss: 2^-110 of a normal step's, so that sums lie on both sides of 2^-126.
    Each record's product and each addition rounds once to 2^-149 at most."""
    k = 2.0 ** -110
    feat = torch.zeros((3, D, D, D, C), device="cuda")
    if C == 16:
        h = _t(np.random.default_rng(1).normal(0, 0.5, (3, C)))
        ref, got = (_pipeline((0, 1, 2), C, feat=feat, head=q) for q in (h, h * k))
    else:
        full = lambda v: (lambda bp: torch.full((bp.R, 3), v, device="cuda"))  # noqa: E731
        ref, got = (_pipeline((0, 1, 2), C, feat=feat, target=full(q)) for q in (0.25, 0.25 * k))
    want, have = ref.grad_feat.double() * k, got.grad_feat.double()
    small = (want.abs() < 2.0 ** -126) & (want != 0)
    assert small.sum().item() > 1000
    # a cell's runs, its partial sums and classes: at most 4096 roundings to 2^-149
    assert ((have - want).abs() <= 2.0 ** -149 * 4096 + want.abs() * 2.0 ** -20).all()
    assert (have[small] != 0).float().mean().item() > 0.9
