"""GPU checks of the deterministic gradient reduction where its records and
stretches change shape: few cells with long runs, targets whose rays all miss
(first, between and last), single rays, 3 and 16 channels, with the TSDF's
records and without.  Every term of the feature gradient is made non-negative
(colours >= 0 against targets of 0, a head >= 0), so that each sum's own value
bounds its rounding."""
import numpy as np
import pytest
import torch
from test_gpu_batch import _t

from sailor_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


def _steps(D, C, sizes, train_tsdf):
    from sailor_gb300.batch import BatchPipeline
    w = syn.make_batch_workload(seed=5, n_frames=2, views=(2, 3), view_res=(64, 96), n_prims=8, D=D, trunc=0.06,
                                n_targets=len(sizes), target_res=(40, 41), target_S=(32, 64, 128))
    rng = np.random.default_rng(D + C)
    rays, targets = [], []
    for t, n in zip(w["targets"], sizes):
        o, d = t["ori"], t["dir"]
        if n < 0:  # all rays away from the volume
            o, d = o[:-n], -d[:-n]
        else:
            at = np.sort(rng.permutation(len(o))[:n])
            o, d = o[at], d[at]
        rays.append((o, d))
        targets.append((t["frame"], len(o), t["S"]))
    feat = _t(rng.random((2, D, D, D, C)))
    head = _t(rng.random((3, C))) if C != 3 else None
    out = []
    for deterministic in (False, True):
        bp = BatchPipeline([[d.shape for d in fr["depth"]] for fr in w["frames"]], targets, D=D, rate=4, C=C, W_hits=96,
                           deterministic=deterministic)
        bp.load_views(w["frames"], w["vol_bbox"], w["voxel_size"], w["trunc_weight"])
        bp.load_rays(rays)
        bp.set_fields(feat=feat, head=head, target_rgb=torch.zeros((bp.R, 3), device="cuda"))
        bp.render_args(float(w["voxel_size"][0]) * w["trunc_weight"], sdf_s=0.02, t_thres=1e-4)
        bp.train_tsdf = train_tsdf
        bp.train_step()
        torch.cuda.synchronize()
        out.append(bp)
    return out


@pytest.mark.parametrize("train_tsdf", [False, True])
@pytest.mark.parametrize("C", [3, 16])
@pytest.mark.parametrize("D,sizes", [(32, (1500, 1500)), (64, (-40, 700, -1, 1, -33, 300, -64)), (32, (1,)),
                                     (64, (33, -5, 1600))])
def test_runs_against_atomics(D, C, sizes, train_tsdf):
    ref, det = _steps(D, C, sizes, train_tsdf)
    assert int(det.status[0]) == 0
    z = det.reduction_sizes()
    for a, b in zip((det.out_rgb, det.out_depth, det.out_ws, det.out_alpha, det.out_loss),
                    (ref.out_rgb, ref.out_depth, ref.out_ws, ref.out_alpha, ref.out_loss)):
        assert torch.equal(a, b)
    g, h = det.grad_feat.double(), ref.grad_feat.double()
    assert (h >= 0).all() and (g >= 0).all()
    # both sides: at most one rounding per sample and per level of the sums
    n = z["slots"] + 64
    assert ((g - h).abs() <= 2 * n * 2.0 ** -24 * h).all()
    if z["records"]:
        assert h.max() > 0 and 0 < z["cells"] <= z["records"] <= z["slots"]
    if train_tsdf:
        m = ref.grad_tsdf.abs().max().item()
        assert (det.grad_tsdf - ref.grad_tsdf).abs().max().item() <= 1e-5 * m
    again = det.grad_feat.clone()
    det.zero_grads()
    det.train_step()
    torch.cuda.synchronize()
    assert torch.equal(again, det.grad_feat)
