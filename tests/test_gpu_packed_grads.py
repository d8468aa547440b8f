"""GPU checks of the packed renders' gradients against the unpacked ones': the
per-sample density gradients bit for bit, the TSDF grid's, and the training
entry points' (deterministic: bit for bit)."""
import ctypes as Ct

import pytest
import torch
from test_gpu_batch import D, _pipeline, work  # noqa: F401  (work: fixture)

pytestmark = pytest.mark.gpu


def _packed(bp):
    from sailor_gb300 import _native as N
    p = torch.full((bp.B, D, D, D, 4), float("nan"), device="cuda")
    N.check(N.lib.sg_pack_fields(Ct.byref(bp.tree), Ct.byref(bp.seg), Ct.byref(bp.args), N.ptr(p), N.stream()), "pack")
    return p


@pytest.mark.parametrize("C", [3, 16])
@pytest.mark.parametrize("rand_const", [0.0, 0.5, 6.0, -4.0])
def test_adjoint(work, C, rand_const):  # noqa: F811
    from sailor_gb300 import _native as N
    bp = _pipeline(work, C=C)
    bp.render_args(float(work["voxel_size"][0]) * work["trunc_weight"], sdf_s=0.01, t_thres=1e-4, rand_const=rand_const)
    g = torch.Generator(device="cuda").manual_seed(1)
    up = [torch.randn((bp.R, 3), generator=g, device="cuda")] + [torch.randn(bp.R, generator=g, device="cuda") for _ in range(3)]
    got = []
    for pk in (None, _packed(bp)):
        gf, gt = torch.zeros_like(bp.feat), torch.zeros_like(bp.tsdf)
        gs, gr = torch.empty((bp.R, bp.S), device="cuda"), torch.empty((bp.R, bp.S, 3), device="cuda")
        N.check(N.lib.sg_render_packed_bwd(Ct.byref(bp.tree), Ct.byref(bp.seg), Ct.byref(bp.args), N.ptr(pk),
                                           *[N.ptr(u) for u in up], N.ptr(gf), N.ptr(gt), N.ptr(gs), N.ptr(gr), N.stream()),
                "bwd")
        got.append((gs, gr, gf, gt))
    a, b = got
    assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1]) and b[0].abs().max().item() > 0
    for k in (2, 3):  # atomics: the order of additions alone
        m = a[k].abs().max().item()
        assert m > 0 and (a[k] - b[k]).abs().max().item() <= 1e-5 * m


@pytest.mark.parametrize("tsdf", [False, True])
@pytest.mark.parametrize("C", [3, 16])
def test_training(work, C, tsdf):  # noqa: F811
    from sailor_gb300 import _native as N
    bp = _pipeline(work, C=C)
    scale = 2.0 / (3.0 * bp.R)
    res = {}
    for name, pk in (("grid", None), ("packed", _packed(bp))):
        for det in (True, False):
            outs = [torch.empty((bp.R, 3), device="cuda")] + [torch.empty(bp.R, device="cuda") for _ in range(4)]
            gf, gt = torch.zeros_like(bp.feat), torch.zeros_like(bp.tsdf) if tsdf else None
            if det:
                N.check(N.lib.sg_render_packed_train_det(
                    Ct.byref(bp.tree), Ct.byref(bp.seg), Ct.byref(bp.args), N.ptr(pk), len(bp._groups), bp._det_groups,
                    bp._det_group_S, N.ptr(bp.target_rgb), scale, *[N.ptr(o) for o in outs], N.ptr(gf), N.ptr(gt),
                    N.ptr(bp.det_ws), bp.det_ws.numel(), bp.record_capacity, N.ptr(bp.status), N.stream()), "det")
            else:
                for seg, args in bp._group_launch:
                    N.check(N.lib.sg_render_packed_train(Ct.byref(bp.tree), Ct.byref(seg), Ct.byref(args), N.ptr(pk),
                                                         N.ptr(bp.target_rgb), scale, *[N.ptr(o) for o in outs], N.ptr(gf),
                                                         N.ptr(gt), N.stream()), "train")
            res[name, det] = outs + [gf] + ([gt] if tsdf else [])
    torch.cuda.synchronize()
    for a, b in zip(res["grid", True], res["packed", True]):
        assert torch.equal(a, b)
    for k, (a, b) in enumerate(zip(res["grid", False], res["packed", False])):
        m = a.abs().max().item()
        assert torch.equal(a, b) if k < 5 else (m > 0 and (a - b).abs().max().item() <= 1e-5 * m)
