"""GPU checks of the renders over packed fields (sg_pack_fields,
sg_render_packed_*) against the same renders over the grids."""
import ctypes

import pytest
import torch
from test_gpu_batch import D, RATE, _pipeline, work  # noqa: F401  (work: fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C", [3, 16])
@pytest.mark.parametrize("rand_const", [0.0, 0.5, 1.0, 6.0, -4.0])
def test_packed_taps_match_grid_taps(work, C, rand_const):
    """Renders from the packed fields against renders from the grids, on the
    same rows, bit for bit; jitters outside [0, 1] move samples off their
    nodes, to cells that are not packed."""
    from sailor_gb300 import _native as N
    bp = _pipeline(work, C=C)
    trunc_m = float(work["voxel_size"][0]) * work["trunc_weight"]
    bp.render_args(trunc_m, sdf_s=0.01, t_thres=1e-4, rand_const=rand_const)
    packed = torch.full((bp.B, D, D, D, 4), float("nan"), device="cuda")
    N.check(N.lib.sg_pack_fields(ctypes.byref(bp.tree), ctypes.byref(bp.seg), ctypes.byref(bp.args), N.ptr(packed), N.stream()),
            "pack")
    g = torch.randn((bp.R, 3), generator=torch.Generator(device="cuda").manual_seed(1), device="cuda")
    got = {}
    for name, pk in (("grid", None), ("packed", packed)):
        outs = [torch.empty((bp.R, 3), device="cuda")] + [torch.empty(bp.R, device="cuda") for _ in range(3)]
        N.check(N.lib.sg_render_packed_fwd(ctypes.byref(bp.tree), ctypes.byref(bp.seg), ctypes.byref(bp.args), N.ptr(pk),
                                           *[N.ptr(o) for o in outs], None, None, N.stream()), "fwd")
        gf, gt = torch.zeros_like(bp.feat), torch.zeros_like(bp.tsdf)
        gs, gr = torch.empty((bp.R, bp.S), device="cuda"), torch.empty((bp.R, bp.S, 3), device="cuda")
        N.check(N.lib.sg_render_packed_bwd(ctypes.byref(bp.tree), ctypes.byref(bp.seg), ctypes.byref(bp.args), N.ptr(pk),
                                           N.ptr(g), None, None, None, N.ptr(gf), N.ptr(gt), N.ptr(gs), N.ptr(gr),
                                           N.stream()), "bwd")
        got[name] = outs + [gr, gf]
    torch.cuda.synchronize()
    a, b = got["packed"], got["grid"]
    for k in range(5):
        assert torch.equal(a[k], b[k]), k
    m = b[5].abs().max().item()
    assert m > 0 and (a[5] - b[5]).abs().max().item() <= 1e-5 * m  # atomics: order alone
    # packed voxels: the bricks of nodes and the voxels beside them, no others
    node = bp.brick_node.view(bp.B, bp.Dt, bp.Dt, bp.Dt) >= 0
    fine = node.repeat_interleave(RATE, 1).repeat_interleave(RATE, 2).repeat_interleave(RATE, 3)
    want = torch.nn.functional.max_pool3d(fine[:, None].float(), 3, 1, 1)[:, 0] > 0
    assert torch.equal(~torch.isnan(packed).any(-1), want)


def test_packed_fields_refused():
    """No packed path for features on another geometry or bricks that are no
    power of two; a misaligned buffer is an invalid argument."""
    from sailor_gb300 import _native as N
    from sailor_gb300.batch import BatchPipeline
    bp = BatchPipeline([[(16, 16)]], [(0, 64, 32)], D=24, rate=6, C=3, W_hits=32)
    bp.render_args(0.04)
    buf = torch.empty(24 ** 3 * 4 + 4, device="cuda")
    call = lambda t: N.lib.sg_pack_fields(ctypes.byref(bp.tree), ctypes.byref(bp.seg), ctypes.byref(bp.args), N.ptr(t),  # noqa
                                          N.stream())
    assert bp.packed is None and call(buf) == 4
    bp = BatchPipeline([[(16, 16)]], [(0, 64, 32)], D=24, rate=4, C=3, W_hits=32)
    bp.render_args(0.04)
    assert call(buf[1:]) == 1
    other = bp.voxel_size.clone()
    bp.args.feat_vs = other.data_ptr()
    assert call(buf) == 4


def test_head_of_voxels_matches_float64(work):  # noqa: F811
    """Rendered colour with a 16-channel head against the same samples,
    weights and features in float64 (head of the tapped features).  Per
    sample: 16 roundings per voxel, 8 of the tap and 3 of the weights, of sums
    of |head| |feature|; the weights (sum at most 1) and the densities they
    come from are those of the 32-bit render, so they carry the bound of the
    existing chain test (1e-5)."""
    bp = _pipeline(work)
    z = torch.empty((bp.R, bp.S), device="cuda")
    node = torch.empty((bp.R, bp.S), dtype=torch.int32, device="cuda")
    bp.forward(z, node)
    gs, gr = torch.empty((bp.R, bp.S), device="cuda"), torch.empty((bp.R, bp.S, 3), device="cuda")
    ones = torch.ones((bp.R, 3), device="cuda")
    bp.backward(ones, grad_sigma=gs, grad_rgb=gr)  # grad_rgb = the compositing weight of each sample
    from sailor_gb300.fields import grid_gather
    worst = 0.0
    for t, (f, n, S) in enumerate(bp.targets):
        a, b = bp.ray_slices[t]
        fe = grid_gather(bp.feat[f:f + 1], bp.ori[a:b][None], bp.dirs[a:b][None], z[a:b, :S][None].contiguous(),
                         bp.vol_bbox[f:f + 1], bp.voxel_size[f:f + 1])[0]
        rgb = ((fe.double() @ bp.head.double().T) * gr[a:b, :S, :1].double()).sum(1)
        worst = max(worst, (bp.out_rgb[a:b].double() - rgb).abs().max().item())
    tol = (2 * 27 + 128) * 2.0 ** -24 * bp.head.abs().sum(1).max().item() * bp.feat.abs().max().item()
    assert worst <= min(tol, 1e-4), (worst, tol)
