"""GPU checks of the intersection's rows where their shapes can go wrong: row
widths off 16 bytes, ray counts off the warp, rays along axes and planes, and
camera segments whose pixels are or are not walked in tiles."""
import ctypes

import numpy as np
import pytest
import torch
from test_gpu_parity import _t, case  # noqa: F401  (case: fixture)

from sailor_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


def _rays(kind, B, n, bb, rng):
    lo, hi = bb[:, None, :, 0], bb[:, None, :, 1]
    inside = lo + (hi - lo) * rng.random((B, n, 3))
    if kind == "axes":
        axes = np.array([[1, 0, 0], [-1, 0, 0], [0, 1, 0], [0, -1, 0], [0, 0, 1], [0, 0, -1], [0.6, 0.8, 0],
                         [0, -0.8, 0.6], [0.8, 0, -0.6], [1e-7, 1, 0], [1e-22, 0.6, 0.8]], np.float32)
        d = axes[rng.integers(0, len(axes), (B, n))]
        if n > 8:  # on the voxel planes exactly
            vs = (hi - lo)[..., :1] / 63.0
            inside[:, : n // 2] = lo + np.round((inside[:, : n // 2] - lo) / vs) * vs + vs * 0.5
    else:
        d = rng.normal(size=(B, n, 3))
        d /= np.linalg.norm(d, axis=-1, keepdims=True)
    return (inside - d * (hi - lo).max() * 1.5).astype(np.float32), d.astype(np.float32)


@pytest.mark.parametrize("kind", ["random", "axes"])
@pytest.mark.parametrize("n", [1, 31, 33, 2000])
def test_rows_match_the_warp_variant(case, kind, n):  # noqa: F811
    """Rows, padding, t-intervals, valid lengths and status against the
    variant that tests every occupied child (its rows padded by a pass of
    their own), bit for bit."""
    from sailor_gb300 import autotune
    octree = case["g"]["octree"]
    B = case["ref"]["vol_bbox"].shape[0]
    o, d = _rays(kind, B, n, case["ref"]["vol_bbox"], np.random.default_rng(n))
    saved, outs = autotune.current(), []
    try:
        for wv in (0, 1):
            autotune.set_knob("isect_warp", wv)
            for W in (1, 3, 5, 33, 130, 1024, 2050):
                for mode in ((-1, False, -1), (2, False, -1), (-1, True, 2)):
                    rows = octree.voxel_traversal(_t(o), _t(d), W, 0, *mode)
                    torch.cuda.synchronize()
                    outs.append([x.clone() for x in rows] + [octree._status.clone()])
    finally:
        for k, v in saved.items():
            autotune.set_knob(k, v)
    half = len(outs) // 2
    for a, b in zip(outs[:half], outs[half:]):
        for x, y in zip(a, b):
            assert torch.equal(x, y)


@pytest.mark.parametrize("sizes", [[(64, 32), (40, 8)], [(40, 20), (33, 17), (16, 12)], [(8, 4), (7, 9), (24, 16)]])
def test_camera_segments_match_ray_buffers(sizes):
    """Camera segments (tiled where width, height and place allow it) against
    the same rays from buffers."""
    from sailor_gb300 import _native as N
    from sailor_gb300.batch import BatchPipeline
    w = syn.make_batch_workload(seed=9, n_frames=2, views=(2, 3), view_res=(96,), n_prims=8, D=64, trunc=0.04,
                                n_targets=len(sizes), target_res=(32, 32), target_S=(32,))
    view_hw = [[d.shape for d in fr["depth"]] for fr in w["frames"]]
    bp = BatchPipeline(view_hw, [(t % 2, a * b, 32) for t, (a, b) in enumerate(sizes)], D=64, rate=4, C=3, W_hits=96,
                       target_widths=[a for a, _ in sizes])
    bp.load_views(w["frames"], w["vol_bbox"], w["voxel_size"], w["trunc_weight"])
    Ks = [syn.intrinsics(32).astype(np.float32) * np.array([[a / 32, 1, a / 32], [1, b / 32, b / 32], [1, 1, 1]])
          for a, b in sizes]
    bp.load_cameras(Ks, [t["R"] for t in w["targets"]], [t["T"] for t in w["targets"]])
    bp.build()
    bp.intersect()
    torch.cuda.synchronize()
    ref = [x.clone() for x in (bp.hit_count, bp.valid_len, bp.hit_idx, bp.hit_t0, bp.hit_t1)]
    assert ref[0].max().item() > 3
    for x in (bp.hit_count, bp.valid_len, bp.hit_idx, bp.hit_t0, bp.hit_t1):
        x.fill_(-7)
    N.check(N.lib.sg_intersect_segments(ctypes.byref(bp.tree), ctypes.byref(bp.seg), N.ptr(bp.ori), N.ptr(bp.dirs),
                                        bp.W, N.ptr(bp.hit_idx), N.ptr(bp.hit_t0), N.ptr(bp.hit_t1),
                                        N.ptr(bp.valid_len), N.ptr(bp.hit_count), N.ptr(bp.status), N.stream()), "i")
    torch.cuda.synchronize()
    used = torch.arange(bp.W, device="cuda")[None] < ref[0][:, None]
    assert torch.equal(bp.hit_count, ref[0]) and torch.equal(bp.valid_len, ref[1])
    for a, b in zip((bp.hit_idx, bp.hit_t0, bp.hit_t1), ref[2:]):
        assert torch.equal(a[used], b[used])
