"""Projection of points into the source views and the gather of per-view 2D
feature maps at the projections: the step of SRONet's render after sampling.

Drop-ins, with the reference's arguments and results:

* ``proj_persp`` for ``utils_render.proj_persp``
  (utils_render/utils_render.py:380-414);
* ``forward_sample_feature`` for ``BasicRenNet.forward_sample_feature``
  (SRONet/BasicRenNet.py:245-259): four ``F.grid_sample`` calls
  (bilinear, align_corners=True, zero padding) and the clamped depth
  difference t_psdf;

and the fused form ``project_sample_features``, both steps in one launch
(the projected grids never leave the SM).  Every call runs
``sg_project_gather`` of ``libsailor_gb300.so`` on the current CUDA stream;
there is no CPU path.  Feature maps are read through their strides, so NCHW
tensors and channels-last ones (``memory_format=torch.channels_last``, read
in whole texel rows) both work; with many points a map in another layout is
rewritten channels-last first.
"""
import ctypes as C

import torch

from . import _native as N

__all__ = ["proj_persp", "forward_sample_feature", "project_sample_features"]

PSDF_CLIP = 0.01  # clamp of proj_z - sampled depth (BasicRenNet.py:250)


def _f32(t, name):
    if not isinstance(t, torch.Tensor) or not t.is_cuda:
        raise RuntimeError(f"{name} input must be a cuda tensor")
    if t.dtype != torch.float32:
        raise RuntimeError(f"{name} must be float32, got {t.dtype}")
    return t


def _cams(K, R, T, n_images):
    K = _f32(K, "K").reshape(n_images, 9).contiguous()
    R = _f32(R, "R").reshape(n_images, 9).contiguous()
    T = _f32(T, "T").reshape(n_images, 3).contiguous()
    return K, R, T


# A thread per item walks the channels of a map that is not channels-last
# through scattered 4-byte loads, near points sharing them; rows of a
# channels-last map are read whole.  Rewriting costs a pass over the map and
# about 10 us of calls, so it is done from CHANNELS_LAST_FROM points a pixel on,
# more with few channels (8 / C; 3 below 8, never below 6), and where the output
# is large enough to hide the calls.  Measured, direct against rewritten, on
# samples along rays (two maps a call) / on a raster of neighbouring pixels, 4
# images of 512^2, us:
#   C   8: 1 point a pixel 160 and 160 /  66 and  87;  2: 309 and 214 / -
#   C  16: 0.5             178 and 172 /  63 and  95;     1: 329 and 207 / 105 and 117
#   C  32: 0.25            235 and 221 /  79 and 128;   0.5: 426 and 245 / 148 and 143
#   C  68: 0.25            419 and 532 / 187 and 290;   0.5: 788 and 588 / 323 and 318
#   C   5: 5 points a pixel 439 and 469; C 6: 2: 213 and 237, 3: 316 and 304
# (the raster of few channels is what rewriting loses on, by less than the direct
# walk has gained there) and, where the calls count, one image of 512^2, C 16: 0.5
# (2^21 values) 50 and 66, 1 (2^22) 87 and 65.
CHANNELS_LAST_FROM = 0.4
CHANNELS_LAST_WORK = 1 << 22


def _rewrites(n, Cm, pixels, N_pts):
    """Whether n maps of Cm channels, not channels-last, are rewritten for N_pts points each."""
    if Cm < 6 or n * N_pts * Cm < CHANNELS_LAST_WORK:
        return False
    return N_pts >= CHANNELS_LAST_FROM * pixels * (max(1.0, 20.0 / Cm) if Cm >= 8 else 7.5)


def _channels_last(img):
    """A copy of a [n, C, H, W] map in channels-last order ([n, H, W, C]
    contiguous), or None where the kernel does not take the size or the memory
    has no room for one (the map is then gathered through its strides)."""
    n, Cm, H, W = img.shape
    try:
        out = torch.empty((n, H, W, Cm), device=img.device)
    except torch.OutOfMemoryError:
        return None
    rc = N.lib.sg_channels_last(N.ptr(img), (C.c_longlong * 4)(*img.stride()), n, Cm, H, W, N.ptr(out), N.stream())
    if rc == N.SG_ERR_UNSUPPORTED:
        return None
    N.check(rc, "channels_last")
    return out


def _maps(a, imgs, N_pts):
    """The [n_images, C, H, W] maps and their [n_images, N, C] outputs into the
    arguments; returns the outputs, and what has to live until the launch."""
    for img in imgs:
        if img.dim() != 4:
            raise RuntimeError("feature maps must be [n_images, C, H, W]")
        _f32(img, "feature map")
    try:
        return _fill_maps(a, imgs, N_pts, True)
    except torch.OutOfMemoryError:
        pass
    return _fill_maps(a, imgs, N_pts, False)  # the copies of maps before an output that had no room are gone


def _fill_maps(a, imgs, N_pts, rewrite):
    outs, keep = [], []
    for i, img in enumerate(imgs):
        n, Cm, H, W = img.shape
        out = torch.empty((n, N_pts, Cm), device=img.device)
        src, strides = img, img.stride()
        if rewrite and img.stride(1) != 1 and _rewrites(n, Cm, H * W, N_pts):
            rows = _channels_last(img)
            if rows is not None:
                src, strides = rows, (H * W * Cm, 1, W * Cm, Cm)
        m = a.maps[i]
        m.data = src.data_ptr()
        for k in range(4):
            m.stride[k] = strides[k]
        m.C, m.H, m.W = Cm, H, W
        m.out = out.data_ptr()
        outs.append(out)
        keep += [img, src]
    a.n_maps = len(imgs)
    return outs, keep


def _launch(a, keep):
    N.check(N.lib.sg_project_gather(C.byref(a), N.stream()), "project_gather")
    return keep


def _persp_args(a, points, K, R, T, p_depths, n_views, depth_thres, min_d, max_d, res):
    pts = _f32(points, "points")
    if pts.dim() != 3 or pts.shape[1] != 3:
        raise RuntimeError("points must be [batch, 3, N]")
    n_images = K.shape[0] if K.dim() == 3 else K.numel() // 9
    Bp = pts.shape[0]
    if p_depths is not None:
        div = n_views  # proj_persp repeats the points over the views
        if Bp * n_views != n_images:
            raise RuntimeError(f"points batch {Bp} x {n_views} views != {n_images} cameras")
    elif Bp == n_images:
        div = 1
    elif Bp == 1:
        div = n_images  # broadcast
    else:
        raise RuntimeError(f"points batch {Bp} does not broadcast against {n_images} cameras")
    Kc, Rc, Tc = _cams(K, R, T, n_images)
    a.points = pts.data_ptr()
    a.points_stride[0], a.points_stride[1], a.points_stride[2] = pts.stride(0), pts.stride(1), pts.stride(2)
    a.points_div = div
    keep = [pts, Kc, Rc, Tc]
    if p_depths is not None:
        pd = _f32(p_depths, "p_depths")
        a.p_depths = pd.data_ptr()
        a.p_depths_stride[0], a.p_depths_stride[1] = pd.stride(0), pd.stride(-1)
        keep.append(pd)
    a.K, a.R, a.T = Kc.data_ptr(), Rc.data_ptr(), Tc.data_ptr()
    a.n_images, a.num_points = n_images, pts.shape[2]
    a.depth_thres, a.min_d, a.max_d = float(depth_thres), float(min_d), float(max_d)
    a.half_res = float(int(res) // 2)
    a.psdf_map = -1
    return keep


def proj_persp(points, K, R, T, p_depths, n_views, depth_thres=0.01, min_d=0.1, max_d=4.0, res=512):
    """points [batch, 3, N]; K, R [batch*n_views, 3, 3]; T [batch*n_views, 3, 1]
    -> (ori_pts [n_images, 3, N] = R p + T, grids [n_images, 2, N] in
    [-1, 1] (-2: behind depth_thres, or p_depth outside [min_d, max_d]),
    depth [n_images, 1, N] (-2 for the latter))."""
    a = N.SgProjGather()
    keep = _persp_args(a, points, K, R, T, p_depths, n_views, depth_thres, min_d, max_d, res)
    dev = points.device
    n, Np = a.n_images, a.num_points
    ori = torch.empty((n, 3, Np), device=dev)
    grids = torch.empty((n, 2, Np), device=dev)
    depth = torch.empty((n, 1, Np), device=dev)
    a.ori_pts, a.grids, a.depth = ori.data_ptr(), grids.data_ptr(), depth.data_ptr()
    _launch(a, keep)
    return ori, grids, depth


def forward_sample_feature(feats_geo, depths, feats_rgb, rgbs_n, xy, z):
    """Maps [n_images, C, H, W]; xy [n_images, N, 1, 2] grids; z [n_images, 1, N]
    -> (geo [n_images, N, Cg], rgb feats [n_images, N, Cr], t_psdf
    [n_images, N, 1] = clamp(z - depth sample, -0.01, 0.01) / 0.01, rgbs
    [n_images, N, 3])."""
    grid = _f32(xy, "xy")
    n = grid.shape[0]
    Np = grid.numel() // (2 * n)
    g = grid.reshape(n, Np, 2).contiguous()
    zz = _f32(z, "z").reshape(n, Np).contiguous()
    a = N.SgProjGather()
    a.grids_in, a.depth_in = g.data_ptr(), zz.data_ptr()
    a.n_images, a.num_points = n, Np
    psdf = torch.empty((n, Np, 1), device=g.device)
    a.psdf_map, a.psdf_clip, a.psdf_scale, a.psdf = 1, PSDF_CLIP, 1.0 / PSDF_CLIP, psdf.data_ptr()
    outs, maps = _maps(a, (feats_geo, depths, feats_rgb, rgbs_n), Np)
    _launch(a, [g, zz] + maps)
    return outs[0], outs[2], psdf, outs[3]


def project_sample_features(points, K, R, T, p_depths, n_views, feats_geo, depths, feats_rgb, rgbs_n,
                            depth_thres=0.01, min_d=0.1, max_d=4.0, res=512, want_grids=False):
    """proj_persp + forward_sample_feature in one launch.  Returns
    (proj_z [n_images, 1, N], geo, rgb feats, t_psdf, rgbs) as the two
    reference calls give them, and the grids [n_images, 2, N] when
    want_grids."""
    a = N.SgProjGather()
    keep = _persp_args(a, points, K, R, T, p_depths, n_views, depth_thres, min_d, max_d, res)
    dev = points.device
    n, Np = a.n_images, a.num_points
    depth = torch.empty((n, 1, Np), device=dev)
    a.depth = depth.data_ptr()
    grids = None
    if want_grids:
        grids = torch.empty((n, 2, Np), device=dev)
        a.grids = grids.data_ptr()
    psdf = torch.empty((n, Np, 1), device=dev)
    a.psdf_map, a.psdf_clip, a.psdf_scale, a.psdf = 1, PSDF_CLIP, 1.0 / PSDF_CLIP, psdf.data_ptr()
    outs, maps = _maps(a, (feats_geo, depths, feats_rgb, rgbs_n), Np)
    _launch(a, keep + maps)
    res_ = (depth, outs[0], outs[2], psdf, outs[3])
    return res_ + (grids,) if want_grids else res_
