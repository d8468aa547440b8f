"""Performance cases: what programs that use sailor_gb300 have it do.

Each kind below is one way the package is used, through its public entry
points.  ``listed()`` holds the sizes of the package's own workloads and of
SRONet's rendering loop (16384-ray chunks, 4 views of 512^2, 128^3 volumes
with 4^3 bricks, 48 samples); ``draw()`` gives other sizes of the same
ranges.  Scenes are unions of capsules and ellipsoids in a 2 m cube seen by
cameras on a 2.5 m ring, as ``sailor_gb300.synthetic`` makes them, ray-cast
here on the GPU.
"""
import math

import numpy as np
import torch
import torch.nn.functional as F

from sailor_gb300 import fields, nerf, views
from sailor_gb300 import synthetic as syn
from sailor_gb300 import voxel_encoding as VE
from sailor_gb300 import voxel_encoding_helper as H
from sailor_gb300.batch import BatchPipeline
from sailor_gb300.pipeline import FramePipeline

DEV = "cuda"


def listed():
    return [
        # Training on many frames at once, the step replayed from a CUDA graph:
        # half the frames and targets of the batched workload, the same sizes.
        dict(name="train_4f", kind="train", frames=4, vmin=4, vmax=8, vres="512,768,1024", D=256, rate=8, C=16,
             targets=8, tmin=256, tmax=1024, S="32,48,64,96,128", W=256, tsdf=False, graph=True),
        # The same on small frames: many short launches.
        dict(name="train_small", kind="train", frames=3, vmin=2, vmax=4, vres="256,384", D=128, rate=8, C=16,
             targets=5, tmin=128, tmax=256, S="32,48,64,96,128", W=256, tsdf=False, graph=True),
        # Full-resolution rendering of one frame on resident buffers: fusion,
        # tree and one fused render.
        dict(name="frame_1024", kind="frame", views=4, res=1024, D=512, rate=8, target=1024, S=96, Dc=256, W=1024),
        # SRONet per frame: fusion over the data-driven box, coarse volume, tree.
        dict(name="build_128", kind="build", batch=1, views=4, res=512, D=128, rate=4),
        # SRONet per chunk of a target's rays: intersection, sampling, sort.
        dict(name="rays_16k", kind="rays", batch=1, views=4, res=512, D=128, rate=4, rays=16384, S=48, shade=False),
        # A whole 512^2 target through the drop-in calls, density and colour
        # from dense grids.
        dict(name="rays_512", kind="rays", batch=1, views=4, res=512, D=256, rate=8, rays=262144, S=64, shade=True),
        # Forward and adjoint of 2^20 random rays, upstream gradients on every output.
        dict(name="diff_1m", kind="diff", views=4, res=512, D=256, rate=8, rays=1 << 20, S=96, C=16, W=256),
        # Field gathers and exact compositing under autograd.
        dict(name="fields_grad", kind="fields", D=256, C=16, rays=1 << 17, S=96),
        # Multi-level tree: build, depth-first traversal, fine sampling.
        dict(name="octree_512", kind="octree", views=4, res=512, D=256, levels=4, rays=262144, S=64, Wf=512),
        # FastNerf's occupancy network.
        dict(name="nerf_4m", kind="nerf", points=1 << 22, views=3, geo=False),
        # Projection into the views and the 2D feature gather: a whole target,
        # channels-last maps.
        dict(name="project_nhwc", kind="project", views=4, res=512, Cg=32, Cr=32, rays=262144, S=32, nhwc=True),
        # The same for one chunk of rays, maps as a convolution leaves them.
        dict(name="project_nchw", kind="project", views=4, res=512, Cg=32, Cr=32, rays=16384, S=48, nhwc=False),
    ]


def draw(rng):
    def span(lo, hi):  # spread over the logarithm
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["train", "frame", "build", "rays", "diff", "fields", "octree", "nerf", "project", "composite"])
    if kind == "train":
        big, tsdf = rng.random() < 0.5, rng.random() < 0.5
        S = rng.choice(["32", "48,128", "32,48,64,96,128", "17,80"])
        # The step behind a ray's last sample is 1e10 long: its density
        # gradient is that times a difference of equal sums, rounding alone
        # unless the sample fills its warp.
        S = rng.choice(["32", "64,128", "32,64,96,128"]) if tsdf else S
        return dict(kind=kind, frames=rng.randint(1, 4), vmin=2, vmax=rng.randint(2, 8),
                    vres="512,768,1024" if big else "200,256,384", D=256 if big else rng.choice([64, 128]),
                    rate=rng.choice([4, 8]), C=rng.choice([3, 16, 16]), targets=rng.randint(1, 8), tmin=64,
                    tmax=span(128, 800), S=S, W=256, tsdf=tsdf, graph=rng.random() < 0.5)
    if kind == "frame":
        return dict(kind=kind, views=rng.randint(2, 6), res=span(256, 1024), D=rng.choice([128, 256, 512]), rate=8,
                    target=span(96, 1024), S=rng.randint(24, 128), Dc=rng.choice([64, 256]), W=512)
    if kind == "build":
        return dict(kind=kind, batch=rng.randint(1, 3), views=rng.randint(2, 6), res=span(200, 1024),
                    D=rng.choice([64, 128, 256]), rate=rng.choice([2, 4, 8]))
    if kind == "rays":
        return dict(kind=kind, batch=rng.randint(1, 2), views=4, res=512, D=rng.choice([128, 256]),
                    rate=rng.choice([4, 8]), rays=span(1000, 262144), S=rng.randint(24, 128),
                    shade=rng.random() < 0.5)
    if kind == "diff":
        return dict(kind=kind, views=4, res=512, D=rng.choice([128, 256]), rate=8, rays=span(4000, 1 << 20),
                    S=32 * rng.randint(1, 3), C=rng.choice([3, 16]), W=256)
    if kind == "fields":
        return dict(kind=kind, D=rng.choice([64, 128, 256]), C=rng.choice([3, 4, 8, 16]), rays=span(1000, 1 << 17),
                    S=rng.randint(24, 96))
    if kind == "octree":
        return dict(kind=kind, views=4, res=512, D=rng.choice([128, 256]), levels=rng.randint(3, 4),
                    rays=span(2000, 262144), S=rng.randint(24, 96), Wf=512)
    if kind == "nerf":
        return dict(kind=kind, points=span(1000, 1 << 22), views=rng.randint(1, 6), geo=rng.random() < 0.3)
    if kind == "project":
        return dict(kind=kind, views=rng.randint(2, 6), res=span(128, 512), Cg=rng.choice([16, 30, 32]),
                    Cr=rng.choice([8, 16, 32]), rays=span(500, 32768), S=rng.randint(24, 96),
                    nhwc=rng.random() < 0.5)
    return dict(kind="composite", rays=span(1000, 262144), S=rng.randint(24, 96), C=rng.choice([3, 8, 16, 30]),
                occ=rng.random() < 0.5, presorted=rng.random() < 0.5)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _dev(a, dt=torch.float32):
    return torch.as_tensor(np.ascontiguousarray(a)).to(DEV, dt)


def _cast(prims, K, R, T, res):
    """z-depth [res, res] (float64, 0: nothing) of the union of primitives."""
    f64 = dict(dtype=torch.float64, device=DEV)
    v, u = torch.meshgrid(torch.arange(res, **f64), torch.arange(res, **f64), indexing="ij")
    Ki, Rt = torch.as_tensor(np.linalg.inv(K), **f64), torch.as_tensor(R, **f64)
    d = (torch.stack([u, v, torch.ones_like(u)], -1) @ Ki.T) @ Rt
    o = torch.as_tensor(-R.T @ T, **f64)

    def sphere(ol, dl, r):
        a, b, c = (dl * dl).sum(-1), (dl * ol).sum(-1), (ol * ol).sum() - r * r
        q = b * b - a * c
        t = (-b - torch.sqrt(q.clamp(min=0))) / a
        return torch.where((q >= 0) & (t > 1e-6), t, torch.inf)

    best = torch.full((res, res), torch.inf, **f64)
    for p in prims:
        if p[0] == "capsule":
            a, b, r = torch.as_tensor(p[1], **f64), torch.as_tensor(p[2], **f64), float(p[3])
            ba, oa = b - a, o - a
            baba, bard, baoa = (ba * ba).sum(), d @ ba, (ba * oa).sum()
            A = baba * (d * d).sum(-1) - bard * bard
            Bq = baba * (d @ oa) - baoa * bard
            h = Bq * Bq - A * (baba * (oa * oa).sum() - baoa * baoa - r * r * baba)
            tb = (-Bq - torch.sqrt(h.clamp(min=0))) / A.clamp(min=1e-12)
            y = baoa + tb * bard
            t = torch.minimum(sphere(o - a, d, r), sphere(o - b, d, r))
            t = torch.where((h >= 0) & (y > 0) & (y < baba) & (tb > 1e-6), tb, t)
        else:
            Q, radii = torch.as_tensor(p[3], **f64), torch.as_tensor(p[2], **f64)
            t = sphere((o - torch.as_tensor(p[1], **f64)) @ Q / radii, d @ Q / radii, 1.0)
        best = torch.minimum(best, t)
    return torch.where(torch.isfinite(best), best, 0.0)


def _view(prims, K, R, T, res, g):
    """Depth (N(0, 5 mm) noise, 2 % dropout, uint16 x 1e-4 m) and packed uint8 colour."""
    z = _cast(prims, K, R, T, res)
    z = z + torch.randn(z.shape, generator=g, device=DEV, dtype=torch.float64) * 0.005 * (z > 0)
    z[torch.rand(z.shape, generator=g, device=DEV) < 0.02] = 0.0
    depth = (torch.round(z * 10000.0).clamp(0, 65535) / 10000.0).float()
    rgb = torch.randint(0, 256, (3, res, res), generator=g, device=DEV).float()
    return depth, rgb, rgb[2] * 65536.0 + rgb[1] * 256.0 + rgb[0]


def _frame(rng, n_views, sizes, g, n_prims=12):
    prims = syn.random_primitives(rng, n_prims)
    fr = dict(K=[], RT=[], depth=[], color=[], rgb=[])
    for R, T in syn.ring_cameras(n_views, phase=rng.uniform(0, 2 * math.pi)):
        res = int(rng.choice(sizes))
        K = syn.intrinsics(res)
        depth, rgb, packed = _view(prims, K, R, T, res, g)
        fr["K"].append(K.astype(np.float32))
        fr["RT"].append(np.concatenate([R, T[:, None]], 1).astype(np.float32))
        fr["depth"].append(depth)
        fr["color"].append(packed)
        fr["rgb"].append(rgb)
    return fr


def _box(D, batch=1, trunc=0.03):
    vs = np.float32(2.0) / np.float32(D - 1)
    return (np.tile(np.array([[-1.0, 1.0]] * 3, np.float32), (batch, 1, 1)), np.full((batch, 1), vs, np.float32),
            float(np.float32(trunc) / vs))


def _camera(rng):
    a = rng.uniform(0, 2 * math.pi)
    return syn.look_at((2.5 * math.cos(a), 2.5 * math.sin(a), rng.uniform(0.6, 1.6)))


def _camera_rays(rng, n):
    """n consecutive rays (rows of pixels about the image's middle) of a
    target camera: one 512^2 image, or a square image where n is more."""
    res = max(512, math.isqrt(n - 1) + 1)
    R, T = _camera(rng)
    K = syn.intrinsics(res)
    rays = VE.rays_calculating(_dev(K).view(1, 1, 3, 3), _dev(R).view(1, 1, 3, 3), _dev(T).view(1, 1, 3), res, 0)
    at = (res * res - n) // 2
    rays = rays.view(-1, 6)[at:at + n]
    return rays[None, :, :3].contiguous(), rays[None, :, 3:].contiguous()


def _aimed_rays(g, n, half=1.0):
    """Rays from a 3 m sphere aimed at uniform points of a cube about the origin."""
    o = torch.randn((n, 3), generator=g, device=DEV)
    o = o * (3.0 / o.norm(dim=-1, keepdim=True))
    d = (torch.rand((n, 3), generator=g, device=DEV) * 2.0 - 1.0) * half - o
    return o, d / d.norm(dim=-1, keepdim=True)


# ---------------------------------------------------------------------------
# train: BatchPipeline.train_step
# ---------------------------------------------------------------------------
def _train_sizes(c):
    """Target image edges and samples: fixed by the case alone."""
    S = [int(s) for s in c["S"].split(",")]
    lo, hi, n = c["tmin"], c["tmax"], c["targets"]
    edge = [int(round((lo + (hi - lo) * (k + 1) / n) / 8) * 8) for k in range(n)]
    edge = [edge[(5 * k + 2) % n] if math.gcd(5, n) == 1 else edge[k] for k in range(n)]
    return [(k % c["frames"], edge[k], S[k % len(S)]) for k in range(n)]


def _prep_train(c, seed):
    rng, g = np.random.default_rng(seed), _gen(seed)
    shape = np.random.default_rng(c["frames"] * 31 + c["D"])  # view counts and sizes: the case's, not the seed's
    sizes = [int(s) for s in c["vres"].split(",")]
    frames = []
    for _ in range(c["frames"]):
        nv = int(shape.integers(c["vmin"], c["vmax"] + 1))
        fr = dict(K=[], RT=[], depth=[], color=[])
        prims = syn.random_primitives(rng, 12)
        for R, T in syn.ring_cameras(nv, phase=rng.uniform(0, 2 * math.pi)):
            res = int(shape.choice(sizes))
            K = syn.intrinsics(res)
            depth, _, packed = _view(prims, K, R, T, res, g)
            fr["K"].append(K.astype(np.float32))
            fr["RT"].append(np.concatenate([R, T[:, None]], 1).astype(np.float32))
            fr["depth"].append(depth)
            fr["color"].append(packed)
        frames.append(fr)
    tg = _train_sizes(c)
    bp = BatchPipeline([[tuple(d.shape) for d in fr["depth"]] for fr in frames], [(f, e * e, s) for f, e, s in tg],
                       D=c["D"], rate=c["rate"], C=c["C"], W_hits=c["W"], train_tsdf=c["tsdf"],
                       target_widths=[e for _, e, _ in tg], device=DEV)
    bbox, vs, tw = _box(c["D"], c["frames"])
    bp.load_views(frames, bbox, vs.reshape(-1), tw)
    cams = [_camera(rng) for _ in tg]
    bp.load_cameras([syn.intrinsics(e) for _, e, _ in tg], [R for R, _ in cams], [T for _, T in cams])
    bp.feat.normal_(0.0, 0.1, generator=g)
    bp.set_fields(head=torch.randn((3, c["C"]), generator=g, device=DEV) * 0.5,
                  target_rgb=torch.rand((bp.R, 3), generator=g, device=DEV))
    bp.render_args(float(vs[0, 0]) * tw, sdf_s=0.005, t_thres=1e-4, rand_seed=12)
    return dict(bp=bp, graph=bp.capture(warmup=1) if c["graph"] else None)


def _run_train(s):
    bp = s["bp"]
    if s["graph"] is not None:
        s["graph"].replay()
    else:
        bp.train_step()
    out = dict(tsdf=bp.tsdf, weight=bp.weight, color=bp.colorv, occ0=bp.occ0, occ1=bp.occ1, rgb=bp.out_rgb,
               depth=bp.out_depth, ws=bp.out_ws, alpha=bp.out_alpha, loss=bp.out_loss, grad_feat=bp.grad_feat)
    if bp.train_tsdf:
        out["grad_tsdf"] = bp.grad_tsdf
    return out


def _work_train(c):
    tg, V = _train_sizes(c), c["D"] ** 3 * c["frames"]
    sizes = [int(s) for s in c["vres"].split(",")]
    pix = c["frames"] * 0.5 * (c["vmin"] + c["vmax"]) * sum(s * s for s in sizes) / len(sizes)
    R, RS = sum(e * e for _, e, _ in tg), sum(e * e * s for _, e, s in tg)
    # the samples touch about 5 % of the voxels of the grids (features and their gradient, TSDF)
    return dict(bytes=16 * V + 8 * pix + 40 * R + 0.05 * V * (8 * c["C"] + 4),
                flops=60 * V + 0.2 * RS * (8 * 2 * (c["C"] + 1) * 2 + 100))


# ---------------------------------------------------------------------------
# frame: FramePipeline.build + render
# ---------------------------------------------------------------------------
def _prep_frame(c, seed):
    rng, g = np.random.default_rng(seed), _gen(seed)
    fr = _frame(rng, c["views"], [c["res"]], g, n_prims=24)
    bbox, vs, tw = _box(c["D"], trunc=0.02 if c["D"] >= 512 else 0.03)
    n = c["target"] ** 2
    R, T = _camera(rng)
    rays = VE.rays_calculating(_dev(syn.intrinsics(c["target"])).view(1, 1, 3, 3), _dev(R).view(1, 1, 3, 3),
                               _dev(T).view(1, 1, 3), c["target"], 0).view(1, n, 6)
    pipe = FramePipeline(1, c["D"], c["rate"], n, c["S"], W_hits=c["W"], device=DEV)
    return dict(pipe=pipe, K=_dev(np.stack(fr["K"]))[None], RT=_dev(np.stack(fr["RT"]))[None],
                col=torch.stack(fr["color"])[None], dep=torch.stack(fr["depth"])[None], bb=_dev(bbox), vs=_dev(vs),
                tw=tw, o=rays[..., :3].contiguous(), d=rays[..., 3:].contiguous(),
                grid=torch.rand((1,) + (c["Dc"],) * 3 + (3,), generator=g, device=DEV), gbb=_dev(bbox),
                gvs=torch.full((1, 1), 2.0 / (c["Dc"] - 1), device=DEV), trunc=float(vs[0, 0]) * tw)


def _run_frame(s):
    p = s["pipe"]
    p.build(s["K"], s["RT"], s["col"], s["dep"], s["bb"], s["vs"], s["tw"])
    rgb, depth, ws, alpha = p.render(s["o"], s["d"], s["grid"], s["gbb"], s["gvs"], s["trunc"])
    return dict(tsdf=p.tsdf, weight=p.weight, color=p.color, occ0=p.occ0, occ1=p.occ1, rgb=rgb, depth=depth, ws=ws,
                alpha=alpha)


def _work_frame(c):
    V, R = c["D"] ** 3, c["target"] ** 2
    return dict(bytes=16 * V + 8 * c["views"] * c["res"] ** 2 + 48 * R + 0.05 * (V * 4 + c["Dc"] ** 3 * 12),
                flops=15 * c["views"] * V + 0.2 * R * c["S"] * 200)


# ---------------------------------------------------------------------------
# build: integrate_depths + OcTreeOptions.init_octree
# ---------------------------------------------------------------------------
def _volumes(batch, D, rate, levels=2):
    vols, cnts = [], []
    for k in range(levels):
        vols.append(torch.full((batch,) + (D // rate ** k,) * 3, -1, dtype=torch.int32, device=DEV))
        cnts.append(torch.zeros((batch, 1), dtype=torch.int32, device=DEV))
    return vols, cnts


def _prep_build(c, seed):
    rng, g = np.random.default_rng(seed), _gen(seed)
    frs = [_frame(rng, c["views"], [c["res"]], g) for _ in range(c["batch"])]

    def cat(k):
        return [x for fr in frs for x in fr[k]]

    depth = torch.stack(cat("depth"))
    return dict(inputs=(torch.stack(cat("rgb")), depth, (depth > 0).float(), _dev(np.stack(cat("K"))),
                        _dev(np.stack(cat("RT")))),
                vols=_volumes(c["batch"], c["D"], c["rate"]), batch=c["batch"], D=c["D"], rate=c["rate"],
                tw=_box(c["D"])[2])


def _build(s, **box):
    occ, cnt, tsdf, color, _, bbox, vs = H.integrate_depths(
        s["inputs"], s["vols"], batch_size=s["batch"], _tsdf_th_low=13.5, _tsdf_th_high=13.5, _level_volumes=2,
        _volume_res_rate=s["rate"], _trunc_weight=s["tw"], **box)
    tree = H.OcTreeOptions(levels=2, batch_size=s["batch"], rate=s["rate"], vol_dim=s["D"], device="cuda:0")
    tree.init_octree(occ, cnt, vs, bbox)
    return occ, cnt, tsdf, color, bbox, vs, tree


def _run_build(s):
    occ, cnt, tsdf, color, bbox, vs, tree = _build(s)
    return dict(occ0=occ[0], occ1=occ[1], cnt0=cnt[0], cnt1=cnt[1], tsdf=tsdf, color=color, bbox=bbox, vs=vs)


def _work_build(c):
    V, P = c["batch"] * c["D"] ** 3, c["batch"] * c["views"] * c["res"] ** 2
    return dict(bytes=12 * V + 16 * P, flops=15 * c["views"] * V)


# ---------------------------------------------------------------------------
# rays: ray_intersection -> sampling -> sort (-> density, colour, compositing)
# ---------------------------------------------------------------------------
def _prep_rays(c, seed):
    s = _prep_build(c, seed)
    bbox, vs, _ = _box(c["D"], c["batch"])
    s["bb"], s["vs"] = _dev(bbox), _dev(vs)
    _, _, tsdf, _, _, _, tree = _build(s, vol_bbox=s["bb"], voxel_size=s["vs"])
    rng, g = np.random.default_rng(seed + 1), _gen(seed + 1)
    rays = [_camera_rays(rng, c["rays"]) for _ in range(c["batch"])]
    s.update(tree=tree, tsdf=tsdf, o=torch.cat([o for o, _ in rays]), d=torch.cat([d for _, d in rays]), S=c["S"],
             noise=torch.full((c["batch"], c["rays"], c["S"]), 0.5, device=DEV), trunc=float(vs[0, 0]) * s["tw"],
             grid=torch.rand((c["batch"],) + (c["D"],) * 3 + (3,), generator=g, device=DEV) if c["shade"] else None)
    return s


def _run_rays(s):
    t, o, d = s["tree"], s["o"], s["d"]
    idx, t0, t1, vl = t.ray_intersection(o, d, 0)
    si, sz = t.ray_voxels_points_sampling_coarse(idx, t0, t1, s["noise"], vl, 0, s["S"])
    srt, pos = t.sort_sampling(sz)
    out = dict(idx=idx, t0=t0, t1=t1, vl=vl, si=si, sz=sz, srt=srt, pos=pos)
    if s["grid"] is not None:
        sigma = fields.tsdf_density(s["tsdf"], o, d, sz, s["bb"], s["vs"], s["trunc"], 0.005)
        rgb = fields.grid_gather(s["grid"], o, d, sz, s["bb"], s["vs"])
        out.update(zip(("rgb", "depth", "ws", "alpha"),
                       H.volume_render(sz, pos, sigma[..., None], rgb, 1e-4, False)))
    return out


def _work_rays(c):
    R = c["batch"] * c["rays"]
    more = c["batch"] * c["D"] ** 3 * 0.05 * 16 + R * (c["S"] * 16 * 2 + 24) if c["shade"] else 0
    return dict(bytes=R * (24 + 1024 * 12 + 4 + c["S"] * (4 + 8 + 8)) + more, flops=R * c["S"] * 60)


# ---------------------------------------------------------------------------
# diff: BatchPipeline.intersect / forward / backward on random rays
# ---------------------------------------------------------------------------
def _prep_diff(c, seed):
    rng, g = np.random.default_rng(seed), _gen(seed)
    fr = _frame(rng, c["views"], [c["res"]], g)
    fr.pop("rgb")
    n, S = c["rays"], c["S"]
    bp = BatchPipeline([[tuple(d.shape) for d in fr["depth"]]], [(0, n, S)], D=c["D"], rate=c["rate"], C=c["C"],
                       W_hits=c["W"], train_tsdf=True, device=DEV, deterministic=False)
    bbox, vs, tw = _box(c["D"])
    bp.load_views([fr], bbox, vs.reshape(-1), tw)
    bp.load_rays([_aimed_rays(g, n)])
    bp.feat.normal_(0.0, 0.1, generator=g)
    bp.set_fields(head=torch.randn((3, c["C"]), generator=g, device=DEV) * 0.5)
    bp.render_args(float(vs[0, 0]) * tw, sdf_s=0.005, t_thres=1e-4, rand_seed=17)
    bp.build()
    return dict(bp=bp, g_rgb=torch.randn((n, 3), generator=g, device=DEV),
                g_depth=torch.randn(n, generator=g, device=DEV), g_ws=torch.zeros(n, device=DEV),
                g_alpha=torch.randn(n, generator=g, device=DEV), gs=torch.empty((n, S), device=DEV),
                gr=torch.empty((n, S, 3), device=DEV))


def _run_diff(s):
    bp = s["bp"]
    bp.intersect()
    rgb, depth, ws, alpha = bp.forward()
    bp.backward(s["g_rgb"], s["g_depth"], s["g_ws"], s["g_alpha"], grad_sigma=s["gs"], grad_rgb=s["gr"])
    return dict(rgb=rgb, depth=depth, ws=ws, alpha=alpha, grad_sigma=s["gs"], grad_rgb=s["gr"],
                grad_feat=bp.grad_feat, grad_tsdf=bp.grad_tsdf)


def _work_diff(c):
    R, S, V = c["rays"], c["S"], c["D"] ** 3
    return dict(bytes=R * (24 + 24 + 24 + 16 * S) + V * 4 * (c["C"] + 1) * 1.05,
                flops=0.25 * R * S * (8 * 2 * (c["C"] + 1) * 3 + 200))


# ---------------------------------------------------------------------------
# fields: tsdf_density and grid_gather into volume_render_exact, and back
# ---------------------------------------------------------------------------
def _prep_fields(c, seed):
    rng, g = np.random.default_rng(seed), _gen(seed)
    D, C, n, S = c["D"], c["C"], c["rays"], c["S"]
    bbox, vs, tw = _box(D)
    # a sphere's truncated distance, roughened
    ax = torch.linspace(-1.0, 1.0, D, device=DEV)
    r = 0.6 + 0.1 * rng.random()
    dist = (ax[:, None, None] ** 2 + ax[None, :, None] ** 2 + ax[None, None, :] ** 2).sqrt() - r
    tsdf = (dist / 0.03 + 0.05 * torch.randn(dist.shape, generator=g, device=DEV)).clamp(-1.0, 1.0)[None]
    o, d = _aimed_rays(g, n, 0.3)
    # stratified samples from 8 cm in front of the sphere to 12 cm inside
    b = (o * d).sum(-1)
    q = (b * b - (o * o).sum(-1) + r * r).clamp(min=0.0).sqrt()
    k = torch.arange(S, device=DEV) + torch.rand((n, S), generator=g, device=DEV)
    z = (-b - q)[:, None] - 0.08 + k * (0.2 / S)
    return dict(tsdf=tsdf.requires_grad_(), feat=(torch.randn((1, D, D, D, C), generator=g, device=DEV) *
                                                  0.1).requires_grad_(), o=o[None], d=d[None], z=z[None].contiguous(),
                pos=torch.arange(S, dtype=torch.int32, device=DEV).expand(1, n, S).contiguous(), bb=_dev(bbox),
                vs=_dev(vs), trunc=float(vs[0, 0]) * tw,
                up=[torch.randn((1, n, k), generator=g, device=DEV) for k in (C, 1, 1, 1)])


def _run_fields(s):
    sigma = fields.tsdf_density(s["tsdf"], s["o"], s["d"], s["z"], s["bb"], s["vs"], s["trunc"], 0.005)
    feat = fields.grid_gather(s["feat"], s["o"], s["d"], s["z"], s["bb"], s["vs"])
    outs = H.volume_render_exact(s["z"], s["pos"], sigma[..., None], feat, 1e-4, False)
    gt, gf = torch.autograd.grad(outs, (s["tsdf"], s["feat"]), s["up"])
    return dict(feats=outs[0], depth=outs[1], ws=outs[2], alpha=outs[3], grad_tsdf=gt, grad_feat=gf)


def _work_fields(c):
    n, S, V, C = c["rays"], c["S"], c["D"] ** 3, c["C"]
    return dict(bytes=n * (24 + 8 * S + 8 * (C + 3)) + V * 4 * (C + 1) * 1.1, flops=n * S * (8 * 2 * (C + 1) * 2 + 12 * C + 150))


def _taps64(bb, vs, D, pt):
    u = (pt - bb[0, :, 0].double()) / vs.double().reshape(-1)[0]
    i0 = torch.floor(u)
    f, i0 = u - i0, i0.long()
    idx, w = [], []
    for k in range(8):
        b = torch.tensor([(k >> 2) & 1, (k >> 1) & 1, k & 1], device=pt.device)
        i = i0 + b
        ok = ((i >= 0) & (i < D)).all(-1)
        i = i.clamp(0, D - 1)
        idx.append((i[..., 0] * D + i[..., 1]) * D + i[..., 2])
        w.append(torch.where(b.bool(), f, 1.0 - f).prod(-1) * ok)
    return torch.stack(idx, -1), torch.stack(w, -1)


def _composite64(z, sg, t_thres, occ):
    """Compositing in 64 bits over sorted rows z, sg [n, S]: weights, alphas, transmittance before
    each sample, the step to the next depth and which samples count."""
    S = z.shape[1]
    valid = z >= 0
    delta = torch.cat([z[:, 1:] - z[:, :-1], torch.full_like(z[:, :1], 1e10)], 1)
    al = torch.where(valid, sg if occ else 1.0 - torch.exp(-sg * delta), 0.0)
    after = torch.cumprod(1.0 - al, 1)
    before = torch.cat([torch.ones_like(after[:, :1]), after[:, :-1]], 1)
    below = valid & (after < t_thres)
    stop = torch.where(below.any(1), below.int().argmax(1), S)
    use = valid & (torch.arange(S, device=z.device)[None] <= stop[:, None]) & (z[:, -1:] >= 0)
    return torch.where(use, al * before, 0.0), al, before, delta, use


def _exact_fields(c, seed):
    s = _prep_fields(c, seed)
    D, C, n = c["D"], c["C"], c["rays"]
    tsdf, feat = s["tsdf"].detach().double().reshape(-1), s["feat"].detach().double().reshape(-1, C)
    k = s["trunc"] / 0.005
    outs = [torch.empty((1, n, m), dtype=torch.float64, device=DEV) for m in (C, 1, 1, 1)]
    gt, gf = torch.zeros_like(tsdf), torch.zeros_like(feat)
    step = max(1, (1 << 20) // c["S"])
    for a in range(0, n, step):
        b = min(n, a + step)
        z = s["z"][0, a:b].double()
        pt = s["o"][0, a:b, None].double() + s["d"][0, a:b, None].double() * z[..., None]
        idx, w8 = _taps64(s["bb"], s["vs"], D, pt)
        sig01 = torch.sigmoid(-(tsdf[idx] * w8).sum(-1) * k)
        fe = sum(feat[idx[..., q]] * w8[..., q, None] for q in range(8))
        w, al, before, delta, use = _composite64(z, sig01 / 0.005, 1e-4, False)
        v = torch.cat([fe, z[..., None], torch.ones_like(z)[..., None], al[..., None]], -1)
        tot = (w[..., None] * v).sum(1)
        for o_, t_ in zip(outs, tot.split([C, 1, 1, 1], 1)):
            o_[0, a:b] = t_
        up = torch.cat([x[0, a:b] for x in s["up"]], -1).double()[:, None]
        rest = tot[:, None] - torch.cumsum(w[..., None] * v, 1)
        Ta = (before * (1.0 - al))[..., None]
        vt = torch.cat([v[..., :-1], 2.0 * al[..., None]], -1)
        gs = torch.where(use, delta * (up * (Ta * vt - rest)).sum(-1), 0.0)
        gd = gs / 0.005 * (-k * sig01 * (1.0 - sig01))
        gfe = w[..., None] * up[..., :C]
        for q in range(8):
            gt.index_add_(0, idx[..., q].reshape(-1), (gd * w8[..., q]).reshape(-1))
            gf.index_add_(0, idx[..., q].reshape(-1), (gfe * w8[..., q, None]).reshape(-1, C))
    return dict(feats=outs[0], depth=outs[1], ws=outs[2], alpha=outs[3], grad_tsdf=gt.view(s["tsdf"].shape),
                grad_feat=gf.view(s["feat"].shape))


# ---------------------------------------------------------------------------
# composite: volume_render (with gradients) / volume_render_infer
# ---------------------------------------------------------------------------
def _prep_composite(c, seed):
    g = _gen(seed)
    n, S, C = c["rays"], c["S"], c["C"]
    z = torch.rand((1, n, S), generator=g, device=DEV) * 2.0 + 1.0
    z, pos = z.sort(-1)
    if not c["presorted"]:  # as sampling leaves it: sort positions into the unsorted samples
        perm = torch.rand((1, n, S), generator=g, device=DEV).argsort(-1)
        z = z.gather(-1, perm)
        z[:, : n // 16] = -1.0  # rays without samples
        pos = z.sort(-1).indices
    else:
        pos = torch.arange(S, device=DEV).expand(1, n, S)
    sg = torch.rand((1, n, S, 1), generator=g, device=DEV)
    sg = sg * 0.3 if c["occ"] else 4.0 + sg * 16.0  # densities: every ray ends before its last sample
    train = not c["presorted"] and C <= 16
    return dict(z=z.contiguous(), pos=pos.to(torch.int32).contiguous(), occ=c["occ"], train=train,
                infer=c["presorted"] and c["occ"], sg=sg.requires_grad_(train),
                ft=torch.randn((1, n, S, C), generator=g, device=DEV).requires_grad_(train),
                up=[torch.randn((1, n, k), generator=g, device=DEV) for k in (C, 1, 1, 1)])


def _run_composite(s):
    if s["infer"]:
        return dict(zip(("rgb", "depth", "ws", "alpha"), H.volume_render_infer(s["z"], s["sg"], s["ft"])))
    if not s["train"]:
        return dict(zip(("rgb", "depth", "ws", "alpha"),
                        H.volume_render(s["z"], s["pos"], s["sg"], s["ft"], 1e-4, s["occ"])))
    outs = H.volume_render_exact(s["z"], s["pos"], s["sg"], s["ft"], 1e-4, s["occ"])
    gs, gf = torch.autograd.grad(outs, (s["sg"], s["ft"]), s["up"])
    return dict(rgb=outs[0], depth=outs[1], ws=outs[2], alpha=outs[3], grad_sigma=gs, grad_feats=gf)


def _work_composite(c):
    n, S, C = c["rays"], c["S"], c["C"]
    train = not c["presorted"] and C <= 16
    return dict(bytes=n * S * 4 * (C + 2 + (not c["presorted"])) * (1.8 if train else 1) + n * 4 * (C + 3),
                flops=n * S * (2 * C + 20) * (3 if train else 1))


def _exact_composite(c, seed):
    s = _prep_composite(c, seed)
    pos = s["pos"][0].long()
    z, sg = s["z"][0].double().gather(1, pos), s["sg"].detach()[0, ..., 0].double().gather(1, pos)
    ft = s["ft"].detach()[0].double().gather(1, pos[..., None].expand(s["ft"].shape[1:]))
    w, al, before, delta, use = _composite64(z, sg, 1e-4, s["occ"])
    v = torch.cat([ft, z[..., None], torch.ones_like(z)[..., None], al[..., None]], -1)
    tot, C = (w[..., None] * v).sum(1), c["C"]
    out = dict(rgb=tot[None, :, :C], depth=tot[None, :, C:C + 1], ws=tot[None, :, C + 1:C + 2],
               alpha=tot[None, :, C + 2:])
    if s["train"]:
        up = torch.cat([x[0] for x in s["up"]], -1).double()[:, None]
        rest = tot[:, None] - torch.cumsum(w[..., None] * v, 1)
        vt = torch.cat([v[..., :-1], 2.0 * al[..., None]], -1)
        if s["occ"]:
            gs = (up * (before[..., None] * vt - rest / (1.0 - al)[..., None])).sum(-1)
        else:
            gs = delta * (up * ((before * (1.0 - al))[..., None] * vt - rest)).sum(-1)
        gs = torch.where(use, gs, 0.0)
        gf = w[..., None] * up[..., :C]
        out["grad_sigma"] = torch.zeros_like(gs).scatter(1, pos, gs)[None, ..., None]
        out["grad_feats"] = torch.zeros_like(gf).scatter(1, pos[..., None].expand_as(gf), gf)[None]
    return out


# ---------------------------------------------------------------------------
# octree: multi-level tree
# ---------------------------------------------------------------------------
def _prep_octree(c, seed):
    rng, g = np.random.default_rng(seed), _gen(seed)
    fr = _frame(rng, c["views"], [c["res"]], g)
    bbox, vs, tw = _box(c["D"])
    vols, cnts = _volumes(1, c["D"], 2, c["levels"])
    VE.integrate_in_box(vols[0], cnts[0], _dev(np.stack(fr["K"]))[None], _dev(np.stack(fr["RT"]))[None],
                        torch.stack(fr["color"])[None], torch.stack(fr["depth"])[None], _dev(bbox), _dev(vs), 1.0, tw,
                        13.5, 13.5, 0)
    VE.build_multi_res_volumes(vols, cnts, c["levels"], 2, 0)
    o, d = _camera_rays(rng, c["rays"])
    return dict(pristine=[v.clone() for v in vols], vols=vols, cnts=cnts, bb=_dev(bbox), vs=_dev(vs), o=o, d=d,
                noise=torch.rand((1, c["rays"], c["S"]), generator=g, device=DEV), levels=c["levels"], D=c["D"],
                S=c["S"], Wf=c["Wf"])


def _run_octree(s):
    for v, p in zip(s["vols"], s["pristine"]):  # the build writes node ids over the occupancy
        v.copy_(p)
    t = H.OcTreeOptions(levels=s["levels"], batch_size=1, rate=2, vol_dim=s["D"], n_max_hits=s["Wf"],
                        device="cuda:0")
    t.init_octree(s["vols"], s["cnts"], s["vs"], s["bb"])
    idx, t0, t1, vl, ic, c0, c1 = t.ray_intersection(s["o"], s["d"], 1, only_voxel_traversal=False)
    si, sz = t.ray_voxels_sampling_points(idx, t0, t1, vl, s["noise"], 1, s["S"])
    return dict(idx=idx, t0=t0, t1=t1, vl=vl, idx_c=ic, t0_c=c0, t1_c=c1, si=si, sz=sz)


def _work_octree(c):
    wc = c["D"] * 3 // 2 ** (c["levels"] - 2)
    return dict(bytes=c["rays"] * (24 + 12 * (wc + c["Wf"]) + c["S"] * 12) + 3 * 4 * c["D"] ** 3 * 8 / 7,
                flops=c["rays"] * c["S"] * 60)


# ---------------------------------------------------------------------------
# nerf: FastNerf's occupancy network
# ---------------------------------------------------------------------------
_NERF_LAYERS = ((0, 18, 64), (1216, 64, 64), (5376, 64, 64), (9536, 64, 64))


def _prep_nerf(c, seed):
    g, V, n = _gen(seed), c["views"], c["points"]
    return dict(params=(torch.randn(22521, generator=g, device=DEV) * 0.2).half(),
                z=torch.rand((1, V, n, 1), generator=g, device=DEV) * 2.5 + 0.5,
                t=torch.rand((1, V, n, 1), generator=g, device=DEV) * 2.0 - 1.0,
                geo=torch.randn((1, V, n, 16), generator=g, device=DEV) * 0.5, n=n, V=V, want=c["geo"])


def _run_nerf(s):
    r = nerf.infer_density(s["z"], s["t"], s["geo"], s["params"], 1, s["n"], s["V"], 0, s["want"])
    return dict(density=r[0], geo=r[1]) if s["want"] else dict(density=r)


def _work_nerf(c):
    n, V = c["points"], c["views"]
    return dict(bytes=n * (V * (72 + (32 if c["geo"] else 0)) + 4) + 45042,
                flops=2 * n * (V * (18 * 64 + 3 * 4096 + 18 * 16 + 128) + 2 * 4096 + 64))


def _exact_nerf(c, seed):
    s = _prep_nerf(c, seed)
    p = s["params"].double()

    def lin(x, off, i, o):
        return x @ p[off:off + i * o].view(o, i).T + p[off + i * o:off + i * o + o]

    dens = torch.empty((1, 1, s["n"]), dtype=torch.float64, device=DEV)
    geo = torch.empty((1, s["V"], s["n"], 8), dtype=torch.float64, device=DEV) if s["want"] else None
    for a in range(0, s["n"], 1 << 19):
        e = min(s["n"], a + (1 << 19))
        # the network's inputs are float16
        x = torch.cat([s["z"][0, :, a:e], s["t"][0, :, a:e], s["geo"][0, :, a:e]], -1).half().double()
        h = x
        for off, i, o in _NERF_LAYERS:
            h = torch.relu(lin(h, off, i, o))
        h = h.mean(0)
        h = torch.relu(lin(h, 13696, 64, 64))
        h = torch.relu(lin(h, 13696 + 4160, 64, 64))
        dens[0, 0, a:e] = torch.sigmoid(lin(h, 13696 + 8320, 64, 1))[:, 0]
        if geo is not None:
            geo[0, :, a:e] = torch.relu(lin(torch.relu(lin(x, 22081, 18, 16)), 22081 + 304, 16, 8))
    return dict(density=dens, geo=geo) if s["want"] else dict(density=dens)


# ---------------------------------------------------------------------------
# project: projection into the views and the 2D feature gather
# ---------------------------------------------------------------------------
def _smooth(shape, g, res, lo, hi):
    """A smooth random image in [lo, hi]: 16 x 16 values, interpolated."""
    x = torch.rand(shape + (16, 16), generator=g, device=DEV)
    return lo + (hi - lo) * F.interpolate(x, size=(res, res), mode="bilinear", align_corners=True)


def _prep_project(c, seed):
    rng, g = np.random.default_rng(seed), _gen(seed)
    V, res, S = c["views"], c["res"], c["S"]
    cams = syn.ring_cameras(V, phase=rng.uniform(0, 2 * math.pi))
    o, d = _camera_rays(rng, c["rays"])
    z = (torch.rand((c["rays"], S), generator=g, device=DEV) * 2.0 + 1.5).sort(-1).values
    pts = (o[0, :, None] + d[0, :, None] * z[..., None]).reshape(1, -1, 3).permute(0, 2, 1)
    maps = [torch.randn((V, c["Cg"], res, res), generator=g, device=DEV), _smooth((V, 1), g, res, 1.5, 3.5),
            torch.randn((V, c["Cr"], res, res), generator=g, device=DEV),
            torch.rand((V, 3, res, res), generator=g, device=DEV)]
    if c["nhwc"]:
        maps = [m.contiguous(memory_format=torch.channels_last) for m in maps]
    return dict(pts=pts, K=_dev(syn.intrinsics(res)).expand(V, 3, 3).contiguous(),
                R=_dev(np.stack([R for R, _ in cams])), T=_dev(np.stack([T for _, T in cams])).view(V, 3, 1),
                pd=z.reshape(1, 1, -1), V=V, res=res, maps=maps)


def _run_project(s):
    z, geo, feats, psdf, rgbs = views.project_sample_features(s["pts"], s["K"], s["R"], s["T"], s["pd"], s["V"],
                                                              *s["maps"], res=s["res"])
    return dict(z=z, geo=geo, feats=feats, psdf=psdf, rgbs=rgbs)


def _work_project(c):
    n, V, ch = c["rays"] * c["S"], c["views"], c["Cg"] + c["Cr"] + 4
    return dict(bytes=4 * (n * 4 + n * V * (ch + 1) + V * ch * c["res"] ** 2), flops=n * V * (ch * 8 + 60))


def _exact_project(c, seed):
    s = _prep_project(c, seed)
    V, n, half = s["V"], s["pts"].shape[2], float(s["res"] // 2)
    outs = [torch.empty((V, n, m.shape[1]), dtype=torch.float64, device=DEV) for m in s["maps"]]
    zs = torch.empty((V, 1, n), dtype=torch.float64, device=DEV)
    step = 1 << 20
    for v in range(V):
        maps = [m[v:v + 1].double().contiguous() for m in s["maps"]]
        K, R, T = (s[k][v].double() for k in "KRT")
        for a in range(0, n, step):
            e = min(n, a + step)
            cam = R @ s["pts"][0, :, a:e].double() + T
            dz = torch.where(cam[2] < 0.01, 1.0, cam[2])
            xy = ((K @ (cam / dz))[:2] - half) / half
            pd = s["pd"][0, 0, a:e]
            off = (pd < 0.1) | (pd > 4.0)
            xy = torch.where((cam[2] < 0.01) | off, -2.0, xy)
            zs[v, 0, a:e] = torch.where(off, -2.0, cam[2])
            for m, o_ in zip(maps, outs):
                o_[v, a:e] = F.grid_sample(m, xy.T.reshape(1, -1, 1, 2), mode="bilinear", padding_mode="zeros",
                                           align_corners=True)[0, :, :, 0].T
    psdf = (zs[:, 0, :, None] - outs[1]).clamp(-0.01, 0.01) / 0.01
    return dict(z=zs, geo=outs[0], feats=outs[2], psdf=psdf, rgbs=outs[3])


# ---------------------------------------------------------------------------
_PREP = dict(train=_prep_train, frame=_prep_frame, build=_prep_build, rays=_prep_rays, diff=_prep_diff,
             fields=_prep_fields, composite=_prep_composite, octree=_prep_octree, nerf=_prep_nerf,
             project=_prep_project)
_RUN = dict(train=_run_train, frame=_run_frame, build=_run_build, rays=_run_rays, diff=_run_diff, fields=_run_fields,
            composite=_run_composite, octree=_run_octree, nerf=_run_nerf, project=_run_project)
_WORK = dict(train=_work_train, frame=_work_frame, build=_work_build, rays=_work_rays, diff=_work_diff,
             fields=_work_fields, composite=_work_composite, octree=_work_octree, nerf=_work_nerf,
             project=_work_project)
# The chains from depth images to rendered rays choose pixels, cells and
# sample positions in 32 bits, step by step: they have no 64-bit value.
_EXACT = dict(fields=_exact_fields, composite=_exact_composite, nerf=_exact_nerf, project=_exact_project)


def prepare(case, seed):
    with torch.no_grad():
        s = _PREP[case["kind"]](case, seed)
    s["kind"] = case["kind"]
    return s


def run(state):
    return _RUN[state["kind"]](state)


def work(case):
    return _WORK[case["kind"]](case)


def exact(case, seed):
    f = _EXACT.get(case["kind"])
    if f is None:
        return None
    with torch.no_grad():
        return f(case, seed)
