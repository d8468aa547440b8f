"""GPU checks of the dense-grid gathers, their adjoint and compositing where
rows change shape: channel counts over the vector widths, addresses off 16
bytes, sample counts off the warp, cells at and beyond the grid's faces."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -24


def _off(a, pad):
    """a on the device, `pad` floats behind a 16-byte boundary."""
    buf = torch.zeros(a.size + 4, device="cuda")
    v = buf[pad:pad + a.size].reshape(a.shape)
    v.copy_(torch.from_numpy(a))
    return v


def _grid_case(C, B, Nr, S, rng):
    """Rays through a grid of D^3 voxels; positions, voxel size and bounds are
    multiples of 2^-10 below 2^4, so cells and fractions carry no rounding."""
    D, vs = 9, 0.25
    q = lambda a, s: (np.round(a * s) / s).astype(np.float32)
    bb = np.zeros((B, 3, 2), np.float32)
    bb[:, :, 0] = q(rng.uniform(-1, 0, (B, 3)), 64)
    bb[:, :, 1] = bb[:, :, 0] + (D - 1) * vs
    ori = q(rng.uniform(-1, 1, (B, Nr, 3)), 32)
    d = q(rng.uniform(-1, 1, (B, Nr, 3)), 8)
    z = q(np.sort(rng.uniform(0, 3, (B, Nr, S)), -1), 16)
    z[rng.random(z.shape) < 0.2] = -1.0
    z[:, 0] = -1.0
    grid = rng.normal(size=(B, D, D, D, C)).astype(np.float32)
    pt = ori[:, :, None].astype(np.float64) + d[:, :, None] * z[..., None].astype(np.float64)
    u = (pt - bb[:, None, None, :, 0]) / vs
    i0 = np.floor(u).astype(np.int64)
    f = u - i0
    corners = []
    for c in range(8):
        b = np.array([(c >> 2) & 1, (c >> 1) & 1, c & 1])
        i = i0 + b
        w = np.prod(np.where(b, f, 1 - f), -1) * ((i >= 0) & (i < D)).all(-1) * (z >= 0)
        i = np.clip(i, 0, D - 1)
        corners.append((w, ((np.arange(B)[:, None, None] * D + i[..., 0]) * D + i[..., 1]) * D + i[..., 2]))
    return D, np.full(B, vs, np.float32), bb, ori, d, z, grid, corners


@pytest.mark.parametrize("C,pad", [(1, 0), (1, 3), (3, 0), (4, 0), (4, 1), (8, 0), (8, 2), (16, 0), (16, 1)])
@pytest.mark.parametrize("B,Nr,S", [(1, 1, 1), (1, 7, 33), (2, 33, 5), (2, 130, 32)])
def test_gather_and_scatter_rows(C, pad, B, Nr, S):
    from sailor_gb300 import _native as N
    rng = np.random.default_rng(C * 100 + S)
    D, vs, bb, ori, d, z, grid, corners = _grid_case(C, B, Nr, S, rng)
    gout = rng.normal(size=(B, Nr, S, C)).astype(np.float32)
    g, gr, out, gg = _off(grid, pad), _off(gout, pad), _off(gout * 0 + 7, pad), _off(grid * 0 + 1, pad)
    to, td, tz, tb, tv = (torch.from_numpy(a).cuda() for a in (ori, d, z, bb, vs))
    geo = (N.ptr(to), N.ptr(td), N.ptr(tz), B, Nr, S)
    N.check(N.lib.sg_grid_gather(*geo, N.ptr(g), D, C, N.ptr(tb), N.ptr(tv), 0, 1.0, 1.0, N.ptr(out), N.stream()), "g")
    N.check(N.lib.sg_grid_scatter(*geo, N.ptr(gr), None, D, C, N.ptr(tb), N.ptr(tv), 0, 1.0, 1.0, N.ptr(gg),
                                  N.stream()), "s")
    flat = grid.reshape(-1, C).astype(np.float64)
    ref = sum(w[..., None] * flat[v] for w, v in corners)
    mag = sum(w[..., None] * np.abs(flat[v]) for w, v in corners)
    # three roundings a weight, one a term
    assert (np.abs(out.cpu().numpy() - ref) <= 11 * EPS * mag).all()
    rs, ms, cnt = np.ones_like(flat), np.ones_like(flat), np.zeros((len(flat), 1))
    for w, v in corners:
        np.add.at(rs, v.ravel(), (w[..., None] * gout).reshape(-1, C))
        np.add.at(ms, v.ravel(), (w[..., None] * np.abs(gout)).reshape(-1, C))
        np.add.at(cnt, v.ravel(), (w.reshape(-1, 1) != 0).astype(float))
    assert (np.abs(gg.cpu().numpy().reshape(-1, C) - rs) <= (cnt + 4) * EPS * ms).all()


def _composite_ref(z, order, sg, feats, t_thres, mode, g, exact):
    """One ray in 64 bits; the samples that count are those of the walk in 32
    bits.  Returns outputs, gradients and whether the walk came within 1e-4 of
    the threshold (where a last bit of alpha could decide)."""
    S, C = feats.shape
    out = [np.zeros(C), 0.0, 0.0, 0.0]
    gf, gs = np.zeros((S, C)), np.zeros(S)
    if z[order[-1]] < 0:
        return out, gf, gs, False
    zs = z[order]
    steps, T, near, stop = [], np.float32(1), False, -1
    for i, s in enumerate(order):
        if zs[i] < 0:
            continue
        if mode == 0:
            if i == S - 1:
                dl = 1e10
            else:
                m = next((q for q in range(i + 1, S) if zs[q] > 0), S - 1)
                dl = float(np.float32(zs[m] - zs[i]))
            al = np.float32(1 - np.float32(np.exp(-np.float64(np.float32(sg[s] * np.float32(dl))))))
        else:
            dl, al = 0.0, sg[s]
        steps.append((s, float(zs[i]), dl, float(al), float(T)))
        T = np.float32(T * np.float32(1 - al))
        near = near or abs(T - t_thres) <= 1e-4 * t_thres
        if T < t_thres:
            stop = s
            break
    f64 = feats.astype(np.float64)
    val = [np.concatenate([[1.0, zz, al], f64[s]]) for s, zz, _, al, _ in steps]  # ws, depth, alpha, features
    w = [al * tb for _, _, _, al, tb in steps]
    tot = sum(a * v for a, v in zip(w, val))
    out = [tot[3:], tot[1], tot[0], tot[2]]
    gv = np.concatenate([[g[2], g[1], g[3]], g[0]]).astype(np.float64)
    pre = np.zeros_like(tot)
    for (s, zz, dl, al, tb), wi, v in zip(steps, w, val):
        pre = pre + wi * v
        if not exact and s == stop:
            continue
        suf, Ta = tot - pre, tb * (1 - al)
        dv = v.copy()
        dv[2] = 2 * al
        if mode == 0:
            gs[s] = dl * (gv @ (Ta * dv - suf) + (0 if exact else 4 * gv[0] * (1 - tot[0])))
        elif exact:
            gs[s] = gv @ (tb * dv - suf / (1 - al))
        else:
            gs[s] = gv @ (Ta * dv - suf) / (1 - al)
        gf[s] = wi * g[0]
    return out, gf, gs, near


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("C,pad", [(1, 0), (2, 0), (3, 0), (4, 0), (4, 1), (5, 0), (6, 0), (8, 2), (12, 0), (13, 0),
                                   (16, 0), (16, 1), (24, 0), (30, 0), (31, 0), (32, 1)])
def test_composite_rows(C, pad, mode):
    from sailor_gb300 import _native as N
    t_thres = 0.02
    for S in (1, 5, 32, 33, 96, 100, 128):
        rng = np.random.default_rng(1000 * C + S + mode)
        R = 19
        z = np.sort(rng.uniform(0.2, 2.0, (R, S)), -1).astype(np.float32)
        z[rng.random((R, S)) < 0.15] = -1.0
        z[::2, -1] = 2.5
        z[3, : S // 2] = -1.0  # nothing in front
        order = np.stack([rng.permutation(S) for _ in range(R)]).astype(np.int32)
        z = np.take_along_axis(z, np.argsort(order, -1), -1)  # position i holds sample order[i]
        # rays that end early, late and never
        top = np.array([0.9, 0.05, 0.3, 0.6])[np.arange(R) % 4][:, None]
        al = (rng.random((R, S)) * top).astype(np.float32)
        sg = al if mode else (al * 20).astype(np.float32)
        feats = rng.normal(size=(R, S, C)).astype(np.float32)
        g = [rng.normal(size=(R, C)), rng.normal(size=R), rng.normal(size=R), rng.normal(size=R)]
        g = [a.astype(np.float32) for a in g]
        ft = _off(feats, pad)
        tz, to, ts = (torch.from_numpy(a).cuda() for a in (z, order, sg))
        tg = [torch.from_numpy(a).cuda() for a in g]
        outs = [torch.full((R, C), 9.0, device="cuda")] + [torch.full((R,), 9.0, device="cuda") for _ in range(3)]
        N.check(N.lib.sg_composite_fwd(N.ptr(tz), N.ptr(to), N.ptr(ts), N.ptr(ft), R, S, C, t_thres, mode,
                                       *[N.ptr(o) for o in outs], N.stream()), "fwd")
        exacts = (0, 1) if C <= 16 else ()
        grads = {}
        for exact in exacts:
            gf, gs = _off(feats * 0 + 9, pad), torch.full((R, S), 9.0, device="cuda")
            N.check(N.lib.sg_composite_bwd(*[N.ptr(a) for a in tg], *[N.ptr(o) for o in outs], N.ptr(tz),
                                           N.ptr(to), N.ptr(ts), N.ptr(ft), R, S, C, t_thres, mode, exact,
                                           N.ptr(gf), N.ptr(gs), N.stream()), "bwd")
            torch.cuda.synchronize()
            grads[exact] = (gf.cpu().numpy(), gs.cpu().numpy())
        got = [o.cpu().numpy() for o in outs]
        # a weight's error: the roundings of its transmittance, and in density
        # mode those of each factor 1 - alpha (expf within 2 units, one subtraction)
        wtol = (S + 2) * EPS * (1 if mode else 6)
        far = 0
        for r in range(R):
            for exact in exacts or (1,):
                ref, rgf, rgs, near = _composite_ref(z[r], order[r], sg[r], feats[r], t_thres, mode,
                                                     [a[r] for a in g], exact)
                if near:
                    continue
                far += 1
                mags = [np.abs(feats[r]).max(), 2.5, 1.0, 1.0]
                for a, b, m in zip(got, ref, mags):
                    assert np.abs(a[r] - b).max() <= S * m * (wtol + S * EPS), (S, r)
                if not exacts:
                    continue
                gf, gs = grads[exact]
                assert np.abs(gf[r] - rgf).max() <= wtol * np.abs(g[0][r]).max() + EPS, (S, r, exact)
                # a bracket g . (T v - suffix): S weighted terms of at most M each,
                # divided by 1 - alpha > 0.1 or times the step
                M = abs(g[2][r]) * 5 + abs(g[1][r]) * 2.5 + 2 * abs(g[3][r]) + np.abs(g[0][r]).sum() * mags[0]
                tol = S * M * (wtol + (S + C + 8) * EPS)
                tol = tol * (10 if mode else 2.5) * np.ones(S)
                if mode == 0:
                    tol[order[r, -1]] *= 1e10 / 2.5  # behind the last position the step is 1e10
                assert (np.abs(gs[r] - rgs) <= tol).all(), (S, r, exact)
        assert far > R // 2
