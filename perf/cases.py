"""What this library's users have it do, as timed cases over the device entry points.

Each case is one call of an operator a CT reconstruction is made of, on device-resident
data: forward projection (FP) and backprojection (BP) in the three geometries, the
general3D ray projectors, one OSC iteration, the TV descent and the FDK pre-filter.
Volumes are random-ellipsoid phantoms, sinograms the ellipsoids' analytic line
integrals, counts are Poisson; everything is drawn from the seed alone.
"""
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "mex-cuda-ct_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from mexct import ops  # noqa: E402

SAD = 1000.0
PAR, FAN, CONE = 0, 1, 2


def listed():
    return [
        # A full-size cone-beam scan, projected and backprojected: the two halves of
        # every iterative update and the whole cost of simulating / FDK-reconstructing it.
        {"name": "fp_cone_512x720", "op": "fp", "geom": CONE, "W": 512, "H": 512, "views": 720,
         "half": False},
        {"name": "bp_cone_512x720", "op": "bp", "geom": CONE, "W": 512, "H": 512, "views": 720,
         "half": False},
        # Parallel-beam (synchrotron) projection and stacked-fan backprojection of a
        # medium scan: the geometries whose rays stay in one slice.
        {"name": "fp_par_384x512", "op": "fp", "geom": PAR, "W": 384, "H": 384, "views": 512,
         "half": False},
        {"name": "bp_fan_384x512", "op": "bp", "geom": FAN, "W": 384, "H": 384, "views": 512,
         "half": False},
        # The smallest problems (a preview volume, one of many in a batch): launches
        # and latency.
        {"name": "fp_cone_64x90", "op": "fp", "geom": CONE, "W": 64, "H": 64, "views": 90,
         "half": False},
        {"name": "bp_cone_64x90", "op": "bp", "geom": CONE, "W": 64, "H": 64, "views": 90,
         "half": False},
        # An odd-sized region of interest with volume and sinogram stored in FP16.
        {"name": "fp_fan_half_243x201x361", "op": "fp", "geom": FAN, "W": 243, "H": 201,
         "views": 361, "half": True},
        # One OSC iteration of a few-view reconstruction: 60 views in 10 subsets.
        {"name": "osc_cone_256x60", "op": "osc", "geom": CONE, "W": 256, "H": 256, "views": 60,
         "subsets": 10},
        # The TV descent after it (20 steps, the reference's count).
        {"name": "tv_256", "op": "tv", "W": 256, "H": 256, "steps": 20},
        # The Hamming pre-filter of an FDK reconstruction.
        {"name": "prefilter_cone_384x512", "op": "prefilter", "geom": CONE, "W": 384, "views": 512,
         "filter": "hamming"},
        # A helical scan through the general3D ray projectors, end points per view.
        {"name": "g3d_fp_256x360", "op": "g3d_fp", "W": 256, "H": 256, "det_w": 256, "det_h": 256,
         "views": 360},
        {"name": "g3d_bp_256x360", "op": "g3d_bp", "W": 256, "H": 256, "det_w": 256, "det_h": 256,
         "views": 360},
    ]


def draw(rng):
    op = rng.choice(["fp", "fp", "bp", "bp", "osc", "tv", "prefilter", "g3d_fp", "g3d_bp"])

    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    if op in ("fp", "bp"):
        geom = rng.choice([PAR, FAN, CONE])
        W = size(64, 512 if geom == CONE else 400)
        H = max(16, int(W * rng.uniform(0.5, 1.0)))
        return {"op": op, "geom": geom, "W": W, "H": H, "views": rng.randint(60, 720),
                "half": rng.random() < 0.25}
    if op == "osc":
        views, W = rng.randint(40, 180), size(64, 256)
        return {"op": op, "geom": rng.choice([PAR, FAN, CONE]), "W": W,
                "H": max(16, int(W * rng.uniform(0.5, 1.0))), "views": views,
                "subsets": rng.randint(4, 12)}
    if op == "tv":
        W = size(64, 400)
        return {"op": op, "W": W, "H": max(16, int(W * rng.uniform(0.5, 1.0))), "steps": 20}
    if op == "prefilter":
        return {"op": op, "geom": rng.choice([PAR, FAN, CONE]), "W": size(64, 512),
                "views": rng.randint(60, 720),
                "filter": rng.choice(["ramp", "shepp-logan", "cosine", "hamming", "hann"])}
    W = size(64, 256)
    return {"op": op, "W": W, "H": max(16, int(W * rng.uniform(0.5, 1.0))),
            "det_w": max(32, int(W * rng.uniform(0.8, 1.2))),
            "det_h": max(32, int(W * rng.uniform(0.5, 1.2))), "views": rng.randint(60, 360)}


# ---------------------------------------------------------------------------
# Inputs.
# ---------------------------------------------------------------------------
def _ellipsoids(rng, W, H, count=10):
    """(centre, semi-axes, rotation, value) in voxels, inside the field of view."""
    out = []
    for _ in range(count):
        scale = np.array([W, W, H], dtype=np.float64)
        c = rng.uniform(-0.3, 0.3, 3) * scale
        a = np.maximum(rng.uniform(0.05, 0.3, 3) * W, 4.0)
        q, _ = np.linalg.qr(rng.normal(size=(3, 3)))
        out.append((c, a, q, float(rng.uniform(0.2, 2.0)) / W))
    return out


def _form(a, q):
    return (q / (a * a)) @ q.T  # points p with p^T M p <= 1


def _axis(n, **kw):
    return torch.arange(n, **kw) - (n - 1) / 2


def _volume(ells, W, H):
    """The phantom (H, W, W) = (z, y, x), float32."""
    kw = dict(device="cuda", dtype=torch.float32)
    vol = torch.zeros((H, W, W), **kw)
    x, z = _axis(W, **kw), _axis(H, **kw)
    for c, a, q, v in ells:
        M = _form(a, q)
        X, Y, Z = (x - c[0])[None, None, :], (x - c[1])[None, :, None], (z - c[2])[:, None, None]
        r = M[0, 0] * X * X + M[1, 1] * Y * Y + 2 * M[0, 1] * X * Y
        r = r + M[2, 2] * Z * Z + Z * (2 * M[0, 2] * X + 2 * M[1, 2] * Y)
        vol += v * (r <= 1)
    return vol


def _chords(ells, s, d):
    """Line integrals of the ellipsoids along s + t d (tuples of broadcastable tensors)."""
    norm = torch.sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2])
    out = 0.0
    for c, a, q, v in ells:
        M = _form(a, q)
        p = [s[i] - c[i] for i in range(3)]
        Md = [sum(M[i, j] * d[j] for j in range(3)) for i in range(3)]
        Mp = [sum(M[i, j] * p[j] for j in range(3)) for i in range(3)]
        dd = sum(d[i] * Md[i] for i in range(3))
        dp = sum(p[i] * Md[i] for i in range(3))
        pp = sum(p[i] * Mp[i] for i in range(3))
        disc = torch.clamp(dp * dp - dd * (pp - 1), min=0)
        out = out + v * 2 * torch.sqrt(disc) / dd * norm
    return out


def _sinogram(ells, geom, W, H, angles):
    """Analytic projections (views, H, W) of the ellipsoids, float32."""
    kw = dict(device="cuda", dtype=torch.float64)
    u, v = _axis(W, **kw)[None, None, :], _axis(H, **kw)[None, :, None]
    out = torch.empty((len(angles), H, W), device="cuda")
    per = max(1, (1 << 22) // (W * H))  # views at once
    for i in range(0, len(angles), per):
        b = torch.from_numpy(angles[i:i + per]).to(**kw)[:, None, None]
        cb, sb = torch.cos(b), torch.sin(b)
        if geom == PAR:
            s = (SAD * cb - u * sb, SAD * sb + u * cb, v)
            d = (-2 * SAD * cb, -2 * SAD * sb, 0 * v)
        else:
            s = (SAD * cb, SAD * sb, v if geom == FAN else 0 * v)
            d = (-2 * SAD * cb - 2 * u * sb, -2 * SAD * sb + 2 * u * cb,
                 0 * v if geom == FAN else 2 * v)
        out[i:i + per] = _chords(ells, s, d)
    return out


def _angles(views, turns=1.0):
    return np.linspace(0.0, 2 * np.pi * turns, views).astype(np.float32)


def _helix(case, gen):
    """End points (views, 6, det_h, det_w) of a 2-turn helix of pitch one volume height."""
    W, H, views = case["det_w"], case["det_h"], case["views"]
    kw = dict(device="cuda", dtype=torch.float32)
    u, v = 2 * _axis(W, **kw)[None, :], 2 * _axis(H, **kw)[:, None]
    pts = torch.empty((views, 6, H, W), **kw)
    jitter = torch.rand((views, 2, H, W), generator=gen, **kw) * 0.1 - 0.05
    zsrc = (torch.arange(views, **kw) / max(views - 1, 1) - 0.5) * 2 * case["H"]
    pts[:, 0], pts[:, 1], pts[:, 3] = SAD, 0.0, -SAD
    pts[:, 2] = zsrc[:, None, None]
    pts[:, 4] = u + jitter[:, 0]
    pts[:, 5] = zsrc[:, None, None] + v + jitter[:, 1]
    return pts


def _subset_order(n, first):
    """A subset order that visits every subset once, far subsets first."""
    step = next(s for s in range(max(1, n // 2), n + 1) if math.gcd(s, n) == 1)
    return np.array([(first + step * i) % n for i in range(n)], dtype=np.int32)


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    op, W = case["op"], case["W"]
    H = case.get("H", W)
    s = dict(case)
    dt = torch.float16 if case.get("half") else torch.float32
    ells = _ellipsoids(rng, W, H)
    if op == "fp":
        s["angles"] = _angles(case["views"])
        s["vol"] = _volume(ells, W, H).to(dt)
        s["out"] = torch.empty((case["views"], H, W), device="cuda", dtype=dt)
    elif op == "bp":
        s["angles"] = _angles(case["views"])
        s["sino"] = _sinogram(ells, case["geom"], W, H, s["angles"]).to(dt)
        s["out"] = torch.empty((H, W, W), device="cuda", dtype=dt)
    elif op == "osc":
        s["angles"] = _angles(case["views"])
        line = _sinogram(ells, case["geom"], W, H, s["angles"])
        s["pre"] = torch.full_like(line, 1e5)
        s["post"] = torch.poisson(1e5 * torch.exp(-line), generator=gen)
        vol = _volume(ells, W, H)
        k = torch.nn.functional.avg_pool3d(vol[None, None], 5, 1, 2)[0, 0]
        s["mu0"] = (0.8 * k + 1e-4).contiguous()  # a partly converged image
        s["mu"] = s["mu0"].clone()
        s["picks"] = _subset_order(case["subsets"], int(rng.integers(0, case["subsets"])))
    elif op == "tv":
        noise = torch.randn((H, W, W), device="cuda", generator=gen)
        s["vol"] = _volume(ells, W, H) + noise * (0.05 / W)
        s["out"] = torch.empty_like(s["vol"])
        s["c"] = 0.002 * float(torch.linalg.vector_norm(s["vol"]))
    elif op == "prefilter":
        s["angles"] = _angles(case["views"])
        s["sino"] = _sinogram(ells, case["geom"], W, W, s["angles"])
        s["out"] = torch.empty_like(s["sino"])
    else:
        s["angles"] = _angles(case["views"], 2.0)
        s["pts"] = _helix(case, gen)
        if op == "g3d_fp":
            s["vol"] = _volume(ells, W, H)
            s["out"] = torch.empty((case["views"], case["det_h"], case["det_w"]), device="cuda")
        else:
            s["sino"] = torch.empty((case["views"], case["det_h"], case["det_w"]), device="cuda")
            per = max(1, (1 << 22) // (case["det_w"] * case["det_h"]))  # views at once
            for i in range(0, case["views"], per):
                b = torch.from_numpy(s["angles"][i:i + per]).double().cuda()[:, None, None]
                cb, sb = torch.cos(b), torch.sin(b)
                p = s["pts"][i:i + per].double().transpose(0, 1)
                a = (p[0] * cb - p[1] * sb, p[1] * cb + p[0] * sb, p[2])
                e = (p[3] * cb - p[4] * sb, p[4] * cb + p[3] * sb, p[5])
                s["sino"][i:i + per] = _chords(ells, a, [e[j] - a[j] for j in range(3)])
            s["out"] = torch.empty((H, W, W), device="cuda")
    return s


def run(s):
    op = s["op"]
    if op == "fp":
        return ops.fp_dev(s["vol"], SAD, s["angles"], s["geom"], out=s["out"])
    if op == "bp":
        return ops.bp_dev(s["sino"], SAD, s["angles"], s["geom"], out=s["out"])
    if op == "osc":
        s["mu"].copy_(s["mu0"])
        return ops.osc_iter_dev(s["mu"], s["pre"], s["post"], s["subsets"], s["picks"],
                                s["angles"], SAD, s["geom"])
    if op == "tv":
        return ops.tvmin3d_dev(s["vol"], s["c"], s["steps"], out=s["out"])
    if op == "prefilter":
        return ops.prefilter_dev(s["sino"], s["angles"], s["geom"], SAD, s["filter"],
                                 out=s["out"])
    if op == "g3d_fp":
        return ops.g3d_fp_dev(s["vol"], s["angles"], s["pts"], out=s["out"])
    return ops.g3d_bp_dev(s["sino"], s["angles"], s["pts"], s["W"], s["H"], out=s["out"])


def _mean_chord(W, H):
    """A ray's mean length through the volume, in voxels (all pixels of a W x H face)."""
    return 0.92 * W


def work(case):
    op, W = case["op"], case["W"]
    H = case.get("H", W)
    N, V = W * W * H, case.get("views", 0)
    es = 2 if case.get("half") else 4
    if op in ("fp", "bp"):
        M = W * H * V
        if op == "bp":
            # bilinear interpolation and one weighted sum per voxel and view
            return {"bytes": es * (N + M), "flops": N * V * (8 if case["geom"] == CONE else 4)}
        # a ray's sum over the cells that it crosses needs each tap's weight once: trilinear
        # (cone) or bilinear samples, one per voxel length
        return {"bytes": es * (N + M),
                "flops": M * _mean_chord(W, H) * (16 if case["geom"] == CONE else 8)}
    if op == "osc":
        M = W * H * V
        return {"bytes": 4 * (2 * N + 2 * M),
                "flops": 2 * M * _mean_chord(W, H) * 8 + 2 * N * V * 8}
    if op == "tv":
        return {"bytes": 8 * N * case["steps"], "flops": 30 * N * case["steps"]}
    if op == "prefilter":
        n = max(64, 1 << (2 * W - 1).bit_length())
        # one real FFT pair per detector row
        return {"bytes": 8 * W * W * V, "flops": W * V * 5.0 * n * math.log2(n)}
    M = case["det_w"] * case["det_h"] * V
    return {"bytes": 4 * (N + 7 * M), "flops": M * _mean_chord(W, H) * 16}


# ---------------------------------------------------------------------------
# The same results in 64 bits.  A ray's end points, its clip to the volume and its
# sample count are binary32 decisions of the operators' definition and are rounded so
# here; positions, weights and sums are in FP64.
# ---------------------------------------------------------------------------
_MOST = 6e10  # samples or voxel updates that fit the time


def _r(x):
    return x.float().double()


def _clip(s, e, half, step):
    """(entry point, step vector, sample count) of rays s -> e, as binary32 gives them."""
    d = [_r(e[i] - s[i]) for i in range(3)]
    lo, hi = torch.zeros_like(d[0]), torch.ones_like(d[0])
    for i in range(3):
        live = d[i].abs() >= 1e-5
        a1, a2 = _r(_r(-half[i] - s[i]) / d[i]), _r(_r(half[i] - s[i]) / d[i])
        lo = torch.where(live, torch.maximum(lo, torch.minimum(a1, a2)), lo)
        hi = torch.where(live, torch.minimum(hi, torch.maximum(a1, a2)), hi)
    c = [_r(lo * d[i] + s[i]) for i in range(3)]
    p = [_r(hi * d[i] + s[i]) for i in range(3)]
    q = [_r(p[i] - c[i]) for i in range(3)]
    t = _r(q[0] * q[0] + _r(q[1] * q[1]))
    dist = _r(torch.sqrt(_r(q[2] * q[2] + t)))
    n = torch.where(dist > 0, torch.ceil(_r(dist / step)), torch.zeros_like(dist))
    m = [_r(_r(q[i] / dist) * step) for i in range(3)]
    m = [torch.where(dist > 0, x, torch.zeros_like(x)) for x in m]
    return c, m, torch.where(torch.isfinite(n), n, torch.zeros_like(n)).long()


def _std_rays(geom, W, H, b):
    kw = dict(device="cuda", dtype=torch.float64)
    u, v = torch.broadcast_tensors(_axis(W, **kw)[None, :], _axis(H, **kw)[:, None])
    cb, sb = float(np.float32(math.cos(float(b)))), float(np.float32(math.sin(float(b))))
    one = torch.ones_like(u)
    if geom == PAR:
        us, uc = _r(u * sb), _r(u * cb)
        s = [_r(SAD * cb - us), _r(SAD * sb + uc), v]
        e = [_r(-SAD * cb - us), _r(-SAD * sb + uc), v]
        return s, e
    um = _r(_r(u * 2 * SAD) / SAD)
    vm = _r(_r(v * 2 * SAD) / SAD)
    s = [_r(SAD * cb * one), _r(SAD * sb * one), v if geom == FAN else 0 * v]
    e = [_r(-SAD * cb - _r(um * sb)), _r(um * cb + _r(-SAD * sb * one)), v if geom == FAN else vm]
    return s, e


def _march(vol, c, d, n, half, border):
    """Sum of the trilinear samples c + k d, k < n, of vol (1, 1, Z, Y, X) in FP64."""
    size = (vol.shape[4], vol.shape[3], vol.shape[2])
    c, d, n = [x.reshape(-1) for x in c], [x.reshape(-1) for x in d], n.reshape(-1)
    k0 = torch.zeros_like(c[0])
    if border:  # all other samples are zeros
        k0, k1 = _crossing(c, d, n, half)
        n = (k1 - k0).long()
    out = torch.zeros_like(c[0])
    live = n.nonzero()[:, 0]
    c, d, n, k0 = [x[live] for x in c], [x[live] for x in d], n[live], k0[live]
    top = int(n.max()) if n.numel() else 0
    block = max(1, (1 << 25) // max(1, n.numel()))
    acc = torch.zeros_like(k0)
    for j0 in range(0, top, block):
        j = torch.arange(j0, min(top, j0 + block), device="cuda", dtype=torch.float64)[None, :]
        k = k0[:, None] + j
        g = torch.stack([((c[i][:, None] + k * d[i][:, None]) + (half[i] - 0.5))
                         * (2.0 / (size[i] - 1)) - 1 for i in range(3)], -1)
        f = torch.nn.functional.grid_sample(vol, g[None, None], mode="bilinear",
                                            padding_mode="zeros" if border else "border",
                                            align_corners=True)[0, 0, 0]
        acc += torch.where(j < n[:, None], f, torch.zeros_like(f)).sum(1)
    out[live] = acc
    return out


def _exact_fp(vol, geom, angles, border, step):
    H, W = vol.shape[0], vol.shape[1]
    half = (W / 2, W / 2, H / 2)
    out = torch.empty((len(angles), H, W), device="cuda", dtype=torch.float64)
    if geom == CONE:
        v5 = vol[None, None]
        for i, b in enumerate(angles):
            c, d, n = _clip(*_std_rays(geom, W, H, b), half, step)
            out[i] = _march(v5, c, d, n, half, border).reshape(H, W) * step
        return out
    # the rays of a column share their path through every slice: one sparse matrix per view
    flat = vol.reshape(H, W * W).T.contiguous()
    for i, b in enumerate(angles):
        s, e = _std_rays(geom, W, H, b)
        c, d, n = _clip([x[:1] for x in s], [x[:1] for x in e], half, step)
        k = torch.arange(int(n.max()), device="cuda", dtype=torch.float64)[None, :]
        live = (k < n[0][:, None]).reshape(-1)
        row = torch.arange(W, device="cuda")[:, None].expand(W, k.shape[1]).reshape(-1)[live]
        p = [(c[j][0][:, None] + k * d[j][0][:, None] + (W / 2 - 0.5)).reshape(-1)[live]
             for j in range(2)]
        f = [torch.floor(x) for x in p]
        w = [p[j] - f[j] for j in range(2)]
        rows, cols, vals = [], [], []
        for dx in (0, 1):
            for dy in (0, 1):
                ix, iy = f[0].long() + dx, f[1].long() + dy
                wt = (w[0] if dx else 1 - w[0]) * (w[1] if dy else 1 - w[1])
                if border:
                    wt = wt * ((ix >= 0) & (ix < W) & (iy >= 0) & (iy < W))
                rows.append(row)
                cols.append(iy.clamp(0, W - 1) * W + ix.clamp(0, W - 1))
                vals.append(wt)
        A = torch.sparse_coo_tensor(torch.stack([torch.cat(rows), torch.cat(cols)]),
                                    torch.cat(vals), (W, W * W)).coalesce().to_sparse_csr()
        out[i] = (A @ flat).T * step
    return out


def _taps(c, n, border):
    """Lower / upper tap and weights of texture coordinate c (texel centres at i + 0.5)."""
    c = c.clamp(-4.0, n + 4.0) - 0.5
    i = torch.floor(c)
    w1 = c - i
    w0 = 1 - w1
    i = i.long()
    if border:
        w0 = w0 * ((i >= 0) & (i < n))
        w1 = w1 * ((i + 1 >= 0) & (i + 1 < n))
    return i.clamp(0, n - 1), (i + 1).clamp(0, n - 1), w0, w1


def _exact_bp(views, geom, angles, border=False):
    """Voxel-driven backprojections (H, W, W) of several sinograms at once, in FP64."""
    _, H, W = views[0].shape
    hw = W // 2 - 1
    kw = dict(device="cuda", dtype=torch.float64)
    i = torch.arange(W, device="cuda")
    inside = ((i - hw)[None, :] ** 2 + (i - hw)[:, None] ** 2 < hw * hw).reshape(-1).nonzero()[:, 0]
    x, y = (inside % W).double() - (hw + 0.5), (inside // W).double() - (hw + 0.5)
    z = torch.arange(H, **kw)[None, :]
    v0 = (H - 1) / 2
    acc = [torch.zeros((inside.numel(), H), **kw) for _ in views]
    for k, b in enumerate(angles):
        cb, sb = float(np.float32(math.cos(float(b)))), float(np.float32(math.sin(float(b))))
        t = y * cb - x * sb
        U = torch.ones_like(t) if geom == PAR else SAD / (SAD - (x * cb + y * sb))
        i0, i1, w0, w1 = _taps(t * U + hw + 1, W, border)
        w = U * U
        w0, w1 = (w * w0)[:, None], (w * w1)[:, None]
        if geom == CONE:
            r0, r1, a0, a1 = _taps((z - v0) * U[:, None] + v0 + 0.5, H, border)
        for out, sino in zip(acc, views):
            p = sino[k].double().T.contiguous()  # (W, H): a detector column is a row
            if geom == CONE:
                col = p[i0] * w0 + p[i1] * w1
                out += a0 * torch.gather(col, 1, r0) + a1 * torch.gather(col, 1, r1)
            else:
                out += p[i0] * w0 + p[i1] * w1
    full = []
    for a in acc:
        v = torch.zeros((W * W, H), **kw)
        v[inside] = a
        full.append(v.T.reshape(H, W, W))
    return full, inside


def _exact_osc(s):
    mu, n = s["mu0"].double(), s["subsets"]
    W = s["W"]
    for sel in s["picks"]:
        keep = slice(int(sel), None, n)
        ang = s["angles"][keep]
        if len(ang):
            line = _exact_fp(mu, s["geom"], ang, True, 0.5)
            ehat = s["pre"][keep].double() * torch.exp(-line)
            (num, den), inside = _exact_bp([ehat - s["post"][keep].double(), ehat * line],
                                           s["geom"], ang, True)
        else:
            num = den = torch.zeros_like(mu)
            inside = _exact_bp([s["pre"][:0]], s["geom"], [])[1]
        new = mu + mu * num / den
        new = torch.where(new > 0, new, torch.zeros_like(new))
        flat = mu.reshape(-1, W * W).clone()
        flat[:, inside] = new.reshape(-1, W * W)[:, inside]
        mu = flat.reshape(mu.shape)
    return mu


def _exact_tv(s):
    x = s["vol"].double()
    for _ in range(s["steps"]):
        q = x[1:, 1:, 1:]
        a, b, c = q - x[1:, 1:, :-1], q - x[1:, :-1, 1:], q - x[:-1, 1:, 1:]
        r = 1 / (1e-6 + torch.sqrt(a * a + b * b + c * c))
        g = torch.zeros_like(x)
        inner = (slice(None, -1),) * 3
        g[1:-1, 1:-1, 1:-1] = (((a + b + c) * r)[inner] - (a * r)[:-1, :-1, 1:]
                               - (b * r)[:-1, 1:, :-1] - (c * r)[1:, :-1, :-1])
        x = x - (float(np.float32(s["c"])) / torch.linalg.vector_norm(g)) * g
    return x


def _exact_prefilter(s):
    W, V, geom, ang = s["W"], s["views"], s["geom"], s["angles"].astype(np.float64)
    order = max(64, 1 << (2 * W - 1).bit_length())
    n = np.arange(order // 2 + 1)
    h = np.zeros(order)
    h[0] = 0.25
    odd = n[n % 2 == 1]
    h[odd] = -1.0 / (np.pi * odd) ** 2
    h[(order - odd) % order] = h[odd]
    filt = 2 * np.real(np.fft.rfft(h))
    w = 2 * np.pi * n[1:] / order
    f = s["filter"]
    if f == "shepp-logan":
        filt[1:] *= np.sin(w / 2) / (w / 2)
    elif f == "cosine":
        filt[1:] *= np.cos(w / 2)
    elif f == "hamming":
        filt[1:] *= 0.54 + 0.46 * np.cos(w)
    elif f == "hann":
        filt[1:] *= (1 + np.cos(w)) / 2
    alpha = np.arctan((np.arange(W) - W / 2 + 0.5) / SAD) if geom != PAR else np.zeros(W)
    if np.all(np.diff(ang) >= 0):
        alpha = -alpha
    delta = abs(alpha[-1] - alpha[0]) / 2
    eps = max(abs(float(s["angles"][-1] - s["angles"][0])) - (np.pi + 2 * delta), 0.0)

    def S(b):
        return np.where(np.abs(b) < 0.5, 0.5 * (1 + np.sin(np.pi * b)), np.where(b >= 0.5, 1.0, 0.0))

    def B(a):
        return 2 * delta - 2 * a + eps

    beta = np.abs(s["angles"] - s["angles"][0]).astype(np.float64)[:, None]
    with np.errstate(all="ignore"):
        park = 0.5 * (S(beta / B(alpha) - 0.5) + S((beta - 2 * delta + 2 * alpha - eps) / B(alpha) + 0.5)
                      - S((beta - np.pi + 2 * alpha) / B(-alpha) - 0.5)
                      - S((beta - np.pi - 2 * delta - eps) / B(-alpha) + 0.5))
    db = np.diff(s["angles"], prepend=s["angles"][:1]).astype(np.float64) / 2
    db[0] = float(s["angles"][1] - s["angles"][0]) / 2
    kw = dict(device="cuda", dtype=torch.float64)
    U = (torch.arange(W, **kw) + 1 - (W - 1) * 0.5)[None, :]
    Vv = (torch.arange(W, **kw) + 1 - (W - 1) * 0.5)[:, None]
    cosw = torch.ones((W, W), **kw)
    if geom != PAR:
        cosw = SAD / torch.sqrt(SAD * SAD + U * U + (Vv * Vv if geom == CONE else 0 * Vv))
    filt, park = torch.from_numpy(filt).cuda(), torch.from_numpy(park).cuda()
    out = torch.empty((V, W, W), **kw)
    for i in range(V):
        g = s["sino"][i].double() * cosw * park[i][None, :]
        out[i] = torch.fft.irfft(torch.fft.rfft(g, order) * filt, order)[:, :W] * float(db[i])
    return out


def _g3d_rays(s, i):
    cb = float(np.float32(math.cos(float(s["angles"][i]))))
    sb = float(np.float32(math.sin(float(s["angles"][i]))))
    p = s["pts"][i].double()
    a = [_r(p[0] * cb - _r(p[1] * sb)), _r(p[1] * cb + _r(p[0] * sb)), p[2]]
    e = [_r(p[3] * cb - _r(p[4] * sb)), _r(p[4] * cb + _r(p[3] * sb)), p[5]]
    return a, e


def _crossing(c, d, n, half):
    """The samples [k0, k1) of rays c + k d, k < n, that can touch the volume (a sample or
    two more at each end)."""
    k0, k1 = torch.zeros_like(c[0]), n.double()
    for i in range(3):
        a, b = (-half[i] - 1 - c[i]) / d[i], (half[i] + 1 - c[i]) / d[i]
        still = d[i] == 0
        far = still & (c[i].abs() > half[i] + 1)
        k0 = torch.where(still, k0, torch.maximum(k0, torch.floor(torch.minimum(a, b))))
        k1 = torch.where(still, k1, torch.minimum(k1, torch.ceil(torch.maximum(a, b)) + 1))
        k1 = torch.where(far, torch.zeros_like(k1), k1)
    return k0, torch.maximum(k0, k1)


def _exact_g3d_bp(s):
    """The two-corner scatter; its positions advance in binary32 (their floor is the
    definition of the voxel), its deposits are summed in FP64."""
    W, H = s["W"], s["H"]
    half = (W / 2, W / 2, H / 2)
    out = torch.zeros(H * W * W, device="cuda", dtype=torch.float64)
    org = torch.tensor([-W / 2, -W / 2, -H / 2], device="cuda")[:, None]
    size = torch.tensor([W, W, H], device="cuda")[:, None]
    per = max(1, (1 << 23) // (s["det_w"] * s["det_h"]))  # views at once
    for v0 in range(0, s["views"], per):
        rays = []
        for i in range(v0, min(s["views"], v0 + per)):
            c, d, n = _clip(*_g3d_rays(s, i), half, 0.5)
            k0, k1 = _crossing(c, d, n, half)
            hit = (k1 > k0) & (s["sino"][i] != 0)
            rays.append((torch.stack([x[hit] for x in c]).float(),
                         torch.stack([x[hit] for x in d]).float(), k1[hit].long(),
                         s["sino"][i][hit] * 0.5))
        pos, step = (torch.cat([r[j] for r in rays], 1) for j in (0, 1))
        n, ps = (torch.cat([r[j] for r in rays]) for j in (2, 3))
        for k in range(int(n.max()) if n.numel() else 0):
            if k % 32 == 0:  # rays that have ended leave
                live = (n > k).nonzero()[:, 0]
                pos, step, n, ps = pos[:, live], step[:, live], n[live], ps[live]
            f = pos - org
            lo, up = torch.floor(f), torch.ceil(f)
            ok = (((lo >= 0) & (up < size)).all(0) & (k < n)).nonzero()[:, 0]
            f, lo, up = f[:, ok], lo[:, ok], up[2, ok]
            w = (f - lo) + 0.5
            pxy = ps[ok] * w[0] * w[1]
            base = lo[0].long() + W * lo[1].long()
            out.index_add_(0, base + W * W * lo[2].long(), (pxy * (1.0 - w[2])).double())
            out.index_add_(0, base + W * W * up.long(), (pxy * w[2]).double())
            pos = pos + step
    return out.reshape(H, W, W)


def exact(case, seed):
    op, W = case["op"], case["W"]
    H, V = case.get("H", W), case.get("views", 0)
    if op == "fp" and W * W * H * V * (1.3 if case["geom"] == CONE else 0.5) > _MOST:
        return None
    if op == "bp" and W * W * H * V * 0.5 > _MOST:
        return None
    if op in ("g3d_fp", "g3d_bp") and 2.6 * case["det_w"] * case["det_h"] * V * W > _MOST:
        return None
    s = prepare(case, seed)
    if op == "fp":
        return _exact_fp(s["vol"].double(), case["geom"], s["angles"], False,
                         1.0 if case["geom"] == CONE else 0.5)
    if op == "bp":
        return _exact_bp([s["sino"]], case["geom"], s["angles"])[0][0]
    if op == "osc":
        return _exact_osc(s)
    if op == "tv":
        return _exact_tv(s)
    if op == "prefilter":
        return _exact_prefilter(s)
    if op == "g3d_fp":
        vol, half = s["vol"].double()[None, None], (W / 2, W / 2, H / 2)
        out = torch.empty(s["out"].shape, device="cuda", dtype=torch.float64)
        for i in range(V):
            c, d, n = _clip(*_g3d_rays(s, i), half, 0.5)
            out[i] = _march(vol, c, d, n, half, True).reshape(out[i].shape) * 0.5
        return out
    return _exact_g3d_bp(s)
