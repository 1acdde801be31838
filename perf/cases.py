"""The calls this framework's speed is measured on: slanted-plane PatchMatch
stereo over its range of sizes, both arithmetics, the inpainting variant and
the batched call; the matching cost alone and its adjoint; TSDF fusion; and
the cost-volume baseline.

Images are seeded slanted-plane scenes of the kind the benchmark and the tests
use (Voronoi cells of planes, blurred-noise texture, the right view resampled
through the true disparity, salt noise and a gain/bias mismatch between the
views), made on the GPU.  The context (``PMHuberStereo``, ``TSDFVolume``) is
kept between calls, as a program that processes a stream of pairs keeps it.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from cvt_gb300 import params as P
from cvt_gb300.autograd import asw_cost
from cvt_gb300.gcv import StereoGCVFilter
from cvt_gb300.stereo import PMHuberStereo
from cvt_gb300.tsdf import TSDFVolume

DEV = "cuda"


def listed():
    stereo = {"kind": "stereo", "preset": "baseline", "patch": 17, "pd": 250, "trace": False}
    return [
        # the smallest call: a preview-sized pair, where launches and latency count
        dict(stereo, name="stereo_64x48", w=64, h=48, dmax=12.0, planes=3, iters=3),
        # a small pair of odd size, integer outputs (winners, validity) included
        dict(stereo, name="stereo_321x243", w=321, h=243, dmax=48.0, planes=6, iters=5, trace=True),
        # the plain configuration: VGA, 3 iterations
        dict(stereo, name="stereo_640x480", w=640, h=480, dmax=64.0, planes=8, iters=3),
        # the headline configuration: a driving-camera pair, 8 iterations
        dict(stereo, name="stereo_1242x375", w=1242, h=375, dmax=128.0, planes=16, iters=8),
        # the largest pair of the batched configuration
        dict(stereo, name="stereo_1920x1080", w=1920, h=1080, dmax=256.0, planes=24, iters=3),
        # the reference's own arithmetic, constants and random streams
        dict(stereo, name="stereo_exact_450x375", preset="reference", w=450, h=375, dmax=64.0, planes=8, iters=3,
             trace=True),
        # the inpainting variant (occlusion-masked smoother, 100 steps)
        {"name": "inpaint_450x375", "kind": "inpaint", "preset": "baseline", "patch": 17, "w": 450, "h": 375,
         "dmax": 64.0, "planes": 8, "iters": 6},
        # pairs of uneven size and disparity range in one batched call
        {"name": "batch_4_uneven", "kind": "batch", "preset": "baseline", "patch": 17, "iters": 3, "w": 320, "h": 240,
         "wmax": 640, "hmax": 480, "pairs": 4},
        # the cost of a fixed plane field (evaluation alone, as a learner or a validator calls it)
        {"name": "cost_640x480", "kind": "cost", "preset": "baseline", "patch": 17, "w": 640, "h": 480, "dmax": 64.0,
         "planes": 8},
        # training: forward and backward of the cost for planes and both images
        {"name": "adjoint_640x480", "kind": "adjoint", "preset": "baseline", "patch": 17, "w": 640, "h": 480,
         "dmax": 64.0, "planes": 8},
        # fusion of a depth map into a volume, and the ray cast of it
        {"name": "tsdf_256", "kind": "tsdf", "n": 256, "w": 640, "h": 480},
        # the comparison baseline: every disparity of the headline pair, both views
        {"name": "gcv_1242x375", "kind": "gcv", "w": 1242, "h": 375, "dmax": 128.0, "planes": 16},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["stereo"] * 5 + ["inpaint", "batch", "cost", "adjoint", "tsdf", "gcv"])
    if kind == "tsdf":
        return {"kind": kind, "n": rng.randrange(48, 257), "w": _log(rng, 64, 640), "h": _log(rng, 48, 480)}
    w, h = _log(rng, 64, 1920), _log(rng, 48, 1080)
    if kind in ("inpaint", "batch", "cost", "adjoint"):
        w, h = _log(rng, 64, 640), _log(rng, 48, 480)
    case = {"kind": kind, "w": w, "h": h}
    if kind == "gcv":
        case.update(w=min(w, 1242), h=min(h, 375), dmax=float(rng.randrange(16, 129)), planes=rng.randrange(3, 17))
        return case
    case.update(preset=rng.choice(["baseline", "baseline", "reference"]), patch=rng.choice([7, 9, 13, 17, 17, 17]))
    if kind == "batch":
        case.update(preset="baseline", iters=rng.randrange(2, 4), wmax=640, hmax=480, pairs=rng.randrange(2, 5))
        return case
    case.update(dmax=float(rng.randrange(8, max(9, min(257, w // 4 + 1)))), planes=rng.randrange(2, 25))
    if kind == "adjoint":
        case["preset"] = "baseline"       # the adjoint is of the FAST arithmetic
    if kind in ("stereo", "inpaint"):
        # no more than the largest listed pair's work
        most = 1920 * 1080 * 3 // (w * h)
        case["iters"] = rng.randrange(1, max(2, min(8, most) + 1))
        if case["preset"] == "reference":
            case["iters"] = max(1, min(case["iters"], most // 2))
    if kind == "stereo":
        case.update(pd=rng.choice([250, 250, 100, 31]), trace=rng.random() < 0.5)
    return case


# ------------------------------------------------------------------ scenes --
def _texture(g, h, w):
    n = torch.rand((3, 1, h + 10, w + 10), generator=g, device=DEV)
    r = torch.arange(-5, 6, device=DEV, dtype=torch.float32)
    k = torch.exp(-0.5 * (r / 1.5) ** 2)
    k = k / k.sum()
    n = torch.nn.functional.conv2d(n, k.view(1, 1, 1, 11))
    n = torch.nn.functional.conv2d(n, k.view(1, 1, 11, 1))[:, 0]
    lo, hi = n.amin((1, 2), True), n.amax((1, 2), True)
    return (n - lo) / (hi - lo)                       # (3, h, w) in [0, 1]


def _scene(seed, w, h, nplanes, dmax, salt=0.02, gain=0.05):
    """left, right (H, W, 4) float32 and the left view's planes (H, W, 3)."""
    g = torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + w * 31 + h)
    rnd = lambda *s: torch.rand(s, generator=g, device=DEV)
    sx, sy = rnd(nplanes) * w, rnd(nplanes) * h
    ab = (rnd(nplanes, 2) - 0.5) * 0.3
    # slopes shrunk until the plane stays within [0, dmax] near its site
    ab = ab * min(1.0, 2.0 * dmax / (0.15 * (w + h)))
    c = (0.1 + 0.8 * rnd(nplanes)) * dmax - ab[:, 0] * sx - ab[:, 1] * sy
    yy, xx = torch.meshgrid(torch.arange(h, device=DEV, dtype=torch.float32),
                            torch.arange(w, device=DEV, dtype=torch.float32), indexing="ij")
    best = torch.full((h, w), float("inf"), device=DEV)
    lab = torch.zeros((h, w), dtype=torch.long, device=DEV)
    for i in range(nplanes):
        d = (xx - sx[i]) ** 2 + (yy - sy[i]) ** 2
        m = d < best
        best, lab = torch.where(m, d, best), torch.where(m, torch.full_like(lab, i), lab)
    dr = torch.full((h, w), -1.0, device=DEV)         # right-view disparity: nearest surface wins
    for i in range(nplanes):
        xl = (xx + ab[i, 1] * yy + c[i]) / (1.0 - ab[i, 0])
        xi = xl.round().clamp(0, w - 1).long()
        d = (xl - xx).clamp(0.0, dmax)
        ok = (xl >= 0) & (xl <= w - 1) & (lab.gather(1, xi) == i)
        dr = torch.where(ok & (d > dr), d, dr)
    dr = dr.clamp_min(0.0)
    tex = _texture(g, h, w)
    xs = (xx + dr).clamp(0, w - 1)
    x0 = xs.floor()
    a = xs - x0
    i0 = x0.long()
    i1 = (i0 + 1).clamp_max(w - 1)
    right = tex.gather(2, i0.expand(3, h, w)) * (1 - a) + tex.gather(2, i1.expand(3, h, w)) * a
    left = tex
    left = torch.where(rnd(h, w) < salt, torch.ones_like(left), left)
    right = torch.where(rnd(h, w) < salt, torch.ones_like(right), right)
    right = (right * (1.0 + (rnd(3, 1, 1) - 0.5) * 2 * gain) + (rnd(3, 1, 1) - 0.5) * 2 * gain).clamp(0, 1)
    one = torch.ones((1, h, w), device=DEV)
    rgba = lambda t: torch.cat([t, one]).permute(1, 2, 0).contiguous()
    planes = torch.stack([ab[:, 0][lab], ab[:, 1][lab], c[lab]], -1)
    return rgba(left), rgba(right), planes


def _params(case, **kw):
    preset = P.PRESET_BASELINE if case["preset"] == "baseline" else P.PRESET_REFERENCE
    return P.default_params(preset, patchsize=case["patch"], **kw)


def _plane_field(seed, planes):
    """Planes near the truth: (a, b) off by 0.01, c by 1 px, as a learner's are."""
    g = torch.Generator(device=DEV).manual_seed(int(seed) + 17)
    noise = torch.randn(planes.shape, generator=g, device=DEV)
    pl = planes + noise * torch.tensor([0.01, 0.01, 1.0], device=DEV)
    return torch.cat([pl, torch.zeros_like(pl[..., :1])], -1).contiguous()


def _states(planes):
    """(s0, s1, s2, -) of left-view planes: x' = x - d."""
    z = torch.zeros_like(planes[..., 0])
    return torch.stack([1.0 - planes[..., 0], -planes[..., 1], -planes[..., 2], z], -1).contiguous()


# ------------------------------------------------------------ TSDF inputs --
def _tsdf_inputs(case, seed):
    n, w, h = case["n"], case["w"], case["h"]
    g = np.random.default_rng(int(seed))
    ext = 2.0                                          # metres per side, centred at z = 2
    vox = ext / n
    g2w = np.array([[vox, 0, 0, -ext / 2], [0, vox, 0, -ext / 2], [0, 0, vox, 1.0], [0, 0, 0, 1]], np.float32)
    f = 0.9 * w
    K = np.array([[f, 0, (w - 1) / 2], [0, f, (h - 1) / 2], [0, 0, 1]], np.float32)
    E = np.eye(4, dtype=np.float32)
    E[:3, 3] = (g.random(3) - 0.5) * 0.1
    # a sphere in front of a wall, as the camera sees it
    cx, cy, cz = (g.random(3) - 0.5) * 0.4 + np.array([0, 0, 2.0])
    v, u = np.mgrid[0:h, 0:w].astype(np.float64)
    dirs = np.stack([(u - K[0, 2]) / f, (v - K[1, 2]) / f, np.ones_like(u)], -1)
    cam = np.array([cx, cy, cz]) + E[:3, 3]
    b = dirs @ cam
    a = (dirs * dirs).sum(-1)
    disc = b * b - a * (cam @ cam - 0.25)
    t = (b - np.sqrt(np.maximum(disc, 0))) / a
    depth = np.where(disc > 0, t, 2.8).astype(np.float32)
    return g2w, K, E, depth


# ----------------------------------------------------------------- prepare --
def prepare(case, seed):
    kind = case["kind"]
    if kind == "tsdf":
        g2w, K, E, depth = _tsdf_inputs(case, seed)
        n = case["n"]
        vol = TSDFVolume(g2w, n, n, n, truncation=0.08)
        return {"case": case, "vol": vol, "K": K, "E": E, "depth": torch.from_numpy(depth).to(DEV)}
    if kind == "batch":
        g = np.random.default_rng(int(seed))
        # sizes belong to the case, images to the seed
        sizes = np.random.default_rng(case["pairs"] * 1000 + case["w"] + case["h"])
        pairs = []
        for _ in range(case["pairs"]):
            w = int(sizes.integers(case["w"], case["wmax"] + 1))
            h = int(sizes.integers(case["h"], case["hmax"] + 1))
            dmax = float(sizes.integers(min(16, w // 4), w // 4 + 1))
            left, right, _ = _scene(int(g.integers(1 << 30)), w, h, 6, dmax)
            pairs.append((left, right, dmax))
        return {"case": case, "stereo": PMHuberStereo(params=_params(case, iterations=case["iters"])), "pairs": pairs}
    left, right, planes = _scene(seed, case["w"], case["h"], case["planes"], case["dmax"])
    if kind == "gcv":
        return {"case": case, "left": left, "right": right, "gcv": StereoGCVFilter()}
    st = {"case": case, "left": left, "right": right}
    if kind == "stereo":
        st["stereo"] = PMHuberStereo(params=_params(case, pd_iterations=case["pd"]))
        st["dmap"] = torch.empty((case["h"], case["w"]), device=DEV)
        st["normals"] = torch.empty((case["h"], case["w"], 4), device=DEV)
    elif kind == "inpaint":
        st["stereo"] = PMHuberStereo(params=_params(case))
        st["dmap"] = torch.empty((case["h"], case["w"]), device=DEV)
    elif kind == "cost":
        st["stereo"] = PMHuberStereo(params=_params(case))
        st["states"] = _states(_plane_field(seed, planes))
    elif kind == "adjoint":
        g = torch.Generator(device=DEV).manual_seed(int(seed) + 29)
        st["stereo"] = PMHuberStereo(params=_params(case))
        st["field"] = _plane_field(seed, planes).requires_grad_(True)
        st["left"].requires_grad_(True)
        st["right"].requires_grad_(True)
        st["dcost"] = torch.randn(planes.shape[:2], generator=g, device=DEV)
    return st


# --------------------------------------------------------------------- run --
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "stereo":
        trace = {} if case["trace"] else None
        s["stereo"].depthMap(s["dmap"], s["left"], s["right"], case["patch"], case["dmax"], case["iters"], 4,
                             normalmap=s["normals"], trace=trace)
        return {"disparity": s["dmap"], "normals": s["normals"], **(trace or {})}
    if kind == "inpaint":
        return s["stereo"].depthMapInpaint(s["dmap"], s["left"], s["right"], case["patch"], case["dmax"],
                                           case["iters"], 4)
    if kind == "batch":
        # the maps are passed back: the same inputs replay the captured graph
        s["outs"] = s["stereo"].depthMapBatched(s["pairs"], s.get("outs"))
        return list(s["outs"])
    if kind == "cost":
        return s["stereo"].cost(s["left"], s["right"], s["states"])
    if kind == "adjoint":
        cost = asw_cost(s["stereo"], s["left"], s["right"], s["field"])
        dl, dr, dp = torch.autograd.grad(cost, (s["left"], s["right"], s["field"]), s["dcost"])
        return {"cost": cost.detach(), "dleft": dl, "dright": dr, "dplanes": dp}
    if kind == "tsdf":
        s["vol"].clear()
        s["vol"].addDepthMap(s["K"], s["E"], s["depth"])
        cast = s["vol"].rayCastDepthMap(s["K"], s["E"], case["w"], case["h"], scale=-1.0)
        # volume() is a view of the volume's own memory; a copy outlives it
        return {"volume": s["vol"].volume().clone(), "cast": cast}
    # gcv: cam0 is the right image (a match of cam1's x lies at x - d)
    fused, d0, d1 = s["gcv"].apply(s["right"], s["left"], 0.0, case["dmax"], 1.0)
    return {"fused": fused, "d0": d0, "d1": d1}


# -------------------------------------------------------------------- work --
def _taps(w, h, p):
    """In-image window taps of all pixels."""
    nx = sum(min(x + p, w - 1) - max(x - p, 0) + 1 for x in range(w))
    ny = sum(min(y + p, h - 1) - max(y - p, 0) + 1 for y in range(h))
    return nx * ny


def work(case):
    """Each image read once and each result written once; operations of the
    algorithm.  A tap's matching terms are 55 operations and its bilateral
    weight 20; a pass tests, per pixel and view, the planes of the 3x3
    neighbourhood (their terms are common to the windows that test them) and
    about ten planes of its own: the smoothed one, six random neighbours, a
    random plane and two refinements; a smoother step is 80 per pixel."""
    kind = case["kind"]
    if kind == "tsdf":
        v = case["n"] ** 3
        return {"bytes": v * 8.0 + case["w"] * case["h"] * 8.0, "flops": v * 24.0}
    if kind == "batch":
        sizes = np.random.default_rng(case["pairs"] * 1000 + case["w"] + case["h"])
        out = {"bytes": 0.0, "flops": 0.0}
        for _ in range(case["pairs"]):
            w = int(sizes.integers(case["w"], case["wmax"] + 1))
            h = int(sizes.integers(case["h"], case["hmax"] + 1))
            sizes.integers(min(16, w // 4), w // 4 + 1)
            one = work({"kind": "stereo", "w": w, "h": h, "patch": case["patch"], "iters": case["iters"], "pd": 250})
            out = {k: out[k] + one[k] for k in out}
        return out
    w, h = case["w"], case["h"]
    n = w * h
    if kind == "gcv":
        # per pixel, view and disparity: cost 40, twelve box sums 48, the guided filter's solve 90, apply 12
        return {"bytes": n * (32.0 + 9.0), "flops": 2.0 * n * case["dmax"] * 190.0}
    taps = _taps(w, h, case["patch"])
    if kind == "cost":
        return {"bytes": n * (32.0 + 16.0 + 4.0), "flops": taps * 75.0}
    if kind == "adjoint":
        return {"bytes": n * (48.0 + 4.0 + 4.0 + 48.0), "flops": taps * (75.0 + 160.0)}
    passes = 2.0 * case["iters"]
    pd = case.get("pd", 100)
    return {"bytes": n * (32.0 + 20.0),
            "flops": passes * (taps * (11 * 55.0 + 20.0 + 8 * 5.0) + n * pd * 80.0) + 2.0 * taps * 75.0}


# ------------------------------------------------------------------- exact --
def _grad64(img):
    """(dx, dy, dxy, dyx) of the grey image, zero outside."""
    gray = img[..., 0] * 0.2126 + img[..., 1] * 0.7152 + img[..., 2] * 0.0722
    b = torch.nn.functional.pad(gray, (1, 1, 1, 1))
    h, w = gray.shape
    at = lambda dx, dy: b[1 + dy:1 + dy + h, 1 + dx:1 + dx + w]
    dx = (at(1, 0) - at(-1, 0)) * 0.5 + (at(1, -1) - at(-1, -1)) * 0.25 + (at(1, 1) - at(-1, 1)) * 0.25
    dy = (at(0, 1) - at(0, -1)) * 0.5 + (at(-1, 1) - at(-1, -1)) * 0.25 + (at(1, 1) - at(1, -1)) * 0.25
    return torch.stack([dx, dy, at(1, 1) - at(-1, -1), at(-1, 1) - at(1, -1)], -1)


def _window(case, img1, img2, g1, g2, s):
    """For every window offset: the pixels whose tap is in both images, and
    the tap's weight and matching cost there (64 bits)."""
    prm = _params(case)
    p, w, h = case["patch"], case["w"], case["h"]
    al, cm, gm = prm.color_alpha, prm.color_maxdiff, prm.grad_maxdiff
    for dy in range(-p, p + 1):
        for dx in range(-p, p + 1):
            y0, y1, x0, x1 = max(0, -dy), min(h, h - dy), max(0, -dx), min(w, w - dx)
            if y0 >= y1 or x0 >= x1:
                continue
            c = (slice(y0, y1), slice(x0, x1))
            q = (slice(y0 + dy, y1 + dy), slice(x0 + dx, x1 + dx))
            qx = torch.arange(x0 + dx, x1 + dx, device=DEV, dtype=torch.float64)[None, :]
            qy = torch.arange(y0 + dy, y1 + dy, device=DEV, dtype=torch.float64)[:, None]
            xp = s[c][..., 0] * qx + s[c][..., 1] * qy + s[c][..., 2]
            ok = (xp >= 0) & (xp < w)
            xi = xp.detach().floor().clamp(0, w - 1)
            a = (xp - xi)[..., None]
            i0 = xi.long()
            i1 = (i0 + 1).clamp_max(w - 1)
            row = torch.arange(y0 + dy, y1 + dy, device=DEV)[:, None].expand_as(i0)
            lerp = lambda t: t[row, i0] * (1 - a) + t[row, i1] * a
            cc = (img1[q][..., :3] - lerp(img2)[..., :3]).abs().clamp_max(cm).sum(-1)
            gc = (g1[q] - lerp(g2)).abs().clamp_max(gm).sum(-1)
            prof = prm.color_weight
            if prm.weight_profile == P.PROFILE_SMOOTHSTEP:
                t = min(max(math.hypot(dx, dy) / 26.0, 0.0), 1.0)
                prof = t * t * (3 - 2 * t) * 1.5 * prm.color_weight + 5.0
            wt = torch.exp(-(img1[c][..., :3] - img1[q][..., :3]).abs().sum(-1) * prof)
            yield c, ok, wt, al * cc + (1 - al) * gc


def _sums64(case, img1, img2, s):
    h, w = case["h"], case["w"]
    S = torch.zeros((h, w), dtype=torch.float64, device=DEV)
    R = torch.zeros_like(S)
    with torch.no_grad():
        for c, ok, wt, cost in _window(case, img1, img2, _grad64(img1), _grad64(img2), s):
            wv = torch.where(ok, wt, torch.zeros_like(wt))
            S[c] += wv
            R[c] += wv * cost
    return S, R


def exact(case, seed):
    kind = case["kind"]
    if kind == "tsdf":
        return _exact_tsdf(case, seed)
    if kind not in ("cost", "adjoint"):
        return None                     # the winners of thousands of comparisons: no 64-bit value
    left, right, planes = _scene(seed, case["w"], case["h"], case["planes"], case["dmax"])
    field = _plane_field(seed, planes)
    if kind == "cost":
        img1, img2, s = left.double(), right.double(), _states(field).double()
        S, R = _sums64(case, img1, img2, s)
        return torch.where(S > 1.1, R / S, torch.full_like(S, 1e5))
    g = torch.Generator(device=DEV).manual_seed(int(seed) + 29)
    dcost = torch.randn(planes.shape[:2], generator=g, device=DEV).double()
    img1, img2, pl = left.double(), right.double(), field.double()
    S, R = _sums64(case, img1, img2, _states(pl))
    good = S > 1.1
    cost = torch.where(good, R / S.clamp_min(1e-300), torch.full_like(S, 1e5))
    u = torch.where(good, dcost / S.clamp_min(1e-300), torch.zeros_like(S))
    img1.requires_grad_(True)
    img2.requires_grad_(True)
    pl.requires_grad_(True)
    g1, g2 = _grad64(img1.detach()).requires_grad_(True), _grad64(img2.detach()).requires_grad_(True)
    # d(R/S) = (dR - C dS) / S, tap by tap
    for c, ok, wt, ct in _window(case, img1, img2, g1, g2, _states(pl)):
        (torch.where(ok, u[c] * wt * (ct - cost[c]), torch.zeros_like(wt))).sum().backward()
    for img, gi in ((img1, g1), (img2, g2)):
        gi_of = _grad64(img)
        gi_of.backward(gi.grad)
    drop = lambda t: torch.cat([t[..., :3], torch.zeros_like(t[..., :1])], -1)
    return {"cost": cost, "dleft": drop(img1.grad), "dright": drop(img2.grad), "dplanes": drop(pl.grad)}


def _exact_tsdf(case, seed):
    g2w, K, E, depth = _tsdf_inputs(case, seed)
    n, w, h = case["n"], case["w"], case["h"]
    K4 = np.eye(4)
    K4[:3, :3] = K
    T = K4 @ E.astype(np.float64) @ g2w.astype(np.float64)
    r = torch.arange(n, device=DEV, dtype=torch.float64)
    z, y, x = r[:, None, None], r[None, :, None], r[None, None, :]
    px, py, pz = (T[i, 0] * x + T[i, 1] * y + T[i, 2] * z + T[i, 3] for i in range(3))
    u, v = px / pz, py / pz
    d = torch.from_numpy(depth).to(DEV).double()
    seen = (u >= 0) & (v >= 0) & (u < w) & (v < h)
    ui, vi = u.floor().clamp(0, w - 1).long(), v.floor().clamp(0, h - 1).long()
    sdf = d[vi, ui] - pz
    trunc = float(np.float32(0.08))
    hit = seen & (d[vi, ui] > 0) & (pz > 0) & (sdf.abs() <= trunc)
    val = torch.where(hit, sdf / trunc, torch.ones_like(sdf))
    return {"volume": torch.stack([val, hit.double()], -1), "cast": None}
