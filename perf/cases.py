"""The renderer's workloads as a user's program runs them, through the public entry points.

A case names one call (`kind`) and its sizes. Scenes follow the distributions of
`fuzzy_ellipses.synthetic`: means uniform in a cube, axis scales log-uniform in [5, 30] mm with a
random rotation, log-weights N(0, 0.5^2), cameras on a sphere looking at the origin.

kinds
  call       `render_forward`: one camera per call, poses as host arrays (the plain drop-in)
  grad       `render` with autograd: one camera, gradients to means, precisions and log-weights
  batch      `Batch.forward`: many scenes and cameras planned once, one launch sequence per pass
  host       `Batch.forward_host`: pinned host Gaussians in, pinned host images out
  step       a shape-from-silhouette step: `Batch.forward`, `silhouette_bce`, `Batch.backward`
  features   `render_features`: per-Gaussian colours or descriptors blended into the image
  pixels     `render_pixels`: pixel rows over many poses, with optical flow
  rasterize  `rasterize`: the reference's own signature (its binning, 8x8 tiles)

`exact` leaves out depths: where a pixel's Gaussians all lie below the density cut-off the
renderer's depth is that of the ones its tile lists, which the uncut formula does not describe.
It leaves out `rasterize` as well, whose binning cuts Gaussians at a few pixels.
"""

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "fuzzy-ellipses_gb300"))
import fuzzy_ellipses as fe  # noqa: E402

BETA2, BETA3 = 21.4, 2.66
SCALE_LO, SCALE_HI = 0.005, 0.03
MEAN_SCALE = (SCALE_HI - SCALE_LO) / math.log(SCALE_HI / SCALE_LO)


def listed():
    vga = {"h": 480, "w": 640, "f": 600.0, "spread": 0.3, "dist": 1.0}
    return [
        # One 200x200 camera of a 40-Gaussian object: the smallest call, where latency counts.
        {"name": "call_small", "kind": "call", "n": 40, "h": 200, "w": 200, "f": 200.0,
         "spread": 0.1, "dist": 0.5},
        # One 640x480 camera of a 1000-Gaussian scene: the ordinary plain call.
        {"name": "call_vga", "kind": "call", "n": 1000, **vga},
        # A dense scene at 1280x720: more Gaussians than the row-by-row binning takes, so the
        # emission and radix sort run.
        {"name": "call_large", "kind": "call", "n": 24000, "h": 720, "w": 1280, "f": 900.0,
         "spread": 0.5, "dist": 1.5},
        # One view of an optimisation loop written in torch autograd.
        {"name": "grad_small", "kind": "grad", "n": 200, "h": 128, "w": 128, "f": 128.0,
         "spread": 0.1, "dist": 0.6},
        # 16 cameras of 640x480 around one scene, in the configuration tuned for it.
        {"name": "batch_views", "kind": "batch", "scenes": 1, "views": 16, "n": 1000,
         "heavy": True, "tile": "16x16", **vga},
        # 256 uneven scenes (8 to 512 Gaussians), 1 to 8 poses each, sides 64, 128 or 256.
        {"name": "batch_scenes", "kind": "batch", "scenes": 256, "views": 0, "n": 0,
         "heavy": False, "tile": "16x16", "h": 0, "w": 0, "f": 0.0, "spread": 0.1, "dist": 0.5},
        # The 16 cameras from host memory to host memory, with the tile shape tuned for the link.
        {"name": "host_views", "kind": "host", "scenes": 1, "views": 16, "n": 1000,
         "heavy": False, "tile": "32x8", **vga},
        # The reference's optimisation step: 20 silhouettes of 128x128, 200 Gaussians.
        {"name": "step_small", "kind": "step", "views": 20, "n": 200, "h": 128, "w": 128,
         "f": 128.0, "spread": 0.1, "dist": 0.6, "heavy": False, "tile": "16x16"},
        # The same step over 16 views of 640x480 and 1000 Gaussians.
        {"name": "step_views", "kind": "step", "views": 16, "n": 1000, "heavy": True,
         "tile": "16x16", **vga},
        # Descriptors of 16 values blended into an image of odd sides.
        {"name": "features_16", "kind": "features", "n": 1000, "features": 16, "h": 479,
         "w": 637, "f": 600.0, "spread": 0.3, "dist": 1.0},
        # Every other pixel of 16 cameras as one pixel list, with flow to the neighbouring poses.
        {"name": "pixels_flow", "kind": "pixels", "n": 1000, "views": 16, "step": 2,
         "shuffled": False, **vga},
        # The reference's own call on a 640x480 camera.
        {"name": "rasterize_vga", "kind": "rasterize", "n": 1000, "h": 480, "w": 640,
         "f": 600.0},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _side(rng, lo, hi):
    return int(round(_log(rng, lo, hi)))


def draw(rng):
    kind = rng.choice(["call", "call", "grad", "batch", "batch", "host", "step", "features",
                       "pixels", "rasterize"])
    room = rng.random() < 0.5  # a table-top object, or a scene a metre away
    c = {"kind": kind, "spread": 0.3 if room else 0.1, "dist": 1.0 if room else 0.5}
    tile = rng.choice(["16x16", "16x16", "32x8", "8x8"])
    if kind in ("call", "rasterize", "features", "grad"):
        c["h"], c["w"] = _side(rng, 64, 720), _side(rng, 64, 1280)
        c["n"] = int(_log(rng, 20, 24000 if kind in ("call", "rasterize") else 4000))
        if kind == "features":
            c["features"] = int(_log(rng, 1, 65))
    else:
        c["h"], c["w"] = _side(rng, 64, 480), _side(rng, 64, 640)
        c["n"], c["views"] = int(_log(rng, 20, 2000)), int(_log(rng, 1, 33))
        if kind in ("batch", "host", "step"):
            c["tile"], c["heavy"] = tile, rng.random() < 0.5
        if kind in ("batch", "host"):
            c["scenes"] = 1
            if rng.random() < 0.5:  # uneven scenes
                c.update(scenes=int(_log(rng, 4, 256)), views=0, n=0, h=0, w=0)
        if kind == "pixels":
            c["step"], c["shuffled"] = rng.randint(1, 4), rng.random() < 0.5
    c["f"] = float(max(c["h"], c["w"]))
    # no more evaluations than the largest listed case has
    while _evaluations(c) > 1.5e8:
        if c.get("views", 0) > 1:
            c["views"] //= 2
        else:
            c["n"] = max(20, c["n"] // 2)
            c["h"], c["w"] = max(64, c["h"] * 3 // 4), max(64, c["w"] * 3 // 4)
    return c


# ---- inputs ------------------------------------------------------------------------------------

def _rotations(rng, n):
    q = rng.standard_normal((n, 4))
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    return q, _quat_to_rot(q)


def _quat_to_rot(q):
    w, x, y, z = q[:, 0], q[:, 1], q[:, 2], q[:, 3]
    return np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                     2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                     2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)],
                    1).reshape(-1, 3, 3)


def _scales(rng, n):
    return np.exp(rng.uniform(math.log(SCALE_LO), math.log(SCALE_HI), (n, 3)))


def _factor(rots, scales):
    cov = np.einsum("nij,nj,nkj->nik", rots, scales ** 2, rots)
    lower = np.linalg.inv(np.linalg.cholesky(cov))
    return np.triu(np.transpose(lower, (0, 2, 1)))


def _gaussians(rng, n, spread):
    """(means, prec, logw) as float32 arrays."""
    means = rng.uniform(-spread, spread, (n, 3))
    prec = _factor(_rotations(rng, n)[1], _scales(rng, n))
    return (means.astype(np.float32), prec.astype(np.float32),
            rng.normal(0.0, 0.5, n).astype(np.float32))


def _directions(rng, n):
    d = rng.standard_normal((n, 3))
    return d / np.linalg.norm(d, axis=1, keepdims=True)


def _look_at(centers):
    """Quaternions (scalar first) of cameras at `centers` looking at the origin."""
    f = -centers / np.linalg.norm(centers, axis=1, keepdims=True)
    up = np.where(np.abs(f[:, 2:]) > 0.99, [[0.0, 1.0, 0.0]], [[0.0, 0.0, 1.0]])
    right = np.cross(f, up)
    right /= np.linalg.norm(right, axis=1, keepdims=True)
    rot = np.stack([right, np.cross(f, right), f], 1)
    quats = []
    for r in rot:  # the quaternion's largest component first
        t = [1 + r[0, 0] + r[1, 1] + r[2, 2], 1 + r[0, 0] - r[1, 1] - r[2, 2],
             1 - r[0, 0] + r[1, 1] - r[2, 2], 1 - r[0, 0] - r[1, 1] + r[2, 2]]
        k = int(np.argmax(t))
        a, b, c = r[2, 1] - r[1, 2], r[0, 2] - r[2, 0], r[1, 0] - r[0, 1]
        d, e, g = r[1, 0] + r[0, 1], r[0, 2] + r[2, 0], r[2, 1] + r[1, 2]
        q = np.array([[t[0], a, b, c], [a, t[1], d, e], [b, d, t[2], g], [c, e, g, t[3]]][k])
        quats.append(q / np.linalg.norm(q))
    return np.array(quats).astype(np.float32)


def _cameras(rng, n, dist):
    centers = dist * _directions(rng, n)
    return _look_at(centers), centers.astype(np.float32)


def _rng(case, seed):
    return np.random.default_rng([int(seed), 20240611])


def _scene_tables(case, rng):
    """Concatenated Gaussians, the scene list and the view list of a batch; without sizes in the
    case, uneven ones."""
    parts, scenes, views, off = [], [], [], 0
    sizes = np.random.default_rng(case["scenes"])  # a plan's sizes are part of the case
    for si in range(case["scenes"]):
        if case["n"]:
            n, k, h, w, f = case["n"], case["views"], case["h"], case["w"], case["f"]
        else:
            n = int(round(math.exp(sizes.uniform(math.log(8), math.log(512)))))
            k, h = int(sizes.integers(1, 9)), int(sizes.choice([64, 128, 256]))
            w = h
            f = float(h)
        parts.append(_gaussians(rng, n, case["spread"]))
        scenes.append((off, n))
        off += n
        for q, t in zip(*_cameras(rng, k, case["dist"])):
            views.append(dict(scene=si, height=h, width=w, fx=f, fy=f, cx=w / 2, cy=h / 2,
                              quat=q, trans=t))
    return [np.concatenate(x) for x in zip(*parts)], scenes, views


def _gpu(x):
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


def _tile(case):
    w, h = case["tile"].split("x")
    return int(w), int(h)


def _pixel_rows(case, rng):
    v, u = np.mgrid[0:case["h"]:case["step"], 0:case["w"]:case["step"]]
    u, v = u.ravel() - case["w"] / 2, v.ravel() - case["h"] / 2
    rows = np.empty((case["views"], u.size, 4), np.float32)
    rows[:, :, 0], rows[:, :, 1], rows[:, :, 2] = u, v, 1.0
    rows[:, :, 3] = np.arange(case["views"])[:, None]
    rows = rows.reshape(-1, 4)
    return rows[rng.permutation(len(rows))] if case["shuffled"] else rows


def _step_inputs(case, seed):
    """Model Gaussians, views and target silhouettes of an optimisation step: the targets are the
    silhouettes (alpha > 0.5) of a scene whose jittered copy the model is."""
    rng = _rng(case, seed)
    n = case["n"]
    means = rng.uniform(-case["spread"], case["spread"], (n, 3))
    rots, scales = _rotations(rng, n)[1], _scales(rng, n)
    logw = rng.normal(0.0, 0.5, n).astype(np.float32)
    truth = means.astype(np.float32), _factor(rots, scales).astype(np.float32), logw
    model = ((means + rng.normal(0.0, 0.01, (n, 3))).astype(np.float32),
             _factor(rots, scales * rng.uniform(0.8, 1.2, (n, 3))).astype(np.float32), logw)
    quats, trans = _cameras(rng, case["views"], case["dist"])
    views = [dict(scene=0, height=case["h"], width=case["w"], fx=case["f"], fy=case["f"],
                  cx=case["w"] / 2, cy=case["h"] / 2, quat=q, trans=t)
             for q, t in zip(quats, trans)]
    truth = [_gpu(x) for x in truth]
    target = torch.cat([(_density(*truth, _camera_rays(v, torch.float32), v["trans"]) >
                         math.log(2.0)).float() for v in views])
    return [_gpu(x) for x in model], views, target


def _legacy_inputs(case, seed):
    rng = _rng(case, seed)
    n, h, w, f = case["n"], case["h"], case["w"], case["f"]
    z = rng.uniform(0.7, 1.3, n)
    means = np.stack([rng.uniform(-0.6, 0.6, n) * z, rng.uniform(-0.6, 0.6, n) * z * h / w, z], 1)
    v, u = np.mgrid[0:h, 0:w]
    rays = np.stack([(u - w / 2) / f, (v - h / 2) / f, np.ones((h, w))], -1).reshape(-1, 3)
    arrays = (means, _scales(rng, n), _rotations(rng, n)[0], rng.normal(0.0, 0.5, n), rays,
              np.eye(3), np.zeros(3))
    return [_gpu(x.astype(np.float32)) for x in arrays] + [h, w, f, f, w / 2, h / 2, 0.01, 4.5]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "rasterize":
        return kind, _legacy_inputs(case, seed)
    if kind == "step":
        gaussians, views, target = _step_inputs(case, seed)
        plan = fe.Batch([(0, case["n"])], views, tile=_tile(case), heavy_first=case["heavy"],
                        keep_binning=True)
        ends = torch.arange(1, case["views"] + 1, device="cuda") * (case["h"] * case["w"])
        stats = torch.empty(3 * plan.n_pixels, device="cuda")
        return kind, plan, gaussians, target, ends, stats
    rng = _rng(case, seed)
    if kind in ("batch", "host"):
        arrays, scenes, views = _scene_tables(case, rng)
        plan = fe.Batch(scenes, views, tile=_tile(case), heavy_first=case["heavy"])
        if kind == "batch":
            return kind, plan, [_gpu(x) for x in arrays]
        images = [torch.empty(plan.n_pixels).pin_memory() for _ in range(2)]
        return kind, plan, [torch.from_numpy(x).pin_memory() for x in arrays], images
    gaussians = [_gpu(x) for x in _gaussians(rng, case["n"], case["spread"])]
    if kind == "pixels":
        poses = np.concatenate(_cameras(rng, case["views"], case["dist"]), 1)
        return kind, gaussians, _gpu(_pixel_rows(case, rng)), 1.0 / case["f"], _gpu(poses)
    quats, trans = _cameras(rng, 1, case["dist"])
    h, w, f = case["h"], case["w"], case["f"]
    camera = (f, f, w / 2, h / 2, quats[0], trans[0], h, w)
    if kind == "features":
        return kind, gaussians, _gpu(rng.standard_normal((case["n"], case["features"]))
                                     .astype(np.float32)), camera
    if kind == "grad":
        cotangents = _cotangents(case, rng, gaussians, _view(camera))
        for x in gaussians:
            x.requires_grad_()
        return kind, gaussians, camera, cotangents
    return kind, gaussians, camera


def _cotangents(case, rng, gaussians, view):
    """Loss cotangents: a depth term where the object is seen, an alpha term everywhere."""
    h, w = case["h"], case["w"]
    seen = _density(*gaussians, _camera_rays(view, torch.float32), view["trans"]) > math.log(2.0)
    seen = seen.reshape(h, w).float()
    gd, ga = (_gpu(rng.standard_normal((h, w)).astype(np.float32)) for _ in range(2))
    return gd * seen / seen.sum().clamp(min=1.0), (ga + 0.5 * seen) / (h * w)


def run(state):
    kind = state[0]
    if kind == "call":
        _, gaussians, camera = state
        depth, alpha = fe.render_forward(*gaussians, *camera)
        return {"depth": depth, "alpha": alpha}
    if kind == "grad":
        _, gaussians, camera, cotangents = state
        depth, alpha = fe.render(*gaussians, *camera)
        gm, gp, gw = torch.autograd.grad((depth, alpha), gaussians, cotangents)
        return {"depth": depth.detach(), "alpha": alpha.detach(), "means": gm, "prec": gp,
                "logw": gw}
    if kind == "batch":
        _, plan, gaussians = state
        depth, alpha = plan.forward(*gaussians)
        return {"depth": depth, "alpha": alpha}
    if kind == "host":
        _, plan, gaussians, images = state
        depth, alpha = plan.forward_host(*gaussians, *images)
        return {"depth": depth, "alpha": alpha}
    if kind == "step":
        _, plan, gaussians, target, ends, stats = state
        depth, alpha = plan.forward(*gaussians, stats=stats)
        loss, galpha = fe.silhouette_bce(alpha, target, ends)
        gm, gp, gw = plan.backward(*gaussians, depth, alpha, stats, None, galpha)
        return {"loss": loss, "alpha": alpha, "means": gm, "prec": gp, "logw": gw}
    if kind == "features":
        _, gaussians, features, camera = state
        m, p, w = gaussians
        depth, alpha, out = fe.render_features(m, p, w, features, *camera)
        return {"depth": depth, "alpha": alpha, "features": out}
    if kind == "pixels":
        _, gaussians, rows, inv_f, poses = state
        depth, alpha, _, _, after, before = fe.render_pixels(*gaussians, rows, inv_f, poses,
                                                             flow=True)
        return {"depth": depth, "alpha": alpha, "next": after, "previous": before}
    depth, alpha = fe.rasterize(*state[1])
    return {"depth": depth, "alpha": alpha}


# ---- what a pass cannot do without -------------------------------------------------------------

def _footprint(case, n, h, w, f, views):
    """(pixel, Gaussian) pairs within the density cut-off of 1e-7, estimated from the scene's
    distribution: an ellipse of k sigma per Gaussian, the part of the cube inside the image."""
    k2 = 2.0 * math.log(1e7)
    scale = f / case["dist"]
    inside = 1.0
    for side in (h, w):
        inside *= min(1.0, side / (2 * scale * case["spread"] + 1e-9))
    area = min(float(h * w), math.pi * k2 * (MEAN_SCALE * scale) ** 2)
    return n * views * area * inside


def _sizes(case):
    """(evaluations, pixels, Gaussians) of one pass."""
    kind = case["kind"]
    if kind == "rasterize":
        n, pix = case["n"], case["h"] * case["w"]
        k = 3.0 if n <= 1000 else 0.75 if n <= 5000 else 0.5
        # the reference's focal length, from the tangent of the full field of view
        focal = case["w"] / 2 / abs(math.tan(2 * math.atan(case["w"] / 2 / case["f"])))
        radius = max(3.0, k * SCALE_HI / 2 * focal)
        return n * min(float(pix), (2 * radius + 4) ** 2), pix, n
    if kind in ("batch", "host") and not case["n"]:
        scenes, n, k = case["scenes"], 504 / math.log(64), 4.5
        pix = scenes * k * (64 ** 2 + 128 ** 2 + 256 ** 2) / 3
        each = sum(_footprint(case, n, s, s, float(s), k) for s in (64, 128, 256)) / 3
        return scenes * each, pix, scenes * n
    views = case.get("views", 1)
    pix = case["h"] * case["w"] * views
    evals = _footprint(case, case["n"], case["h"], case["w"], case["f"], views)
    if kind == "pixels":
        pix, evals = pix / case["step"] ** 2, evals / case["step"] ** 2
    return evals, pix, case["n"]


def _evaluations(case):
    return _sizes(case)[0] * (3 if case["kind"] in ("grad", "step") else
                              2 if case["kind"] == "features" else 1)


def work(case):
    evals, pix, n = _sizes(case)
    kind = case["kind"]
    # Per evaluation: 22 multiply-adds and 3 transcendentals forward, 47 and 3 backward.
    nbytes, flops = 52.0 * n + 8.0 * pix, 47.0 * evals
    if kind in ("grad", "step"):
        nbytes += 52.0 * n + (8.0 if kind == "grad" else 4.0) * pix
        flops += 97.0 * evals
    elif kind == "features":
        nbytes += 4.0 * case["features"] * (pix + n)
        flops += 2.0 * case["features"] * evals
    elif kind == "pixels":
        nbytes += (16.0 + 16.0) * pix
    elif kind == "rasterize":
        nbytes += 12.0 * pix
    return {"bytes": nbytes, "flops": flops}


# ---- the same outputs in 64 bits, from the formulas --------------------------------------------

_CHUNK = 1 << 24  # (ray, Gaussian) pairs evaluated at a time


def _camera_rays(view, dtype=torch.float64):
    h, w = view["height"], view["width"]
    v, u = torch.meshgrid(torch.arange(h, device="cuda", dtype=dtype),
                          torch.arange(w, device="cuda", dtype=dtype), indexing="ij")
    cam = torch.stack([(u - view["cx"]) / view["fx"], (v - view["cy"]) / view["fy"],
                       torch.ones_like(u)], -1).reshape(-1, 3)
    return cam @ _rotation(view["quat"], dtype)


def _rotation(quat, dtype=torch.float64):
    q = np.asarray(quat, np.float64)[None]
    return torch.from_numpy(_quat_to_rot(q / np.linalg.norm(q))[0]).to("cuda", dtype)


def _peaks(means, prec, logw, rays, center):
    """Ray parameter and log density of every Gaussian's peak along every ray: (P, N) each."""
    n = means.shape[0]
    upper = torch.triu(prec)
    t = torch.as_tensor(np.asarray(center), device="cuda", dtype=means.dtype)
    a = (rays @ upper.permute(1, 0, 2).reshape(3, 3 * n)).reshape(-1, n, 3)
    b = torch.einsum("ni,nij->nj", means - t, upper)
    vsv = a.square().sum(-1)
    psv = (a * b).sum(-1)
    z = psv / vsv
    return z, logw - 0.5 * (a * z[..., None] - b).square().sum(-1)


def _density(means, prec, logw, rays, center):
    """Sum of the Gaussians' peak densities along every ray."""
    out = torch.empty(rays.shape[0], device="cuda", dtype=means.dtype)
    rows = max(1, _CHUNK // means.shape[0])
    for i in range(0, rays.shape[0], rows):
        out[i:i + rows] = _peaks(means, prec, logw, rays[i:i + rows], center)[1].exp().sum(-1)
    return out


def _weights(z, s):
    """Softmax weights (P, N) of the Gaussians in front of the camera."""
    logit = torch.where(z > 0, BETA3 * s - BETA2 * z, torch.full_like(z, -math.inf))
    return torch.softmax(logit, -1)


def _doubles(arrays):
    return [(x if torch.is_tensor(x) else _gpu(x)).detach().double() for x in arrays]


def _view(camera):
    fx, fy, cx, cy, quat, trans, h, w = camera
    return dict(height=h, width=w, fx=fx, fy=fy, cx=cx, cy=cy, quat=quat, trans=trans)


def _exact_grad(case, seed):
    _, gaussians, camera, (gd, ga) = prepare(case, seed)
    view = _view(camera)
    params = [x.requires_grad_() for x in _doubles(gaussians)]
    rays = _camera_rays(view)
    gd, ga = gd.double().reshape(-1), ga.double().reshape(-1)
    alphas = []
    rows = max(1, _CHUNK // case["n"])
    for i in range(0, rays.shape[0], rows):
        z, s = _peaks(*params, rays[i:i + rows], view["trans"])
        alpha = -torch.expm1(-s.exp().sum(-1))
        depth = (_weights(z, s) * z).sum(-1)
        ((depth * gd[i:i + rows]).sum() + (alpha * ga[i:i + rows]).sum()).backward()
        alphas.append(alpha.detach())
    return {"depth": None, "alpha": torch.cat(alphas).reshape(case["h"], case["w"]),
            "means": params[0].grad, "prec": params[1].grad, "logw": params[2].grad}


def _exact_step(case, seed):
    gaussians, views, target = _step_inputs(case, seed)
    params = [x.requires_grad_() for x in _doubles(gaussians)]
    per = case["h"] * case["w"]
    rows = max(1, _CHUNK // case["n"])
    losses, alphas, clip = [], [], 3e-8
    for k, view in enumerate(views):
        rays, total = _camera_rays(view), 0.0
        t = target[k * per:(k + 1) * per].double()
        for i in range(0, per, rows):
            density = _peaks(*params, rays[i:i + rows], view["trans"])[1].exp().sum(-1)
            a = (-torch.expm1(-density)).clamp(clip, 1 - clip)
            ti = t[i:i + rows]
            loss = -(ti * a.log() + (1 - ti) * (1 - a).log()).sum() / per
            loss.backward()
            total += loss.detach()
            alphas.append(-torch.expm1(-density.detach()))
        losses.append(total)
    return {"loss": torch.stack(losses), "alpha": torch.cat(alphas), "means": params[0].grad,
            "prec": params[1].grad, "logw": params[2].grad}


def exact(case, seed):
    kind = case["kind"]
    if kind == "rasterize":
        return None
    if kind == "grad":
        return _exact_grad(case, seed)
    if kind == "step":
        return _exact_step(case, seed)
    rng = _rng(case, seed)
    if kind in ("batch", "host"):
        arrays, scenes, views = _scene_tables(case, rng)
        m, p, w = _doubles(arrays)
        alphas = []
        for v in views:
            o, n = scenes[v["scene"]]
            alphas.append(-torch.expm1(-_density(m[o:o + n], p[o:o + n], w[o:o + n],
                                                 _camera_rays(v), v["trans"])))
        return {"depth": None, "alpha": torch.cat(alphas)}
    state = prepare(case, seed)
    gaussians = _doubles(state[1])
    if kind == "pixels":
        rows, poses = state[2], state[4].cpu().numpy()
        alpha = torch.empty(rows.shape[0], device="cuda", dtype=torch.float64)
        for k in range(case["views"]):
            at = (rows[:, 3] == k).nonzero()[:, 0]
            cam = rows[at, :3].double() * torch.tensor([state[3], state[3], 1.0], device="cuda",
                                                       dtype=torch.float64)
            density = _density(*gaussians, cam @ _rotation(poses[k, :4]), poses[k, 4:])
            alpha[at] = -torch.expm1(-density)
        return {"depth": None, "alpha": alpha, "next": None, "previous": None}
    view = _view(state[-1])
    alpha = -torch.expm1(-_density(*gaussians, _camera_rays(view), view["trans"]))
    return {"depth": None, "alpha": alpha.reshape(case["h"], case["w"]), "features": None}
