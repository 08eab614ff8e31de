"""Performance cases of the Gaussian rasterizer: the calls a user's program
makes, over the range of sizes it makes them with.

``listed()`` names the cases, ``draw(rng)`` gives another one of the same
ranges, ``prepare`` builds what the program holds before the call (scene,
cameras, upstream gradients, all on the GPU), ``run`` is one pass through the
public entry points, ``work`` the bytes and operations no implementation can
avoid, ``exact`` the outputs in 64 bits by plain torch.

The scenes follow the benchmark's distributions (``word2world_b200.scenes``),
drawn on the GPU so that making one is quick.
"""
import math

import torch

from word2world_b200 import _C, voxel
from word2world_b200.batch import BatchRenderer, Scene, View
from word2world_b200.camera import orbit_camera, orbit_views
from word2world_b200.renderer import GaussianParams, Renderer, _render_gaussians_inline

DEV = "cuda"
PLANES = {0: 1, 1: 4, 2: 9, 3: 16}


def _render(name, kind, P, width, height, degree, views, layout):
    return {"name": name, "kind": kind, "P": P, "width": width, "height": height, "degree": degree, "views": views,
            "layout": layout}


def listed():
    return [
        # a viewer's preview of a fresh, small scene: one image, no gradients; launches and latency are all of it
        _render("preview_1k_128", "render", 1000, 128, 128, 0, 1, "shell"),
        # the trainer's step on the scene it starts from: 4 orbit views, SH degree 3, one backward
        _render("train_16k_256", "train", 16384, 256, 256, 3, 4, "shell"),
        # a step while the scene grows, image and count of no round size, a lower degree
        _render("train_50k_397x211", "train", 50021, 397, 211, 1, 1, "ball"),
        # the trainer's own frame (800 x 800) and the degree its render call passes (0)
        _render("train_100k_800", "train", 100000, 800, 800, 0, 1, "ball"),
        # the densified scene: the headline step, 4 views
        _render("train_500k_512", "train", 500000, 512, 512, 3, 4, "ball"),
        # the same scene looked at without training (validation images, turntables)
        _render("render_500k_512", "render", 500000, 512, 512, 3, 1, "ball"),
        # the largest scene and image of the multi-scene workload
        _render("train_1m_1024", "train", 1000000, 1024, 1024, 3, 1, "ball"),
        # the function on activated tensors with the forward's true derivative, a loss on colour, depth and alpha
        _render("inline_exact_30k_300x400", "inline", 30000, 300, 400, 2, 1, "ball"),
        # a serving batch: scenes of uneven size and resolution, forward and backward in one call each
        {"name": "batch_6_scenes", "kind": "batch", "P": 60000, "scenes": 6, "views": 2, "width": 256, "height": 512},
        # the sort stage as an entry point of its own
        {"name": "sort_20m", "kind": "sort", "n": 20000000, "tiles": 4096},
        # mesh extraction's occupancy field
        {"name": "voxel_64_20k", "kind": "voxel", "P": 20000, "resolution": 64, "blocks": 8, "relax": 0.1},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["render", "train", "train", "train", "inline", "batch", "sort", "voxel"])
    if kind == "sort":
        return {"kind": kind, "n": _log(rng, 50000, 20000000), "tiles": _log(rng, 64, 4096)}
    if kind == "voxel":
        return {"kind": kind, "P": _log(rng, 1000, 50000), "resolution": rng.randint(32, 96),
                "blocks": rng.randint(4, 10), "relax": round(rng.uniform(0.0, 0.3), 3)}
    if kind == "batch":
        return {"kind": kind, "P": _log(rng, 5000, 100000), "scenes": rng.randint(2, 8), "views": rng.randint(1, 3),
                "width": _log(rng, 100, 512), "height": _log(rng, 100, 512)}
    while True:
        case = {"kind": kind, "P": _log(rng, 1000, 200000 if kind == "inline" else 1000000),
                "width": _log(rng, 96, 1024), "height": _log(rng, 96, 1024), "degree": rng.randint(0, 3),
                "views": rng.choice([1, 1, 2, 4]) if kind == "train" else 1, "layout": rng.choice(["shell", "ball"])}
        if case["views"] * case["P"] * (1 + case["width"] * case["height"] / 262144) <= 4000000:
            return case


# ---- inputs -----------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _scene(P, layout, g):
    """Raw parameters (mean, sh_dc, sh_ac, opacity, svec, quaternion) as ``scenes.make_scene`` distributes them."""
    n = lambda *s: torch.randn(*s, device=DEV, generator=g)
    u = lambda *s: torch.rand(*s, device=DEV, generator=g)
    unit = torch.nn.functional.normalize(n(P, 3), dim=1)
    mean = unit * 0.5 + 0.05 * n(P, 3) if layout == "shell" else unit * (0.6 * u(P, 1).pow(1.0 / 3.0))
    return [mean, 0.5 + 0.2 * n(P, 1, 3), 0.05 * n(P, 15, 3), u(P, 1) * 4 - 2, u(P, 3) * 2 - 5,
            torch.nn.functional.normalize(n(P, 4), dim=1)]


def _camera_tensors(cam):
    t = lambda a: torch.from_numpy(a.copy()).to(DEV)
    return t(cam.viewmatrix), t(cam.projmatrix), t(cam.campos)


def _cameras(case, seed):
    return orbit_views(max(1, case["views"]), 2.5, case["width"], case["height"], azimuth0_deg=17.0 * (seed % 21))


def _batch_items(case, g, seed):
    """The scenes' raw parameters and the (scene, camera) items of a serving batch, of uneven sizes."""
    raws, items = [], []
    for s in range(case["scenes"]):
        raws.append(_scene(max(64, case["P"] * (s + 1) // case["scenes"] + 13 * s), "ball" if s % 2 else "shell", g))
        w, h = (case["width"], case["height"]) if s % 2 else (case["height"], case["height"])
        for v in range(case["views"]):
            items.append((s, orbit_camera(360.0 * v / case["views"] + 31.0 * s + seed % 7, 0.0, 2.5, w, h)))
    return raws, items


def _activated(raw):
    mean, dc, ac, opacity, svec, quat = raw
    o, s, r, sh = _C.activate(opacity, svec, quat, dc, ac)
    return mean, o, s, r, sh


def prepare(case, seed):
    g, kind = _gen(seed), case["kind"]
    if kind == "sort":
        p = torch.arange(1, case["tiles"] + 1, device=DEV, dtype=torch.float64).pow(-1.2)
        cdf = torch.cumsum(p / p.sum(), 0)
        tile = torch.searchsorted(cdf, torch.rand(case["n"], device=DEV, generator=g, dtype=torch.float64))
        depth = torch.rand(case["n"], device=DEV, generator=g) * 4 + 0.5
        keys = (tile.clamp_(max=case["tiles"] - 1) << 32) | depth.view(torch.int32).long()
        bits = 32 + max(1, (case["tiles"] - 1).bit_length())
        return {"kind": kind, "keys": keys, "vals": torch.arange(case["n"], device=DEV, dtype=torch.int32),
                "bits": bits}
    if kind == "voxel":
        return dict(_voxel_inputs(case, g), kind=kind, case=case)
    if kind == "batch":
        raws, items = _batch_items(case, g, seed)
        scenes = [Scene(*_activated(r)) for r in raws]
        views = [View(s, cam) for s, cam in items]
        grads = [torch.randn(3, cam.height, cam.width, device=DEV, generator=g) for _, cam in items]
        return {"kind": kind, "scenes": scenes, "views": views, "grads": grads,
                "renderer": BatchRenderer(reuse_buffers=True)}
    raw = _scene(case["P"], case["layout"], g)
    cams = _cameras(case, seed)
    up = [torch.randn(3, c.height, c.width, device=DEV, generator=g) for c in cams]
    state = {"kind": kind, "case": case, "cams": cams, "tensors": [_camera_tensors(c) for c in cams], "up": up}
    if kind == "inline":
        state["inputs"] = [t.detach().requires_grad_(True) for t in _activated(raw)]
        state["screen"] = torch.zeros_like(raw[0], requires_grad=True)
        state["up1"] = [torch.randn(1, case["height"], case["width"], device=DEV, generator=g) for _ in range(2)]
        state["bg"] = torch.ones(3, device=DEV)
        return state
    params = GaussianParams(*[t.requires_grad_(kind == "train") for t in raw])
    state["renderer"] = Renderer(params, sh_degree=case["degree"])
    return state


def _voxel_inputs(case, g):
    P = case["P"]
    means = torch.rand(P, 3, device=DEV, generator=g) * 2 - 1
    rot = _rotation(torch.nn.functional.normalize(torch.randn(P, 4, device=DEV, generator=g), dim=1))
    L = rot * (0.02 + 0.13 * torch.rand(P, 1, 3, device=DEV, generator=g))
    S = L @ L.transpose(1, 2)
    covs = torch.stack([S[:, 0, 0], S[:, 0, 1], S[:, 0, 2], S[:, 1, 1], S[:, 1, 2], S[:, 2, 2]], 1).contiguous()
    return {"means": means, "covs": covs, "opacities": torch.rand(P, 1, device=DEV, generator=g)}


# ---- one pass ---------------------------------------------------------------

def _view(renderer, cam, tensors):
    view, proj, campos = tensors
    return renderer.render(cam.fovx, cam.fovy, view, proj, campos, cam.width, cam.height)


def run(state):
    kind = state["kind"]
    if kind == "sort":
        keys, vals = _C.sort_pairs_u64(state["keys"], state["vals"], 0, state["bits"])
        return {"keys": keys, "vals": vals}
    if kind == "voxel":
        c = state["case"]
        return voxel.voxel_field(state["means"], state["covs"], state["opacities"], c["resolution"], c["blocks"],
                                 c["relax"])
    if kind == "batch":
        br = state["renderer"]
        res = br.forward(state["scenes"], state["views"])
        out = br.backward(res, state["grads"])
        got = {k: out[k] for k in ("means3D", "opacities", "scales", "rotations", "shs")}
        return dict(got, color=torch.cat([c.reshape(-1) for c in res.color]), radii=torch.cat(res.radii),
                    means2D=torch.cat(out["means2D"]))
    if kind == "inline":
        cam, (view, proj, campos) = state["cams"][0], state["tensors"][0]
        mean, opacity, scales, rots, shs = state["inputs"]
        color, radii, depth, alpha = _render_gaussians_inline(
            mean, state["screen"], shs, None, opacity, scales, rots, None, state["bg"], 1, view, proj, cam.tanfovx,
            cam.tanfovy, state["case"]["degree"], campos, image_height=cam.height, image_width=cam.width,
            grad_mode="exact")
        grads = torch.autograd.grad([color, depth, alpha], state["inputs"] + [state["screen"]],
                                    [state["up"][0]] + state["up1"])
        return {"color": color, "depth": depth, "alpha": alpha, "radii": radii, "grads": list(grads)}
    renderer = state["renderer"]
    if kind == "render":
        with torch.no_grad():
            out = _view(renderer, state["cams"][0], state["tensors"][0])
        return {"image": out["image"], "available": out["available_pts"]}
    outs = [_view(renderer, c, t) for c, t in zip(state["cams"], state["tensors"])]
    images = [o["image"] for o in outs]
    grads = torch.autograd.grad(images, renderer.params.parameters() + [o["accum_grads"] for o in outs], state["up"])
    return {"images": images, "available": [o["available_pts"] for o in outs], "grads": list(grads)}


# ---- what a pass cannot do without ---------------------------------------------

# A pixel in front of the scene blends Gaussians until its transmittance falls
# from 1 to 1e-4: about 64 at the scenes' mean alpha; a pair costs about 20
# operations in the forward and 60 in the backward, a Gaussian about 600 to
# project and 900 in its backward.
_PAIRS, _FWD, _BWD, _G_FWD, _G_BWD = 64, 20, 60, 600, 900


def work(case):
    kind = case["kind"]
    if kind == "sort":
        return {"bytes": 24 * case["n"], "flops": 0}
    if kind == "voxel":
        R, B = case["resolution"], case["blocks"]
        near = case["P"] * ((1 + 2 * case["relax"]) / B) ** 3
        return {"bytes": 40 * case["P"] + 4 * R ** 3, "flops": 30 * near * R ** 3}
    if kind == "batch":
        sizes = [max(64, case["P"] * (s + 1) // case["scenes"] + 13 * s) for s in range(case["scenes"])]
        px = [case["height"] * (case["width"] if s % 2 else case["height"]) for s in range(case["scenes"])]
        # parameters read and their gradients written once per scene, screen-space gradients, radii and images per view
        v = case["views"]
        return {"bytes": 4 * sum(P * (59 + 59 + 4 * v) + 6 * v * n for P, n in zip(sizes, px)),
                "flops": v * sum(P * (_G_FWD + _G_BWD) + n * _PAIRS * (_FWD + _BWD) for P, n in zip(sizes, px))}
    P, n, v = case["P"], case["width"] * case["height"], case["views"]
    read = 11 + 3 * PLANES[case["degree"]]
    if kind == "render":
        return {"bytes": 4 * (P * read + 3 * n) + P, "flops": P * _G_FWD + n * _PAIRS * _FWD}
    return {"bytes": 4 * (P * (59 + 59) + v * (3 * P + 6 * n)) + v * P,
            "flops": v * (P * (_G_FWD + _G_BWD) + n * _PAIRS * (_FWD + _BWD))}


# ---- the same in 64 bits -------------------------------------------------------

def _rotation(q):
    r, x, y, z = q.unbind(1)
    return torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - r * z), 2 * (x * z + r * y),
                        2 * (x * y + r * z), 1 - 2 * (x * x + z * z), 2 * (y * z - r * x),
                        2 * (x * z - r * y), 2 * (y * z + r * x), 1 - 2 * (x * x + y * y)], 1).view(-1, 3, 3)


def _sh_basis(x, y, z, c20):
    x2, y2, z2 = x * x, y * y, z * z
    one = torch.ones_like(x)
    return torch.stack([
        0.28209479177387814 * one, -0.4886025119029199 * y, 0.4886025119029199 * z, -0.4886025119029199 * x,
        1.0925484305920792 * x * y, -1.0925484305920792 * y * z, c20 * (2 * z2 - x2 - y2),
        -1.0925484305920792 * x * z, 0.5462742152960396 * (x2 - y2),
        -0.5900435899266435 * y * (3 * x2 - y2), 2.890611442640554 * x * y * z,
        -0.4570457994644658 * y * (4 * z2 - x2 - y2), 0.3731763325901154 * z * (2 * z2 - 3 * x2 - 3 * y2),
        -0.4570457994644658 * x * (4 * z2 - x2 - y2), 1.445305721320277 * z * (x2 - y2),
        -0.5900435899266435 * x * (x2 - 3 * y2)], 1)


def _project(mean, opacity, scales, rots, shs, view, proj, campos, focal, W, H, degree):
    """Per Gaussian: (NDC x and y, pixel position, conic, opacity, colour, depth), plus the discrete side
    (visible, 2-D covariance, determinant)."""
    R = _rotation(rots)
    S = (R * scales.square().unsqueeze(1)) @ R.transpose(1, 2)
    h = torch.cat([mean, torch.ones_like(mean[:, :1])], 1)
    t = h @ view
    tx, ty, tz = t[:, 0] / t[:, 3], t[:, 1] / t[:, 3], t[:, 2] / t[:, 3]
    rx, ry = tx / tz, ty / tz
    sq = (rx * rx + ry * ry) / (W / (2 * focal)) ** 2
    shrink = torch.where(sq > 1, torch.rsqrt(sq.clamp(min=1)), torch.ones_like(sq))
    tx, ty = rx * shrink * tz, ry * shrink * tz
    right, up, fwd = view[:3, 0], view[:3, 1], view[:3, 2]
    jx = focal * (right / tz[:, None] - tx[:, None] * fwd / tz[:, None] ** 2)
    jy = focal * (up / tz[:, None] - ty[:, None] * fwd / tz[:, None] ** 2)
    Sx, Sy = (S @ jx[:, :, None])[..., 0], (S @ jy[:, :, None])[..., 0]
    cxx, cxy, cyy = (jx * Sx).sum(1), (jx * Sy).sum(1), (jy * Sy).sum(1)
    det = cxx * cyy - cxy * cxy
    visible = (tz > 1) & (det.abs() >= 1e-8)
    det_s = torch.where(visible, det, torch.ones_like(det))
    conic = torch.stack([cyy, -cxy, cxx], 1) / det_s[:, None]
    c = h @ proj
    ndc = c[:, :3] / (c[:, 3:4] + 0.00001)
    size = torch.tensor([W, H], device=mean.device, dtype=mean.dtype)
    pix = (ndc[:, :2] + 1) * 0.5 * size - 0.5
    d = mean - campos
    d = d / d.square().sum(1, keepdim=True).sqrt()
    basis = _sh_basis(d[:, 0], d[:, 1], d[:, 2], 0.3)[:, :PLANES[degree]]
    rgb = (basis[:, :, None] * shs[:, :PLANES[degree]]).sum(1) + 0.5
    flat = torch.cat([pix, conic, opacity.reshape(-1, 1), rgb, ndc[:, 2:3]], 1)
    return ndc, flat, visible, (cxx, cyy, det), S


def _lists(flat, visible, cov, W, H):
    """Sorted tile lists: (radii, Gaussian ids, first and one-past-last entry of every tile), with the reference's
    key emission: a Gaussian writes the tiles of its integer-radius rectangle from its allocated slot on, and the
    lowest index keeps a slot that several write."""
    gw, gh = (W + 15) // 16, (H + 15) // 16
    cxx, cyy, det = cov
    mx, my, o = flat[:, 0], flat[:, 1], flat[:, 5]
    half = (cxx + cyy) * 0.5
    ymax = half + (half * half - det).clamp(min=0.1).sqrt()
    on = visible & ~(o <= 0.0039)
    mr = torch.minimum((2 * ymax * (o * 255).clamp(min=1e-30).log()).clamp(min=0).sqrt(), 3 * ymax.sqrt())
    mr = torch.where(on, mr, torch.zeros_like(mr))
    radii = torch.where(on, mr.ceil(), torch.zeros_like(mr)).long()
    low = lambda c: ((c - mr) / 16).trunc().clamp(min=0)
    top = lambda c, n: ((c + mr + 15) / 16).trunc().clamp(max=n)
    alloc = ((top(mx, gw) - low(mx)).clamp(min=0) * (top(my, gh) - low(my)).clamp(min=0)).long()
    rf = radii.double()
    x0, x1 = ((mx - rf) / 16).floor().clamp(0, gw).long(), ((mx + rf) / 16).ceil().clamp(0, gw).long()
    y0, y1 = ((my - rf) / 16).floor().clamp(0, gh).long(), ((my + rf) / 16).ceil().clamp(0, gh).long()
    emit = (x1 - x0).clamp(min=0) * (y1 - y0).clamp(min=0)
    gone = radii <= 0
    alloc, emit = alloc.masked_fill(gone, 0), emit.masked_fill(gone, 0)
    end = torch.cumsum(alloc, 0)
    total = int(end[-1])
    start = end - alloc
    reach = torch.cummax(start + emit, 0).values
    first = torch.maximum(start, torch.cat([reach.new_zeros(1), reach[:-1]]))
    count = (torch.clamp(start + emit, max=total) - first).clamp(min=0)
    ids = torch.repeat_interleave(torch.arange(len(count), device=DEV), count)
    base = torch.cumsum(count, 0) - count
    k = torch.arange(len(ids), device=DEV) - base[ids] + (first - start)[ids]
    w = (x1 - x0)[ids]
    tile = (y0[ids] + k // w) * gw + x0[ids] + k % w
    depth = flat[:, 9].float().view(torch.int32).long()[ids]
    order = torch.sort((tile << 32) | depth, stable=True).indices
    bounds = torch.searchsorted(tile[order], torch.arange(gw * gh + 1, device=DEV))
    return radii, ids[order], bounds


def _blend(flat, ids, bounds, W, H, up, clamp_grad):
    """(colour, depth, alpha) images, white background, and with ``up`` (upstream gradients of the three, None for
    none) the gradient of ``flat``; ``clamp_grad``: whether alpha's ceiling of 0.99 stops gradients."""
    gw, gh = (W + 15) // 16, (H + 15) // 16
    out = flat.new_zeros(5, gh * 16, gw * 16)
    grad = torch.zeros_like(flat)
    u = flat.new_zeros(5, gh * 16, gw * 16)
    if up is not None:
        u[:, :H, :W] = torch.cat([g.double() if g is not None else flat.new_zeros(1, H, W) for g in up])
    length = (bounds[1:] - bounds[:-1]).tolist()
    px = torch.arange(256, device=DEV)
    order = sorted(range(gw * gh), key=lambda t: -length[t])
    at = 0
    while at < len(order):
        L = max(1, length[order[at]])
        n = max(1, min(len(order) - at, 20000000 // (L * 256)))
        t = torch.tensor(order[at:at + n], device=DEV)
        at += n
        y, x = (t // gw)[:, None] * 16 + px // 16, (t % gw)[:, None] * 16 + px % 16
        pos = bounds[t][:, None] + torch.arange(L, device=DEV)
        live = pos < bounds[t + 1][:, None]
        gid = ids[pos.clamp(max=len(ids) - 1)] if len(ids) else torch.zeros_like(pos)
        e = flat[gid].detach().requires_grad_(up is not None)  # [n, L, 10]
        with torch.set_grad_enabled(up is not None):
            dx, dy = e[:, None, :, 0] - x[:, :, None], e[:, None, :, 1] - y[:, :, None]
            power = -0.5 * (e[:, None, :, 2] * dx * dx + e[:, None, :, 4] * dy * dy) - e[:, None, :, 3] * dx * dy
            power = torch.where(power > 0, power.new_tensor(-500.0), power)
            og = e[:, None, :, 5] * power.exp()
            a = og.clamp(max=0.99) if clamp_grad else og - (og - 0.99).clamp(min=0).detach()
            a = torch.where((a >= 1 / 255) & live[:, None, :], a, torch.zeros_like(a))
            with torch.no_grad():
                keep = torch.cumprod(1 - a, 2) >= 0.0001
            a = torch.where(keep, a, torch.zeros_like(a))
            T = torch.cumprod(1 - a, 2)
            wgt = a * torch.cat([torch.ones_like(T[:, :, :1]), T[:, :, :-1]], 2)
            col = wgt @ torch.cat([e[:, :, 6:10], torch.ones_like(e[:, :, :1])], 2)  # [n, 256, 5]
            res = torch.cat([col[:, :, :3] + T[:, :, -1:], col[:, :, 3:]], 2)
            if up is not None:
                (ge,) = torch.autograd.grad((res * u[:, y, x].permute(1, 2, 0)).sum(), e)
                grad.index_add_(0, gid.reshape(-1), (ge * live[:, :, None]).reshape(-1, 10))
        out[:, y, x] = res.detach().permute(2, 0, 1)
    out = out[:, :H, :W]
    return (out[:3], out[3:4], out[4:5]), grad


def _reference_backward(g, mean, scales, rots, shs, S, rgb, on, view, proj, campos, cam):
    """Per-Gaussian gradients by the reference's formulas (which are not all derivatives of its forward) from the
    gradient ``g`` of the flat 2-D values."""
    W, H = cam.width, cam.height
    g = torch.where(on[:, None], g, torch.zeros_like(g))
    m2 = torch.cat([g[:, :2] * torch.tensor([0.5 * W, 0.5 * H], device=DEV, dtype=torch.float64),
                    torch.zeros_like(g[:, :1])], 1)
    gx, gy, gz = g[:, 2], 0.5 * g[:, 3], g[:, 4]
    h = torch.cat([mean, torch.ones_like(mean[:, :1])], 1)
    v = h @ view
    p = v[:, :3] / (v[:, 3:4] + 1e-8)
    zi = 1 / p[:, 2]
    hx, hy = W / (2 * cam.tanfovx), H / (2 * cam.tanfovy)
    bx, by = 1.3 * cam.tanfovx, 1.3 * cam.tanfovy
    rx, ry = p[:, 0] * zi, p[:, 1] * zi
    px, py = rx.clamp(-bx, bx) * p[:, 2], ry.clamp(-by, by) * p[:, 2]
    inx, iny = (rx.abs() <= bx).double(), (ry.abs() <= by).double()
    right, up, fwd = view[:3, 0], view[:3, 1], view[:3, 2]
    T0 = hx * (right * zi[:, None] - fwd * (px * zi * zi)[:, None])
    T1 = hy * (up * zi[:, None] - fwd * (py * zi * zi)[:, None])
    V0, V1 = (S @ T0[:, :, None])[..., 0], (S @ T1[:, :, None])[..., 0]
    a, b, c = (T0 * V0).sum(1) + 0.3, (T0 * V1).sum(1), (T1 * V1).sum(1) + 0.3
    den = a * c - b * b
    inv = 1 / (den * den + 1e-7)
    ga = inv * (-c * c * gx + 2 * b * c * gy + (den - a * c) * gz)
    gb = inv * 2 * (b * c * gx - (den + 2 * b * b) * gy + a * b * gz)
    gc = inv * (-a * a * gz + 2 * a * b * gy + (den - a * c) * gx)
    outer = lambda s, q, r: s[:, None, None] * q[:, :, None] * r[:, None, :]
    D = outer(ga, T0, T0) + 0.5 * (outer(gb, T0, T1) + outer(gb, T1, T0)) + outer(gc, T1, T1)
    dcov = D * 2 - torch.diag_embed(torch.diagonal(D, dim1=1, dim2=2))
    gT0, gT1 = 2 * V0 * ga[:, None] + V1 * gb[:, None], 2 * V1 * gc[:, None] + V0 * gb[:, None]
    j00, j02, j11, j12 = gT0 @ right, gT0 @ fwd, gT1 @ up, gT1 @ fwd
    gv = torch.stack([inx * (-hx * zi * zi * j02), iny * (-hy * zi * zi * j12),
                      -hx * zi * zi * j00 - hy * zi * zi * j11 + 2 * zi ** 3 * (hx * px * j02 + hy * py * j12)], 1)
    dm = gv @ view[:3, :3].T
    q = h @ proj
    iw = 1 / (q[:, 3] + 1e-7)
    for k in range(2):
        dm = dm + (proj[:3, k] * iw[:, None] - proj[:3, 3] * (q[:, k] * iw * iw)[:, None]) * m2[:, k:k + 1]
    dm = dm + (view[:3, 2] - view[:3, 3] * v[:, 2:3]) * g[:, 9:10]
    cf = g[:, 6:9] * (rgb >= 0)
    rd = mean - campos
    msq = rd.square().sum(1)
    im = (msq + 1e-10).rsqrt()
    with torch.enable_grad():
        d = (rd * im[:, None]).detach().requires_grad_(True)
        basis = _sh_basis(d[:, 0], d[:, 1], d[:, 2], 0.31539156525252005)
        (ag,) = torch.autograd.grad((basis * (shs * cf[:, None, :]).sum(2)).sum(), d)
    dsh = basis.detach()[:, :, None] * cf[:, None, :]
    dm = dm + (msq[:, None] * ag - rd * (rd * ag).sum(1, keepdim=True)) * (im ** 3)[:, None]
    R = _rotation(rots)
    sx, sy, sz = scales.unbind(1)
    A = 2 * (R * scales[:, :, None]) @ torch.triu(dcov).add(torch.triu(dcov, 1).transpose(1, 2))
    dscale = (R * A).sum(2)
    w, x, y, z = rots.unbind(1)
    (a11, a12, a13), (a21, a22, a23), (a31, a32, a33) = [A[:, i].unbind(1) for i in range(3)]
    drot = 4 * torch.stack([
        -sz * (a31 * y * w - a32 * x * w + a33 * x * y) + sy * (a21 * z * w - a22 * x * z + a23 * y * y)
        + sx * (a12 * z * w - a13 * y * w - a11 * y * z),
        sz * (a31 * z * w + a32 * z * z - a33 * y * z) - sy * (a21 * y * w + a22 * x * y + a23 * x * x)
        + sx * (a12 * y * y + a13 * z * w + a11 * x * z),
        -sz * (a31 * x * x + a32 * x * w + a33 * x * z) + sy * (a21 * z * w + a22 * y * y + a23 * y * w)
        - sx * (a12 * x * w + a13 * x * x + a11 * x * y),
        sz * (a31 * x * w - a32 * x * x + a33 * x * y) - sy * (a21 * x * z - a22 * z * w + a23 * y * z)
        + sx * (a12 * y * z - a13 * z * z + a11 * y * y)], 1)
    z3 = lambda t: torch.where(on.view(-1, *[1] * (t.dim() - 1)), t, torch.zeros_like(t))
    return [z3(t) for t in (m2, dm, g[:, 5:6], dscale, drot, dsh)]


def _view64(activated, cam, degree, up=None, mode="reference"):
    """One view of activated parameters in 64 bits: images, radii and gradients
    (means2D, mean, opacity, scales, rots, shs)."""
    tensors = [t.double() for t in _camera_tensors(cam)]
    leaves = [t.double().detach().requires_grad_(mode == "exact") for t in activated]
    mean, opacity, scales, rots, shs = leaves
    ndc, flat, visible, cov, S = _project(mean, opacity, scales, rots, shs, *tensors, cam.focal_x, cam.width,
                                          cam.height, degree)
    with torch.no_grad():
        radii, ids, bounds = _lists(flat, visible, cov, cam.width, cam.height)
    images, g = _blend(flat.detach(), ids, bounds, cam.width, cam.height, up, mode == "exact")
    grads = None
    if up is not None and mode == "exact":
        grads = list(torch.autograd.grad(flat, [ndc] + leaves, g))
        grads[0] = torch.cat([grads[0][:, :2], torch.zeros_like(grads[0][:, :1])], 1)
    elif up is not None:
        grads = _reference_backward(g, mean, scales, rots, shs, S, flat[:, 6:9], radii > 0, *tensors, cam)
    return images, radii, grads


def _activate64(raw):
    mean, dc, ac, opacity, svec, quat = [t.detach().double() for t in raw]
    return mean, torch.sigmoid(opacity), svec.exp(), torch.nn.functional.normalize(quat, dim=1), torch.cat([dc, ac], 1)


def _voxel64(case, inputs):
    R, B, relax = case["resolution"], case["blocks"], case["relax"]
    # which block a voxel and a Gaussian fall in is decided in 32 bits, as the field defines it
    f = lambda v: torch.tensor(v, device=DEV, dtype=torch.float32)
    idx = torch.arange(R, device=DEV, dtype=torch.float32)
    coord = f(-1.0) + f(2.0) * idx / f(float(R - 1))
    bs = f(2.0) / f(float(B))
    blk = ((coord + f(1.0)) / bs).long().clamp(0, B)
    m, o = inputs["means"], inputs["opacities"].reshape(-1).double()
    S = inputs["covs"].double()[:, [0, 1, 2, 1, 3, 4, 2, 4, 5]].view(-1, 3, 3)
    inv = torch.linalg.inv(S)
    x = coord.double()
    out = torch.zeros(R, R, R, device=DEV, dtype=torch.float64)
    at, inside = [], []
    for b in range(B + 1):
        at.append((blk == b).nonzero()[:, 0])
        lo, hi = f(-1.0) + f(float(b)) * bs - bs * f(relax), f(-1.0) + f(float(b + 1)) * bs + bs * f(relax)
        inside.append((m >= lo) & (m <= hi))
    for bz in range(B + 1):
        for by in range(B + 1):
            for bx in range(B + 1):
                ix, iy, iz = at[bx], at[by], at[bz]
                if not (len(ix) and len(iy) and len(iz)):
                    continue
                sel = (inside[bx][:, 0] & inside[by][:, 1] & inside[bz][:, 2]).nonzero()[:, 0]
                pts = torch.stack(torch.meshgrid(x[iz], x[iy], x[ix], indexing="ij")[::-1], -1).view(-1, 1, 3)
                d = pts - m[sel].double()
                power = -0.5 * torch.einsum("vgi,gij,vgj->vg", d, inv[sel], d)
                val = (power.exp() * o[sel]).sum(1)
                out[iz[:, None, None], iy[None, :, None], ix] = val.view(len(iz), len(iy), len(ix))
    return out


def exact(case, seed):
    g, kind = _gen(seed), case["kind"]
    if kind == "sort":
        return None  # whole numbers
    if kind == "voxel":
        return _voxel64(case, _voxel_inputs(case, g))
    if kind == "batch":
        raws, items = _batch_items(case, g, seed)
        # the batch takes activated tensors: those the program holds, in 32 bits
        acts = [_activated(r) for r in raws]
        sums, cols, m2 = [None] * len(raws), [], []
        for s, cam in items:
            up = torch.randn(3, cam.height, cam.width, device=DEV, generator=g)
            images, _, grads = _view64(acts[s], cam, 3, (up, None, None))
            cols.append(images[0].reshape(-1))
            m2.append(grads[0])
            sums[s] = grads[1:] if sums[s] is None else [a + b for a, b in zip(sums[s], grads[1:])]
        got = {n: [s[i] for s in sums] for i, n in enumerate(("means3D", "opacities", "scales", "rotations", "shs"))}
        return dict(got, color=torch.cat(cols), radii=None, means2D=torch.cat(m2))
    if case["P"] * case["width"] * case["height"] > 4e11:
        return None  # the largest scenes and images take longer than a check is worth
    raw = _scene(case["P"], case["layout"], g)
    cams = _cameras(case, seed)
    up = [torch.randn(3, c.height, c.width, device=DEV, generator=g) for c in cams]
    if kind == "inline":
        up1 = [torch.randn(1, case["height"], case["width"], device=DEV, generator=g) for _ in range(2)]
        images, _, (m2, mean, opacity, scales, rots, shs) = _view64(_activated(raw), cams[0], case["degree"],
                                                                    (up[0], up1[0], up1[1]), "exact")
        return {"color": images[0], "depth": images[1], "alpha": images[2], "radii": None,
                "grads": [mean, opacity.reshape(-1, 1), scales, rots, shs, m2]}
    act = _activate64(raw)
    if kind == "render":
        return {"image": _view64(act, cams[0], case["degree"])[0][0], "available": None}
    images, screens, total = [], [], None
    for cam, u in zip(cams, up):
        img, _, grads = _view64(act, cam, case["degree"], (u, None, None))
        images.append(img[0])
        screens.append(grads[0])
        total = grads[1:] if total is None else [a + b for a, b in zip(total, grads[1:])]
    dmean, dop, dscale, drot, dsh = total
    o, s, q, n = act[1], act[2], act[3], raw[5].double().norm(dim=1, keepdim=True)
    dquat = (drot - q * (q * drot).sum(1, keepdim=True)) / n
    return {"images": images, "available": [None] * len(images),
            "grads": [dmean, dsh[:, :1], dsh[:, 1:], dop * o * (1 - o), dscale * s, dquat] + screens}
