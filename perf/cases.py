"""Performance cases of the CT operators: what users have them do, over the range of sizes they do it at.

Each case is one pass through the public entry points (``rasterize_fwd`` / ``rasterize_bwd``,
``voxelize_fwd`` / ``voxelize_bwd``, the fused image and volume losses, the autograd functions,
``BatchedFit``). The fields of a case:

* ``mode``: "forward" (outputs only), "vjp" (outputs and the gradients of fixed adjoints), "fit" (image loss
  against measured projections, TV of the volume, gradients of both), "autograd" (an image loss differentiated
  through ``torch.autograd``), "batched" (several reconstructions' fit steps as one graph);
* ``n`` primitives with log-normal scales around ``scale``; ``beta``, ``uncertainty``: the Beta kernel and the
  variance branch; ``dtype``;
* ``views`` cameras on an orbit with ``height`` x ``width`` detectors (0 views: no projection);
* ``depth`` x ``vheight`` x ``vwidth`` voxels over a unit extent (0: no volume);
* ``recompute`` (autograd): rebuild the projection in the backward instead of keeping it;
* ``scenes`` (batched): reconstructions per step, of decreasing size.
"""

from __future__ import annotations

import math

import torch

import r2splat_b200 as r2s
from r2splat_b200 import autograd as r2s_autograd
from r2splat_b200 import batched, explicit, scenes
from r2splat_b200.cuda import volume_loss_fwd_bwd

LAMBDA_TV = 0.05
SCALE_SIGMA = 0.4
RASTER_TILE, VOXEL_TILE = 16, 8  # tile sizes of the explicit operators: they bound the evaluated samples
EPS = 1e-8
_NAMES = ("means", "quats", "scales", "densities", "beta", "uncertainty")


def _case(name, mode, n, *, views=0, height=0, width=0, depth=0, vheight=0, vwidth=0, scale=0.01, beta=False,
          uncertainty=False, dtype="float32", recompute=False, scenes=1):
    case = {"mode": mode, "n": n, "views": views, "height": height, "width": width, "depth": depth,
            "vheight": vheight, "vwidth": vwidth, "scale": scale, "beta": beta, "uncertainty": uncertainty,
            "dtype": dtype, "recompute": recompute, "scenes": scenes}
    return case if name is None else {"name": name, **case}


def listed():
    return [
        # The smallest fit step (the package's small configuration): launches and host work.
        _case("fit_small", "fit", 2_000, views=4, height=64, width=64, depth=32, vheight=32, vwidth=32, scale=0.03),
        # Double precision with every option on a few primitives: gradient checks and error studies.
        _case("vjp_f64_options", "vjp", 1_500, views=3, height=48, width=56, depth=24, vheight=20, vwidth=28,
              scale=0.05, beta=True, uncertainty=True, dtype="float64"),
        # Stochastic fitting: one projection a step through autograd.
        _case("one_view_autograd", "autograd", 100_000, views=1, height=512, width=512),
        # The same at a high-resolution detector, with the projection rebuilt in the backward to save memory.
        _case("one_view_recompute", "autograd", 300_000, views=1, height=1024, width=1024, scale=0.006,
              recompute=True),
        # Rendering a finished reconstruction from every view of the cone-beam orbit.
        _case("render_ct", "forward", 200_000, views=64, height=512, width=512),
        # Exporting a finished reconstruction as a volume.
        _case("export_volume", "forward", 200_000, depth=256, vheight=256, vwidth=256),
        # A variance-aware Gaussian step on a detector and a volume of odd sizes.
        _case("vjp_variance_ragged", "vjp", 50_021, views=17, height=333, width=517, depth=150, vheight=173,
              vwidth=201, scale=0.012, uncertainty=True),
        # Fitting a volume alone (distillation from a given volume), odd sizes.
        _case("volume_vjp_ragged", "vjp", 120_007, depth=301, vheight=263, vwidth=277),
        # An ordinary Beta fit step.
        _case("fit_beta", "fit", 100_000, views=32, height=384, width=384, depth=192, vheight=192, vwidth=192,
              beta=True),
        # Several small reconstructions stepped together as one graph.
        _case("batched_small", "batched", 40_000, views=16, height=256, width=256, depth=128, vheight=128, vwidth=128,
              scenes=4),
        # The full cone-beam fit step: 200,000 Gaussians, 64 views at 512^2, volume 256^3.
        _case("fit_ct", "fit", 200_000, views=64, height=512, width=512, depth=256, vheight=256, vwidth=256),
        # The largest: 500,000 Beta primitives with uncertainty, 128 views at 768^2, volume 384^3.
        _case("vjp_beta_uncertainty", "vjp", 500_000, views=128, height=768, width=768, depth=384, vheight=384,
              vwidth=384, beta=True, uncertainty=True),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    largest = work(listed()[-1])["flops"]
    while True:
        mode = rng.choice(("forward", "vjp", "fit", "fit", "autograd", "batched"))
        n = log(1_000, 500_000)
        small = mode == "batched"
        if small:
            n = min(n, 60_000)
        halves = "both" if mode in ("fit", "batched") else "raster" if mode == "autograd" else rng.choice(
            ("raster", "voxel", "both"))
        case = _case(None, mode, n)
        if halves != "voxel":
            case["views"] = 1 if mode == "autograd" else log(2, 24 if small else 128)
            case["height"], case["width"] = (log(48, 320 if small else 1024) for _ in range(2))
        if halves != "raster":
            case["depth"], case["vheight"], case["vwidth"] = (log(24, 144 if small else 384) for _ in range(3))
        # Primitives shrink as their number grows: overlapping, but not all over the volume.
        case["scale"] = round(min(0.05, 0.6 / n ** (1.0 / 3.0)) * rng.uniform(0.7, 1.2), 5)
        case["beta"] = rng.random() < 0.35
        case["uncertainty"] = mode in ("vjp", "forward") and rng.random() < 0.4
        if n < 5_000 and mode in ("vjp", "fit") and rng.random() < 0.3:
            case["dtype"] = "float64"
        if mode == "autograd":
            case["recompute"] = rng.random() < 0.5
        if small:
            case["scenes"] = rng.randint(2, 6)
        if work(case)["flops"] <= 0.6 * largest:
            return case


# --------------------------------------------------------------------------- inputs

def _phantom_projections(case, viewmats, Ks, gen, dtype):
    """Measured projections: line integrals through a few ellipsoids plus detector noise."""
    h, w, views = case["height"], case["width"], case["views"]
    dev = viewmats.device
    centres = (torch.rand((6, 3), generator=gen, device=dev) - 0.5) * 0.6
    radii = 0.08 + 0.25 * torch.rand((6, 3), generator=gen, device=dev)
    density = 0.5 + 2.0 * torch.rand((6,), generator=gen, device=dev)
    y, x = torch.meshgrid(torch.arange(h, device=dev) + 0.5, torch.arange(w, device=dev) + 0.5, indexing="ij")
    out = torch.empty((views, h, w), dtype=dtype, device=dev)
    for c in range(views):
        view, K = viewmats[c].float(), Ks[c].float()
        rot, eye = view[:3, :3], -view[:3, :3].T @ view[:3, 3]
        rays = torch.stack(((x - K[0, 2]) / K[0, 0], (y - K[1, 2]) / K[1, 1], torch.ones_like(x)), -1) @ rot
        rays = rays / rays.norm(dim=-1, keepdim=True)
        image = 0.01 * torch.randn((h, w), generator=gen, device=dev)
        for k in range(6):
            d, o = rays / radii[k], (eye - centres[k]) / radii[k]
            a, b, q = (d * d).sum(-1), (d * o).sum(-1), (o * o).sum() - 1.0
            image += density[k] * 2.0 * (b * b - a * q).clamp_min(0).sqrt() / a
        out[c] = image.to(dtype)
    return out


def _inputs(case, seed, index=0):
    """Primitives, cameras, measured projections or adjoints: made from the seed alone."""
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(1_000_003 * int(seed) + index)
    dtype = getattr(torch, case["dtype"])
    n = case["n"]

    def rand(*shape):
        return torch.rand(shape, generator=gen, device=dev, dtype=torch.float64)

    def randn(*shape):
        return torch.randn(shape, generator=gen, device=dev, dtype=torch.float64)

    p = {
        "means": rand(n, 3) - 0.5,
        "quats": randn(n, 4),
        "scales": torch.exp(math.log(case["scale"]) + SCALE_SIGMA * randn(n, 3)),
        "densities": torch.nn.functional.softplus(randn(n)),
        "beta": 0.5 + 3.5 * rand(n) if case["beta"] else None,
        "uncertainty": 0.1 * rand(n) if case["uncertainty"] else None,
    }
    state = {"case": case, "p": {k: None if v is None else v.to(dtype) for k, v in p.items()}}
    backward = case["mode"] != "forward"

    def adjoint(shape, sigma):
        return (sigma * torch.randn(shape, generator=gen, device=dev, dtype=torch.float32)).to(dtype)

    if case["views"]:
        size = (case["views"], case["height"], case["width"])
        focal = 1.171875 * max(size[1:])
        viewmats, Ks = scenes.orbit_cameras(size[0], 3.0, focal, size[2], size[1], dtype=dtype)
        state["viewmats"], state["Ks"] = viewmats.to(dev), Ks.to(dev)
        if case["mode"] in ("fit", "autograd", "batched"):
            state["target"] = _phantom_projections(case, state["viewmats"], state["Ks"], gen, dtype)
        elif backward:
            state["v_image"] = adjoint(size, 1.0)
            state["v_image_var"] = adjoint(size, 0.1) if case["uncertainty"] else None
    if case["depth"]:
        shape = (case["depth"], case["vheight"], case["vwidth"])
        state["ones"] = torch.ones(1, device=dev, dtype=dtype)
        if backward and case["mode"] == "vjp":
            state["v_volume"] = adjoint(shape, 1.0)
            state["v_volume_var"] = adjoint(shape, 0.1) if case["uncertainty"] else None
    return state


def _sub_cases(case):
    """The reconstructions of a batched case: sizes fall by a third from one to the next."""
    out = []
    for k in range(case["scenes"]):
        f = 1.0 / (1.0 + k / 2.0)
        out.append({**case, "mode": "batched", "n": max(500, int(case["n"] * f)),
                    "views": max(2, int(case["views"] * f))})
    return out


def prepare(case, seed):
    if case["mode"] != "batched":
        return _inputs(case, seed)
    fits = []
    for index, sub in enumerate(_sub_cases(case)):
        s = _inputs(sub, seed, index)
        p = s["p"]
        config = batched.SceneConfig(image_size=(sub["height"], sub["width"]),
                                     volume_shape=(sub["depth"], sub["vheight"], sub["vwidth"]), lr=1e-4)
        fits.append(batched.FitScene(p["means"], p["quats"], p["scales"], p["densities"], s["viewmats"], s["Ks"],
                                     s["target"], config, beta=p["beta"]))
    fit = batched.BatchedFit(fits)
    fit.capture()
    return {"case": case, "fit": fit}


# --------------------------------------------------------------------------- one pass

def _gradients(g):
    return {k: getattr(g, k) for k in _NAMES if getattr(g, k) is not None}


def _run_batched(state):
    fit = state["fit"]
    fit.step()
    # Updated parameters, and the first Adam moments: the running mean of all of a step's gradients.
    keys = ("loss", "means", "quats", "scales", "densities", "beta", "adam_m")
    return [{k: getattr(s, k) for k in keys if getattr(s, k) is not None} for s in fit.scenes]


def _run_autograd(state):
    case, p = state["case"], state["p"]
    leaves = {k: v.detach().requires_grad_() for k, v in p.items() if v is not None}
    image = r2s_autograd.rasterize(leaves["means"], leaves["quats"], leaves["scales"], leaves["densities"],
                                   state["viewmats"], state["Ks"], (case["height"], case["width"]),
                                   beta=leaves.get("beta"), recompute=case["recompute"])
    loss = (image - state["target"]).square().mean()
    grads = torch.autograd.grad(loss, list(leaves.values()))
    return {"image": image.detach(), "loss": loss.detach(), "grad": dict(zip(leaves, grads))}


def run(state):
    case = state["case"]
    mode = case["mode"]
    if mode == "batched":
        return _run_batched(state)
    if mode == "autograd":
        return _run_autograd(state)
    p = state["p"]
    prims = (p["means"], p["quats"], p["scales"], p["densities"])
    options = {"beta": p["beta"], "uncertainty": p["uncertainty"]}
    out, grads = {}, []
    if case["views"]:
        size = (case["height"], case["width"])
        if mode == "fit":
            image, ctx, v_image, loss, _ = explicit.rasterize_fwd_with_loss(
                *prims, state["viewmats"], state["Ks"], size, state["target"], **options)
            out["image"], out["image_loss"] = image, loss
            grads.append(r2s.rasterize_bwd(ctx, v_image))
        else:
            image, ctx = r2s.rasterize_fwd(*prims, state["viewmats"], state["Ks"], size, **options)
            out["image"] = image
            if mode == "vjp":
                out["raster"] = _gradients(r2s.rasterize_bwd(ctx, state["v_image"], state["v_image_var"]))
    if case["depth"]:
        shape = (case["depth"], case["vheight"], case["vwidth"])
        volume, ctx = r2s.voxelize_fwd(*prims, shape, volume_extent=(1.0, 1.0, 1.0), **options)
        out["volume"] = volume
        if mode == "fit":
            loss, _, v_volume = volume_loss_fwd_bwd(volume.unsqueeze(0), state["ones"], LAMBDA_TV)
            out["tv_loss"] = loss
            grads.append(r2s.voxelize_bwd(ctx, v_volume[0]))
        elif mode == "vjp":
            out["voxel"] = _gradients(r2s.voxelize_bwd(ctx, state["v_volume"], state["v_volume_var"]))
    if mode == "fit":
        a, b = (_gradients(g) for g in grads)
        out["grad"] = {k: a[k] + b[k] for k in a}
    return out


# --------------------------------------------------------------------------- necessary work

def _samples(case):
    """(projected, voxel) samples inside the primitives' supports: an ellipse or ellipsoid of three standard
    deviations (Gaussian) or of one (Beta) for each primitive and view, for the mean of the log-normal scales."""
    clip = 1.0 if case["beta"] else 3.0
    two = three = 0.0
    if case["views"]:
        focal = 1.171875 * max(case["height"], case["width"])
        sigma = case["scale"] * focal / 3.0
        two = case["n"] * case["views"] * math.pi * (clip * sigma) ** 2 * math.exp(SCALE_SIGMA ** 2)
    if case["depth"]:
        cells = case["depth"] * case["vheight"] * case["vwidth"]
        three = case["n"] * cells * 4.0 / 3.0 * math.pi * (clip * case["scale"]) ** 3 * math.exp(1.5 * SCALE_SIGMA ** 2)
    return two, three


def work(case):
    if case["mode"] == "batched":
        parts = [work({**sub, "mode": "fit"}) for sub in _sub_cases(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    size = 8 if case["dtype"] == "float64" else 4
    backward = case["mode"] != "forward"
    per = 11 + int(case["beta"]) + int(case["uncertainty"])
    planes = 1 + int(case["uncertainty"])
    pixels = case["views"] * case["height"] * case["width"]
    voxels = case["depth"] * case["vheight"] * case["vwidth"]
    values = case["n"] * per + 25 * case["views"] + planes * (pixels + voxels)
    if backward:  # the adjoints or measured projections in, the gradients out
        values += planes * pixels + (planes * voxels if case["mode"] == "vjp" else 0)
        values += case["n"] * per * (2 if case["mode"] == "vjp" and pixels and voxels else 1)
    two, three = _samples(case)
    # Contracted floating-point operations of one sample: value, and the sums of its VJP; the Beta power and its
    # logarithm count as one operation each.
    flops = two * (11 + (30 if backward else 0)) + three * (21 + (48 if backward else 0))
    return {"bytes": float(values * size), "flops": float(flops)}


# --------------------------------------------------------------------------- 64-bit values

_CHUNK = 1 << 23  # samples evaluated at once


def _covariance(quats, scales):
    w, x, y, z = (quats / quats.norm(dim=-1, keepdim=True)).unbind(-1)
    rot = torch.stack((1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                       2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                       2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)), -1).reshape(-1, 3, 3)
    return (rot * scales.square()[:, None, :]) @ rot.transpose(-1, -2)


def _span(mean, radius, tile, count):
    lo = torch.floor(mean / tile - radius / tile).clamp(0, count).long()
    hi = torch.ceil(mean / tile + radius / tile).clamp(0, count).long()
    return lo, hi


def _project(p, view, K, height, width):
    """Centre, 3x3 projected covariance and visibility of matched primitives and cameras."""
    rot = view[:, :3, :3]
    cam = (rot @ p["means"][:, :, None]).squeeze(-1) + view[:, :3, 3]
    x, y, z = cam.unbind(-1)
    visible = z > 0.01
    z = torch.where(visible, z, torch.ones_like(z))
    fx, fy, cx, cy = K[:, 0, 0], K[:, 1, 1], K[:, 0, 2], K[:, 1, 2]
    tx = z * torch.minimum(torch.maximum(x / z, -(cx + 0.15 * width) / fx), (1.15 * width - cx) / fx)
    ty = z * torch.minimum(torch.maximum(y / z, -(cy + 0.15 * height) / fy), (1.15 * height - cy) / fy)
    zero, norm = torch.zeros_like(z), (tx * tx + ty * ty + z * z).sqrt()
    jac = torch.stack((fx / z, zero, -fx * tx / z ** 2, zero, fy / z, -fy * ty / z ** 2, tx / norm, ty / norm,
                       z / norm), -1).reshape(-1, 3, 3)
    full = jac @ rot
    cov = full @ _covariance(p["quats"], p["scales"]) @ full.transpose(-1, -2)
    return fx * x / z + cx, fy * y / z + cy, cov, visible


def _profile(distance, exponent, gaussian):
    if gaussian:
        return torch.exp(-0.5 * distance)
    inside = (distance >= 0) & (distance < 1)
    base = torch.where(inside, 1 - distance, torch.ones_like(distance))
    return torch.where(inside, base.pow(exponent), torch.zeros_like(distance))


def _keep(alpha, limit, mask):
    return torch.where((alpha >= limit) & mask, alpha, torch.zeros_like(alpha))


class _Exact:
    """Projections, volumes and their VJPs in 64 bits over each primitive's tiles."""

    def __init__(self, state):
        self.case = state["case"]
        self.p = {k: None if v is None else v.detach().double() for k, v in state["p"].items()}
        self.gaussian = not self.case["beta"]
        self.clip = 3.0 if self.gaussian else 1.0
        if self.case["views"]:
            self.view, self.K = state["viewmats"].double(), state["Ks"].double()

    def _subset(self, p, n):
        return {k: None if v is None else v[n] for k, v in p.items()}

    # 2D: pairs are (camera, primitive) with the tile rectangle their integer radii cover.
    def pairs_2d(self):
        case, t = self.case, RASTER_TILE
        n, found = case["n"], []
        tx, ty = -(-case["width"] // t), -(-case["height"] // t)
        for c in range(case["views"]):
            idx = torch.arange(n, device="cuda")
            mx, my, cov, visible = _project(self.p, self.view[c].expand(n, 4, 4), self.K[c].expand(n, 3, 3),
                                            case["height"], case["width"])
            rx = torch.ceil(self.clip * (cov[:, 0, 0] + EPS).sqrt())
            ry = torch.ceil(self.clip * (cov[:, 1, 1] + EPS).sqrt())
            x0, x1 = _span(mx, rx, t, tx)
            y0, y1 = _span(my, ry, t, ty)
            ok = visible & (mx + rx > 0) & (mx - rx < case["width"]) & (my + ry > 0) & (my - ry < case["height"])
            ok &= (x1 > x0) & (y1 > y0)
            found.append(torch.stack((torch.full_like(idx, c), idx, x0, y0, x1 - x0, y1 - y0), -1)[ok])
        return torch.cat(found)

    def chunk_2d(self, p, pairs, w, h):
        """alpha [P,H,W] of pairs with w x h tiles each and the flat pixel index (out of the detector: masked)."""
        case, t = self.case, RASTER_TILE
        c, n = pairs[:, 0], pairs[:, 1]
        q = self._subset(p, n)
        mx, my, cov, _ = _project(q, self.view[c], self.K[c], case["height"], case["width"])
        cov = cov + EPS * torch.eye(3, device="cuda", dtype=torch.float64)
        a, b, d = cov[:, 0, 0], cov[:, 0, 1], cov[:, 1, 1]
        det = a * d - b * b
        p11, p12, p22 = d / det, -b / det, a / det
        e, f = cov[:, 0, 2], cov[:, 1, 2]
        ray = cov[:, 2, 2] - (p11 * e * e + 2 * p12 * e * f + p22 * f * f)
        amp = q["densities"] * torch.sqrt(2 * math.pi * ray)
        exponent = None
        if not self.gaussian:
            g = q["beta"]
            amp = amp * torch.exp(torch.lgamma(g + 1) - torch.lgamma(g + 1.5)) / math.sqrt(2.0)
            exponent = (g + 0.5)[:, None, None]
        ix = pairs[:, 2, None] * t + torch.arange(w * t, device="cuda")
        iy = pairs[:, 3, None] * t + torch.arange(h * t, device="cuda")
        dx = (ix + 0.5 - mx[:, None])[:, None, :]
        dy = (iy + 0.5 - my[:, None])[:, :, None]
        s = lambda v: v[:, None, None]  # noqa: E731
        distance = s(p11) * dx * dx + 2 * s(p12) * dx * dy + s(p22) * dy * dy
        mask = (iy < case["height"])[:, :, None] & (ix < case["width"])[:, None, :]
        pixel = (c[:, None, None] * case["height"] + iy[:, :, None]) * case["width"] + ix[:, None, :]
        return _keep(s(amp) * _profile(distance, exponent, self.gaussian), 1e-5, mask), pixel * mask, q

    # 3D: primitives with the tile box their integer radii cover.
    def _map(self, q):
        case = self.case
        dims = torch.tensor([case["vwidth"], case["vheight"], case["depth"]], device="cuda", dtype=torch.float64)
        cov = _covariance(q["quats"], q["scales"]) * (dims[:, None] * dims[None, :])
        return q["means"] * dims + 0.5 * dims, cov + EPS * torch.eye(3, device="cuda", dtype=torch.float64)

    def pairs_3d(self):
        case, t = self.case, VOXEL_TILE
        mean, cov = self._map(self.p)
        radius = torch.ceil(self.clip * torch.diagonal(cov, dim1=-2, dim2=-1).sqrt())
        counts = [-(-case[k] // t) for k in ("vwidth", "vheight", "depth")]
        lo, hi = zip(*(_span(mean[:, k], radius[:, k], t, counts[k]) for k in range(3)))
        size = [h - l for l, h in zip(lo, hi)]
        ok = (size[0] > 0) & (size[1] > 0) & (size[2] > 0)
        return torch.stack((torch.arange(case["n"], device="cuda"), *lo, *size), -1)[ok]

    def chunk_3d(self, p, pairs, w, h, d):
        case, t = self.case, VOXEL_TILE
        q = self._subset(p, pairs[:, 0])
        mean, cov = self._map(q)
        prec = torch.linalg.inv(cov)
        index = [pairs[:, 1 + k, None] * t + torch.arange(m * t, device="cuda") for k, m in enumerate((w, h, d))]
        dx, dy, dz = (index[k] + 0.5 - mean[:, k, None] for k in range(3))
        dx, dy, dz = dx[:, None, None, :], dy[:, None, :, None], dz[:, :, None, None]
        s = lambda i, j: prec[:, i, j, None, None, None]  # noqa: E731
        distance = (s(0, 0) * dx * dx + s(1, 1) * dy * dy + s(2, 2) * dz * dz + 2 * s(0, 1) * dx * dy
                    + 2 * s(0, 2) * dx * dz + 2 * s(1, 2) * dy * dz)
        exponent = None if self.gaussian else q["beta"][:, None, None, None]
        limits = (case["vwidth"], case["vheight"], case["depth"])
        inside = [index[k] < limits[k] for k in range(3)]
        mask = inside[2][:, :, None, None] & inside[1][:, None, :, None] & inside[0][:, None, None, :]
        voxel = ((index[2][:, :, None, None] * limits[1] + index[1][:, None, :, None]) * limits[0]
                 + index[0][:, None, None, :])
        alpha = q["densities"][:, None, None, None] * _profile(distance, exponent, self.gaussian)
        return _keep(alpha, 1e-6 if self.gaussian else 1e-5, mask), voxel * mask, q

    def half(self, dims, shape, adjoints=None):
        """(value, variance) over ``shape``; with ``adjoints(value, variance)`` also the gradients."""
        pairs = self.pairs_2d() if dims == 2 else self.pairs_3d()
        evaluate = self.chunk_2d if dims == 2 else self.chunk_3d
        tile = RASTER_TILE ** 2 if dims == 2 else VOXEL_TILE ** 3
        extents = pairs[:, -dims:]
        chunks = []
        for size in torch.unique(extents, dim=0).tolist():
            rows = pairs[(extents == torch.tensor(size, device="cuda")).all(-1)]
            step = max(1, _CHUNK // (math.prod(size) * tile))
            chunks += [(rows[k:k + step], size) for k in range(0, rows.shape[0], step)]
        total = math.prod(shape)
        value = torch.zeros(total, device="cuda", dtype=torch.float64)
        variance = torch.zeros_like(value) if self.case["uncertainty"] else None
        with torch.no_grad():
            for rows, size in chunks:
                alpha, where, q = evaluate(self.p, rows, *size)
                value.index_add_(0, where.reshape(-1), alpha.reshape(-1))
                if variance is not None:
                    u = q["uncertainty"].reshape(-1, *([1] * dims))
                    variance.index_add_(0, where.reshape(-1), (u * alpha * alpha).reshape(-1))
        value = value.reshape(shape)
        variance = None if variance is None else variance.reshape(shape)
        if adjoints is None:
            return value, variance, None
        v, vv = adjoints(value)
        v, vv = v.reshape(-1), None if vv is None else vv.reshape(-1)
        leaves = {k: None if x is None else x.detach().clone().requires_grad_() for k, x in self.p.items()}
        for rows, size in chunks:
            alpha, where, q = evaluate(leaves, rows, *size)
            total = (v[where] * alpha).sum()
            if vv is not None:
                total = total + (vv[where] * q["uncertainty"].reshape(-1, *([1] * dims)) * alpha * alpha).sum()
            total.backward()
        return value, variance, {k: x.grad for k, x in leaves.items() if x is not None}


def _tv(volume):
    """(lambda times the mean absolute difference, its gradient)."""
    edges = sum(volume.numel() // volume.shape[k] * (volume.shape[k] - 1) for k in range(3))
    grad, loss = torch.zeros_like(volume), 0.0
    for k in range(3):
        diff = volume.diff(dim=k)
        loss = loss + diff.abs().sum()
        m = volume.shape[k] - 1
        grad.narrow(k, 1, m).add_(diff.sign())
        grad.narrow(k, 0, m).sub_(diff.sign())
    return LAMBDA_TV * loss / max(edges, 1), grad * (LAMBDA_TV / max(edges, 1))


def _tile_samples(case):
    """About how many samples the tiles that the primitives' radii cover hold: what is evaluated here."""
    clip, total = 1.0 if case["beta"] else 3.0, 0.0
    if case["views"]:
        reach = 2.0 * clip * case["scale"] * 1.171875 * max(case["height"], case["width"]) / 3.0
        total += case["n"] * case["views"] * (reach + 1.5 * RASTER_TILE) ** 2
    if case["depth"]:
        total += case["n"] * math.prod(2.0 * clip * case["scale"] * case[k] + 1.5 * VOXEL_TILE
                                       for k in ("depth", "vheight", "vwidth"))
    return total


def exact(case, seed):
    if case["mode"] == "batched" or _tile_samples(case) > 2.5e10:
        return None
    state = _inputs(case, seed)
    e = _Exact(state)
    mode, out, grads = case["mode"], {}, []

    def put(key, value, variance):
        out[key] = value if variance is None else (value, variance)

    if case["views"]:
        shape = (case["views"], case["height"], case["width"])
        if mode in ("fit", "autograd"):
            target = state["target"].double()
            adjoints = lambda image: (2.0 * (image - target) / image.numel(), None)  # noqa: E731
        else:
            adjoints = (lambda image: tuple(None if v is None else v.double() for v in (
                state["v_image"], state["v_image_var"]))) if mode == "vjp" else None
        image, variance, g = e.half(2, shape, adjoints)
        put("image", image, variance)
        if mode in ("fit", "autograd"):
            out["image_loss" if mode == "fit" else "loss"] = (image - target).square().mean()
            grads.append(g)
        elif mode == "vjp":
            out["raster"] = g
    if case["depth"]:
        shape = (case["depth"], case["vheight"], case["vwidth"])
        if mode == "fit":
            adjoints = lambda volume: (_tv(volume)[1], None)  # noqa: E731
        else:
            adjoints = (lambda volume: tuple(None if v is None else v.double() for v in (
                state["v_volume"], state["v_volume_var"]))) if mode == "vjp" else None
        volume, variance, g = e.half(3, shape, adjoints)
        put("volume", volume, variance)
        if mode == "fit":
            out["tv_loss"] = _tv(volume)[0]
            grads.append(g)
        elif mode == "vjp":
            out["voxel"] = g
    if grads:
        out["grad"] = {k: sum(g[k] for g in grads) for k in grads[0]}
    return out
