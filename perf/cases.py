"""The work a user of trigrad_b200 has it do, as cases that can be timed and compared.

A case is one call pattern at one size: a viewer that only looks at the image, a fitting loop through autograd, a
fitting loop through the fused step, and the options beside them (packed inputs, blending in tile order, unlimited
layers, near-plane splitting).  Sizes are those of the benchmark configurations (``trigrad_b200/scenes.py``), of the
reference-style fixtures, and ragged ones between them.

Keys of a case: ``scene`` and its size (``triangles`` or ``subdivisions``), ``edge`` / ``spread`` of random triangles,
``width`` x ``height``, ``tile``, ``call`` (which entry point), ``grad`` ("none", "mse": mean squared error of the
image, "both": upstream gradients for image and depth map), ``sort`` (per_pixel_sort), ``layers`` (max_layers).
"""
from __future__ import annotations

import functools
import math

import torch

import trigrad_b200
from trigrad_b200 import scenes, views

DEV = "cuda"


def _case(name, scene, size, width, height, call, grad, edge=0.0, sigma=0.5, spread=0.0, tile=16, sort=True, layers=32,
          u8=False):
    return {"name": name, "scene": scene, "size": size, "width": width, "height": height, "call": call, "grad": grad,
            "edge": edge, "sigma": sigma, "spread": spread, "tile": tile, "sort": sort, "layers": layers, "u8": u8}


def listed():
    return [
        # the smallest calls: a unit-test sized fit (ten squares, 50x50 image, 4x4 tiles) and a thumbnail of a small
        # mesh, looked at and fitted; launches and host time decide here
        _case("fixture fit", "squares", 10, 50, 50, "render", "both", tile=4),
        _case("thumbnail view", "sphere", 3, 256, 256, "render", "none"),
        _case("thumbnail fit", "sphere", 3, 256, 256, "render", "mse"),
        # a small radiance-mesh fit with the parameters kept in the packed 16-byte layout
        _case("small fit, packed", "random", 10_000, 512, 512, "packed", "mse", edge=0.02),
        # the ordinary full-HD scene: a viewer's frame, a fitting step through autograd (the call pattern the headline
        # metric is defined on) and the same step through the fused loss
        _case("hd view", "random", 200_000, 1920, 1080, "render", "none", edge=0.005, sigma=0.7),
        _case("hd fit", "random", 200_000, 1920, 1080, "render", "mse", edge=0.005, sigma=0.7),
        _case("hd step", "random", 200_000, 1920, 1080, "step", "mse", edge=0.005, sigma=0.7),
        # one view of a multi-view optimisation of a fine mesh (triangles of about a pixel, long lists), 8-bit targets
        _case("fine mesh step", "sphere", 8, 1920, 1080, "world", "mse", u8=True),
        # the largest: two million triangles piled up in the middle of a 4K image, lists of thousands of entries
        _case("4k overlap step", "random", 2_000_000, 3840, 2160, "step", "mse", edge=0.01, spread=0.1),
        # blending in tile order, ragged image, gradients of image and depth map
        _case("tile-order fit", "random", 20_000, 1001, 777, "render", "both", edge=0.03, sort=False, layers=64),
        # no limit on the layers, with gradients that are right beyond the first batch
        _case("deep layers fit", "random", 3_000, 637, 421, "corrected", "both", edge=0.35, layers=0),
        # a camera inside the mesh: triangles are split at the near plane before they are rendered
        _case("inside view fit", "inside", 6, 1280, 720, "clip", "both"),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def image(lo, hi):
        h = log(lo, hi)
        return max(lo, min(2 * hi, int(h * rng.choice([1.0, 4 / 3, 16 / 9]) + rng.randint(0, 7)))), h

    kind = rng.choice(["mesh", "random", "random", "step", "step", "packed", "tile", "deep", "inside", "world"])
    tile = rng.choice([16, 16, 16, 8, 32])
    grad = rng.choice(["none", "mse", "both"])
    w, h = image(96, 1440)
    if kind == "mesh":
        c = _case("", "sphere", rng.randint(2, 7), w, h, "render", grad, tile=tile)
    elif kind == "world":
        c = _case("", "sphere", rng.randint(5, 8), w, h, "world", "mse", u8=rng.random() < 0.5)
    elif kind == "inside":
        c = _case("", "inside", rng.randint(4, 7), w, h, "clip", rng.choice(["mse", "both"]))
    elif kind == "deep":
        t = log(300, 4000)
        w, h = image(96, 480)
        c = _case("", "random", t, w, h, rng.choice(["corrected", "render"]), "both",
                  edge=round(math.sqrt(rng.uniform(60, 140) / t), 4), layers=0)
    else:
        t = log(1000, 800_000)
        # about one to four layers on average where the triangles are spread over the image
        edge = round(math.sqrt(rng.uniform(2, 16) / t), 5)
        spread = rng.choice([0.0, 0.0, 0.0, 0.2])
        if kind == "tile":
            t = min(t, 100_000)
            edge = round(math.sqrt(rng.uniform(4, 16) / t), 5)
            c = _case("", "random", t, w, h, "render", grad, edge=edge, sort=False, layers=rng.choice([32, 64, 0]), tile=tile)
        elif kind == "packed":
            c = _case("", "random", t, w, h, "packed", rng.choice(["mse", "both"]), edge=edge, spread=spread)
        elif kind == "step":
            c = _case("", "random", t, w, h, "step", "mse", edge=edge, spread=spread, u8=rng.random() < 0.5,
                      layers=rng.choice([32, 32, 8]))
        else:
            c = _case("", "random", t, w, h, "render", grad, edge=edge, spread=spread, tile=tile, sigma=rng.choice([0.5, 0.7]))
    del c["name"]
    return c


# ---- inputs ------------------------------------------------------------------------------------------------------


@functools.lru_cache(maxsize=8)
def _icosphere(subdivisions):
    """The mesh's topology and undisplaced positions: the same for every seed."""
    pts, faces = scenes.icosphere(subdivisions)
    return torch.from_numpy(pts.astype("float32")).to(DEV), torch.from_numpy(faces).to(DEV)


def _uniform(g, shape, lo=0.0, hi=1.0):
    return lo + (hi - lo) * torch.rand(shape, generator=g, device=DEV)


def _random_triangles(case, g):
    """Equilateral triangles of log-normal size at random places, rotations and depths (scenes.random_triangles)."""
    n = case["size"]
    if case["spread"]:
        centre = case["spread"] * torch.randn((n, 1, 2), generator=g, device=DEV)
    else:
        centre = _uniform(g, (n, 1, 2), -1.0, 1.0)
    radius = case["edge"] * torch.exp(case["sigma"] * torch.randn((n, 1), generator=g, device=DEV)) / math.sqrt(3.0)
    angle = _uniform(g, (n, 1), 0.0, 2 * math.pi) + torch.arange(3, device=DEV) * (2 * math.pi / 3)
    xy = centre + torch.stack([radius * torch.cos(angle), radius * torch.sin(angle)], dim=2)
    depth = _uniform(g, (n, 1), 0.1, 10.0) * (1 + 0.05 * _uniform(g, (n, 3), -1.0, 1.0))
    vertices = torch.cat([xy, depth[..., None], 1 / depth[..., None]], dim=2).reshape(3 * n, 4).contiguous()
    return vertices, torch.arange(3 * n, dtype=torch.int32, device=DEV).reshape(n, 3)


def _squares(case, g):
    """Concentric squares one behind the other (the overlapping-squares fixture), jittered."""
    n = case["size"]
    half = torch.linspace(0.1, 0.9, n, device=DEV) * _uniform(g, (n,), 0.95, 1.05)
    corner = torch.tensor([[-1.0, -1], [1, -1], [1, 1], [-1, 1]], device=DEV)
    xy = half[:, None, None] * corner
    depth = torch.arange(1, n + 1, device=DEV, dtype=torch.float32)[:, None, None].expand(n, 4, 1)
    vertices = torch.cat([xy, depth, 1 / depth], dim=2).reshape(4 * n, 4).contiguous()
    quad = 4 * torch.arange(n, device=DEV, dtype=torch.int32)[:, None, None]
    faces = quad + torch.tensor([[0, 1, 2], [0, 2, 3]], device=DEV, dtype=torch.int32)
    return vertices, faces.reshape(2 * n, 3).contiguous()


def _displaced_sphere(case, g):
    """Unit sphere with smooth radial bumps: sums of plane waves of random directions and phases."""
    pts, faces = _icosphere(case["size"])
    out = torch.zeros(pts.shape[0], device=DEV)
    for octave in range(4):
        k = torch.randn((3, 8), generator=g, device=DEV) * (2.0 * 2 ** octave)
        out += 0.5 ** octave * torch.sin(pts @ k + _uniform(g, (8,), 0, 2 * math.pi)).mean(dim=1)
    return (pts * (1 + 0.1 * out[:, None])).contiguous(), faces


def _camera(case, g, radius):
    a = float(_uniform(g, (1,), 0.0, 2 * math.pi))
    eye = [radius * math.sin(a), 0.0, radius * math.cos(a)]
    target = (0.0, 0.0, 0.0) if radius > 1 else (2 * math.cos(a), 0.3, -2 * math.sin(a))
    p = scenes.perspective(45.0 if radius > 1 else 75.0, 0.1 if radius > 1 else 0.02, 100.0, case["width"], case["height"])
    return (p @ scenes.lookat(eye, target)).astype("float32")


def prepare(case, seed):
    """The tensors and buffers a fitting or viewing program keeps between its calls."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    w, h = case["width"], case["height"]
    s = dict(case)
    if case["scene"] in ("random", "squares"):
        s["vertices"], s["indices"] = (_random_triangles if case["scene"] == "random" else _squares)(case, g)
        lo = 0.1
    else:
        points, s["indices"] = _displaced_sphere(case, g)
        lo = 0.3 if case["call"] == "render" else 0.1
        if case["call"] == "render":
            # small object in front of the viewer, parallel projection: depth 2 - z, as in the benchmark's first scene
            depth = 2.0 - points[:, 2:]
            s["vertices"] = torch.cat([points[:, :2] * 0.75, depth, 1 / depth], dim=1).contiguous()
        else:
            s["points"] = points
            s["pv"] = _camera(case, g, 3.0 if case["scene"] == "sphere" else 0.6)
    nv = (s["vertices"] if "vertices" in s else s["points"]).shape[0]
    s["colors"] = _uniform(g, (nv, 3))
    s["opacities"] = _uniform(g, (nv,), lo, 0.9)
    if case["grad"] == "mse":
        s["target"] = torch.rand((h, w, 4), generator=g, device=DEV)
        if case["u8"]:
            s["target"] = (s["target"] * 255).round().to(torch.uint8)
    elif case["grad"] == "both":
        s["grad_image"] = torch.randn((h, w, 4), generator=g, device=DEV)
        s["grad_depth"] = torch.randn((h, w), generator=g, device=DEV)
    if case["call"] == "packed":
        s["rgba"], s["faces"] = trigrad_b200.pack_mesh(s["colors"], s["opacities"], s["indices"])
    if case["call"] in ("step", "world"):
        s["grads"] = views.GradBuffer.allocate(nv, DEV, position_components=4 if case["call"] == "step" else 3)
        if case["call"] == "world":
            s["accumulator"] = views.PackedGradients(nv, DEV)
    elif case["grad"] != "none":
        for k in ("vertices", "points", "colors", "opacities", "rgba"):
            if k in s:
                s[k].requires_grad_()
    return s


# ---- one pass ----------------------------------------------------------------------------------------------------


def _fused_step(s):
    b = s["grads"]
    b.zero_()
    if s["call"] == "step":
        image = views.l2_view_step(s["vertices"], s["indices"], s["colors"], s["opacities"], s["target"], s["width"],
                                   s["height"], b.points, b.colors, b.opacities, b.loss, s["tile"], s["tile"],
                                   max_layers=s["layers"])
    else:
        image = views.l2_world_view_step(s["points"], s["pv"], s["indices"], s["colors"], s["opacities"], s["target"],
                                         s["width"], s["height"], b.points, b.colors, b.opacities, b.loss, s["tile"],
                                         s["tile"], max_layers=s["layers"], packed=s["accumulator"])
    return image, b.points, b.colors, b.opacities, b.loss


def run(s):
    if s["call"] in ("step", "world"):
        return _fused_step(s)
    size = (s["width"], s["height"], s["tile"], s["tile"])
    options = dict(per_pixel_sort=s["sort"], max_layers=s["layers"])
    if s["grad"] == "none":
        with torch.no_grad():
            return trigrad_b200.render(s["vertices"], s["indices"], s["colors"], s["opacities"], *size, **options)
    if s["call"] == "packed":
        leaves = (s["vertices"], s["rgba"])
        image, depth = trigrad_b200.render_packed(s["vertices"], s["faces"], s["rgba"], *size, **options)
    elif s["call"] == "clip":
        leaves = (s["points"], s["colors"], s["opacities"])
        soup = trigrad_b200.project_clip(s["points"], s["indices"], s["colors"], s["opacities"], s["pv"])
        image, depth = trigrad_b200.render(*soup, *size, **options)
    else:
        leaves = (s["vertices"], s["colors"], s["opacities"])
        function = trigrad_b200.render_corrected if s["call"] == "corrected" else trigrad_b200.render
        image, depth = function(s["vertices"], s["indices"], s["colors"], s["opacities"], *size, **options)
    if s["grad"] == "mse":
        loss = torch.mean((image - s["target"]) ** 2)
        return image, depth, loss, *torch.autograd.grad(loss, leaves)
    return image, depth, *torch.autograd.grad((image, depth), leaves, (s["grad_image"], s["grad_depth"]))


# ---- what a pass cannot do without -------------------------------------------------------------------------------


def _counts(case):
    """(triangles, vertices, blended fragments) of a case; the fragments from the mean triangle area."""
    pixels = case["width"] * case["height"]
    if case["scene"] == "random":
        t, v = case["size"], 3 * case["size"]
        area = math.sqrt(3) / 4 * (case["edge"] * math.exp(case["sigma"] ** 2)) ** 2 / 4 * pixels
        inside = pixels if not case["spread"] else min(1.0, 4 * case["spread"] ** 2) * pixels
        return t, v, min(t * area, 32 * inside)
    if case["scene"] == "squares":
        return 2 * case["size"], 4 * case["size"], 0.35 * case["size"] * pixels
    t, v = 20 * 4 ** case["size"], 10 * 4 ** case["size"] + 2
    return t, v, (1.0 if case["scene"] == "inside" else 0.6) * pixels


def work(case):
    t, v, fragments = _counts(case)
    pixels = case["width"] * case["height"]
    nbytes = 12 * t + 32 * v + 20 * pixels                          # mesh in, image and depth map out
    if case["grad"] != "none":
        upstream = 4 if case["u8"] else 16                          # target or upstream gradient of the image
        nbytes += upstream * pixels + (4 * pixels if case["grad"] == "both" else 0) + 32 * v
    # set-up of a triangle, then interpolation and blending of a fragment, and its gradient
    return {"bytes": nbytes, "flops": 120 * t + fragments * (90 if case["grad"] == "none" else 90 + 330)}


def tolerance(case):
    """Images are 32-bit sums of a few terms.  Gradients sum many pixels in no fixed order, through differences of
    nearly equal barycentric terms on small triangles: 1e-4, the bar of the parity tests, with single values of
    cancelled sums further off."""
    if case["grad"] == "none":
        return {"rel": 1e-5}
    return {"rel": 1e-4, "max": 2e-2}
