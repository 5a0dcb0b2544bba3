"""GPU tests of the public Python entry point (``trigrad_b200.render``) and of the reference leg.

``render`` is exercised the way the reference's own tests call ``trigrad.render``: tensors in, autograd
out.  Results are compared with the CPU oracle, with the golden vectors recorded from the reference's
CUDA build and, when that build is present on the machine, with the reference itself run live.
"""
import os
import sys

import numpy as np
import pytest
import torch

import helpers as Hh
import oracle as O
import trigrad_b200
from trigrad_b200 import scenes as S

pytestmark = pytest.mark.gpu

GOLDEN_DIR = os.path.join(os.path.dirname(__file__), "golden")
sys.path.insert(0, GOLDEN_DIR)
import make_golden as MG  # noqa: E402

GOLDEN = MG.golden_scenes()


def run_render(sc, mode, gi, gd):
    v, i, c, o = Hh.scene_tensors(sc)
    v.requires_grad_(), c.requires_grad_(), o.requires_grad_()
    image, depth = trigrad_b200.render(v, i, c, o, sc.width, sc.height, sc.tile_width, sc.tile_height, mode["thr"],
                                       False, mode["per_pixel_sort"], mode["max_layers"])
    d0 = torch.where(torch.isfinite(depth), depth, torch.zeros_like(depth))
    ((image * Hh.cuda(gi)).sum() + (d0 * Hh.cuda(gd)).sum()).backward()
    return (image.detach().cpu().numpy(), depth.detach().cpu().numpy(), v.grad.cpu().numpy(), c.grad.cpu().numpy(),
            o.grad.cpu().numpy())


@pytest.mark.parametrize("name", list(GOLDEN))
def test_render_matches_reference_golden(name):
    """The product path against vectors recorded from the reference's own CUDA build."""
    sc, mode = GOLDEN[name]
    g = np.load(os.path.join(GOLDEN_DIR, name + ".npz"))
    gi, gd = MG.upstream(sc)
    image, depth, gV, gC, gO = run_render(sc, mode, gi, gd)
    npx = sc.width * sc.height
    diff = np.abs(image.astype(np.float64) - g["image"]).max(axis=2)
    flips = diff > 1e-3
    assert int(flips.sum()) <= max(4, int(5e-4 * npx))
    keep = ~flips
    assert Hh.rel_l2(image[keep], g["image"][keep]) <= 1e-5
    assert np.array_equal(np.isfinite(depth), np.isfinite(g["depthmap"]))
    fin = np.isfinite(depth) & keep
    assert Hh.rel_l2(depth[fin], g["depthmap"][fin]) <= 1e-5
    if mode["per_pixel_sort"] or "layers" in name:
        assert Hh.rel_l2(gV, g["grad_vertices"]) <= 1e-4
        assert Hh.rel_l2(gC, g["grad_colors"]) <= 1e-4
        assert Hh.rel_l2(gO, g["grad_opacities"]) <= 1e-4


def test_render_autograd_matches_oracle_on_config1():
    sc = S.config1_icosphere()
    mode = dict(thr=1 / 256, per_pixel_sort=True, max_layers=32)
    rng = np.random.default_rng(5)
    gi = rng.normal(size=(sc.height, sc.width, 4)).astype(np.float32)
    gd = rng.normal(size=(sc.height, sc.width)).astype(np.float32)
    image, depth, gV, gC, gO = run_render(sc, mode, gi, gd)
    of = O.forward(sc.vertices, sc.indices, sc.colors, sc.opacities, sc.width, sc.height)
    og = O.backward(sc.vertices, sc.indices, sc.colors, sc.opacities, sc.width, sc.height, of, gi, gd)
    assert np.array_equal(image.view(np.uint32), of.image.view(np.uint32))
    assert np.array_equal(depth.view(np.uint32), of.depthmap.view(np.uint32))
    for a, b in zip((gV, gC, gO), og):
        assert Hh.rel_l2(a, b) <= 1e-4


def test_l2_loss_step_matches_oracle_step():
    """The benchmark's step (mean squared error against a seeded target) on config 2."""
    sc = S.config2_random10k()
    v, i, c, o = Hh.scene_tensors(sc)
    v.requires_grad_(), c.requires_grad_(), o.requires_grad_()
    image, _ = trigrad_b200.render(v, i, c, o, sc.width, sc.height)
    loss = torch.mean((image - Hh.cuda(sc.target())) ** 2)
    loss.backward()
    oloss, of, og = O.render_l2(sc)
    assert abs(float(loss.detach()) - oloss) <= 1e-6 * oloss
    for a, b in zip((v.grad, c.grad, o.grad), og):
        assert Hh.rel_l2(a.cpu().numpy(), b) <= 1e-4


def test_record_timing_contract():
    sc = S.config1_icosphere()
    v, i, c, o = Hh.scene_tensors(sc)
    out = trigrad_b200.render(v, i, c, o, sc.width, sc.height, record_timing=True)
    assert len(out) == 3
    assert set(out[2]) == {"init", "per_tile_lists", "sorting", "bary_transforms", "rasterization"}
    assert all(isinstance(t, float) and t >= 0 for t in out[2].values())


def test_zero_triangles_fast_path():
    v = torch.zeros((3, 4), device="cuda", requires_grad=True)
    c = torch.zeros((3, 3), device="cuda", requires_grad=True)
    o = torch.zeros((3,), device="cuda", requires_grad=True)
    i = torch.zeros((0, 3), dtype=torch.int32, device="cuda")
    image, depth = trigrad_b200.render(v, i, c, o, 40, 24)
    assert torch.all(image[..., 3] == 1) and torch.all(image[..., :3] == 0) and torch.all(torch.isinf(depth))
    (image.sum()).backward()
    assert torch.all(v.grad == 0) and torch.all(c.grad == 0) and torch.all(o.grad == 0)


def test_shape_and_dtype_errors():
    sc = S.large_triangles(2)
    v, i, c, o = Hh.scene_tensors(sc)
    with pytest.raises(ValueError):
        trigrad_b200.render(v[:, :3].contiguous(), i, c, o, 32, 32)
    with pytest.raises(TypeError):
        trigrad_b200.render(v.double(), i, c, o, 32, 32)
    with pytest.raises(TypeError):
        trigrad_b200.render(v, i.long(), c, o, 32, 32)
    with pytest.raises(ValueError):
        trigrad_b200.render(v, i, c, o, 64, 64, 64, 64)


@pytest.mark.parametrize("tile", [(0, 16), (16, 0), (0, 0), (-16, 16), (-4, -4), (2 ** 32 + 16, 16), (2 ** 33, 2 ** 33)])
def test_every_entry_point_rejects_tiles_that_are_none(tile):
    from trigrad_b200 import views
    sc = S.large_triangles(2)
    v, i, c, o = Hh.scene_tensors(sc)
    rgba, faces = trigrad_b200.pack_mesh(c, o, i)
    target = torch.rand((32, 32, 4), device="cuda")
    b4, b3 = (views.GradBuffer.allocate(v.shape[0], "cuda", p) for p in (4, 3))
    pv = np.eye(4, dtype=np.float32)
    for call in (lambda: trigrad_b200.render(v, i, c, o, 32, 32, *tile),
                 lambda: trigrad_b200.render_corrected(v, i, c, o, 32, 32, *tile),
                 lambda: trigrad_b200.render_packed(v, faces, rgba, 32, 32, *tile),
                 lambda: trigrad_b200.Renderer.apply(v, i, c, o, 32, 32, *tile),
                 lambda: views.l2_view_step(v, i, c, o, target, 32, 32, b4.points, b4.colors, b4.opacities, b4.loss, *tile),
                 lambda: views.l2_world_view_step(v[:, :3].contiguous(), pv, i, c, o, target, 32, 32, b3.points, b3.colors,
                                                  b3.opacities, b3.loss, *tile)):
        with pytest.raises(ValueError):
            call()
    if max(tile) < 2 ** 31:                  # a mesh without triangles is not binned
        assert trigrad_b200.render(v, i[:0], c, o, 32, 32, *tile)[0].shape == (32, 32, 4)


@pytest.mark.parametrize("triangles", [0, 2])
def test_fused_steps_check_a_mesh_without_triangles_like_any_other(triangles):
    from trigrad_b200 import views
    v, i, c, o = Hh.scene_tensors(S.large_triangles(2))
    i = i[:triangles]
    target = torch.rand((24, 32, 4), device="cuda")

    def step(positions=v, indices=i, colors=c, opacities=o, target=target, tile=16, **k):
        b = views.GradBuffer.allocate(v.shape[0], "cuda", 4)
        views.l2_view_step(positions, indices, colors, opacities, target, 32, 24, b.points, b.colors, b.opacities, b.loss, tile, 16, **k)
        return float(b.loss)

    def world(positions=v[:, :3].contiguous(), pv=np.eye(4), indices=i, colors=c, opacities=o, target=target, tile=16, **k):
        b = views.GradBuffer.allocate(v.shape[0], "cuda", 3)
        views.l2_world_view_step(positions, pv, indices, colors, opacities, target, 32, 24, b.points, b.colors, b.opacities, b.loss,
                                 tile, 16, **k)
        return float(b.loss)

    for call in (step, world):
        assert call() > 0
        assert call(target=(target * 255).to(torch.uint8)) > 0
        for bad in (dict(target=target[:23]), dict(target=target[..., :3].contiguous()), dict(indices=i[:, :2]),
                    dict(tile=65), dict(colors=c[:1]), dict(opacities=o[:, None]), dict(max_layers=0),
                    dict(target=(target * 255).to(torch.uint8), one_kernel=True)):
            with pytest.raises(ValueError):
                call(**bad)
        for bad in (dict(indices=i.long()), dict(target=target.double()), dict(target=target.cpu()), dict(indices=i.cpu()),
                    dict(positions=v.double())):
            with pytest.raises(TypeError):
                call(**bad)
    with pytest.raises(ValueError):
        world(pv=np.eye(3))
    if not triangles:
        with pytest.raises(ValueError):
            step(packed=views.PackedGradients(v.shape[0], "cuda"))


@pytest.mark.parametrize("which", range(4))
def test_gradient_tensors_that_kernels_add_to_are_checked(which):
    from trigrad_b200 import views
    v, i, c, o = Hh.scene_tensors(S.large_triangles(2))
    V, target, points, pv = v.shape[0], torch.rand((24, 32, 4), device="cuda"), v[:, :3].contiguous(), np.eye(4)
    packed = views.PackedGradients(V, "cuda")
    for p, call in ((4, lambda *g: views.l2_view_step(v, i, c, o, target, 32, 24, *g)),
                    (4, lambda *g: views.l2_view_step(v, i, c, o, target, 32, 24, *g, one_kernel=True)),
                    (3, lambda *g: views.l2_world_view_step(points, pv, i, c, o, target, 32, 24, *g)),
                    (3, lambda *g: views.l2_world_view_step(points, pv, i, c, o, target, 32, 24, *g, packed=packed)),
                    (4, lambda *g: packed.unpack(32, 24, *g))):
        b = views.GradBuffer.allocate(V, "cuda", p)
        good = [b.points, b.colors, b.opacities, b.loss]
        call(*good)
        t = good[which]
        bad = [t.double(), t.cpu(), t.flatten()[:-1]]
        if t.dim():
            bad.append(t.repeat_interleave(2, dim=0)[::2])
        for x in bad:
            with pytest.raises((TypeError, ValueError)):
                call(*good[:which], x, *good[which + 1:])
    with pytest.raises(ValueError):
        views.project_backward_native(points, pv, torch.zeros_like(v), torch.zeros((3, V), device="cuda").t())


def test_capacity_regrow_and_reuse():
    """A small scene first, then one with far more (triangle, tile) pairs, then the small one again."""
    small, big = S.large_triangles(2), S.full_screen_layers(50, width=640, height=480)
    for sc in (small, big, small):
        v, i, c, o = Hh.scene_tensors(sc)
        image, _ = trigrad_b200.render(v, i, c, o, sc.width, sc.height, sc.tile_width, sc.tile_height)
        of = O.forward(sc.vertices, sc.indices, sc.colors, sc.opacities, sc.width, sc.height, sc.tile_width,
                       sc.tile_height)
        assert np.array_equal(image.cpu().numpy().view(np.uint32), of.image.view(np.uint32))


def test_non_contiguous_inputs():
    sc = S.config1_icosphere(width=96, height=96)
    v, i, c, o = Hh.scene_tensors(sc)
    vv = torch.zeros((v.shape[0], 8), device="cuda")[:, ::2]
    vv.copy_(v)
    assert not vv.is_contiguous()
    a, _ = trigrad_b200.render(vv, i, c, o, 96, 96)
    b, _ = trigrad_b200.render(v, i, c, o, 96, 96)
    assert torch.equal(a, b)


@pytest.mark.parametrize("tile,one_kernel", [(16, False), (16, True), (32, True)],
                         ids=["two_kernels", "one_kernel", "one_kernel_asked_with_big_tiles"])
def test_fused_l2_view_step_matches_autograd(tile, one_kernel):
    """views.l2_view_step (accumulating; forward + loss-fused backward, or both directions in one compositing
    kernel, which tiles of more than 256 pixels cannot use) against render() + torch autograd."""
    from trigrad_b200 import views
    sc = S.config2_random10k()
    sc.tile_width = sc.tile_height = tile
    V = sc.num_vertices
    gV = torch.zeros((V, 4), device="cuda")
    gC = torch.zeros((V, 3), device="cuda")
    gO = torch.zeros((V,), device="cuda")
    loss = torch.zeros((), device="cuda")
    refs = [torch.zeros_like(gV), torch.zeros_like(gC), torch.zeros_like(gO)]
    ref_loss = 0.0
    rng = np.random.default_rng(17)
    for k in range(2):                                     # two views: accumulation across calls
        verts = sc.vertices.copy()
        verts[:, 0] += 0.01 * k
        target = Hh.cuda(rng.random((sc.height, sc.width, 4), dtype=np.float32))
        v, i, c, o = Hh.cuda(verts), Hh.cuda(sc.indices), Hh.cuda(sc.colors), Hh.cuda(sc.opacities)
        img = views.l2_view_step(v, i, c, o, target, sc.width, sc.height, gV, gC, gO, loss, tile, tile,
                                 one_kernel=one_kernel)
        vv, cc, oo = v.clone().requires_grad_(), c.clone().requires_grad_(), o.clone().requires_grad_()
        image, _ = trigrad_b200.render(vv, i, cc, oo, sc.width, sc.height, tile, tile)
        assert torch.equal(image, img)
        l = torch.mean((image - target) ** 2)
        g = torch.autograd.grad(l, (vv, cc, oo))
        for r, x in zip(refs, g):
            r += x
        ref_loss += float(l)
    torch.cuda.synchronize()
    assert abs(float(loss) - ref_loss) <= 1e-5 * ref_loss
    for a, b in zip((gV, gC, gO), refs):
        assert Hh.rel_l2(a.cpu().numpy(), b.cpu().numpy()) <= 1e-5


def test_negated_views_are_read_as_what_they_are():
    """The imaginary part of a conjugate is a view with a flag; kernels see memory."""
    from trigrad_b200 import views
    sc = S.random_triangles(300, 64, 48, 0.3, 0.4, name="negated", seed=1)
    v, i, c, o = Hh.scene_tensors(sc)

    def negated(t):
        n = torch.complex(torch.zeros_like(t), -t).conj().imag
        assert n.is_neg() and torch.equal(n, t)
        return n

    image, depth = trigrad_b200.render(v, i, c, o, 64, 48)
    for call in (trigrad_b200.render, trigrad_b200.render_corrected, trigrad_b200.Renderer.apply):
        out = call(negated(v), i, negated(c), negated(o), 64, 48)
        assert torch.equal(out[0], image) and torch.equal(out[1], depth)
    x = [t.requires_grad_() for t in (v, c, o)]
    out = trigrad_b200.render(v, i, c, o, 64, 48)
    up = [torch.randn_like(t) for t in out]
    want = torch.autograd.grad(out, x, up, retain_graph=True)
    for a, b in zip(torch.autograd.grad(out, x, [negated(t) for t in up]), want):
        assert Hh.rel_l2(a.cpu().numpy(), b.cpu().numpy()) <= 1e-5      # order of atomics
    target = torch.rand_like(image)
    steps = []
    for t in (target, negated(target)):
        b = views.GradBuffer.allocate(v.shape[0], "cuda", 4)
        views.l2_view_step(v.detach(), i, c.detach(), o.detach(), t, 64, 48, b.points, b.colors, b.opacities, b.loss)
        steps.append(b.flat.cpu().numpy())
    assert Hh.rel_l2(*steps) <= 1e-5
    pv = S.camera_ring(8)[1]
    points = v.detach()[:, :3].contiguous()
    for a, b in zip(trigrad_b200.project_clip(negated(points), i, negated(c.detach()), o.detach(), pv),
                    trigrad_b200.project_clip(points, i, c.detach(), o.detach(), pv)):
        assert torch.equal(a, b)
    assert torch.equal(views.project_native(negated(points), pv), views.project_native(points, pv))


def _reference():
    import build_ref
    try:
        return build_ref.load()
    except Exception:
        return None


@pytest.mark.parametrize("make,sort", [(S.config2_random10k, True), (S.config1_icosphere, True),
                                       (lambda: S.config5_overlap(T=4000, width=320, height=192), True),
                                       (lambda: S.full_screen_layers(60, width=48, height=40), False)])
def test_live_reference_leg(make, sort):
    """Same inputs through the reference's own CUDA build (when present on this machine) and the product."""
    ref = _reference()
    if ref is None:
        pytest.skip("reference build (oracle/_ref) not present")
    sc = make()
    mode = dict(thr=1 / 256, per_pixel_sort=sort, max_layers=32 if sort else 61)
    rng = np.random.default_rng(7)
    gi = rng.normal(size=(sc.height, sc.width, 4)).astype(np.float32)
    gd = rng.normal(size=(sc.height, sc.width)).astype(np.float32)
    v, i, c, o = Hh.scene_tensors(sc)
    r_img, r_depth, r_fw, r_ids, r_off, r_bary, r_ends, _ = ref.render_forward(
        v, i, c, o, sc.width, sc.height, sc.tile_width, sc.tile_height, mode["thr"], True, sort, mode["max_layers"])
    torch.cuda.synchronize()
    from trigrad_b200 import wrapper as Wr
    fwd = Wr.forward_native(v, i, c, o, sc.width, sc.height, sc.tile_width, sc.tile_height, mode["thr"], False, sort,
                            mode["max_layers"])
    image, ends = fwd[0].cpu().numpy(), fwd[7].cpu().numpy()
    # Pixels where the two builds decide differently blend different fragments: a pixel centre on a shared edge
    # (the number of blended fragments differs) or two fragments a few ulp apart in depth (the image differs by
    # far more than rounding).  Their upstream gradient is zeroed on BOTH sides so that the gradient comparison
    # below always runs and covers every other pixel.
    r_image = r_img.cpu().numpy()
    diff = np.abs(image.astype(np.float64) - r_image).max(axis=2)
    flips = (diff > 1e-3) | (ends != r_ends.cpu().numpy())
    # exact-arithmetic yardstick: the fp64 oracle on the same inputs (its own decisions, so pixels where IT blends
    # other fragments than the fp32 builds are set aside as well, outside the flip budget)
    v64, c64, o64 = (np.asarray(x, np.float64) for x in (sc.vertices, sc.colors, sc.opacities))
    of64 = O.forward(v64, sc.indices, c64, o64, sc.width, sc.height, sc.tile_width, sc.tile_height, mode["thr"], sort,
                     mode["max_layers"])
    aside = flips | (of64.ends != ends)
    gi[aside] = 0
    gd[aside] = 0
    r_gV, r_gC, r_gO = ref.render_backward(Hh.cuda(gi), Hh.cuda(gd), v, i, c, o, r_ids, r_off, r_bary, r_img, r_depth,
                                           r_fw, r_ends, sc.width, sc.height, sc.tile_width, sc.tile_height, mode["thr"],
                                           sort, mode["max_layers"])
    torch.cuda.synchronize()
    image, depth, gV, gC, gO = run_render(sc, mode, gi, gd)
    # binning objects: tile ranges bit-exact, lists equal per tile as multisets
    tens = Hh.scene_tensors(sc)
    counts, _, geo, attr = Hh.preprocess(sc, tens)
    tri_off = Hh.scan(counts)
    K = int(tri_off[-1])
    keys, ids = Hh.emit_keys(sc, tri_off, K, tens)
    tiles = Hh.num_tiles(sc)
    skeys, sids = Hh.sort_pairs(keys, ids, 0, 32 + int(np.ceil(np.log2(tiles))))
    off = Hh.tile_ranges(skeys, tiles).cpu().numpy()
    assert np.array_equal(off, r_off.cpu().numpy())
    mine, theirs = sids.cpu().numpy(), r_ids.cpu().numpy()
    for t in range(tiles):
        assert np.array_equal(np.sort(mine[off[t]:off[t + 1]]), np.sort(theirs[off[t]:off[t + 1]]))
    # image and gradients
    npx = sc.width * sc.height
    assert int(flips.sum()) <= max(4, int(5e-4 * npx))
    # Both builds evaluate barycentrics as M*(px,py,1) in fp32; that evaluation carries an absolute
    # error of about eps*(|m0|+|m1|+|m2|) per coordinate, which grows as triangles shrink, and the
    # reference's FMA placement is compiler-chosen.  The bar is 1e-5 where the problem is well
    # conditioned and the conditioning bound otherwise.
    kappa = float(np.median(np.abs(geo.cpu().numpy()[:, :9]).reshape(-1, 3, 3).sum(axis=2)))
    tol = max(1e-5, 4 * 2.0 ** -24 * kappa)
    img_err = Hh.rel_l2(image[~flips], r_image[~flips])
    assert img_err <= tol
    refs = [x.cpu().numpy() for x in (r_gV, r_gC, r_gO)]
    errs = {n: Hh.rel_l2(a, b) for n, a, b in zip(("vertices", "colors", "opacities"), (gV, gC, gO), refs)}
    # How far is each fp32 build from exact arithmetic?  Two differently compiled fp32 evaluations of the same
    # formulas cannot agree better than each of them agrees with the exact result, so the bar of 1e-4 is widened
    # to the reference build's own distance from the fp64 oracle where that is larger (small triangles: the
    # expanded barycentric partials of util.h:415-443 cancel in fp32).  Only in the default mode: outside it the
    # reference's backward is not the gradient and the oracle restates it literally.
    truth = O.backward(v64, sc.indices, c64, o64, sc.width, sc.height, of64, gi.astype(np.float64), gd.astype(np.float64),
                       sc.tile_width, sc.tile_height, sort, mode["max_layers"])
    ref_noise = {n: Hh.rel_l2(b, t) for n, b, t in zip(errs, refs, truth)}
    own_noise = {n: Hh.rel_l2(a, t) for n, a, t in zip(errs, (gV, gC, gO), truth)}
    path = os.environ.get("TG_PARITY_REPORT")
    if path:
        import json
        with open(path, "a") as f:
            f.write(json.dumps(dict(test="live_reference", scene=sc.name, per_pixel_sort=bool(sort), pixels=npx,
                                    flips=int(flips.sum()), set_aside=int(aside.sum()), kappa=kappa, image_tol=tol,
                                    image_rel_l2=img_err, grad_rel_l2_vs_reference_build=errs,
                                    reference_build_vs_fp64=ref_noise, product_vs_fp64=own_noise)) + "\n")
    for name, err in errs.items():
        bar = max(1e-4, 2.0 * ref_noise[name])
        assert err <= bar, f"grad_{name} against the reference's own build: relative L2 error {err:.3e} (bar {bar:.3e})"
        assert own_noise[name] <= bar, f"grad_{name} against exact arithmetic: {own_noise[name]:.3e} (bar {bar:.3e})"


def test_projection_kernels_vs_oracle_and_autograd():
    """tg_project / tg_project_backward against the numpy restatement of the viewer's tensor operations
    (fp64) and against torch autograd on views.project."""
    from trigrad_b200 import views
    mesh = S.displaced_sphere(4)
    pv = S.camera_ring(8)[3]
    pts = Hh.cuda(mesh.points)
    verts = views.project_native(pts, pv)
    ref = O.project(mesh.points.astype(np.float64), pv)
    assert Hh.rel_err(verts.cpu().numpy(), ref) <= 1e-6
    rng = np.random.default_rng(5)
    g = rng.normal(size=ref.shape).astype(np.float32)
    gp = torch.zeros_like(pts)
    views.project_backward_native(pts, pv, Hh.cuda(g), gp, accumulate=False)
    views.project_backward_native(pts, pv, Hh.cuda(g), gp, accumulate=True)          # twice: accumulation
    ref_g = 2 * O.project_vjp(mesh.points.astype(np.float64), pv, g.astype(np.float64))
    assert Hh.rel_l2(gp.cpu().numpy(), ref_g) <= 1e-6
    p = pts.clone().requires_grad_()
    (ga,) = torch.autograd.grad(views.project(p, Hh.cuda(pv)), p, grad_outputs=Hh.cuda(g))
    assert Hh.rel_l2(gp.cpu().numpy(), 2 * ga.cpu().numpy()) <= 1e-5


def test_world_space_view_step_matches_autograd():
    """views.l2_world_view_step (projection kernel, rendering step, projection VJP kernel) against
    render() + torch autograd through views.project."""
    from trigrad_b200 import views
    mesh = S.displaced_sphere(4)
    pv = S.camera_ring(8)[1]
    W, H = 320, 192
    pts, i, c, o = Hh.cuda(mesh.points), Hh.cuda(mesh.indices), Hh.cuda(mesh.colors), Hh.cuda(mesh.opacities)
    V = pts.shape[0]
    target = torch.rand((H, W, 4), device="cuda")
    gP, gC, gO = torch.zeros((V, 3), device="cuda"), torch.zeros((V, 3), device="cuda"), torch.zeros((V,), device="cuda")
    loss = torch.zeros((), device="cuda")
    img = views.l2_world_view_step(pts, pv, i, c, o, target, W, H, gP, gC, gO, loss)
    # reference: the same render-space vertices through render() + autograd, then the VJP of the torch projection
    vv = views.project_native(pts, pv).requires_grad_()
    cc, oo = c.clone().requires_grad_(), o.clone().requires_grad_()
    image, _ = trigrad_b200.render(vv, i, cc, oo, W, H)
    l = torch.mean((image - target) ** 2)
    gv, gc, go = torch.autograd.grad(l, (vv, cc, oo))
    p = pts.clone().requires_grad_()
    (gp,) = torch.autograd.grad(views.project(p, Hh.cuda(pv)), p, grad_outputs=gv)
    torch.cuda.synchronize()
    assert torch.equal(img, image)
    assert abs(float(loss) - float(l)) <= 1e-5 * float(l)
    for a, b in zip((gP, gC, gO), (gp, gc, go)):
        assert Hh.rel_l2(a.cpu().numpy(), b.cpu().numpy()) <= 1e-5


@pytest.mark.parametrize("one_kernel", [False, True])
def test_triangles_without_any_tile_entry(one_kernel):
    """T > 0 but K = 0 (all triangles degenerate): background image, zero gradients, through both step paths."""
    from trigrad_b200 import views
    v = np.array([[0.1, 0.1, 1.0, 1.0]] * 3 + [[-0.5, -0.5, 2.0, 0.5], [0.0, 0.0, 2.0, 0.5], [0.5, 0.5, 2.0, 0.5]], np.float32)
    idx = np.array([[0, 1, 2], [3, 4, 5]], np.int32)
    c = np.full((6, 3), 0.5, np.float32)
    o = np.full((6,), 0.5, np.float32)
    W, H = 37, 21
    image, depth = trigrad_b200.render(Hh.cuda(v), Hh.cuda(idx), Hh.cuda(c), Hh.cuda(o), W, H)
    assert torch.equal(image[..., :3], torch.zeros_like(image[..., :3])) and torch.all(image[..., 3] == 1)
    assert torch.all(torch.isinf(depth))
    gV, gC, gO = torch.zeros((6, 4), device="cuda"), torch.zeros((6, 3), device="cuda"), torch.zeros((6,), device="cuda")
    loss = torch.zeros((), device="cuda")
    target = torch.rand((H, W, 4), device="cuda")
    img = views.l2_view_step(Hh.cuda(v), Hh.cuda(idx), Hh.cuda(c), Hh.cuda(o), target, W, H, gV, gC, gO, loss,
                             one_kernel=one_kernel)
    torch.cuda.synchronize()
    assert torch.equal(img, image)
    assert abs(float(loss) - float(torch.mean((image - target) ** 2))) <= 1e-6
    assert float(gV.abs().max()) == 0 and float(gC.abs().max()) == 0 and float(gO.abs().max()) == 0


def test_packed_accumulator_over_views_and_streams():
    """views.PackedGradients: three views on two streams add into one accumulator that is unpacked once;
    equal to the per-view accumulation of l2_view_step."""
    from trigrad_b200 import views
    sc = S.config2_random10k()
    V = sc.num_vertices
    i, c, o = Hh.cuda(sc.indices), Hh.cuda(sc.colors), Hh.cuda(sc.opacities)
    rng = np.random.default_rng(23)
    vs, ts = [], []
    for k in range(3):
        verts = sc.vertices.copy()
        verts[:, 1] += 0.02 * k
        vs.append(Hh.cuda(verts))
        ts.append(Hh.cuda(rng.random((sc.height, sc.width, 4), dtype=np.float32)))
    ref = [torch.zeros((V, 4), device="cuda"), torch.zeros((V, 3), device="cuda"), torch.zeros((V,), device="cuda")]
    ref_loss = torch.zeros((), device="cuda")
    for v, t in zip(vs, ts):
        views.l2_view_step(v, i, c, o, t, sc.width, sc.height, ref[0], ref[1], ref[2], ref_loss)
    torch.cuda.synchronize()
    packed = views.PackedGradients(V, "cuda")
    side = torch.cuda.Stream()
    for one_kernel in (False, True):
        packed.zero_()
        start = torch.cuda.Event()
        start.record()
        side.wait_event(start)
        for k, (v, t) in enumerate(zip(vs, ts)):
            with torch.cuda.stream(side if k == 1 else torch.cuda.current_stream()):
                views.l2_view_step(v, i, c, o, t, sc.width, sc.height, None, None, None, None, one_kernel=one_kernel,
                                   packed=packed)
        done = torch.cuda.Event()
        done.record(side)
        torch.cuda.current_stream().wait_event(done)
        got = [torch.full((V, 4), 7.0, device="cuda"), torch.full((V, 3), 7.0, device="cuda"), torch.full((V,), 7.0, device="cuda")]
        loss = torch.full((), 7.0, device="cuda")
        packed.unpack(sc.width, sc.height, got[0], got[1], got[2], loss, accumulate=False)     # overwrites
        torch.cuda.synchronize()
        assert abs(float(loss) - float(ref_loss)) <= 1e-5 * float(ref_loss)
        for a, b in zip(got, ref):
            assert Hh.rel_l2(a.cpu().numpy(), b.cpu().numpy()) <= 1e-5


def test_bounded_wait_runs_out_and_is_reported():
    """A device-side wait that nothing satisfies: the look-back warp polls a partition word that is never published,
    gives up after its limit, raises the status word and returns - the launch ends, the context stays usable."""
    import ctypes as C
    from trigrad_b200 import _native as N
    scratch = torch.zeros(8, dtype=torch.int32, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    st = N.lib().tg_selftest_bounded_wait(C.c_void_p(scratch.data_ptr()), 32, C.c_void_p(status.data_ptr()), 8,
                                          C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == N.TG_OK
    torch.cuda.synchronize()
    assert int(status[0]) == 1                      # what TG_ERR_DEVICE_FLAG reports to the host
    assert int(scratch[2]) == 7 and int(scratch[3]) == 2   # the warp still published its (inclusive) word
    # the context is fine: an ordinary render right after it
    sc = S.large_triangles(2)
    v, i, c, o = Hh.scene_tensors(sc)
    image, _ = trigrad_b200.render(v, i, c, o, sc.width, sc.height)
    assert torch.isfinite(image).all()


def test_stale_device_error_word_raises_at_the_next_render_and_in_backward():
    """The error word of a render travels to a pinned slot asynchronously; the next render on the stream, the
    backward of the same render and ``check_device_errors`` must raise when it is set."""
    from trigrad_b200 import wrapper as Wr
    sc = S.large_triangles(2)
    v, i, c, o = Hh.scene_tensors(sc)
    trigrad_b200.render(v, i, c, o, sc.width, sc.height)
    torch.cuda.synchronize()
    st = Wr._state(v.device)
    st.info[st.last_slot, 2] = 3                    # as if a kernel of that render had raised the word
    with pytest.raises(RuntimeError, match="device error word 3"):
        trigrad_b200.render(v, i, c, o, sc.width, sc.height)
    torch.cuda.synchronize()
    st.info[st.last_slot, 2] = 5
    with pytest.raises(RuntimeError, match="device error word 5"):
        trigrad_b200.check_device_errors()
    trigrad_b200.check_device_errors()              # the word was consumed
    vv = v.clone().requires_grad_()
    image, _ = trigrad_b200.render(vv, i, c, o, sc.width, sc.height)
    torch.cuda.synchronize()
    st.info[st.last_slot, 2] = 9
    with pytest.raises(RuntimeError, match="device error word 9"):
        image.sum().backward()
    trigrad_b200.check_device_errors()


def test_render_without_saved_selection_gives_the_same_gradients():
    """Above ``SELECTION_MAX_BYTES`` the forward saves no per-pixel fragment ids and the backward searches the lists."""
    from trigrad_b200 import wrapper as Wr
    sc = S.config2_random10k()
    mode = dict(thr=1 / 256, per_pixel_sort=True, max_layers=32)
    rng = np.random.default_rng(9)
    gi = rng.normal(size=(sc.height, sc.width, 4)).astype(np.float32)
    gd = rng.normal(size=(sc.height, sc.width)).astype(np.float32)
    a = run_render(sc, mode, gi, gd)
    old = Wr.SELECTION_MAX_BYTES
    Wr.SELECTION_MAX_BYTES = 0
    try:
        b = run_render(sc, mode, gi, gd)
    finally:
        Wr.SELECTION_MAX_BYTES = old
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
    for x, y in zip(a[2:], b[2:]):
        assert Hh.rel_l2(x, y) <= 1e-5


def test_uint8_target_matches_the_float_target_it_stands_for():
    """views.l2_view_step with an 8-bit RGBA target against the same call on ``u8.float() / 255``: identical loss and
    gradients up to the run-dependent order of the float atomics."""
    from trigrad_b200 import views
    sc = S.config2_random10k()
    v, i, c, o = Hh.scene_tensors(sc)
    V = sc.num_vertices
    t8 = torch.from_numpy(np.random.default_rng(23).integers(0, 256, (sc.height, sc.width, 4), dtype=np.uint8)).cuda()
    out = []
    for target in (t8, t8.float() / 255):
        gV, gC, gO = torch.zeros((V, 4), device="cuda"), torch.zeros((V, 3), device="cuda"), torch.zeros((V,), device="cuda")
        loss = torch.zeros((), device="cuda")
        views.l2_view_step(v, i, c, o, target, sc.width, sc.height, gV, gC, gO, loss)
        out.append((float(loss), gV.cpu().numpy(), gC.cpu().numpy(), gO.cpu().numpy()))
    assert abs(out[0][0] - out[1][0]) <= 1e-6 * out[1][0]
    for a, b in zip(out[0][1:], out[1][1:]):
        assert Hh.rel_l2(a, b) <= 1e-5
    with pytest.raises(TypeError):
        views.l2_view_step(v, i, c, o, t8.short(), sc.width, sc.height, None, None, None, torch.zeros((), device="cuda"))
    with pytest.raises(ValueError):
        views.l2_view_step(v, i, c, o, t8, sc.width, sc.height, None, None, None, torch.zeros((), device="cuda"), one_kernel=True)


def test_world_space_view_step_with_packed_accumulators_on_two_streams():
    """Two views on two streams, each with its own packed accumulator, adding atomically into one set of world-space
    gradient tensors (``tg_unpack_project_backward``) against the same two views through the unpacked path."""
    from trigrad_b200 import views
    mesh = S.displaced_sphere(4)
    pvs = S.camera_ring(8)
    W, H = 320, 192
    pts, i, c, o = Hh.cuda(mesh.points), Hh.cuda(mesh.indices), Hh.cuda(mesh.colors), Hh.cuda(mesh.opacities)
    V = pts.shape[0]
    targets = [torch.rand((H, W, 4), device="cuda") for _ in range(2)]
    ref = views.GradBuffer.allocate(V, pts.device, 3)
    for k in range(2):
        views.l2_world_view_step(pts, pvs[k + 1], i, c, o, targets[k], W, H, ref.points, ref.colors, ref.opacities, ref.loss)
    got = views.GradBuffer.allocate(V, pts.device, 3)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    packs = [views.PackedGradients(V, pts.device) for _ in range(2)]
    for rounds in range(2):                                  # second round: the accumulators were left zero by the first
        got.zero_()
        torch.cuda.synchronize()
        for k, st in enumerate(streams):
            with torch.cuda.stream(st):
                views.l2_world_view_step(pts, pvs[k + 1], i, c, o, targets[k], W, H, got.points, got.colors, got.opacities,
                                         got.loss, packed=packs[k])
        torch.cuda.synchronize()
        assert abs(float(got.loss) - float(ref.loss)) <= 1e-5 * float(ref.loss)
        for a, b in zip((got.points, got.colors, got.opacities), (ref.points, ref.colors, ref.opacities)):
            assert Hh.rel_l2(a.cpu().numpy(), b.cpu().numpy()) <= 1e-5
        for p in packs:
            assert not bool(p.scratch.any())


@pytest.mark.parametrize("use", ["image", "depth"])
def test_loss_that_uses_only_one_output(use):
    """Autograd hands the unused output's gradient over as None (no zero tensor is made): image-only and depth-only
    losses against the oracle with the other upstream gradient zero."""
    sc = S.config1_icosphere(width=128, height=128)
    rng = np.random.default_rng(3)
    gi = rng.normal(size=(sc.height, sc.width, 4)).astype(np.float32)
    gd = rng.normal(size=(sc.height, sc.width)).astype(np.float32)
    v, i, c, o = Hh.scene_tensors(sc)
    v.requires_grad_(), c.requires_grad_(), o.requires_grad_()
    image, depth = trigrad_b200.render(v, i, c, o, sc.width, sc.height)
    if use == "image":
        (image * Hh.cuda(gi)).sum().backward()
        gd[:] = 0
    else:
        d0 = torch.where(torch.isfinite(depth), depth, torch.zeros_like(depth))
        (d0 * Hh.cuda(gd)).sum().backward()
        gi[:] = 0
    of = O.forward(sc.vertices, sc.indices, sc.colors, sc.opacities, sc.width, sc.height)
    og = O.backward(sc.vertices, sc.indices, sc.colors, sc.opacities, sc.width, sc.height, of, gi, gd)
    for a, b in zip((v.grad, c.grad, o.grad), og):
        if float(np.abs(b).max()) == 0.0:
            assert float(a.abs().max()) == 0.0
        else:
            assert Hh.rel_l2(a.cpu().numpy(), b) <= 1e-4
