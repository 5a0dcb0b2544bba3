"""Renders under torch's transforms: refused where the autograd nodes take no part in them, never silently wrong."""
import numpy as np
import pytest
import torch
import torch.autograd.forward_ad as fwAD
from torch.fx.experimental.proxy_tensor import make_fx

import helpers as Hh
import trigrad_b200
from trigrad_b200 import scenes as S

pytestmark = pytest.mark.gpu

W, H = 64, 48


def _mesh():
    sc = S.random_triangles(300, W, H, 0.3, 0.4, name="transforms", seed=1)
    return Hh.scene_tensors(sc)


def _calls(triangles=300):
    v, i, c, o = _mesh()
    rgba, faces = trigrad_b200.pack_mesh(c, o, i)
    i, faces = i[:triangles], faces[:triangles]
    pv, points = np.eye(4, dtype=np.float32), v[:, :3].contiguous()
    return {
        "render": (lambda x: trigrad_b200.render(v, i, x, o, W, H)[0], c),
        "tile_order": (lambda x: trigrad_b200.render(v, i, x, o, W, H, per_pixel_sort=False, max_layers=0)[0], c),
        "corrected": (lambda x: trigrad_b200.render_corrected(v, i, x, o, W, H, max_layers=0)[0], c),
        "packed": (lambda x: trigrad_b200.render_packed(v, faces, x, W, H)[0], rgba),
        "Renderer": (lambda x: trigrad_b200.Renderer.apply(v, i, x, o, W, H)[0], c),
        "project_clip": (lambda x: trigrad_b200.project_clip(points, i, x, o, pv)[2], c),
    }


NAMES = ["render", "tile_order", "corrected", "packed", "Renderer", "project_clip"]


@pytest.mark.parametrize("triangles", [300, 0])
@pytest.mark.parametrize("name", NAMES)
def test_transforms_that_are_not_supported_are_refused(name, triangles):
    f, x = _calls(triangles)[name]
    with fwAD.dual_level(), pytest.raises(NotImplementedError):
        f(fwAD.make_dual(x, torch.ones_like(x)))
    with pytest.raises(RuntimeError):
        torch.func.grad(lambda y: f(y).sum())(x)
    with pytest.raises(RuntimeError):
        torch.func.vmap(f)(torch.stack([x, x]))
    if triangles or name != "Renderer":          # without triangles that one is plain torch operations
        with pytest.raises(RuntimeError):
            make_fx(f)(x)
    assert f(x).shape == f(x.clone()).shape


@pytest.mark.filterwarnings("ignore::torch.jit.TracerWarning", "ignore::DeprecationWarning")
@pytest.mark.parametrize("triangles", [300, 0])
@pytest.mark.parametrize("name", NAMES)
def test_a_trace_renders_the_inputs_it_is_given(name, triangles):
    f, x = _calls(triangles)[name]
    for grad in (False, True):
        traced = torch.jit.trace(f, (x.clone().requires_grad_(grad),), check_trace=False)
        y = (0.5 * x).requires_grad_(grad)
        a, b = traced(y), f(y)
        assert torch.equal(a, b)
        if grad:
            (ga,), (gb,) = torch.autograd.grad(a.sum(), y), torch.autograd.grad(b.sum(), y)
            assert ga.shape == gb.shape and Hh.rel_l2(ga.cpu().numpy(), gb.cpu().numpy()) <= 1e-5      # order of atomics
