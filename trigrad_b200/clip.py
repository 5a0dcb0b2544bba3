"""Near-plane triangle splitting fused with the world -> render-space projection (``tg_project_clip``).

The reference's notebook clips with a Python loop over triangles (``split_clipped``,
``notebooks/renderer.ipynb``, cell "Clip Test") before dividing by w: a triangle that crosses the plane
``z + w = 0`` in clip space is cut into one or two triangles, one behind it is dropped, and the result is a
triangle soup with interpolated colours and opacities.  ``project_clip`` does the projection, the splitting and the
division in one kernel and is differentiable: its backward (``tg_project_clip_backward``) carries the gradients of
the soup back to world positions, colours and opacities, also through the interpolation parameters.

The soup has a fixed layout: input triangle t owns output triangles 2t and 2t+1 (vertices 6t .. 6t+5); slots that
are not needed hold a degenerate triangle that the rasteriser drops, so nothing is counted or compacted and the
reference's triangle order is kept.
"""
from __future__ import annotations

import numpy as np
import torch
from torch.autograd import Function

from . import _native as N


def _pv_host(pv):
    if isinstance(pv, torch.Tensor):
        pv = pv.detach().cpu().numpy()
    m = np.ascontiguousarray(pv, dtype=np.float32)
    if m.shape != (4, 4):
        raise ValueError("pv must be a 4x4 matrix")
    return m


class ProjectClip(Function):
    """What ``torch.jit.trace`` records of a ``project_clip``."""

    @staticmethod
    def forward(ctx, points, indices, colors, opacities, pv):
        ctx.pv = pv
        ctx.save_for_backward(points, indices, colors, opacities)
        out = N.host().project_clip(points, indices, colors, opacities, pv)
        ctx.mark_non_differentiable(out[1])
        return out

    @staticmethod
    def backward(ctx, grad_vertices, _, grad_colors, grad_opacities):
        gp, gc, go = N.host().project_clip_backward(*ctx.saved_tensors, ctx.pv, grad_vertices, grad_colors, grad_opacities)
        return gp, None, gc, go, None


def project_clip(points: torch.Tensor, indices: torch.Tensor, colors: torch.Tensor, opacities: torch.Tensor, pv):
    """World-space mesh -> render-space triangle soup clipped at the near plane.

        points (V,3) float32, indices (T,3) int32, colors (V,3), opacities (V,), pv: 4x4 projection * view (host)

    Returns ``(vertices (6T,4), indices (2T,3), colors (6T,3), opacities (6T,))`` ready for ``render``; differentiable
    with respect to points, colours and opacities.
    """
    if torch._C._get_tracing_state() is not None:
        return ProjectClip.apply(points, indices, colors, opacities, _pv_host(pv))
    return N.host().project_clip(points, indices, colors, opacities, _pv_host(pv))
