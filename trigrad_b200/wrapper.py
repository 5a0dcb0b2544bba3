"""Python entry point: ``render`` and the ``Renderer`` autograd function.

Mirrors the public interface of the reference (``src/trigrad/wrapper.py:12-158``): same argument
order and defaults, same exceptions (``TypeError`` for device / dtype, ``ValueError`` for shapes and
oversized tiles), same outputs ``(image, depthmap[, timings])`` and the same twelve gradient slots.
The work itself is done by hand-written sm_100a kernels behind the C ABI of
``include/trigrad_b200.h``; allocations, the per-stream state and the autograd nodes are in
``csrc/tg_torch.cpp``.  There is no CPU path.
"""
from __future__ import annotations

from typing import Tuple

import torch
from torch.autograd import Function

from . import _native as N
from .util import create_check

precision = torch.float32
check_tensor = create_check("cuda", precision)

TIMING_KEYS = ("init", "per_tile_lists", "sorting", "bary_transforms", "rasterization")

# In the default mode the forward saves, per pixel, the ids of the fragments it blended (max_layers int32 planes
# of the image size: 265 MB at 1920x1080, 1.06 GB at 3840x2160, alive until the backward of that render has
# run) so that the backward need not search the tile lists again.  A render whose planes would exceed this many
# bytes saves nothing and its backward searches the lists as the reference does (same gradients, slower).
SELECTION_MAX_BYTES = 1 << 30

# With per_pixel_sort (the default) ``render`` lists a (triangle, tile) pair only when the triangle can cover the
# centre of a pixel of that tile - the exact test the reference leaves as a TODO (``render.cu:110``).  A pair that is
# dropped covers no pixel, so image, depth map and gradients are bit-identical either way; only the private tile
# lists are shorter than the reference's.  Tile-order mode keeps the reference's lists because its backward indexes
# them by position.  Set to False to build the reference's lists in every mode.
CULL_TILES = True


def _state(device: torch.device):
    """Workspace, pinned read-back slots and list-length estimate of the current stream of ``device``."""
    index = device.index if device.index is not None else torch.cuda.current_device()
    return N.host().state(index, torch.cuda.current_stream(device).cuda_stream)


def check_device_errors(device=None) -> None:
    """Synchronise the current stream of `device` and raise if the last render on it reported a device error
    word.  ``render`` checks the word of a call when the next call on the same stream returns, and (without
    waiting) when its backward starts; this is the explicit check for the last call of a program."""
    device = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    torch.cuda.current_stream(device).synchronize()
    st = _state(device)
    st.check_error_word(st.last_slot)


def _timings(stage_ms):
    return None if stage_ms is None else {k: ms / 1000.0 for k, ms in zip(TIMING_KEYS, stage_ms)}


def forward_native(vertices, indices, colors, opacities, width, height, tile_width, tile_height,
                   early_stopping_threshold, record_timing, per_pixel_sort, max_layers, save_selection=True,
                   cull_tiles=False, packed_inputs=False):
    """Run the whole forward path.  Returns the public outputs and the state saved for backward.

    ``save_selection=False`` (or planes larger than ``SELECTION_MAX_BYTES``) skips the per-pixel record of the
    blended fragment ids; the backward then searches the tile lists again.  ``cull_tiles`` lists a (triangle, tile)
    pair only if the triangle can cover a pixel centre of the tile (``TG_FORWARD_CULL_TILES``): same image, same
    gradients, shorter lists than the reference's.  ``packed_inputs``: ``indices`` is ``[T,4]`` int32 and ``colors`` is
    ``[V,4]`` (r, g, b, opacity), ``opacities`` is None (``TG_INPUT_PACKED``)."""
    out = N.host().forward(vertices, indices, colors, None if packed_inputs else opacities, width, height, tile_width,
                           tile_height, early_stopping_threshold, record_timing, per_pixel_sort, max_layers,
                           save_selection, cull_tiles, SELECTION_MAX_BYTES)
    return (*out[:9], _timings(out[9]))


# which gradients a render's backward computes (the host path's enumeration)
GRADIENTS_REFERENCE, GRADIENTS_CORRECTED, GRADIENTS_PACKED = range(3)


class RendererOfKind(Function):
    """The autograd function behind ``Renderer``, and behind every render that ``torch.jit.trace`` records: the trace keeps
    a call of it, where it would see nothing of the host path's own nodes.  ``kind``: one of ``GRADIENTS_*``; with
    ``GRADIENTS_PACKED`` the inputs are vertices, faces, rgba, None."""

    @staticmethod
    def forward(ctx, kind, vertices, indices, colors, opacities, width, height, tile_width, tile_height,
                early_stopping_threshold, record_timing, per_pixel_sort, max_layers):
        packed = kind == GRADIENTS_PACKED
        n, _ = vertices.shape
        check_tensor(vertices, "vertices", (n, 4))
        if packed:
            check_tensor(colors, "rgba", (n, 4))
        else:
            check_tensor(colors, "colors", (n, 3))
            check_tensor(opacities, "opacities", (n,))
        n, _ = indices.shape
        check_tensor(indices, "faces" if packed else "indices", (n, 4 if packed else 3), torch.int32)
        if max_layers <= 0:
            max_layers = n + 1
        # an output that was not used downstream arrives in backward as None instead of a tensor of zeros that
        # autograd would have to fill and the kernel to read (the depth map, in the usual image-only loss)
        ctx.set_materialize_grads(False)
        ctx.kind = kind
        timings = None
        if n < 1:
            ctx.layout = None
            image = torch.zeros((height, width, 4), dtype=colors.dtype, device=colors.device)
            image[..., 3] = 1.0
            depthmap = torch.full((height, width), float("inf"), dtype=colors.dtype, device=colors.device)
            ctx.save_for_backward(vertices, colors, opacities)
        else:
            out = N.host().forward(vertices, indices, colors, opacities, width, height, tile_width, tile_height,
                                   early_stopping_threshold, record_timing, per_pixel_sort, max_layers,
                                   kind != GRADIENTS_CORRECTED,
                                   (kind == GRADIENTS_CORRECTED or bool(per_pixel_sort)) and CULL_TILES, SELECTION_MAX_BYTES)
            image, depthmap, timings, ctx.layout = out[0], out[1], _timings(out[9]), out[10]
            # image, depth map, blob, and the selection or, where there is none, the lists
            ctx.save_for_backward(image, depthmap, out[11], None if out[8] is not None else out[3], out[8])
        if record_timing:
            return image, depthmap, timings
        return image, depthmap

    @staticmethod
    def backward(ctx, grad_image, grad_depthmap, grad_timings=None):
        if ctx.layout is None:
            grads = [None if t is None else torch.zeros_like(t) for t in ctx.saved_tensors]
        else:
            grads = N.host().backward(ctx.kind, ctx.layout, *ctx.saved_tensors, grad_image, grad_depthmap)
            if ctx.kind == GRADIENTS_PACKED:
                grads = [*grads, None]
        gV, gC, gO = grads
        return (None, gV, None, gC, gO, None, None, None, None, None, None, None, None)


class Renderer(Function):
    """The autograd function behind ``render``, for callers that use it directly (``Renderer.apply``)."""

    @staticmethod
    def forward(ctx, vertices: torch.Tensor, indices: torch.Tensor, colors: torch.Tensor, opacities: torch.Tensor,
                width: int = 500, height: int = 500, tile_width: int = 16, tile_height: int = 16,
                early_stopping_threshold: float = 1 / 256, record_timing: bool = False, per_pixel_sort: bool = True,
                max_layers: int = 32):
        return RendererOfKind.forward(ctx, GRADIENTS_REFERENCE, vertices, indices, colors, opacities, width, height, tile_width,
                                      tile_height, early_stopping_threshold, record_timing, per_pixel_sort, max_layers)

    @staticmethod
    def backward(ctx, grad_image: torch.Tensor, grad_depthmap: torch.Tensor, grad_timings=None):
        return RendererOfKind.backward(ctx, grad_image, grad_depthmap, grad_timings)[1:]


def finish_render(out, *args):
    """What the host path's ``render`` does not return by itself: stage times as a dict, and nothing while a trace is being
    recorded - the call then goes through a node that the trace sees.  ``args``: those of ``RendererOfKind``."""
    if out is None:
        return RendererOfKind.apply(*args)
    return out[0], out[1], _timings(out[2])


def render(vertices: torch.Tensor, indices: torch.Tensor, colors: torch.Tensor, opacities: torch.Tensor,
           width: int = 500, height: int = 500, tile_width: int = 16, tile_height: int = 16,
           early_stopping_threshold: float = 1 / 256, record_timing: bool = False, per_pixel_sort: bool = True,
           max_layers: int = 32) -> Tuple[torch.Tensor, torch.Tensor] | Tuple[torch.Tensor, torch.Tensor, dict]:
    """Render semi-transparent triangles (same contract as the reference ``trigrad.render``).

        vertices  : (N, 4) float32 CUDA tensor (x'/w', y'/w', z'/w', 1/w') in [-1, 1] clip space
        indices   : (M, 3) int32 triangle vertex indices
        colors    : (N, 3) vertex colours, opacities : (N,) vertex opacities
        per_pixel_sort : sort fragments per pixel (default) or blend in per-tile order
        max_layers     : maximum number of layers composited per pixel, <= 0 for no limit

    Returns ``image`` (height, width, 4) whose alpha channel holds the remaining translucency,
    ``depthmap`` (height, width) and, with ``record_timing``, a dict of stage times in seconds (the call then waits for the GPU,
    and a small render sorts and composites in two kernels, each with its time, where it otherwise does both in one).

    Memory: in the default mode (``per_pixel_sort`` and ``max_layers <= 32``) autograd keeps ``max_layers`` int32
    planes of the image size alive per render until its backward has run (265 MB at 1920x1080), see
    ``SELECTION_MAX_BYTES`` in this module for the switch to the list-searching backward.
    """
    out = N.host().render(GRADIENTS_REFERENCE, vertices, indices, colors, opacities, width, height, tile_width, tile_height,
                          early_stopping_threshold, record_timing, per_pixel_sort, max_layers,
                          bool(per_pixel_sort) and CULL_TILES, SELECTION_MAX_BYTES)
    if record_timing or out is None:
        return finish_render(out, GRADIENTS_REFERENCE, vertices, indices, colors, opacities, width, height, tile_width, tile_height,
                             early_stopping_threshold, record_timing, per_pixel_sort, max_layers)
    return out
