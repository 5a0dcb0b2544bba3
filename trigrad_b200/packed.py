"""Packed 16-byte input layout: faces as ``[T,4]`` int32 and per-vertex attributes as ``[V,4]`` (r, g, b, opacity).

The reference passes colours as ``[V,3]`` and faces as ``[T,3]`` and reads them through packed 3-word types
(``color3``, ``id3``, ``src/trigrad/util.h:457-573``): 12-byte strides that no vector load fits.  A caller that owns
its parameter tensors can keep them in the packed layout instead - one tensor ``rgba`` to optimise instead of
``colors`` and ``opacities`` - and call ``render_packed``: same rasteriser, same results, gradients returned in
the same layout (``tg_unpack_gradients_rgba``).
"""
from __future__ import annotations

import torch

from . import _native as N
from . import wrapper as _w


def pack_mesh(colors: torch.Tensor, opacities: torch.Tensor, indices: torch.Tensor):
    """``(colors [V,3], opacities [V], indices [T,3] int32)`` -> ``(rgba [V,4], faces [T,4] int32)`` (one kernel)."""
    return N.host().pack_mesh(colors, opacities, indices)


def render_packed(vertices: torch.Tensor, faces: torch.Tensor, rgba: torch.Tensor, width: int = 500, height: int = 500,
                  tile_width: int = 16, tile_height: int = 16, early_stopping_threshold: float = 1 / 256,
                  record_timing: bool = False, per_pixel_sort: bool = True, max_layers: int = 32):
    """``render`` for the packed layout: ``faces`` is ``[T,4]`` int32 (fourth column ignored), ``rgba`` is ``[V,4]``
    (r, g, b, opacity).  Same outputs as ``render(vertices, faces[:, :3], rgba[:, :3], rgba[:, 3], ...)``; gradients
    flow to ``vertices`` and ``rgba``."""
    out = N.host().render(_w.GRADIENTS_PACKED, vertices, faces, rgba, None, width, height, tile_width, tile_height,
                          early_stopping_threshold, record_timing, per_pixel_sort, max_layers,
                          bool(per_pixel_sort) and _w.CULL_TILES, _w.SELECTION_MAX_BYTES)
    if record_timing or out is None:
        return _w.finish_render(out, _w.GRADIENTS_PACKED, vertices, faces, rgba, None, width, height, tile_width, tile_height,
                                early_stopping_threshold, record_timing, per_pixel_sort, max_layers)
    return out
