"""``render_corrected``: the reference's ``render`` with gradients that are right in every mode.

The reference's backward kernel is only consistent with its forward in the default mode.  With
``per_pixel_sort=False`` it visits the first ``ends`` list entries front to back although its recurrences are
written for a walk from the last blended fragment to the first and ``ends`` counts blended fragments
(``src/trigrad/render.cu:659-666`` against ``:478-497``); with more than 32 layers it reverses the order inside
each batch of 32 only (``:673-693``).  ``trigrad_b200.render`` reproduces both literally (drop-in means identical
results).  This module is the opt-in alternative: same arguments, same forward results, and a backward
(``tg_blend_backward_corrected``) that differentiates what the forward blended, whatever the mode and the
number of layers.  In the default mode both functions return the same gradients.
"""
from __future__ import annotations

from . import _native as N
from . import wrapper as _w


def render_corrected(vertices, indices, colors, opacities, width=500, height=500, tile_width=16, tile_height=16,
                     early_stopping_threshold=1 / 256, record_timing=False, per_pixel_sort=True, max_layers=32):
    """Same contract as ``trigrad_b200.render`` (and the reference's ``trigrad.render``); the gradients are those of
    the rendered image in every mode, see the module docstring."""
    out = N.host().render(_w.GRADIENTS_CORRECTED, vertices, indices, colors, opacities, width, height, tile_width,
                          tile_height, early_stopping_threshold, record_timing, per_pixel_sort, max_layers, _w.CULL_TILES,
                          _w.SELECTION_MAX_BYTES)
    if record_timing or out is None:
        return _w.finish_render(out, _w.GRADIENTS_CORRECTED, vertices, indices, colors, opacities, width, height, tile_width,
                                tile_height, early_stopping_threshold, record_timing, per_pixel_sort, max_layers)
    return out
