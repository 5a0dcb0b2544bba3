"""What a render keeps for its backward is autograd's: saved-tensor hooks see all of it, and it is freed with the graph."""
import numpy as np
import pytest
import torch

import helpers as Hh
import trigrad_b200
from trigrad_b200 import scenes as S

pytestmark = pytest.mark.gpu

W, H = 200, 120


def _leaves(packed=False):
    sc = S.random_triangles(3000, W, H, 0.2, 0.4, name="saved", seed=4)
    v, i, c, o = Hh.scene_tensors(sc)
    if packed:
        rgba, i = trigrad_b200.pack_mesh(c, o, i)
        return i, [x.requires_grad_() for x in (v, rgba)]
    return i, [x.requires_grad_() for x in (v, c, o)]


CALLS = {
    "render": lambda i, x: trigrad_b200.render(x[0], i, x[1], x[2], W, H),
    "searched": lambda i, x: trigrad_b200.render(x[0], i, x[1], x[2], W, H, 16, 16, 1 / 256, False, True, 40),
    "tile_order": lambda i, x: trigrad_b200.render(x[0], i, x[1], x[2], W, H, 16, 16, 1 / 256, False, False, 64),
    "corrected": lambda i, x: trigrad_b200.render_corrected(x[0], i, x[1], x[2], W, H, 16, 16, 1 / 256, False, True, 0),
    "packed": lambda i, x: trigrad_b200.render_packed(x[0], i, x[1], W, H),
    "Renderer": lambda i, x: trigrad_b200.Renderer.apply(x[0], i, x[1], x[2], W, H),
}


def _loss(out):
    weights = torch.linspace(0.5, 1.5, out[0].numel(), device="cuda").reshape(out[0].shape)
    return (out[0] * weights).sum() + torch.where(torch.isfinite(out[1]), out[1], 0).sum()


def _moved(t):
    """The same values at an address and with strides of its own."""
    room = torch.empty(2 * t.numel() + 1, dtype=t.dtype, device="cuda")
    return room[1:].as_strided(t.shape, [2 * s for s in t.contiguous().stride()]).copy_(t)


@pytest.mark.parametrize("call", list(CALLS))
def test_hooks_see_and_move_all_that_is_saved(call):
    i, leaves = _leaves(call == "packed")
    want = torch.autograd.grad(_loss(CALLS[call](i, leaves)), leaves)
    seen = []

    def pack(t):
        seen.append(t.numel() * t.element_size())
        return t.cpu()

    for unpack in (lambda t: t.cuda(), _moved):
        seen.clear()
        with torch.autograd.graph.saved_tensors_hooks(pack, unpack):
            out = CALLS[call](i, leaves)
        # image and depth map, final weights and ends, records of 160 bytes, and the selection where one is kept
        least = 20 * W * H + 8 * W * H + 160 * i.shape[0]
        if call in ("render", "packed", "Renderer"):
            least += 4 * 32 * W * H
        assert sum(seen) >= least
        for a, b in zip(torch.autograd.grad(_loss(out), leaves), want):
            assert Hh.rel_l2(a.cpu().numpy(), b.cpu().numpy()) <= 1e-5      # sums of atomics, in no fixed order


@pytest.mark.parametrize("call", list(CALLS))
def test_a_hook_that_changes_device_or_size_is_an_error(call):
    i, leaves = _leaves(call == "packed")
    for unpack in (lambda t: t, lambda t: t.cuda().flatten()[:-1] if t.numel() > 1 else t, lambda t: t.cuda().double()):
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t.cpu(), unpack):
            out = CALLS[call](i, leaves)
        loss = _loss((out[0], out[1]))
        with pytest.raises(RuntimeError):
            torch.autograd.grad(loss, leaves)


@pytest.mark.parametrize("call", list(CALLS))
def test_saved_state_is_freed_by_a_backward_that_does_not_keep_the_graph(call):
    i, leaves = _leaves(call == "packed")
    torch.autograd.grad(_loss(CALLS[call](i, leaves)), leaves)          # the stream's own workspaces exist from here on
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    out = CALLS[call](i, leaves)
    loss = _loss(out)
    kept = torch.cuda.memory_allocated() - before
    torch.autograd.grad(loss, leaves, retain_graph=True)
    torch.autograd.grad(loss, leaves)
    with pytest.raises(RuntimeError, match="second time"):
        torch.autograd.grad(loss, leaves)
    assert out[0].grad_fn is not None
    freed = kept - (torch.cuda.memory_allocated() - before)
    assert freed >= 160 * i.shape[0] + (4 * 32 * W * H if call in ("render", "packed", "Renderer") else 0)


@pytest.mark.parametrize("call", list(CALLS))
def test_second_backward_of_a_mesh_without_triangles(call):
    i, leaves = _leaves(call == "packed")
    out = CALLS[call](i[:0], leaves)
    for keep in (True, False):
        for g, x in zip(torch.autograd.grad(out[0].sum(), leaves, retain_graph=keep), leaves):
            assert g.shape == x.shape and not bool(g.any())
    with pytest.raises(RuntimeError, match="second time"):
        torch.autograd.grad(out[0].sum(), leaves)


@pytest.mark.parametrize("call", list(CALLS))
def test_lists_are_kept_only_for_a_backward_that_reads_them(call):
    i, leaves = _leaves(call == "packed")
    sizes = []

    def pack(t):
        sizes.append(t.numel() * t.element_size())
        return t

    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t):
        CALLS[call](i, leaves)
    blob = 8 * W * H + 160 * i.shape[0] + 4 * (13 * 8 + 1) + 5 * 256
    selection = 4 * 32 * W * H if call in ("render", "packed", "Renderer") else 0
    lists = sum(sizes) - 20 * W * H - selection
    if selection:
        assert lists <= blob                  # nothing but final weights, ends, records and offsets
    else:
        assert lists >= 8 * W * H + 160 * i.shape[0] + 4 * i.shape[0]


@pytest.mark.parametrize("triangles, width, height, tile", [(20, 50, 50, 4), (1280, 256, 256, 16), (4000, 120, 100, 16), (300, 40, 40, 2)])
@pytest.mark.parametrize("call", ["render", "tile_order", "corrected"])
def test_small_renders_keep_little_more_than_image_records_and_selection(call, triangles, width, height, tile):
    """A hundred live graphs of calls that may go without the number of list entries, whose lists have room for every pair."""
    sc = S.random_triangles(triangles, width, height, 0.05, 0.4, name="live", seed=4)
    v, i, c, o = Hh.scene_tensors(sc)
    leaves = [x.requires_grad_() for x in (v, c, o)]
    options = dict(tile_order=dict(per_pixel_sort=False), corrected={}, render={})[call]
    function = trigrad_b200.render_corrected if call == "corrected" else trigrad_b200.render
    render = lambda: function(leaves[0], i, leaves[1], leaves[2], width, height, tile, tile, **options)
    with torch.cuda.stream(torch.cuda.Stream()):
        for _ in range(70):
            torch.autograd.grad(render()[0].sum(), leaves)
        torch.cuda.current_stream().synchronize()
        before = torch.cuda.memory_allocated()
        live = [render() for _ in range(100)]
        kept = (torch.cuda.memory_allocated() - before) / len(live)
    tiles = -(-width // tile) * -(-height // tile)
    px = width * height
    rest = 28 * px + 160 * triangles + 4 * (tiles + 1) + 5 * 256
    # the lists: none, up to as much as the rest, or what a call that counts has room for
    lists = 0 if call == "render" else max(rest, 4 * max(2 * triangles, 5 * int(_entries(v, i, c, o, width, height, tile)) // 4) + 4096)
    selection = 4 * 32 * px if call == "render" else 0
    # blocks are rounded up to 512 bytes; of the 20 MB segments that blocks above 1 MB come from, less than 1 MB is given away unsplit
    unsplit = (1 << 20) / ((20 << 20) // selection) if selection > 1 << 20 else 0
    assert kept <= rest + selection + lists + 5 * 512 + unsplit


def _entries(v, i, c, o, width, height, tile):
    out = trigrad_b200.wrapper.forward_native(v.detach(), i, c.detach(), o.detach(), width, height, tile, tile, 1 / 256, False, True, 32)
    return out[3].numel()


def test_a_backward_that_walks_the_lists_needs_them():
    """With a selection the lists may not be there; the corrected gradients walk them all the same."""
    from trigrad_b200 import _native as N
    from trigrad_b200 import wrapper as Wr

    i, (v, c, o) = _leaves()
    out = N.host().forward(v.detach(), i, c.detach(), o.detach(), W, H, 16, 16, 1 / 256, False, True, 32, True, True, Wr.SELECTION_MAX_BYTES)
    image, depth, ids, selection, layout, blob = *out[:2], out[3], out[8], out[10], out[11]
    gi = torch.ones_like(image)
    for kind in (Wr.GRADIENTS_REFERENCE, Wr.GRADIENTS_PACKED):
        N.host().backward(kind, layout, image, depth, blob, None, selection, gi, None)
    with pytest.raises(RuntimeError, match="tile lists"):
        N.host().backward(Wr.GRADIENTS_CORRECTED, layout, image, depth, blob, None, selection, gi, None)
