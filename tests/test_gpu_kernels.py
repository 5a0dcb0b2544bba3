"""Single kernels at the sizes where they change their method: ends of length classes, remainders of chunks."""
import numpy as np
import pytest
import torch

import helpers as Hh
import oracle as O
import trigrad_b200
from trigrad_b200 import scenes as S
from trigrad_b200 import wrapper as Wr

pytestmark = pytest.mark.gpu


def _ordered(depth):
    u = depth.astype(np.float32).view(np.uint32)
    return np.where(u >> 31 != 0, ~u, u | np.uint32(0x80000000)).astype(np.uint64)


@pytest.mark.parametrize("lengths", [[129, 3, 1023, 1024], [1025, 0, 4096, 8191], [8192, 8193, 130], [24575, 24576, 24577]],
                         ids=lambda x: "_".join(map(str, x)))
@pytest.mark.parametrize("depths", ["uniform", "two_layers", "clustered", "empty_clips"])
def test_bucket_sort_of_tile_lists(lengths, depths):
    """Finite depths with a few equal ones; the clustered ones overflow the buckets and take the network."""
    rng = np.random.default_rng(len(lengths) + lengths[0])
    offsets = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    n = int(offsets[-1])
    d = {"uniform": rng.uniform(-3, 10, n), "two_layers": rng.choice([1.0, 4.0], n) + rng.uniform(0, 0.02, n),
         "clustered": 2 + rng.normal(0, 1e-4, n) ** 3, "empty_clips": rng.uniform(0.1, 10, n)}[depths].astype(np.float32)
    d[5::50] = d[4::50][:len(d[5::50])]
    if depths == "empty_clips":
        d[::997] = 1e30
    entries, expect = np.empty(n, np.uint64), np.empty(n, np.uint64)
    for a, b in zip(offsets[:-1], offsets[1:]):
        entries[a:b] = (_ordered(d[a:b]) << np.uint64(32)) | rng.permutation(int(b - a)).astype(np.uint64)
        expect[a:b] = np.sort(entries[a:b])
    dev = Hh.cuda(entries.view(np.int64))
    ids = Hh.sort_tile_lists(dev, Hh.cuda(offsets))
    torch.cuda.synchronize()
    assert np.array_equal(dev.cpu().numpy().view(np.uint64), expect)
    assert np.array_equal(ids.cpu().numpy().view(np.uint32), (expect & np.uint64(0xFFFFFFFF)).astype(np.uint32))


@pytest.mark.parametrize("triangles,edge,width,height,tile,layers", [
    (3000, 0.9, 61, 45, 16, 32),        # long lists, every pixel full early: the rest of the list is filtered
    (3000, 0.9, 40, 33, 32, 8),         # the same with one CTA of 1024 threads, small batches
    (20000, 0.02, 100, 77, 16, 32),     # small triangles: records tested by a lane each, last block cut by the image
    (20000, 0.02, 90, 70, 8, 70),       # several batches
    (129, 0.5, 33, 17, 16, 32),         # lists just beyond what the compositing kernel sorts itself
    (128, 0.5, 33, 17, 16, 32),
    (65, 0.5, 31, 31, 4, 5),
])
def test_forward_methods_agree_with_the_oracle(triangles, edge, width, height, tile, layers):
    sc = S.random_triangles(triangles, width, height, edge, 0.4, name="methods", seed=triangles + tile)
    sc.tile_width = sc.tile_height = tile
    of = O.forward(sc.vertices, sc.indices, sc.colors, sc.opacities, width, height, tile, tile, 1e-6, True, layers)
    for repeat in range(2):             # the second call finds the workspace and the guess of the first
        out = Wr.forward_native(*Hh.scene_tensors(sc), width, height, tile, tile, 1e-6, False, True, layers, cull_tiles=True)
        torch.cuda.synchronize()
        assert np.array_equal(out[7].cpu().numpy(), of.ends)
        assert np.array_equal(out[0].cpu().numpy().view(np.uint32), of.image.view(np.uint32))
        assert np.array_equal(out[1].cpu().numpy().view(np.uint32), of.depthmap.view(np.uint32))
    li = O.build_lists(sc.vertices, sc.indices, width, height, tile, tile, cull=True)
    assert np.array_equal(out[4].cpu().numpy(), li.offsets) and np.array_equal(out[3].cpu().numpy(), li.ids)


@pytest.mark.parametrize("triangles,side,tile", [(4097, 1024, 1), (4096, 1024, 1), (2049, 1024, 1), (65536 + 1, 1024, 4)])
def test_more_pairs_than_a_list_can_hold(triangles, side, tile):
    """Triangles over the whole image, 2^31 to 2^32 + 2^20 pairs: 32-bit sums of them are small numbers or zero.  The call is
    refused and the next one on the stream finds its counters in order."""
    corners = np.array([[-4, -4], [4, -4], [0, 4]], np.float32)
    v = torch.ones((triangles, 3, 4), device="cuda")
    v[..., :2] = Hh.cuda(corners)
    v = v.reshape(-1, 4)
    i = torch.arange(3 * triangles, dtype=torch.int32, device="cuda").reshape(-1, 3)
    c, o = torch.rand((3 * triangles, 3), device="cuda"), torch.rand((3 * triangles,), device="cuda")
    with pytest.raises(RuntimeError, match="pairs"):
        trigrad_b200.render(v, i, c, o, side, side, tile, tile)
    few = slice(0, 7)
    image = trigrad_b200.render(v, i[few], c, o, 64, 48, tile, tile)[0].cpu().numpy()
    of = O.forward(*(x.cpu().numpy() for x in (v, i[few], c, o)), 64, 48, tile, tile)
    assert np.array_equal(image.view(np.uint32), of.image.view(np.uint32))


@pytest.mark.parametrize("triangles", [64, 65, 128, 129, 256, 257])
@pytest.mark.parametrize("per_pixel_sort", [True, False], ids=["per_pixel", "tile_order"])
def test_lists_at_the_ends_of_chunks(triangles, per_pixel_sort):
    """Faint triangles over a whole tile and a part of another, blended to the last one: lists of whole chunks, staged once
    for all batches of 32 layers, and one entry more; forward and corrected backward."""
    sc = S.random_triangles(triangles, 23, 16, 6.0, 0.05, name="chunks", seed=triangles)
    op = (0.05 * sc.opacities).astype(np.float32)
    image_of = lambda v, c, o: O.forward(v, sc.indices, c, o, 23, 16, 16, 16, 0.0, per_pixel_sort, triangles + 1)
    of = image_of(sc.vertices, sc.colors, op)
    v, i, c, o = (Hh.cuda(x) for x in (sc.vertices, sc.indices, sc.colors, op))
    for x in (v, c, o):
        x.requires_grad_()
    image, depth = trigrad_b200.render_corrected(v, i, c, o, 23, 16, 16, 16, 0.0, False, per_pixel_sort, 0)
    assert np.array_equal(image.detach().cpu().numpy().view(np.uint32), of.image.view(np.uint32))
    assert np.array_equal(depth.detach().cpu().numpy().view(np.uint32), of.depthmap.view(np.uint32))
    assert int(of.ends.max()) > min(triangles // 2, 60)
    rng = np.random.default_rng(triangles)
    gi = rng.normal(size=of.image.shape).astype(np.float32)
    f64 = [np.asarray(x, np.float64) for x in (sc.vertices, sc.colors, op)]
    of64 = image_of(*f64)
    assert np.array_equal(of64.ends, of.ends)       # no pixel centre on an edge: both precisions blend the same fragments
    (image * Hh.cuda(gi)).sum().backward()
    og = O.backward(f64[0], sc.indices, f64[1], f64[2], 23, 16, of64, gi.astype(np.float64), np.zeros((16, 23)), 16, 16,
                    per_pixel_sort, triangles + 1, corrected=True)
    for a, b in zip((v, c, o), og):
        assert Hh.rel_l2(a.grad.cpu().numpy(), b) <= 2e-4


@pytest.mark.parametrize("columns", [[1], [1, 6], [6, 7], [7, 7, 7, 1], [8, 7, 6, 5, 4, 3, 2, 1], [2] * 13 + [8], [1] * 31 + [8]],
                         ids=lambda x: f"{len(x)}_layers_{4 * sum(x)}")
@pytest.mark.parametrize("depth_gradient, layers", [(False, 32), (True, 32), (True, 40)])
def test_fragments_that_a_warp_keeps_for_its_next_round(columns, depth_gradient, layers):
    """One warp of 8x4 pixels; layer k is a slanted rectangle over its first columns[k] columns.  With more than 32 layers allowed
    the backward walks the list, in rounds of 4 * columns lanes."""
    W, H, rng = 8, 4, np.random.default_rng(len(columns))
    vertices, faces = [], []
    for k, n in enumerate(columns):
        right, z = 2 * n / W - 1, 1 + 0.1 * k
        depth = z + 0.01 * rng.random(4)
        xy = [(-1.1, -1.1), (right, -1.1), (right, 1.1), (-1.1, 1.1)]
        faces += [[4 * k, 4 * k + 1, 4 * k + 2], [4 * k, 4 * k + 2, 4 * k + 3]]
        vertices += [(x, y, d, 1 / d) for (x, y), d in zip(xy, depth)]
    v, i = np.array(vertices, np.float32), np.array(faces, np.int32)
    c, o = rng.random((len(v), 3), dtype=np.float32), rng.uniform(0.1, 0.5, len(v)).astype(np.float32)
    of = O.forward(v, i, c, o, W, H, 16, 16, 1 / 256, True, layers)
    assert int(of.ends.sum()) == 4 * sum(columns)
    gi = rng.standard_normal((H, W, 4)).astype(np.float32)
    gd = rng.standard_normal((H, W)).astype(np.float32) if depth_gradient else np.zeros((H, W), np.float32)
    og = O.backward(v, i, c, o, W, H, of, gi, np.where(np.isfinite(of.depthmap.reshape(H, W)), gd, 0).astype(np.float32), 16, 16, True, layers)
    leaves = [Hh.cuda(x).requires_grad_() for x in (v, c, o)]
    image, depth = trigrad_b200.render(leaves[0], Hh.cuda(i), leaves[1], leaves[2], W, H, 16, 16, max_layers=layers)
    outputs = [(image, Hh.cuda(gi))] + ([(depth, Hh.cuda(gd))] if depth_gradient else [])
    got = torch.autograd.grad([x for x, _ in outputs], leaves, [g for _, g in outputs])
    for a, b in zip(got, og):
        # sums of at most 32 fragments per vertex; the barycentric partials of triangles this large lose about two digits
        assert Hh.rel_l2(a.cpu().numpy(), b) <= 1e-4


@pytest.mark.parametrize("triangles, tile", [(128, 16), (129, 16), (192, 8), (256, 32), (257, 32)])
def test_lists_that_stay_in_shared_memory_for_all_sweeps(triangles, tile):
    """Every triangle covers the image's one tile or most of it: lists around the number of records that are kept."""
    rng = np.random.default_rng(triangles)
    angle = rng.uniform(0, 2 * np.pi, (triangles, 1)) + np.arange(3) * (2 * np.pi / 3)
    depth = rng.uniform(0.5, 10, (triangles, 1)) * np.ones(3)
    v = np.stack([3 * np.cos(angle), 3 * np.sin(angle), depth, 1 / depth], 2).reshape(-1, 4).astype(np.float32)
    i = np.arange(3 * triangles, dtype=np.int32).reshape(-1, 3)
    c, o = rng.random((len(v), 3), dtype=np.float32), rng.uniform(0.01, 0.03, len(v)).astype(np.float32)
    size = (tile, tile, tile, tile)
    li = O.build_lists(v, i, *size)
    assert li.offsets[-1] == triangles
    gi = rng.standard_normal((tile, tile, 4)).astype(np.float32)
    gd = rng.standard_normal((tile, tile)).astype(np.float32)
    of = O.forward(v, i, c, o, *size, 1 / 256, True, 1000)
    for function, corrected in ((trigrad_b200.render, False), (trigrad_b200.render_corrected, True)):
        og = O.backward(v, i, c, o, tile, tile, of, gi, gd, tile, tile, True, 1000, corrected=corrected)
        leaves = [Hh.cuda(x).requires_grad_() for x in (v, c, o)]
        image, depth = function(leaves[0], Hh.cuda(i), leaves[1], leaves[2], *size, max_layers=1000)
        for a, b in zip(torch.autograd.grad((image, depth), leaves, (Hh.cuda(gi), Hh.cuda(gd))), og):
            # the recurrences' divisions by 1 - opacity, a few hundred in a row, on both sides in 32 bits
            assert Hh.rel_l2(a.cpu().numpy(), b) <= 2e-4


@pytest.mark.parametrize("scale", [3.0, 1e3, 1e5, 3e6, 1e8])
@pytest.mark.parametrize("cull", [False, True])
def test_keys_of_triangles_far_larger_than_the_image(scale, cull):
    """Intersections that miss their border by more than a tile leave polygons that are not convex: keys as the oracle's."""
    rng, T, W, H, tile = np.random.default_rng(int(scale)), 400, 96, 80, 8
    xy = rng.standard_normal((T, 3, 2)) * scale * 10 ** rng.uniform(-2, 0, (T, 3, 1)) + rng.uniform(-1, 1, (T, 1, 2))
    d = rng.uniform(0.5, 10, (T, 3, 1))
    v = np.concatenate([xy, d, 1 / d], 2).reshape(-1, 4).astype(np.float32)
    i = np.arange(3 * T, dtype=np.int32).reshape(-1, 3)
    c, o = rng.random((len(v), 3), dtype=np.float32), rng.random(len(v), dtype=np.float32)
    li = O.build_lists(v, i, W, H, tile, tile, cull=cull)
    assert li.offsets[-1] > 1000
    out = Wr.forward_native(*map(Hh.cuda, (v, i, c, o)), W, H, tile, tile, 1 / 256, False, True, 32, cull_tiles=cull)
    assert np.array_equal(out[4].cpu().numpy(), li.offsets)
    assert np.array_equal(out[3].cpu().numpy()[:li.offsets[-1]], li.ids)


@pytest.mark.parametrize("tile, across, down", [(16, 37, 4), (16, 149, 1), (8, 37, 16), (8, 593, 1), (4, 37, 32), (4, 1185, 1), (16, 1, 1)])
@pytest.mark.parametrize("triangles", [40, 256, 257])
def test_walked_lists_at_the_number_of_tiles_that_chooses_the_sums(tile, across, down, triangles):
    """Eight warps on each of 148 multiprocessors and one tile more; the last column and row of tiles ragged."""
    W, H, rng = tile * across - tile // 2, tile * down - 1, np.random.default_rng(triangles + across)
    angle = rng.uniform(0, 2 * np.pi, (triangles, 1)) + np.arange(3) * (2 * np.pi / 3)
    radius = np.where(np.arange(triangles) % 4 == 0, rng.uniform(0.02, 0.5, triangles), 4.0)[:, None]      # some small, most over all
    centre = np.where(radius < 1, rng.uniform(-1, 1, (triangles, 2)), 0.0)
    depth = rng.uniform(0.5, 10, (triangles, 1)) * np.ones(3)
    v = np.stack([centre[:, :1] + radius * np.cos(angle), centre[:, 1:] + radius * np.sin(angle), depth, 1 / depth], 2)
    v, i = v.reshape(-1, 4).astype(np.float32), np.arange(3 * triangles, dtype=np.int32).reshape(-1, 3)
    c, o = rng.random((len(v), 3), dtype=np.float32), rng.uniform(0.01, 0.03, len(v)).astype(np.float32)
    size = (W, H, tile, tile)
    of = O.forward(v, i, c, o, *size, 1 / 256, True, 1000)
    assert of.ends.min() >= 30
    gi = rng.standard_normal((H, W, 4)).astype(np.float32)
    gd = rng.standard_normal((H, W)).astype(np.float32)
    for function, corrected in ((trigrad_b200.render, False), (trigrad_b200.render_corrected, True)):
        og = O.backward(v, i, c, o, W, H, of, gi, gd, tile, tile, True, 1000, corrected=corrected)
        leaves = [Hh.cuda(x).requires_grad_() for x in (v, c, o)]
        image, depth = function(leaves[0], Hh.cuda(i), leaves[1], leaves[2], *size, max_layers=1000)
        for a, b in zip(torch.autograd.grad((image, depth), leaves, (Hh.cuda(gi), Hh.cuda(gd))), og):
            # as for the lists that stay in shared memory: a few hundred divisions by 1 - opacity, on both sides in 32 bits
            assert Hh.rel_l2(a.cpu().numpy(), b) <= 2e-4
