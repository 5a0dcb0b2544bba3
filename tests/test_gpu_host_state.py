"""The state that the host path keeps per stream: shared by threads, by meshes of different size, and over failed calls."""
import ctypes
import threading

import numpy as np
import pytest
import torch

import helpers as Hh
import oracle as O
import trigrad_b200
from trigrad_b200 import scenes as S
from trigrad_b200 import views

pytestmark = pytest.mark.gpu


class Job:
    """A render and its gradients, through autograd or the fused step, with the oracle-free expectation of a lone call."""

    def __init__(self, triangles, width, height, fused, seed):
        self.size, self.fused = (width, height), fused
        self.v, self.i, self.c, self.o = Hh.scene_tensors(
            S.random_triangles(triangles, width, height, 0.2, 0.4, name="host state", seed=seed))
        self.target = torch.rand((height, width, 4), device="cuda", generator=torch.Generator("cuda").manual_seed(seed))
        with torch.cuda.stream(torch.cuda.Stream()):
            torch.cuda.current_stream().wait_stream(torch.cuda.default_stream())
            self.expected = [t.clone() for t in self.run()]
            torch.cuda.current_stream().synchronize()

    def run(self):
        if self.fused:
            b = views.GradBuffer.allocate(self.v.shape[0], "cuda", 4)
            image = views.l2_view_step(self.v, self.i, self.c, self.o, self.target, *self.size, b.points, b.colors, b.opacities, b.loss)
            return image, b.points, b.colors, b.opacities
        x = [t.detach().requires_grad_() for t in (self.v, self.c, self.o)]
        image, _ = trigrad_b200.render(x[0], self.i, x[1], x[2], *self.size)
        return image.detach(), *torch.autograd.grad(torch.mean((image - self.target) ** 2), x)

    def check(self, got):
        assert torch.equal(got[0], self.expected[0])
        for a, b in zip(got[1:], self.expected[1:]):
            assert Hh.rel_l2(a.cpu().numpy(), b.cpu().numpy()) <= 1e-5      # order of atomics


def test_threads_that_render_on_one_stream():
    """Four threads, two streams: two threads on each, with meshes, images and entry points of their own."""
    jobs = [Job(40, 50, 40, False, 1), Job(20_000, 320, 200, True, 2), Job(3000, 100, 300, False, 3), Job(300, 64, 64, True, 4)]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    results, errors = [[] for _ in jobs], []

    def work(k):
        try:
            with torch.cuda.stream(streams[k % 2]):
                for _ in range(12):
                    results[k].append(jobs[k].run())
                torch.cuda.current_stream().synchronize()
        except BaseException as e:
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for job, got in zip(jobs, results):
        assert len(got) == 12
        for g in got:
            job.check(g)


def test_meshes_of_different_size_take_turns_on_one_accumulator():
    jobs = [Job(50, 64, 64, True, 1), Job(30_000, 400, 300, True, 2), Job(2000, 90, 70, False, 3), Job(60_000, 256, 256, False, 4)]
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream()):
        for k in (0, 1, 0, 2, 3, 0, 1, 3, 2, 0):
            jobs[k].check(jobs[k].run())


@pytest.mark.parametrize("fused", [True, False])
def test_an_accumulator_above_the_limit_is_not_kept(fused):
    """9 million vertices, 288 MB of sums, of which the triangles use the last 3000."""
    small = Job(1000, 64, 64, fused, 5)
    n, used = 9_000_000, small.v.shape[0]
    big = Job.__new__(Job)
    big.size, big.fused, big.target = small.size, fused, small.target
    big.i = small.i + (n - used)
    big.v, big.c, big.o = (torch.zeros((n, *t.shape[1:]), device="cuda") for t in (small.v, small.c, small.o))
    for b, t in zip((big.v, big.c, big.o), (small.v, small.c, small.o)):
        b[n - used:] = t
    small.check(small.run())
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    got = big.run()
    small.check([got[0]] + [t[n - used:] for t in got[1:]])
    assert not any(bool(t[:n - used].any()) for t in got[1:])
    del got
    assert torch.cuda.memory_allocated() - before < 64 << 20
    small.check(small.run())


def test_calls_after_a_failed_call():
    job = Job(3000, 100, 80, True, 6)
    fit = Job(500, 64, 48, False, 7)
    V = job.v.shape[0]
    flat = torch.zeros(8 * V + 2, device="cuda")
    args = (job.v, job.i, job.c, job.o, job.target, *job.size)
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream()):
        for _ in range(2):
            # refused by the unpacking, after the sums have been made: the accumulator is not left zero
            with pytest.raises(RuntimeError, match="aligned"):
                views.l2_view_step(*args, flat[1:4 * V + 1].view(V, 4), flat[4 * V + 1:7 * V + 1].view(V, 3), flat[7 * V + 1:8 * V + 1],
                                   flat[8 * V + 1:].view(()))
            fit.check(fit.run())
            # refused behind the forward
            old, trigrad_b200.wrapper.SELECTION_MAX_BYTES = trigrad_b200.wrapper.SELECTION_MAX_BYTES, 0
            try:
                with pytest.raises(ValueError):
                    job.run()
            finally:
                trigrad_b200.wrapper.SELECTION_MAX_BYTES = old
            # refused ahead of it
            with pytest.raises(RuntimeError):
                trigrad_b200.render(job.v, job.i, job.c, job.o, -1, 8)
            job.check(job.run())


def test_more_streams_than_states_are_kept():
    """The state of the stream used least lately is given back, and made anew when the stream comes back."""
    job = Job(500, 64, 48, False, 8)
    torch.cuda.synchronize()
    handles = []
    for _ in range(140):
        h = ctypes.c_void_p()
        assert int(torch.cuda.cudart().cudaStreamCreate(ctypes.addressof(h))) == 0
        handles.append(h.value)
    results = []
    for h in handles + handles[:3]:
        with torch.cuda.stream(torch.cuda.ExternalStream(h)):
            results.append(job.run())
    torch.cuda.synchronize()
    for got in results:
        job.check(got)
    for h in handles:
        assert int(torch.cuda.cudart().cudaStreamDestroy(h)) == 0


@pytest.mark.parametrize("tile", [16, 8, 32])
@pytest.mark.parametrize("sort, corrected", [(True, False), (False, False), (True, True)])
def test_lists_that_grow_beyond_what_the_calls_before_had(tile, sort, corrected):
    """Small renders behind one with short lists do not wait for the number of entries; the first with long lists gets them
    sorted where they are, later ones as any others, and short ones again go back to not waiting."""
    w, h = 197, 121
    short = S.random_triangles(300, w, h, 0.05, 0.4, name="short", seed=tile)
    long = S.random_triangles(2000, w, h, 0.6, 0.4, name="long", seed=tile + 1)
    rng = np.random.default_rng(5)
    gi, gd = rng.normal(size=(h, w, 4)).astype(np.float32), rng.normal(size=(h, w)).astype(np.float32)
    with torch.cuda.stream(torch.cuda.Stream()):
        outs = []
        for sc in (short, short, short, long, long, long, short, short, long):
            v, i, c, o = Hh.scene_tensors(sc)
            leaves = [t.requires_grad_() for t in (v, c, o)]
            render = trigrad_b200.render_corrected if corrected else trigrad_b200.render
            out = render(leaves[0], i, leaves[1], leaves[2], w, h, tile, tile, per_pixel_sort=sort, max_layers=0 if corrected else 32)
            outs.append((sc, out[0], torch.autograd.grad(out, leaves, (Hh.cuda(gi), Hh.cuda(gd)))))
        torch.cuda.synchronize()
    for sc in (short, long):
        layers = 0 if corrected else 32
        of = O.forward(sc.vertices, sc.indices, sc.colors, sc.opacities, w, h, tile, tile, 1 / 256, sort, layers)
        assert (np.diff(of.lists.offsets).max() > 128) == (sc is long)
        og = O.backward(sc.vertices, sc.indices, sc.colors, sc.opacities, w, h, of, gi, gd, tile, tile, sort, layers,
                        corrected=corrected)
        for image, grads in ((x[1], x[2]) for x in outs if x[0] is sc):
            assert np.array_equal(image.detach().cpu().numpy().view(np.uint32), of.image.view(np.uint32))
            for a, b in zip(grads, og):
                # prefixes subtracted from the final values lose a few bits more, as in the tests of those gradients
                assert Hh.rel_l2(a.cpu().numpy(), b) <= (2e-4 if corrected else 1e-4)


@pytest.mark.parametrize("triangles, capacity, flags", [
    (4097, 4097 * 64, 4 | 32),       # more triangles than the flag is for
    (100, 100 * 64 - 1, 4 | 32),     # a list that could overflow
    (100, 100 * 64, 32),             # host memory that kernels cannot write
])
def test_not_counting_is_refused_where_it_is_not_safe(triangles, capacity, flags):
    from trigrad_b200 import _native as N

    sc = S.random_triangles(triangles, 128, 128, 0.05, 0.4, name="refused")
    out = trigrad_b200.wrapper.forward_native(*Hh.scene_tensors(sc), 128, 128, 16, 16, 1 / 256, False, True, 32)
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())
    lib = N.lib()
    size = lib.tg_forward_workspace_bytes(triangles, 64, capacity)
    ws = torch.empty(size + 256, dtype=torch.uint8, device="cuda")
    info = torch.zeros(4, dtype=torch.int32).pin_memory()
    image, depth, fw, ids, off, geo, attr, ends, sel = out[:9]
    ids = torch.empty(capacity, dtype=torch.int32, device="cuda")
    t = Hh.scene_tensors(sc)
    status = lib.tg_render_forward(*(ptr(x) for x in (t[0], t[1], t[2], t[3])), triangles, 128, 128, 16, 16, 1 / 256, 1, 32, ptr(image),
                                   ptr(depth), ptr(fw), ptr(ends), ptr(sel), ptr(geo), ptr(attr), ptr(ids), capacity, ptr(off),
                                   ctypes.c_void_p((ws.data_ptr() + 255) // 256 * 256), size, ptr(info), None, flags, ctypes.c_void_p(0))
    assert status == 1


@pytest.mark.filterwarnings("ignore:The CUDA Graph is empty")
def test_not_counting_is_refused_while_the_stream_is_captured():
    from trigrad_b200 import _native as N

    T, tiles = 100, 64
    capacity = T * tiles
    t = Hh.scene_tensors(S.random_triangles(T, 128, 128, 0.05, 0.4, name="captured"))
    out = trigrad_b200.wrapper.forward_native(*t, 128, 128, 16, 16, 1 / 256, False, True, 32)
    image, depth, fw, _, off, geo, attr, ends, sel = out[:9]
    want = image.clone()
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())
    lib = N.lib()
    size = lib.tg_forward_workspace_bytes(T, tiles, capacity)
    ws = torch.empty(size + 256, dtype=torch.uint8, device="cuda")
    ids = torch.empty(capacity, dtype=torch.int32, device="cuda")
    info = torch.zeros(4, dtype=torch.int32).pin_memory()
    stream = torch.cuda.Stream()

    def call():
        return lib.tg_render_forward(*(ptr(x) for x in t), T, 128, 128, 16, 16, 1 / 256, 1, 32, ptr(image), ptr(depth), ptr(fw), ptr(ends),
                                     ptr(sel), ptr(geo), ptr(attr), ptr(ids), capacity, ptr(off),
                                     ctypes.c_void_p((ws.data_ptr() + 255) // 256 * 256), size, ptr(info), None, 4 | 32,
                                     ctypes.c_void_p(stream.cuda_stream))

    image.zero_()
    torch.cuda.synchronize()
    launches = lib.tg_launch_count()
    with torch.cuda.stream(stream):
        graph = torch.cuda.CUDAGraph()
        graph.capture_begin()
        status = call()
        graph.capture_end()
    assert status == N.TG_ERR_BAD_ARG and lib.tg_launch_count() == launches
    torch.cuda.synchronize()
    assert not bool(image.any())
    assert call() == N.TG_OK
    torch.cuda.synchronize()
    assert torch.equal(image, want) and not bool(info.any())


def _stacked(n, w, h, seed):
    """n triangles over the whole image, at few depths, so that order is the triangles' in part."""
    rng = np.random.default_rng(seed)
    xy = np.array([[-3, -3], [3, -3], [0, 5]], np.float32) + rng.normal(size=(n, 1, 2)).astype(np.float32) * 0.01
    z = rng.integers(2, 9, size=(n, 1, 1)).astype(np.float32).repeat(3, axis=1)
    v = np.concatenate([xy, z, 1 / z], axis=2).reshape(3 * n, 4)
    c = rng.random((3 * n, 3), dtype=np.float32)
    o = np.full(3 * n, min(0.5, 20 / n), np.float32)
    return [Hh.cuda(np.ascontiguousarray(x)) for x in (v, np.arange(3 * n, dtype=np.int32).reshape(n, 3), c, o)]


@pytest.mark.parametrize("n", [129, 1023, 1024, 1025, 2049, 4096])
@pytest.mark.parametrize("tile", [16, 8, 32])
@pytest.mark.parametrize("sort", [True, False])
def test_long_lists_of_a_call_that_does_not_count(n, tile, sort):
    """The order of a list at the edges of the chunks it is sorted in, all of it seen in tile order, the first layers otherwise."""
    from trigrad_b200 import _native as N

    w, h = 20, 13
    few, many = _stacked(20, w, h, 1), _stacked(n, w, h, n)
    options = dict(tile_width=tile, tile_height=tile, early_stopping_threshold=0.0, per_pixel_sort=sort, max_layers=32 if sort else 0)
    with torch.cuda.stream(torch.cuda.Stream()), torch.no_grad():
        state = N.host().state(0, torch.cuda.current_stream().cuda_stream)
        for _ in range(65):                                   # the stream may have met long lists before
            trigrad_b200.render(*few, w, h, **options)
        before = state.last_slot
        got = trigrad_b200.render(*many, w, h, **options)
        assert state.last_slot == before                      # went without the count
        want = trigrad_b200.render(*many, w, h, record_timing=True, **options)
        assert state.last_slot != before
        torch.cuda.current_stream().synchronize()
    for a, b in zip(got, want):
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))


@pytest.mark.parametrize("n", [1, 31, 33, 64, 65, 127, 128, 129])
@pytest.mark.parametrize("w, h, tile", [(20, 13, 32), (97, 61, 16), (250, 130, 8)])
def test_lists_that_are_not_moved_together(n, w, h, tile):
    """Entries that go straight to their lists, in turn with calls that keep the lists or count on the same workspace."""
    from trigrad_b200 import _native as N

    mesh = _stacked(n, w, h, n)
    size = (w, h, tile, tile)
    gi = torch.rand((h, w, 4), device="cuda", generator=torch.Generator("cuda").manual_seed(n))

    def gradients(function, **options):
        leaves = [x.detach().requires_grad_() for x in (mesh[0], mesh[2], mesh[3])]
        image, _ = function(leaves[0], mesh[1], leaves[1], leaves[2], *size, **options)
        return [image.detach(), *torch.autograd.grad(image, leaves, gi)]

    calls = {"look": lambda: trigrad_b200.render(*mesh, *size), "fit": lambda: gradients(trigrad_b200.render),
             "lists": lambda: gradients(trigrad_b200.render, per_pixel_sort=False),
             "corrected": lambda: gradients(trigrad_b200.render_corrected)}
    with torch.cuda.stream(torch.cuda.Stream()):
        state = N.host().state(0, torch.cuda.current_stream().cuda_stream)
        want = {}
        for name, call in calls.items():
            state_before = state.last_slot
            trigrad_b200.wrapper.forward_native(*_stacked(150, w, h, 9), w, h, tile, tile, 1 / 256, False, True, 32)     # the next call counts
            want[name] = call()
            assert state.last_slot != state_before
        few, long_list = _stacked(3, w, h, 3), ctypes.c_uint32.from_address(state.long_row + 4)

        def after_short_lists():
            with torch.no_grad():
                for _ in range(65):
                    trigrad_b200.render(*few, *size)
            torch.cuda.current_stream().synchronize()

        after_short_lists()
        for name in ("look", "fit", "look", "lists", "look", "corrected", "fit", "look"):
            if n > 128:
                after_short_lists()                           # the call before met long lists
            assert long_list.value == 0
            before = state.last_slot
            got = calls[name]()
            torch.cuda.current_stream().synchronize()
            assert state.last_slot == before                  # went without the count
            assert long_list.value == (n if n > 128 else 0)   # every list has all the triangles
            assert torch.equal(got[0], want[name][0])
            for a, b in zip(got[1:], want[name][1:]):
                if name == "look":
                    assert torch.equal(a, b)
                else:
                    assert Hh.rel_l2(a.cpu().numpy(), b.cpu().numpy()) <= 1e-5      # order of atomics
        trigrad_b200.wrapper.forward_native(*mesh, w, h, tile, tile, 1 / 256, False, True, 32)
        assert torch.equal(trigrad_b200.render(*mesh, *size, record_timing=True)[0], want["look"][0])
        torch.cuda.current_stream().synchronize()


def test_lists_that_change_between_short_and_long():
    """Calls that meet a long list without having counted get rarer, whatever the pattern; where lists stay short, no call counts."""
    from trigrad_b200 import _native as N

    w, h = 64, 64
    few, many = _stacked(20, w, h, 1), _stacked(300, w, h, 2)
    with torch.cuda.stream(torch.cuda.Stream()), torch.no_grad():
        state = N.host().state(0, torch.cuda.current_stream().cuda_stream)

        def counts(mesh):
            before = state.last_slot
            trigrad_b200.render(*mesh, w, h)
            torch.cuda.current_stream().synchronize()
            return state.last_slot != before

        for short in (1, 2, 5, 16):
            uncounted = 0
            for _ in range(40):
                for _ in range(short):
                    counts(few)
                uncounted += not counts(many)
            assert uncounted <= 3
        for _ in range(64):
            counts(few)
        assert not any(counts(few) for _ in range(300))


def _uncounted_routes():
    w, h = 72, 40

    def packed(m, target):
        rgba, faces = trigrad_b200.pack_mesh(m[2], m[3], m[1])
        x = [m[0].detach().requires_grad_(), rgba.requires_grad_()]
        image, depth = trigrad_b200.render_packed(x[0], faces, x[1], w, h)
        return image.detach(), *torch.autograd.grad((image * target).sum() + depth[torch.isfinite(depth)].sum(), x)

    def step(u8):
        def f(m, target):
            b = views.GradBuffer.allocate(m[0].shape[0], "cuda", 4)
            target = (target * 255).to(torch.uint8) if u8 else target
            image = views.l2_view_step(m[0], m[1], m[2], m[3], target, w, h, b.points, b.colors, b.opacities, b.loss)
            return image, b.points, b.colors, b.opacities, b.loss.reshape(1)
        return f

    def world(kept):
        def f(m, target):
            b = views.GradBuffer.allocate(m[0].shape[0], "cuda", 3)
            p = views.PackedGradients(m[0].shape[0], "cuda") if kept else None
            image = views.l2_world_view_step(m[0][:, :3].contiguous(), torch.eye(4), m[1], m[2], m[3], target, w, h, b.points, b.colors,
                                             b.opacities, b.loss, packed=p)
            return image, b.points, b.colors, b.opacities, b.loss.reshape(1)
        return f

    return w, h, {"packed": packed, "step": step(False), "step_u8": step(True), "world": world(False), "world_packed": world(True)}


@pytest.mark.parametrize("route", ["packed", "step", "step_u8", "world", "world_packed"])
def test_every_route_without_the_count(route):
    """Packed inputs and the fused steps, lists short and long, against the same call when it counts."""
    from trigrad_b200 import _native as N

    w, h, routes = _uncounted_routes()
    run = routes[route]
    few, many = _stacked(20, w, h, 1), _stacked(700, w, h, 2)
    target = torch.rand((h, w, 4), device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    state_here = lambda: N.host().state(0, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    want = {}
    with torch.cuda.stream(torch.cuda.Stream()):
        for name, mesh in (("few", few), ("many", many)):
            trigrad_b200.wrapper.forward_native(*many, w, h, 16, 16, 1 / 256, False, True, 32)      # long: the next call counts
            before = state_here().last_slot
            want[name] = run(mesh, target)
            assert state_here().last_slot != before
        torch.cuda.current_stream().synchronize()
    with torch.cuda.stream(torch.cuda.Stream()):
        for _ in range(65):
            run(few, target)
        torch.cuda.current_stream().synchronize()
        before = state_here().last_slot
        got = {"few": run(few, target), "many": run(many, target)}
        assert state_here().last_slot == before
        torch.cuda.current_stream().synchronize()
    for name in want:
        assert torch.equal(got[name][0], want[name][0])
        for a, b in zip(got[name][1:], want[name][1:]):
            assert Hh.rel_l2(a.cpu().numpy(), b.cpu().numpy()) <= 1e-5      # order of atomics


def test_states_that_share_a_row_of_the_table_of_long_lists():
    """More states have been made than the table has rows: a word that one state's kernel writes is another's to find."""
    from trigrad_b200 import _native as N

    w, h = 50, 40
    few, many = _stacked(20, w, h, 1), _stacked(400, w, h, 2)
    want = {name: trigrad_b200.render(*m, w, h, record_timing=True)[0] for name, m in (("few", few), ("many", many))}
    torch.cuda.synchronize()
    handles = []

    def new_stream():
        s = ctypes.c_void_p()
        assert int(torch.cuda.cudart().cudaStreamCreate(ctypes.addressof(s))) == 0
        handles.append(s.value)
        return s.value

    first = new_stream()
    row = N.host().state(0, first).long_row
    for _ in range(600):
        second = new_stream()
        if N.host().state(0, second).long_row == row:
            break
        assert N.host().state(0, first).long_row == row             # the one used least lately is given back: not this one
    else:
        raise AssertionError("no two states share a row")
    state = {h_: N.host().state(0, h_) for h_ in (first, second)}

    def counts(handle, name):
        before = state[handle].last_slot
        with torch.cuda.stream(torch.cuda.ExternalStream(handle)), torch.no_grad():
            image = trigrad_b200.render(*(few if name == "few" else many), w, h)[0]
            torch.cuda.current_stream().synchronize()
        assert torch.equal(image, want[name])
        return state[handle].last_slot != before

    for handle in (first, second):
        while counts(handle, "few"):
            pass
    assert not counts(first, "many")
    assert counts(second, "few")                   # found the other's word
    for _ in range(6):
        for handle in (first, second, first):
            counts(handle, "many")
            counts(handle, "few")
    torch.cuda.synchronize()
    for handle in handles:
        assert int(torch.cuda.cudart().cudaStreamDestroy(handle)) == 0
