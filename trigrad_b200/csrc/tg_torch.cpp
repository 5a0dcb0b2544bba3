// Host path of the Python entry points: argument checks, allocations, the per-stream state and the autograd nodes, in
// C++ over the C ABI of include/trigrad_b200.h.
//
// A small render is over in 40 us on the GPU; issued from Python (a dozen torch.empty calls, a ctypes call with 31
// arguments, a Python autograd Function whose backward has to take the interpreter lock in the engine's thread) one
// pass of it took 100 us forward only and 360 us with gradients.  Here one call does all of it, without the lock.
//
// The kernels are reached through the shared library that trigrad_b200/_native.py loads (bind() gets its path), so this
// module holds no device code.
#include <dlfcn.h>

#include <algorithm>
#include <atomic>
#include <list>
#include <memory>
#include <mutex>
#include <tuple>
#include <vector>

#include <ATen/Parallel.h>
#include <ATen/TracerMode.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/extension.h>

#include "../../include/trigrad_b200.h"

namespace py = pybind11;
using at::Tensor;
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

namespace {

// ---- the library ---------------------------------------------------------------------------------------------------
struct Api {
#define TG_FN(name) decltype(&tg_##name) name = nullptr;
#define TG_FUNCTIONS(F)                                                                                              \
    F(last_error) F(status_string) F(selection_planes) F(forward_workspace_bytes) F(render_forward)                  \
    F(render_step_l2) F(backward_scratch_bytes) F(blend_backward) F(blend_backward_corrected) F(blend_backward_l2)   \
    F(blend_backward_l2_u8) F(unpack_gradients) F(unpack_gradients_rgba) F(project) F(project_backward)              \
    F(project_clip) F(project_clip_backward) F(clear_gradients) F(unpack_project_backward) F(pack_inputs)
    TG_FUNCTIONS(TG_FN)
#undef TG_FN
};
Api g;
PyObject* g_native_error = nullptr;   // trigrad_b200._native.NativeError
PyObject* g_check_tensor = nullptr;   // trigrad_b200.util check, called to raise the error of a failed check

void bind(const std::string& path, py::object native_error, py::object check_tensor) {
    void* h = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
    if (!h) throw std::runtime_error(std::string("cannot load ") + path + ": " + dlerror());
#define TG_FN(name)                                                                             \
    g.name = reinterpret_cast<decltype(&tg_##name)>(dlsym(h, "tg_" #name));                      \
    if (!g.name) throw std::runtime_error(path + " does not export tg_" #name);
    TG_FUNCTIONS(TG_FN)
#undef TG_FN
    g_native_error = native_error.release().ptr();
    g_check_tensor = check_tensor.release().ptr();
}

// A failed library call, thrown without the interpreter lock and translated into NativeError where the lock is held.
// A std::runtime_error, so that the autograd engine reports it as a RuntimeError (NativeError's base) as well.
struct LibraryError : std::runtime_error {
    std::string stage, detail;
    int status;
    LibraryError(const char* s, int st, const std::string& d)
        : std::runtime_error(std::string("trigrad_b200 ") + s + " failed: status " + std::to_string(st) + " (" + d + ")"),
          stage(s), detail(d), status(st) {}
};
void check(const char* stage, int status) {
    if (status == TG_OK) return;
    std::string detail = g.last_error();
    if (detail.empty()) detail = g.status_string(status);
    throw LibraryError(stage, status, detail);
}

// ---- argument checks -----------------------------------------------------------------------------------------------
// Device, dtype, then shape; the error itself (type and text) is raised by the Python helper.  Needs the lock.
void need(const Tensor& t, const char* name, std::initializer_list<int64_t> shape, at::ScalarType type = at::kFloat) {
    if (t.is_cuda() && t.scalar_type() == type && t.sizes() == at::IntArrayRef(shape.begin(), shape.size())) return;
    py::tuple want(shape.size());
    size_t k = 0;
    for (int64_t s : shape) want[k++] = py::int_(s);
    const char* dt = type == at::kFloat ? "float32" : type == at::kInt ? "int32" : "uint8";
    py::reinterpret_borrow<py::object>(g_check_tensor)(t, name, want, py::module_::import("torch").attr(dt));
    throw py::value_error(std::string(name) + ": wrong tensor");
}
// A tensor that kernels write or add to, taken as so many consecutive floats.  None where a call can do without.
void need_out(const Tensor& t, const char* name, int64_t numel) {
    if (!t.defined()) return;
    if (!t.is_cuda() || t.scalar_type() != at::kFloat) throw py::type_error(std::string(name) + " must be a float32 tensor on cuda");
    if (!t.is_contiguous() || t.numel() < numel)
        throw py::value_error(std::string(name) + " must be contiguous, with " + std::to_string(numel) + " elements");
}
// First dimension of a matrix argument (what `n, _ = t.shape` gives).
int64_t rows(const Tensor& t, const char* name) {
    if (t.dim() != 2) throw py::value_error(std::string(name) + " must have two dimensions");
    return t.size(0);
}
void need_no_proxies() {
    TORCH_CHECK(!c10::impl::TorchDispatchModeTLS::any_modes_set() ||
                    !c10::impl::TorchDispatchModeTLS::get_mode(c10::impl::TorchDispatchModeKey::PROXY),
                "trigrad_b200 cannot be traced by make_fx");
}
// Transforms that the autograd nodes here do not take part in: left alone they would drop tangents or see no kernel at all.
void need_no_transform(std::initializer_list<const Tensor*> differentiable) {
    for (const Tensor* t : differentiable)
        TORCH_CHECK_NOT_IMPLEMENTED(!t->defined() || !t->_fw_grad(/*level=*/0).defined(),
                                    "trigrad_b200 does not implement forward-mode automatic differentiation");
    TORCH_CHECK(!c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode),
                "trigrad_b200 cannot be used inside torch.func transforms (vmap, grad, jvp, jacrev, ...)");
    need_no_proxies();
}
int need_int(int64_t v) {
    TORCH_CHECK(v >= 0 && v <= INT32_MAX, "size out of range");
    return (int)v;
}
// The product as the caller's 64-bit numbers have it (the reference's check); the sign is view_of's to look at.
void need_tile(int64_t tw, int64_t th) {
    int64_t area = 0;
    if (__builtin_mul_overflow(tw, th, &area) ? (tw < 0) == (th < 0) : area > 1024)
        throw py::value_error("tile_width * tile_height must be <= 1024");
}

// Its values in memory, in order: a negated view (torch._neg_view, the imaginary part of a conjugate) is not that.
Tensor plain(const Tensor& t) { return (t.is_neg() ? t.resolve_neg() : t).contiguous(); }

template <class T>
T* data(const Tensor& t) { return t.defined() ? static_cast<T*>(t.data_ptr()) : nullptr; }

// ---- per (device, stream) state ------------------------------------------------------------------------------------
// Workspace, pinned read-back slots and the estimate of the number of list entries.  `use` is held while a forward call
// issues its work: two threads that render on one stream take turns (the workspace holds one render's lists).
struct DeviceState {
    static constexpr int kSlots = 256;
    std::mutex use;
    Tensor workspace, info;      // info [slots,4] int32 pinned: K, longest list, error word, slots
    int slot = 0, last_slot = -1;
    int64_t k_estimate = 0;
    bool short_lists = false;          // the last forward had no tile list beyond TG_SHORT_LIST entries
    // image and tile size of the last successful forward, whose counters and tables the workspace still holds; W = 0: none
    int ready[4] = {0, 0, 0, 0};

    // Packed gradient accumulator, kept zero between calls (`accumulator_zero`: the last call left it so): the kernel that
    // unpacks it zeroes what it reads, so that no call clears 32 bytes per vertex first.
    Tensor accumulator;
    bool accumulator_zero = false;

    explicit DeviceState(at::Device device) {
        workspace = at::empty({0}, at::TensorOptions().dtype(at::kByte).device(device));
        info = at::zeros({kSlots, 4}, at::TensorOptions().dtype(at::kInt)).pin_memory();
    }
    int32_t* words(int s) { return info.data_ptr<int32_t>() + 4 * s; }
    int next_slot() {
        const int s = slot;
        slot = (slot + 1) % kSlots;
        return s;
    }
    // Raise if the kernels of the call that used slot `s` raised the device error word (a bounded wait ran out inside a
    // kernel, so its outputs are not valid).  The word arrives by an asynchronous copy at the end of that call: it is
    // certain to be there once a later event of the same stream has completed.
    void check_error_word(int s) {
        if (s < 0) return;
        const int32_t stale = words(s)[2];
        if (!stale) return;
        words(s)[2] = 0;
        throw std::runtime_error("trigrad_b200: an earlier render reported device error word " + std::to_string(stale) +
                                 " (a bounded wait ran out inside a kernel); its outputs are not valid");
    }
    // Whether a call can do without the number of entries on the host (TG_NO_COUNT): the lists of the last few calls that counted
    // were short, no kernel of a call that did not has said otherwise since (in `long_row`), and the room for every pair of
    // triangle and tile is small.  28 bytes each, so 14 MB.  The wait was the length of the binning and a trip over PCIe in
    // every small call (B200: ten squares, 50x50, forward and backward 99 -> 84 us; 1280 triangles, 256x256, forward 25.3 ->
    // 19.9, with a loss and backward 171 -> 161), by overlap with the calls around it: a caller that waits for every image gains
    // nothing here.
    // "The last few": one at first, twice as many (up to kCountedMax) each time a call that did not count met a long list, which
    // costs it 100 to 200 us where lists have 3300 entries (see sort_words in tg_blend.cu).  So a program whose lists change
    // between short and long pays that a few times and not at every change, and one that has long lists now and then keeps most
    // of the gain (short and such lists in turn, 160x160: 538 us a call when one short call was enough, 108 now, 110 with every
    // call waiting).
    // Such a kernel may write its word after the state is gone, so the rows are nobody's to free: a fixed table, whose rows
    // states that come and go share.  A word that another state's kernel wrote costs a few calls that wait.
    int32_t* const long_row = next_long_row();
    static int32_t* next_long_row() {
        constexpr int kRows = 2 * 128;
        static Tensor& table = *new Tensor(at::zeros({kRows, 4}, at::TensorOptions().dtype(at::kInt)).pin_memory());
        static std::atomic<unsigned> next{0};
        return table.data_ptr<int32_t>() + 4 * (next++ % kRows);
    }
    static constexpr int64_t kNoCountPairs = int64_t(1) << 19;
    static constexpr int kCountedMax = 64;
    int counted_short = 0, counted_needed = 1;
    bool no_count(int64_t T, int64_t tiles) {
        volatile int32_t* longest = long_row + 1;
        if (*longest) {
            *longest = 0;
            short_lists = false;
            counted_short = 0;
            counted_needed = std::min(2 * counted_needed, kCountedMax);
        }
        return counted_short >= counted_needed && T <= TG_NO_COUNT_TRIANGLES && T * tiles <= kNoCountPairs && tiles <= kNoCountTiles;
    }
    void counted(bool all_short) {
        short_lists = all_short;
        counted_short = all_short ? std::min(counted_short + 1, kCountedMax) : 0;
    }
    static constexpr int64_t kNoCountTiles = 1184;
    // After a forward call that used slot `s` has returned: it waited for work recorded after the previous call's on
    // this stream, so the previous call's error word has arrived.
    void finish_call(int s) {
        const int prev = last_slot;
        last_slot = s;
        if (prev != s) check_error_word(prev);
    }
    void* workspace_of(size_t bytes, size_t* have) {
        if ((size_t)workspace.numel() < bytes + 256) {
            workspace = at::empty({(int64_t)(bytes + bytes / 4 + 512)}, workspace.options());
            ready[0] = 0;
        }
        const uintptr_t p = (uintptr_t)workspace.data_ptr(), base = (p + 255) / 256 * 256;
        *have = (size_t)workspace.numel() - (base - p);
        return (void*)base;
    }
};

// The state's accumulator for the time of one backward (under `use`), or a fresh one where it would keep more than
// kAccumulatorMax bytes alive.
constexpr size_t kAccumulatorMax = size_t(256) << 20;
struct Accumulator {
    DeviceState& state;
    Tensor t;
    bool kept;
    Accumulator(DeviceState& s, size_t bytes, const at::TensorOptions& byte_options) : state(s), kept(bytes <= kAccumulatorMax) {
        if (!kept) {
            t = at::zeros({(int64_t)bytes}, byte_options);
            return;
        }
        if (!state.accumulator.defined() || (size_t)state.accumulator.numel() < bytes) {
            state.accumulator = at::zeros({(int64_t)bytes}, byte_options);
        } else if (!state.accumulator_zero) {
            state.accumulator.zero_();
        }
        state.accumulator_zero = false;
        t = state.accumulator;
    }
    void unpacked() { state.accumulator_zero = kept; }       // by a kernel with TG_UNPACK_CLEAR
};

// At most kStates of them: a program that keeps making streams gives back the workspace of the one not used for longest.
constexpr size_t kStates = 128;
struct StateEntry {
    int device;
    cudaStream_t stream;
    std::shared_ptr<DeviceState> state;
};
std::mutex g_states_lock;
std::list<StateEntry>& states() {
    static auto* s = new std::list<StateEntry>();   // never destroyed: its tensors must not outlive the CUDA context
    return *s;
}
std::shared_ptr<DeviceState> state_of(int device, cudaStream_t stream) {
    std::lock_guard<std::mutex> lock(g_states_lock);
    auto& all = states();
    for (auto it = all.begin(); it != all.end(); ++it)
        if (it->device == device && it->stream == stream) {
            if (it != all.begin()) all.splice(all.begin(), all, it);
            return it->state;
        }
    all.push_front({device, stream, std::make_shared<DeviceState>(at::Device(at::kCUDA, (at::DeviceIndex)device))});
    if (all.size() > kStates) all.pop_back();
    return all.front().state;
}

struct Where {      // device made current for the scope, its current stream
    c10::cuda::CUDAGuard guard;
    int device;
    cudaStream_t stream;
    explicit Where(const Tensor& t) : guard(t.device()), device(t.get_device()) {
        stream = c10::cuda::getCurrentCUDAStream(device).stream();
    }
};

// ---- forward -------------------------------------------------------------------------------------------------------
struct View {       // the arguments of a render that are not tensors
    int W, H, tw, th;
    double thr;
    bool sort;
    int layers;
    int tiles() const { return ((W + tw - 1) / tw) * ((H + th - 1) / th); }
    int64_t pixels() const { return (int64_t)W * H; }
};

// What a forward leaves for its backward: sizes and places (`Layout`), and two tensors - final weights, ends, records
// and tile offsets in one allocation (`blob`), and the selection, or the lists where there is none.  Between the passes they belong to
// autograd (SavedVariable, ctx.save_for_backward), which may move them; so places are offsets, never addresses.
struct Layout {
    View v;
    int V = 0, T = 0, planes = 0;
    int64_t K = 0;
    size_t final_w = 0, ends = 0, geo = 0, attr = 0, offsets = 0, bytes = 0;      // of blob

    Layout() = default;
    Layout(const View& view, int n_vertices, int n_triangles) : v(view), V(n_vertices), T(n_triangles) {
        const size_t px = (size_t)v.pixels();
        auto take = [&](size_t n) { const size_t at = bytes; bytes += (n + 255) / 256 * 256; return at; };
        final_w = take(4 * px);
        ends = take(4 * px);
        geo = take(4 * (size_t)T * TG_GEO_WORDS);
        attr = take(4 * (size_t)T * TG_ATTR_WORDS);
        offsets = take(4 * ((size_t)v.tiles() + 1));
    }
};
struct Saved {
    Layout l;
    Tensor blob, ids, selection;
    template <class X>
    X* at(size_t place) const { return reinterpret_cast<X*>(data<char>(blob) + place); }
    float* final_w() const { return at<float>(l.final_w); }
    float* geo() const { return at<float>(l.geo); }
    float* attr() const { return at<float>(l.attr); }
    int32_t* ends() const { return at<int32_t>(l.ends); }
    int32_t* offsets() const { return at<int32_t>(l.offsets); }
    int32_t* id_list() const { return data<int32_t>(ids); }
    int32_t* sel() const { return data<int32_t>(selection); }
};

struct ForwardOut {
    Tensor image, depthmap;
    Saved saved;
    std::vector<float> stage_ms;    // five, when asked for
};

struct L2Step {     // forward, loss and gradients in one call (tg_render_step_l2)
    const float* target;
    float *loss, *gV, *gC, *gO;
    int mode;
    void* scratch;
    size_t scratch_bytes;
};

// `opacities` undefined: packed inputs (indices [T,4], colors [V,4]).  Called without the interpreter lock.
// `count`: whether the caller needs the number of list entries (otherwise Layout::K may be the room for them).
//   kAlways                it does
//   kUnlessSmall           it needs neither it nor the lists: tile offsets and ids may be left unwritten
//   kUnlessSmallKeepLists  it may walk the lists later, where there is no selection
// Where the lists are left unwritten Saved::ids is undefined, and backward() refuses to walk them.
enum class Count { kAlways, kUnlessSmall, kUnlessSmallKeepLists };
ForwardOut forward(const Tensor& vertices_, const Tensor& indices_, const Tensor& colors_, const Tensor& opacities_,
                   const View& v, bool record_timing, bool save_selection, bool cull, int64_t selection_max_bytes, Count count,
                   const L2Step* step = nullptr) {
    const Tensor vertices = plain(vertices_), indices = plain(indices_), colors = plain(colors_);
    const bool packed = !opacities_.defined();
    const Tensor opacities = packed ? Tensor() : plain(opacities_);
    const Where w(vertices);
    const int T = need_int(indices.size(0)), V = need_int(vertices.size(0));
    const auto options = vertices.options().requires_grad(false);
    ForwardOut out;
    out.image = at::empty({v.H, v.W, 4}, options);
    out.depthmap = at::empty({v.H, v.W}, options);
    // a trace records the Python function around this call, for which its outputs have to be known; nothing else
    at::tracer::impl::NoTracerDispatchMode untraced;
    Saved& s = out.saved;
    s.l = Layout(v, V, T);
    s.blob = at::empty({(int64_t)s.l.bytes}, options.dtype(at::kByte));
    const int64_t planes = save_selection ? g.selection_planes(v.sort ? 1 : 0, v.layers) : 0;
    if (planes > 0 && planes * v.pixels() * 4 <= selection_max_bytes) {
        s.l.planes = (int)planes;
        s.selection = at::empty({planes, v.H, v.W}, options.dtype(at::kInt));
    }
    if (record_timing) out.stage_ms.resize(5);
    const unsigned fixed_flags = (cull ? TG_FORWARD_CULL_TILES : 0u) | (packed ? TG_INPUT_PACKED : 0u) | TG_INFO_MAPPED;
    const auto state = state_of(w.device, w.stream);
    std::lock_guard<std::mutex> lock(state->use);
    // Without the count the lists have room for every pair, however few there are.  Where they are kept for a backward that is
    // let be up to as much as the graph keeps anyway (image, depth map, blob), so a live graph at most doubles, by 2 MB at most;
    // beyond it the call counts.  (Corrected gradients, forward and backward, B200: 604 triangles, 142x104, a third of the rest,
    // 90 us without the count against 99 with it; 1140, 346x192, six tenths, 135 against 139.)
    const bool lists_small = count != Count::kUnlessSmallKeepLists || s.selection.defined() ||
                             4 * (int64_t)T * v.tiles() <= 20 * v.pixels() + (int64_t)s.l.bytes;
    const bool no_count = state->no_count(T, v.tiles()) && count != Count::kAlways && lists_small && !record_timing && !step &&
                          c10::cuda::currentStreamCaptureStatusMayInitCtx() == c10::cuda::CaptureStatus::None;
    const unsigned lists_unused = count == Count::kUnlessSmall || s.selection.defined() ? TG_LISTS_UNUSED : 0u;
    int64_t cap = no_count ? (int64_t)T * v.tiles()
                           : std::max<int64_t>(state->k_estimate + state->k_estimate / 4 + 1024, 2 * (int64_t)T + 1024);
    while (true) {
        s.ids = at::empty({cap}, options.dtype(at::kInt));
        size_t have = 0;
        void* ws = state->workspace_of(g.forward_workspace_bytes(T, v.tiles(), (uint32_t)cap), &have);
        const int key[4] = {v.W, v.H, v.tw, v.th};
        const bool ready = std::equal(key, key + 4, state->ready);
        state->ready[0] = 0;                     // until this call has succeeded
        const unsigned flags = fixed_flags | (ready ? TG_WORKSPACE_READY : 0u) |
                               (no_count ? TG_NO_COUNT | lists_unused : state->short_lists && !step ? TG_EXPECT_SHORT_LISTS : 0u);
        const int slot = no_count ? -1 : state->next_slot();
        int32_t* info = no_count ? state->long_row : state->words(slot);
        float* ms = record_timing ? out.stage_ms.data() : nullptr;
        const double n = 4.0 * v.pixels();
        const int status =
            step ? g.render_step_l2(data<float>(vertices), data<int32_t>(indices), data<float>(colors), data<float>(opacities),
                                    T, V, v.W, v.H, v.tw, v.th, (float)v.thr, v.layers, step->target, (float)(2.0 / n),
                                    (float)(1.0 / n), step->loss, data<float>(out.image), data<float>(out.depthmap),
                                    s.final_w(), s.ends(), s.geo(), s.attr(), s.id_list(), (uint32_t)cap, s.offsets(),
                                    step->gV, step->gC, step->gO, step->mode, ws, have, step->scratch,
                                    step->scratch_bytes, (uint32_t*)info, ms, flags, w.stream)
                 : g.render_forward(data<float>(vertices), data<int32_t>(indices), data<float>(colors),
                                    data<float>(opacities), T, v.W, v.H, v.tw, v.th, (float)v.thr, v.sort ? 1 : 0,
                                    v.layers, data<float>(out.image), data<float>(out.depthmap), s.final_w(), s.ends(),
                                    s.sel(), s.geo(), s.attr(), s.id_list(), (uint32_t)cap, s.offsets(), ws, have, (uint32_t*)info, ms, flags, w.stream);
        if (no_count) {
            check("render_forward", status);
            std::copy(key, key + 4, state->ready);
            state->check_error_word(state->last_slot);       // of an earlier call that counted; may yet arrive
            s.l.K = cap;
            if (lists_unused) s.ids = Tensor();
            return out;
        }
        s.l.K = (uint32_t)info[0];
        if (status == TG_ERR_CAPACITY) {
            cap = s.l.K + s.l.K / 4 + 1024;              // what the call says it needs
            continue;
        }
        check(step ? "render_step_l2" : "render_forward", status);
        std::copy(key, key + 4, state->ready);
        state->counted((uint32_t)info[1] <= TG_SHORT_LIST);
        state->finish_call(slot);
        state->k_estimate = std::max<int64_t>(s.l.K, (uint32_t)info[3]);
        return out;
    }
}

// ---- backward ------------------------------------------------------------------------------------------------------
enum class Kind { kReference, kCorrected, kPacked };

// Raise when the forward's error word has arrived by now and is set (no waiting here): lists built by a kernel whose
// bounded wait ran out must not be walked.
void check_last_forward(const Where& w) {
    const auto state = state_of(w.device, w.stream);
    state->check_error_word(state->last_slot);
}

// Gradients in the order of the inputs: vertices, colours, opacities - or vertices, rgba with packed inputs.
std::vector<Tensor> backward(Kind kind, const Saved& s, const Tensor& image, const Tensor& depthmap, Tensor gi, Tensor gd) {
    const Where w(image);
    check_last_forward(w);
    TORCH_CHECK(s.ids.defined() || (s.selection.defined() && kind != Kind::kCorrected),
                "this backward walks the tile lists, which the forward did not leave");
    const auto options = image.options().requires_grad(false);
    std::vector<Tensor> out;
    const View& v = s.l.v;
    const int V = s.l.V;
    out.push_back(at::empty({V, 4}, options));
    if (kind == Kind::kPacked) {
        out.push_back(at::empty({V, 4}, options));
    } else {
        out.push_back(at::empty({V, 3}, options));
        out.push_back(at::empty({V}, options));
    }
    if (!gi.defined() && !gd.defined()) {
        for (auto& t : out) t.zero_();
        return out;
    }
    gi = gi.defined() ? plain(gi) : at::zeros_like(image);      // only the depth map was used downstream
    gd = gd.defined() ? plain(gd) : Tensor();                  // none: taken as zero by the kernel
    const size_t nscratch = g.backward_scratch_bytes(V);
    const auto state = state_of(w.device, w.stream);
    std::lock_guard<std::mutex> lock(state->use);
    if (kind == Kind::kCorrected) {
        const Tensor scratch = at::empty({(int64_t)nscratch}, options.dtype(at::kByte));
        check("blend_backward_corrected",
              g.blend_backward_corrected(s.geo(), s.attr(), s.id_list(), s.offsets(), V, v.W, v.H, v.tw, v.th, v.sort, v.layers,
                                         data<float>(gi), data<float>(gd), data<float>(image), data<float>(depthmap),
                                         s.final_w(), s.ends(), data<float>(out[0]), data<float>(out[1]), data<float>(out[2]),
                                         0, scratch.data_ptr(), nscratch, w.stream));
        return out;
    }
    Accumulator sums(*state, nscratch, options.dtype(at::kByte));
    check("blend_backward", g.blend_backward(s.geo(), s.attr(), s.id_list(), s.offsets(), V, v.W, v.H, v.tw, v.th, v.sort,
                                             v.layers, data<float>(gi), data<float>(gd), data<float>(image),
                                             data<float>(depthmap), s.final_w(), s.ends(), s.sel(), nullptr, nullptr, nullptr,
                                             TG_ACCUMULATE_PACKED, sums.t.data_ptr(), nscratch, w.stream));
    if (kind == Kind::kPacked)
        check("unpack_gradients_rgba", g.unpack_gradients_rgba(sums.t.data_ptr(), nscratch, V, 0.f, nullptr, data<float>(out[0]),
                                                               data<float>(out[1]), TG_UNPACK_CLEAR, w.stream));
    else
        check("unpack_gradients", g.unpack_gradients(sums.t.data_ptr(), nscratch, V, 0.f, nullptr, data<float>(out[0]),
                                                     data<float>(out[1]), data<float>(out[2]), TG_UNPACK_CLEAR, w.stream));
    sums.unpacked();
    return out;
}

// A tensor that autograd kept: what was saved, or what a saved-tensor hook made of it in between, which only has to have
// the same device, type and number of elements (`at_least`: or more of them).
Tensor kept(Tensor t, at::Device device, at::ScalarType type, int64_t numel, bool at_least = false) {
    TORCH_CHECK(t.defined() && t.device() == device && t.scalar_type() == type &&
                    (at_least ? t.numel() >= numel : t.numel() == numel),
                "a tensor saved for backward came back with another device, type or size");
    t = plain(t);
    return ((uintptr_t)t.data_ptr() & 15) != 0 ? t.clone() : t;      // the kernels load 16 bytes at a time
}
struct Kept {
    Tensor image, depthmap;
    Saved saved;
};
Kept kept_all(const Layout& l, const Tensor& image, const Tensor& depthmap, const Tensor& blob, const Tensor& ids,
              const Tensor& selection) {
    const int64_t px = l.v.pixels();
    const at::Device d = image.device();
    return {kept(image, d, at::kFloat, 4 * px), kept(depthmap, d, at::kFloat, px),
            {l, kept(blob, d, at::kByte, (int64_t)l.bytes), l.planes > 0 ? Tensor() : kept(ids, d, at::kInt, l.K, true),
             l.planes > 0 ? kept(selection, d, at::kInt, l.planes * px) : Tensor()}};
}

struct RenderBackward : public Node {
    Kind kind = Kind::kReference;
    Layout layout;
    SavedVariable image, depthmap;           // outputs of this node
    SavedVariable blob, ids, selection;      // the lists or the selection
    struct Shape { at::DimVector sizes; at::TensorOptions options; };
    std::vector<Shape> zeros;                // mesh without triangles: nothing saved, the gradients' shapes
    bool released = false;
    std::mutex lock;

    std::string name() const override { return "RenderBackward"; }
    variable_list apply(variable_list&& grads) override {
        std::lock_guard<std::mutex> hold(lock);
        variable_list out;
        TORCH_CHECK(!released, torch::autograd::ERR_BACKWARD_TWICE);
        if (!zeros.empty()) {
            for (const auto& z : zeros) out.push_back(at::zeros(z.sizes, z.options));
            return out;
        }
        const Tensor im = image.unpack(shared_from_this()), dm = depthmap.unpack(shared_from_this()), bl = blob.unpack(),
                     li = ids.unpack(), se = selection.unpack();
        at::AutoDispatchBelowADInplaceOrView below_autograd;
        const Kept k = kept_all(layout, im, dm, bl, li, se);
        for (auto& t : backward(kind, k.saved, k.image, k.depthmap, grads[0], grads[1])) out.push_back(std::move(t));
        return out;
    }
    void release_variables() override {
        std::lock_guard<std::mutex> hold(lock);
        released = true;
        for (SavedVariable* s : {&image, &depthmap, &blob, &ids, &selection}) s->reset_data();
    }
};

struct ImageAndDepth {
    Tensor image, depthmap;
    std::vector<float> stage_ms;
};

// Forward with the gradient node attached when gradients are wanted.  Without the interpreter lock.
ImageAndDepth render_graph(Kind kind, const Tensor& vertices, const Tensor& indices, const Tensor& colors,
                           const Tensor& opacities, View v, bool record_timing, bool cull_tiles,
                           int64_t selection_max_bytes) {
    const int64_t T = indices.size(0);
    if (v.layers <= 0) v.layers = need_int(T + 1);
    const bool wants_grad = at::GradMode::is_enabled() && (vertices.requires_grad() || colors.requires_grad() ||
                                                           (opacities.defined() && opacities.requires_grad()));
    std::shared_ptr<RenderBackward> node;
    if (wants_grad) {
        node = std::shared_ptr<RenderBackward>(new RenderBackward(), torch::autograd::deleteNode);
        node->kind = kind;
        if (kind == Kind::kPacked) node->set_next_edges(torch::autograd::collect_next_edges(vertices, colors));
        else node->set_next_edges(torch::autograd::collect_next_edges(vertices, colors, opacities));
    }
    ImageAndDepth r;
    Saved saved;
    {
        at::AutoDispatchBelowADInplaceOrView below_autograd;
        if (T < 1) {
            const c10::cuda::CUDAGuard guard(colors.device());
            const auto options = colors.options().requires_grad(false);
            r.image = at::zeros({v.H, v.W, 4}, options);
            r.image.select(2, 3).fill_(1.0);
            r.depthmap = at::full({v.H, v.W}, INFINITY, options);
            if (node) {
                for (const Tensor* t : {&vertices, &colors, &opacities})
                    if (t->defined()) node->zeros.push_back({at::DimVector(t->sizes()), t->options().requires_grad(false)});
            }
        } else {
            // the corrected gradients walk the lists themselves and need no selection; nor does a render nobody differentiates
            ForwardOut f = forward(vertices, indices, colors, opacities, v, record_timing,
                                   wants_grad && kind != Kind::kCorrected, cull_tiles, selection_max_bytes,
                                   wants_grad ? Count::kUnlessSmallKeepLists : Count::kUnlessSmall);
            r.image = std::move(f.image);
            r.depthmap = std::move(f.depthmap);
            r.stage_ms = std::move(f.stage_ms);
            saved = std::move(f.saved);
        }
    }
    if (node) {
        torch::autograd::set_history(r.image, node);
        torch::autograd::set_history(r.depthmap, node);
        if (saved.blob.defined()) {
            node->layout = saved.l;
            node->image = SavedVariable(r.image, /*is_output=*/true);
            node->depthmap = SavedVariable(r.depthmap, /*is_output=*/true);
            node->blob = SavedVariable(saved.blob, false);
            if (saved.selection.defined()) node->selection = SavedVariable(saved.selection, false);
            else node->ids = SavedVariable(saved.ids, false);
        }
    }
    return r;
}

// ---- fused mean-squared-error step ---------------------------------------------------------------------------------
struct Grads {      // where a step's gradients and loss go: the three tensors and the loss, or a packed accumulator
    Tensor vertices, colors, opacities, loss, packed;
};

Tensor l2_step(const Tensor& vertices, const Tensor& indices, const Tensor& colors, const Tensor& opacities,
               const Tensor& target_, const View& v, const Grads& to, bool one_kernel, bool cull,
               int64_t selection_max_bytes) {
    const at::AutoDispatchBelowADInplaceOrView below_autograd;
    const Where w(vertices);
    const int V = need_int(vertices.size(0));
    const Tensor target = plain(target_);
    const size_t nscratch = g.backward_scratch_bytes(V);
    const bool packed = to.packed.defined();
    const double n = 4.0 * v.pixels();
    const auto byte_options = vertices.options().dtype(at::kByte).requires_grad(false);
    if (one_kernel) {
        const Tensor scratch = packed ? to.packed : at::empty({(int64_t)nscratch}, byte_options);
        L2Step step;
        step.target = data<float>(target);
        step.mode = packed ? TG_ACCUMULATE_PACKED : 1;
        step.loss = packed ? nullptr : data<float>(to.loss);
        step.gV = packed ? nullptr : data<float>(to.vertices);
        step.gC = packed ? nullptr : data<float>(to.colors);
        step.gO = packed ? nullptr : data<float>(to.opacities);
        step.scratch = scratch.data_ptr();
        step.scratch_bytes = (size_t)scratch.numel();
        return forward(vertices, indices, colors, opacities, v, false, false, cull, 0, Count::kAlways, &step).image;
    }
    const ForwardOut f = forward(vertices, indices, colors, opacities, v, false, true, cull, selection_max_bytes, Count::kUnlessSmall);
    const Saved& s = f.saved;
    TORCH_CHECK_VALUE(s.selection.defined(), "the fused L2 backward needs per_pixel_sort=True and max_layers <= 32");
    auto backward_into = [&](const Tensor& sums) {
        check("blend_backward_l2",
              target.scalar_type() == at::kByte
                  ? g.blend_backward_l2_u8(s.geo(), s.attr(), s.id_list(), s.offsets(), V, v.W, v.H, v.tw, v.th, 1, v.layers,
                                           data<uint8_t>(target), (float)(2.0 / n), (float)(1.0 / n), nullptr,
                                           data<float>(f.image), data<float>(f.depthmap), s.final_w(), s.ends(), s.sel(), nullptr,
                                           nullptr, nullptr, TG_ACCUMULATE_PACKED, sums.data_ptr(), (size_t)sums.numel(), w.stream)
                  : g.blend_backward_l2(s.geo(), s.attr(), s.id_list(), s.offsets(), V, v.W, v.H, v.tw, v.th, 1, v.layers,
                                        data<float>(target), (float)(2.0 / n), (float)(1.0 / n), nullptr,
                                        data<float>(f.image), data<float>(f.depthmap), s.final_w(), s.ends(), s.sel(), nullptr,
                                        nullptr, nullptr, TG_ACCUMULATE_PACKED, sums.data_ptr(), (size_t)sums.numel(), w.stream));
    };
    if (packed) {
        backward_into(to.packed);
        return f.image;
    }
    const auto state = state_of(w.device, w.stream);
    std::lock_guard<std::mutex> lock(state->use);
    Accumulator sums(*state, nscratch, byte_options);
    backward_into(sums.t);
    check("unpack_gradients", g.unpack_gradients(sums.t.data_ptr(), nscratch, V, (float)(1.0 / n), data<float>(to.loss),
                                                 data<float>(to.vertices), data<float>(to.colors), data<float>(to.opacities),
                                                 1 | TG_UNPACK_CLEAR, w.stream));
    sums.unpacked();
    return f.image;
}

// ---- projection ----------------------------------------------------------------------------------------------------
struct Matrix { float m[16]; };

Tensor project(const Tensor& points_, const Matrix& pv) {
    const at::AutoDispatchBelowADInplaceOrView below_autograd;
    const Tensor points = plain(points_);
    const Where w(points);
    const Tensor out = at::empty({points.size(0), 4}, points.options().requires_grad(false));
    check("project", g.project(data<float>(points), need_int(points.size(0)), pv.m, data<float>(out), w.stream));
    return out;
}

void project_backward(const Tensor& points_, const Matrix& pv, const Tensor& grad_vertices_, const Tensor& grad_points,
                      bool accumulate) {
    const at::AutoDispatchBelowADInplaceOrView below_autograd;
    const Tensor points = plain(points_), grad_vertices = plain(grad_vertices_);
    const Where w(points);
    check("project_backward", g.project_backward(data<float>(points), need_int(points.size(0)), pv.m,
                                                 data<float>(grad_vertices), data<float>(grad_points), accumulate, w.stream));
}

Tensor world_step(const Tensor& points_, const Matrix& pv, const Tensor& indices, const Tensor& colors,
                  const Tensor& opacities, const Tensor& target, const View& v, const Grads& to, bool one_kernel,
                  int64_t selection_max_bytes) {
    const at::AutoDispatchBelowADInplaceOrView below_autograd;
    const Tensor points = plain(points_);
    const Where w(points);
    const Tensor vertices = project(points, pv);
    if (!to.packed.defined()) {
        Grads inner = to;
        inner.vertices = at::zeros_like(vertices);
        const Tensor image = l2_step(vertices, indices, colors, opacities, target, v, inner, one_kernel, true,
                                     selection_max_bytes);
        project_backward(points, pv, inner.vertices, to.vertices, true);
        return image;
    }
    const Tensor image = l2_step(vertices, indices, colors, opacities, target, v, to, one_kernel, true, selection_max_bytes);
    check("unpack_project_backward",
          g.unpack_project_backward(to.packed.data_ptr(), (size_t)to.packed.numel(), need_int(points.size(0)),
                                    data<float>(points), pv.m, (float)(1.0 / (4.0 * v.pixels())), data<float>(to.loss),
                                    data<float>(to.vertices), data<float>(to.colors), data<float>(to.opacities), w.stream));
    return image;
}

// ---- projection with near-plane splitting --------------------------------------------------------------------------
std::vector<Tensor> project_clip_backward(const Tensor& points, const Tensor& indices, const Tensor& colors,
                                          const Tensor& opacities, const Matrix& pv, const Tensor& grad_vertices,
                                          const Tensor& grad_colors, const Tensor& grad_opacities) {
    at::AutoDispatchBelowADInplaceOrView below_autograd;
    const Tensor p = plain(points), i = plain(indices), c = plain(colors), o = plain(opacities);
    const Where w(p);
    const int64_t T = i.size(0);
    const auto options = p.options().requires_grad(false);
    auto upstream = [&](const Tensor& t, at::IntArrayRef shape) { return t.defined() ? plain(t) : at::zeros(shape, options); };
    const Tensor gv = upstream(grad_vertices, {6 * T, 4}), gc = upstream(grad_colors, {6 * T, 3}), go = upstream(grad_opacities, {6 * T});
    std::vector<Tensor> out = {at::empty_like(p), at::empty_like(c), at::empty_like(o)};
    check("clear_gradients", g.clear_gradients(data<float>(out[0]), data<float>(out[1]), data<float>(out[2]), need_int(p.size(0)),
                                               w.stream));
    check("project_clip_backward",
          g.project_clip_backward(data<float>(p), data<int32_t>(i), data<float>(c), data<float>(o), need_int(T), pv.m,
                                  data<float>(gv), data<float>(gc), data<float>(go), data<float>(out[0]),
                                  data<float>(out[1]), data<float>(out[2]), w.stream));
    return out;
}

struct ProjectClipBackward : public Node {
    SavedVariable points, indices, colors, opacities;
    Matrix pv;
    std::mutex lock;

    std::string name() const override { return "ProjectClipBackward"; }
    variable_list apply(variable_list&& grads) override {
        std::lock_guard<std::mutex> hold(lock);
        return project_clip_backward(points.unpack().detach(), indices.unpack(), colors.unpack().detach(),
                                     opacities.unpack().detach(), pv, grads[0], grads[1], grads[2]);
    }
    void release_variables() override {
        std::lock_guard<std::mutex> hold(lock);
        points.reset_data(); indices.reset_data(); colors.reset_data(); opacities.reset_data();
    }
};

std::tuple<Tensor, Tensor, Tensor, Tensor> project_clip(const Tensor& points_, const Tensor& indices_, const Tensor& colors_,
                                                        const Tensor& opacities_, const Matrix& pv) {
    const Tensor points = plain(points_), indices = plain(indices_), colors = plain(colors_),
                 opacities = plain(opacities_);
    std::shared_ptr<ProjectClipBackward> node;
    if (at::GradMode::is_enabled() && (points.requires_grad() || colors.requires_grad() || opacities.requires_grad())) {
        node = std::shared_ptr<ProjectClipBackward>(new ProjectClipBackward(), torch::autograd::deleteNode);
        node->set_next_edges(torch::autograd::collect_next_edges(points, colors, opacities));
        node->points = SavedVariable(points, false);
        node->indices = SavedVariable(indices, false);
        node->colors = SavedVariable(colors, false);
        node->opacities = SavedVariable(opacities, false);
        node->pv = pv;
    }
    Tensor ov, oi, oc, oo;
    {
        at::AutoDispatchBelowADInplaceOrView below_autograd;
        const Where w(points);
        const int64_t T = indices.size(0);
        const auto options = points.options().requires_grad(false);
        ov = at::empty({6 * T, 4}, options);
        oi = at::empty({2 * T, 3}, options.dtype(at::kInt));
        oc = at::empty({6 * T, 3}, options);
        oo = at::empty({6 * T}, options);
        check("project_clip", g.project_clip(data<float>(points), data<int32_t>(indices), data<float>(colors),
                                             data<float>(opacities), need_int(T), pv.m, data<float>(ov), data<int32_t>(oi),
                                             data<float>(oc), data<float>(oo), w.stream));
    }
    if (node) {
        torch::autograd::set_history(ov, node);
        torch::autograd::set_history(oc, node);
        torch::autograd::set_history(oo, node);
    }
    return {ov, oi, oc, oo};
}

// ---- what Python sees ----------------------------------------------------------------------------------------------
// Checks with the interpreter lock, work without it.
using Optional = std::optional<Tensor>;
Tensor or_none(const Optional& t) { return t ? *t : Tensor(); }

// `binned` false: a mesh without triangles, which no kernel sees; its tile size is not looked at.
View view_of(bool binned, int64_t W, int64_t H, int64_t tw, int64_t th, double thr, bool sort, int64_t layers) {
    need_int(W);
    need_int(H);
    if (binned) {
        if (tw < 1 || th < 1) throw py::value_error("tile_width and tile_height must be positive");
        need_tile(tw, th);                       // so both fit an int
        // fewer than 2^31 tiles, and pixels on a side with the last tile rounded up
        if (W > INT32_MAX - tw || H > INT32_MAX - th || ((W + tw - 1) / tw) * ((H + th - 1) / th) >= INT32_MAX)
            throw py::value_error("too many tiles");
    } else {
        tw = th = 1;
    }
    return {(int)W, (int)H, (int)tw, (int)th, thr, sort, (int)std::clamp<int64_t>(layers, INT32_MIN, INT32_MAX)};
}

Matrix matrix_of(const py::buffer& b) {
    const py::buffer_info i = b.request();
    if (i.itemsize != 4 || i.format != py::format_descriptor<float>::format() || i.size != 16)
        throw py::value_error("pv must be a 4x4 matrix");
    Matrix m;
    std::copy_n(static_cast<const float*>(i.ptr), 16, m.m);
    return m;
}

py::object py_render(int kind, const Tensor& vertices, const Tensor& indices, const Tensor& colors,
                     const Optional& opacities_, int64_t W, int64_t H, int64_t tw, int64_t th, double thr, bool timing,
                     bool sort, int64_t layers, bool cull, int64_t selection_max_bytes) {
    need_tile(tw, th);
    if (torch::jit::tracer::isTracing()) return py::none();          // the caller's autograd function is what a trace can hold
    const Tensor opacities = or_none(opacities_);
    need_no_transform({&vertices, &colors, &opacities});
    const int64_t V = rows(vertices, "vertices");
    need(vertices, "vertices", {V, 4});
    if ((Kind)kind == Kind::kPacked) {
        need(colors, "rgba", {V, 4});
        need(indices, "faces", {rows(indices, "faces"), 4}, at::kInt);
    } else {
        need(colors, "colors", {V, 3});
        need(opacities, "opacities", {V});
        need(indices, "indices", {rows(indices, "indices"), 3}, at::kInt);
    }
    const View v = view_of(indices.size(0) > 0, W, H, tw, th, thr, sort, layers);
    ImageAndDepth r;
    {
        py::gil_scoped_release nogil;
        r = render_graph((Kind)kind, vertices, indices, colors, opacities, v, timing, cull, selection_max_bytes);
    }
    if (!timing) return py::make_tuple(std::move(r.image), std::move(r.depthmap));
    return py::make_tuple(std::move(r.image), std::move(r.depthmap),
                          r.stage_ms.empty() ? py::object(py::none()) : py::cast(r.stage_ms));
}

// The separate tensors a caller of the forward alone gets: views of the one allocation.
Tensor part(const Saved& s, size_t place, at::ScalarType type, at::IntArrayRef shape) {
    int64_t n = 4;
    for (int64_t d : shape) n *= d;
    return s.blob.narrow(0, (int64_t)place, n).view(type).view(shape);
}

// opacities None: packed inputs
py::object py_forward(const Tensor& vertices, const Tensor& indices, const Tensor& colors, const Optional& opacities,
                      int64_t W, int64_t H, int64_t tw, int64_t th, double thr, bool timing, bool sort, int64_t layers,
                      bool save_selection, bool cull, int64_t selection_max_bytes) {
    need_no_proxies();
    const View v = view_of(true, W, H, tw, th, thr, sort, layers);
    ForwardOut f;
    Tensor fw, ids, off, geo, attr, ends;
    {
        py::gil_scoped_release nogil;
        at::AutoDispatchBelowADInplaceOrView below_autograd;
        f = forward(vertices, indices, colors, or_none(opacities), v, timing, save_selection, cull, selection_max_bytes, Count::kAlways);
        const Saved& s = f.saved;
        const Layout& l = s.l;
        at::tracer::impl::NoTracerDispatchMode untraced;
        fw = part(s, l.final_w, at::kFloat, {v.H, v.W});
        ids = s.ids.narrow(0, 0, l.K);
        off = part(s, l.offsets, at::kInt, {v.tiles() + 1});
        geo = part(s, l.geo, at::kFloat, {l.T, TG_GEO_WORDS});
        attr = part(s, l.attr, at::kFloat, {l.T, TG_ATTR_WORDS});
        ends = part(s, l.ends, at::kInt, {v.H, v.W});
    }
    return py::make_tuple(f.image, f.depthmap, fw, ids, off, geo, attr, ends,
                          f.saved.selection.defined() ? py::cast(f.saved.selection) : py::object(py::none()),
                          timing ? py::cast(f.stage_ms) : py::object(py::none()), f.saved.l, f.saved.blob);
}

// `blob`, `ids` and `selection` as forward returned them with `layout`; the lists are not looked at when there is a selection.
py::list py_backward(int kind, const Layout& layout, const Tensor& image, const Tensor& depthmap, const Tensor& blob,
                     const Optional& ids, const Optional& selection, const Optional& gi, const Optional& gd) {
    std::vector<Tensor> out;
    {
        py::gil_scoped_release nogil;
        at::AutoDispatchBelowADInplaceOrView below_autograd;
        const Kept k = kept_all(layout, image, depthmap, blob, or_none(ids), or_none(selection));
        at::tracer::impl::NoTracerDispatchMode untraced;
        out = backward((Kind)kind, k.saved, k.image, k.depthmap, or_none(gi), or_none(gd));
    }
    return py::cast(out);
}

void need_mesh(const Tensor& positions, const char* name, int64_t components, const Tensor& indices, const Tensor& colors,
               const Tensor& opacities) {
    const int64_t V = rows(positions, name);
    need(positions, name, {V, components});
    need(colors, "colors", {V, 3});
    need(opacities, "opacities", {V});
    need(indices, "indices", {rows(indices, "indices"), 3}, at::kInt);
}

Tensor py_l2_step(const Tensor& vertices, const Tensor& indices, const Tensor& colors, const Tensor& opacities,
                  const Tensor& target, int64_t W, int64_t H, int64_t tw, int64_t th, double thr, int64_t layers,
                  const Optional& gV, const Optional& gC, const Optional& gO, const Optional& loss, const Optional& packed,
                  bool one_kernel, bool cull, int64_t selection_max_bytes, const py::object& pv) {
    const bool world = !pv.is_none();
    need_mesh(vertices, world ? "points" : "vertices", world ? 3 : 4, indices, colors, opacities);
    need(target, "target", {H, W, 4}, target.scalar_type() == at::kByte && !one_kernel ? at::kByte : at::kFloat);
    need_tile(tw, th);
    const View v = view_of(true, W, H, tw, th, thr, true, layers);
    const Grads to = {or_none(gV), or_none(gC), or_none(gO), or_none(loss), or_none(packed)};
    const int64_t V = vertices.size(0);
    if (world || !to.packed.defined()) {
        need_out(to.vertices, world ? "grad_points" : "grad_vertices", (world ? 3 : 4) * V);
        need_out(to.colors, "grad_colors", 3 * V);
        need_out(to.opacities, "grad_opacities", V);
        need_out(to.loss, "loss", 1);
    }
    const Matrix m = world ? matrix_of(pv.cast<py::buffer>()) : Matrix{};
    py::gil_scoped_release nogil;
    return world ? world_step(vertices, m, indices, colors, opacities, target, v, to, one_kernel, selection_max_bytes)
                 : l2_step(vertices, indices, colors, opacities, target, v, to, one_kernel, cull, selection_max_bytes);
}

Tensor py_project(const Tensor& points, const py::buffer& pv) {
    need(points, "points", {rows(points, "points"), 3});
    const Matrix m = matrix_of(pv);
    py::gil_scoped_release nogil;
    return project(points, m);
}

void py_project_backward(const Tensor& points, const py::buffer& pv, const Tensor& gv, const Tensor& gp, bool accumulate) {
    const int64_t V = rows(points, "points");
    need(points, "points", {V, 3});
    need(gv, "grad_vertices", {V, 4});
    need(gp, "grad_points", {V, 3});
    need_out(gp, "grad_points", 3 * V);
    const Matrix m = matrix_of(pv);
    py::gil_scoped_release nogil;
    project_backward(points, m, gv, gp, accumulate);
}

py::tuple py_project_clip(const Tensor& points, const Tensor& indices, const Tensor& colors, const Tensor& opacities,
                          const py::buffer& pv) {
    need_no_transform({&points, &colors, &opacities});
    need_mesh(points, "points", 3, indices, colors, opacities);
    const Matrix m = matrix_of(pv);
    std::tuple<Tensor, Tensor, Tensor, Tensor> r;
    {
        py::gil_scoped_release nogil;
        r = project_clip(points, indices, colors, opacities, m);
    }
    return py::make_tuple(std::get<0>(r), std::get<1>(r), std::get<2>(r), std::get<3>(r));
}

py::list py_project_clip_backward(const Tensor& points, const Tensor& indices, const Tensor& colors, const Tensor& opacities,
                                  const py::buffer& pv, const Optional& gv, const Optional& gc, const Optional& go) {
    const Matrix m = matrix_of(pv);
    std::vector<Tensor> out;
    {
        py::gil_scoped_release nogil;
        at::tracer::impl::NoTracerDispatchMode untraced;
        out = project_clip_backward(points, indices, colors, opacities, m, or_none(gv), or_none(gc), or_none(go));
    }
    return py::cast(out);
}

py::tuple py_pack_mesh(const Tensor& colors_, const Tensor& opacities_, const Tensor& indices_) {
    const int64_t V = rows(colors_, "colors"), T = rows(indices_, "indices");
    need(colors_, "colors", {V, 3});
    need(opacities_, "opacities", {V});
    need(indices_, "indices", {T, 3}, at::kInt);
    Tensor rgba, faces;
    {
        py::gil_scoped_release nogil;
        const at::AutoDispatchBelowADInplaceOrView below_autograd;
        const Tensor colors = plain(colors_), opacities = plain(opacities_), indices = plain(indices_);
        const Where w(colors);
        rgba = at::empty({V, 4}, colors.options().requires_grad(false));
        faces = at::empty({T, 4}, indices.options());
        check("pack_inputs", g.pack_inputs(data<float>(colors), data<float>(opacities), data<int32_t>(indices), need_int(V),
                                           need_int(T), data<float>(rgba), data<int32_t>(faces), w.stream));
    }
    return py::make_tuple(rgba, faces);
}

void py_unpack_gradients(const Tensor& scratch, int64_t V, int64_t W, int64_t H, const Tensor& gV, const Tensor& gC,
                         const Tensor& gO, const Optional& loss, bool accumulate) {
    need_out(gV, "grad_vertices", 4 * V);
    need_out(gC, "grad_colors", 3 * V);
    need_out(gO, "grad_opacities", V);
    need_out(or_none(loss), "loss", 1);
    py::gil_scoped_release nogil;
    const Where w(gV);
    check("unpack_gradients",
          g.unpack_gradients(scratch.data_ptr(), (size_t)scratch.numel(), need_int(V), (float)(1.0 / (4.0 * W * H)),
                             data<float>(or_none(loss)), data<float>(gV), data<float>(gC), data<float>(gO), accumulate,
                             w.stream));
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    py::register_exception_translator([](std::exception_ptr p) {
        try {
            if (p) std::rethrow_exception(p);
        } catch (const LibraryError& e) {
            const py::object error = py::reinterpret_borrow<py::object>(g_native_error)(e.stage, e.status, e.detail);
            PyErr_SetObject(g_native_error, error.ptr());
        }
    });
    py::class_<Layout>(m, "Layout");
    py::class_<DeviceState, std::shared_ptr<DeviceState>>(m, "DeviceState")
        .def_readonly("info", &DeviceState::info)
        .def_readonly("last_slot", &DeviceState::last_slot)
        .def_readonly("k_estimate", &DeviceState::k_estimate)
        .def_property_readonly("long_row", [](const DeviceState& s) { return (uintptr_t)s.long_row; })
        .def("check_error_word", &DeviceState::check_error_word);
    m.def("bind", &bind);
    m.def("state", [](int device, int64_t stream) { return state_of(device, (cudaStream_t)stream); });
    m.def("render", &py_render);
    m.def("forward", &py_forward);
    m.def("backward", &py_backward);
    m.def("l2_step", &py_l2_step);
    m.def("project", &py_project);
    m.def("project_backward", &py_project_backward);
    m.def("project_clip", &py_project_clip);
    m.def("project_clip_backward", &py_project_clip_backward);
    m.def("pack_mesh", &py_pack_mesh);
    m.def("unpack_gradients", &py_unpack_gradients);
}
