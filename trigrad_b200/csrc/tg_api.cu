// Whole forward path behind one C entry point (stages 1-6 sequenced on the caller's stream).
#include <atomic>
#include <chrono>

#include <sched.h>

#include "tg_radix.cuh"

namespace {

constexpr uint32_t kNotArrived = 0xffffffffu;

inline size_t align_up(size_t x, size_t a = 256) { return (x + a - 1) / a * a; }

// Carves the caller's workspace; the same function sizes it.
struct ForwardWorkspace {
    tg_host::BinBuffers bin = {};
    uint32_t* long_list;       // work lists of the per-tile sort; only their six head words need clearing
    size_t total;

    ForwardWorkspace(void* base, int tiles, uint32_t cap) {
        size_t off = 0;
        auto take = [&](size_t bytes) {
            void* p = base ? (void*)((char*)base + off) : nullptr;
            off += align_up(bytes ? bytes : 1);
            return p;
        };
        const bool device_scan = tiles > tg::kTileScanByLastCta;
        bin.entries = (uint64_t*)take(sizeof(uint64_t) * (size_t)cap);
        bin.pairs = (uint4*)take(sizeof(uint4) * (size_t)cap);
        bin.tables = (float4*)take(sizeof(float4) * ((size_t)tiles + 1));     // tiles_x + tiles_y <= tiles + 1
        bin.info = (uint32_t*)take(sizeof(uint32_t) * 3);
        // everything from `status` up to the head of the work lists must be zero when the kernels start: one clear
        bin.status = (uint32_t*)take(sizeof(uint32_t) * 4);
        bin.counters = (uint32_t*)take(sizeof(uint32_t) * 2);
        bin.tile_scan_scratch = take(device_scan ? tg_scan_scratch_bytes(tiles) : 0);
        bin.tile_counts = (uint32_t*)take(sizeof(uint32_t) * (size_t)tiles);
        long_list = (uint32_t*)take(tg_host::tile_sort_scratch_bytes(tiles));
        bin.clear = bin.status;
        bin.clear_words = base ? (size_t)(long_list + 6 - bin.clear) : 0;
        bin.tile_order = (uint32_t*)take(sizeof(uint32_t) * (size_t)tiles);
        if (device_scan) bin.tile_order = nullptr;
        total = off;
    }
};

// One reusable event per (thread, device): marks "K has reached the host".
int scratch_event(cudaEvent_t* out) {
    constexpr int kMaxDevices = 64;
    static thread_local cudaEvent_t events[kMaxDevices] = {};
    int dev = 0;
    TG_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) {
        tg_host::set_error("device index %d outside the supported range", dev);
        return TG_ERR_BAD_ARG;
    }
    if (events[dev] == nullptr) TG_CUDA(cudaEventCreateWithFlags(&events[dev], cudaEventDisableTiming));
    *out = events[dev];
    return TG_OK;
}

struct StageTimer {
    cudaEvent_t ev[6];
    int n = 0;
    bool on;
    cudaStream_t s;
    StageTimer(bool enable, cudaStream_t stream) : on(enable), s(stream) {
        if (on) for (auto& e : ev) cudaEventCreate(&e);
    }
    void mark() { if (on && n < 6) cudaEventRecord(ev[n++], s); }
    ~StageTimer() { if (on) for (auto& e : ev) cudaEventDestroy(e); }
};

}  // namespace

// Everything before compositing: per-triangle records, tile offsets, sorted tile lists (timer marks 0-3).
static int build_tile_lists(const float* vertices, const int32_t* indices, const float* colors, const float* opacities,
                            int T, int W, int H, int tw, int th, int max_layers, float* tri_geo, float* tri_attr,
                            int32_t* sorted_ids, uint32_t list_capacity, int32_t* offsets, void* workspace,
                            size_t workspace_bytes, uint32_t* info_host, unsigned flags, StageTimer& timer,
                            uint32_t** device_status, const uint32_t** tile_order_out, cudaStream_t s) {
    TG_REQUIRE(T >= 0 && W > 0 && H > 0 && tw > 0 && th > 0, "sizes");
    TG_REQUIRE(tw * th <= 1024, "tile_width * tile_height must be <= 1024");
    TG_REQUIRE(max_layers >= 1, "max_layers must be >= 1");
    TG_REQUIRE(workspace && info_host && offsets, "null pointer");
    TG_REQUIRE(((uintptr_t)workspace & 255) == 0, "workspace must be 256-byte aligned");
    TG_REQUIRE(list_capacity < 0x80000000u, "list capacity must stay below 2^31");
    const int tiles_x = (W + tw - 1) / tw, tiles_y = (H + th - 1) / th;
    const int tiles = tiles_x * tiles_y;
    TG_REQUIRE((flags & ~(unsigned)(TG_FORWARD_CULL_TILES | TG_INPUT_PACKED | TG_INFO_MAPPED)) == 0, "unknown flag");
    const bool packed = (flags & TG_INPUT_PACKED) != 0;
    const bool device_scan = tiles > tg::kTileScanByLastCta;
    // beyond 65536 tiles the lists are the reference's
    const bool cull = (flags & TG_FORWARD_CULL_TILES) != 0 && !device_scan;
    const ForwardWorkspace ws(workspace, tiles, list_capacity);
    // the only kernel of this path that can raise the error word is the scan
    *device_status = device_scan ? ws.bin.status : nullptr;
    *tile_order_out = nullptr;
    if (workspace_bytes < ws.total) {
        tg_host::set_error("forward workspace: need %zu bytes, got %zu", ws.total, workspace_bytes);
        return TG_ERR_WORKSPACE;
    }
    info_host[0] = kNotArrived;     // K < 2^31, so this value means "K has not landed yet"
    info_host[1] = 0;
    info_host[2] = 0;
    info_host[3] = 0;
    TG_REQUIRE(list_capacity == 0 || sorted_ids != nullptr, "null sorted_ids");
    // mapped: the binning kernel writes K where the host looks; otherwise a copy brings it
    const bool mapped = (flags & TG_INFO_MAPPED) != 0 && T > 0;
    cudaEvent_t k_ready = nullptr;
    if (!mapped)
        if (int st = scratch_event(&k_ready)) return st;

    timer.mark();                                                    // [0] start of "init"
    timer.mark();                                                    // [1] start of "bary_transforms"
    // per-triangle records, (triangle, tile) pairs with their depth keys, tile offsets
    int st = tg_host::bin_triangles(vertices, indices, colors, opacities, T, W, H, tw, th, tri_geo, tri_attr, ws.bin,
                                    offsets, list_capacity, mapped ? info_host : nullptr, cull, packed, s);
    if (st) return st;
    timer.mark();                                                    // [2] start of "per_tile_lists"
    if (!mapped) {
        // [3] first: the host watches the word K arrives in
        TG_CUDA(cudaMemcpyAsync(&info_host[3], ws.bin.info + 2, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
        TG_CUDA(cudaMemcpyAsync(&info_host[0], ws.bin.info, 2 * sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
        TG_CUDA(cudaEventRecord(k_ready, s));
    }
    // The entries move to their tiles while K travels to the host: the kernel does nothing when K exceeds the capacity,
    // and nothing that reads them is launched before K has been checked.
    st = tg_host::scatter_entries(ws.bin, list_capacity, offsets, tiles, T, s);
    if (st) return st;
    // K arrives in (preferably pinned) host memory.  Watching the word itself is quicker than
    // waking up from cudaEventSynchronize (the compositing kernels cannot be launched before K is known, so every
    // microsecond here is an idle GPU once the entry writer has finished); after a bounded while, or for pageable
    // memory where the copy has completed by now anyway, the event (the stream, without a copy) is waited for in the ordinary way, which also
    // surfaces any error of the kernels before it.
    {
        const volatile uint32_t* watched = info_host;
        const auto t0 = std::chrono::steady_clock::now();
        for (uint32_t spins = 1; *watched == kNotArrived; ++spins) {
#if defined(__x86_64__)
            __builtin_ia32_pause();
#endif
            // after a short pure spin the core is offered to other runnable threads between looks (several ranks or
            // issuing threads per core: a waiter must not hold up the thread whose launches it is waiting behind)
            if (spins > 2048) sched_yield();
            if ((spins & 0xfffu) == 0 && std::chrono::steady_clock::now() - t0 > std::chrono::milliseconds(200)) break;
        }
        std::atomic_thread_fence(std::memory_order_acquire);
        if (info_host[0] == kNotArrived) TG_CUDA(mapped ? cudaStreamSynchronize(s) : cudaEventSynchronize(k_ready));
    }
    if (info_host[0] == kNotArrived) {
        tg_host::set_error("the number of list entries never reached the host");
        return TG_ERR_CUDA;
    }
    const uint32_t K = info_host[0];
    // the longest-list word carries "a launch order of the tiles was written" in its top bit
    const bool have_order = (info_host[1] & tg::kOrderWrittenBit) != 0 && info_host[1] != UINT32_MAX;
    if (info_host[1] != UINT32_MAX) info_host[1] &= ~tg::kOrderWrittenBit;
    *tile_order_out = have_order ? ws.bin.tile_order : nullptr;
    const uint32_t slots = info_host[3];            // K and the holes of culled pairs
    if (K > list_capacity || slots > list_capacity) {
        info_host[0] = K > slots ? K : slots;
        tg_host::set_error("%u entries and culled pairs exceed the list capacity %u", info_host[0], list_capacity);
        return TG_ERR_CAPACITY;
    }
    timer.mark();                                                    // [3] start of "sorting"
    if (K > 0) {
        st = tg_host::sort_tile_lists(ws.bin.entries, offsets, tiles, sorted_ids, ws.long_list, true, false, info_host[1], s);
        if (st) return st;
    }
    return TG_OK;
}

// Stage times from the timer's six marks (synchronises), then the device error word.
static int finish_timing(StageTimer& timer, float* stage_ms_host, const uint32_t* info_host, cudaStream_t s) {
    if (!stage_ms_host) return TG_OK;
    TG_CUDA(cudaStreamSynchronize(s));
    float ms[5];
    for (int i = 0; i < 5; i++) TG_CUDA(cudaEventElapsedTime(&ms[i], timer.ev[i], timer.ev[i + 1]));
    stage_ms_host[0] = ms[0];   // init
    stage_ms_host[1] = ms[2];   // per_tile_lists: K read-back + entry emission
    stage_ms_host[2] = ms[3];   // sorting: per-tile sort
    stage_ms_host[3] = ms[1];   // bary_transforms: preprocess + scan + tile counts and offsets
    stage_ms_host[4] = ms[4];   // rasterization
    if (info_host[2]) {
        tg_host::set_error("device error word = %u", info_host[2]);
        return TG_ERR_DEVICE_FLAG;
    }
    return TG_OK;
}

extern "C" {

size_t tg_forward_workspace_bytes(int T, int tiles, uint32_t list_capacity) {
    if (tiles < 0) tiles = 0;
    (void)T;
    return ForwardWorkspace(nullptr, tiles, list_capacity).total;
}

int tg_render_forward(const float* vertices, const int32_t* indices, const float* colors, const float* opacities, int T,
                      int W, int H, int tw, int th, float thr, int per_pixel_sort, int max_layers, float* image,
                      float* depthmap, float* final_weights, int32_t* ends, int32_t* selection, float* tri_geo,
                      float* tri_attr, int32_t* sorted_ids, uint32_t list_capacity, int32_t* offsets, void* workspace,
                      size_t workspace_bytes, uint32_t* info_host, float* stage_ms_host, unsigned flags,
                      tg_stream_t stream) {
    TG_REQUIRE(image && depthmap && final_weights && ends, "null pointer");
    cudaStream_t s = (cudaStream_t)stream;
    StageTimer timer(stage_ms_host != nullptr, s);
    uint32_t* device_status = nullptr;
    const uint32_t* tile_order = nullptr;
    int st = build_tile_lists(vertices, indices, colors, opacities, T, W, H, tw, th, max_layers, tri_geo, tri_attr,
                              sorted_ids, list_capacity, offsets, workspace, workspace_bytes, info_host, flags, timer, &device_status, &tile_order, s);
    if (st) return st;
    timer.mark();                                                    // [4] start of "rasterization"
    tg_host::set_tile_order(tile_order, info_host[1]);      // with the longest list: long lists are streamed
    st = tg_blend_forward(tri_geo, tri_attr, sorted_ids, offsets, W, H, tw, th, thr, per_pixel_sort, max_layers, image,
                          depthmap, final_weights, ends, selection, stream);
    tg_host::set_tile_order(nullptr);
    if (st) return st;
    timer.mark();                                                    // [5] end
    // device error word: valid on the host once the stream has been synchronised
    if (device_status) TG_CUDA(cudaMemcpyAsync(&info_host[2], device_status, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    return finish_timing(timer, stage_ms_host, info_host, s);
}

int tg_render_step_l2(const float* vertices, const int32_t* indices, const float* colors, const float* opacities, int T,
                      int V, int W, int H, int tw, int th, float thr, int max_layers, const float* target,
                      float grad_scale, float loss_scale, float* loss_out, float* image, float* depthmap,
                      float* final_weights, int32_t* ends, float* tri_geo, float* tri_attr, int32_t* sorted_ids,
                      uint32_t list_capacity, int32_t* offsets, float* grad_vertices, float* grad_colors,
                      float* grad_opacities, int accumulate, void* workspace, size_t workspace_bytes, void* scratch,
                      size_t scratch_bytes, uint32_t* info_host, float* stage_ms_host, unsigned flags,
                      tg_stream_t stream) {
    TG_REQUIRE(image && depthmap && final_weights && ends && target, "null pointer");
    TG_REQUIRE(tw * th <= 256 && max_layers <= 32, "the one-kernel step needs tiles of at most 256 pixels and max_layers <= 32");
    cudaStream_t s = (cudaStream_t)stream;
    StageTimer timer(stage_ms_host != nullptr, s);
    uint32_t* device_status = nullptr;
    const uint32_t* tile_order = nullptr;
    int st = build_tile_lists(vertices, indices, colors, opacities, T, W, H, tw, th, max_layers, tri_geo, tri_attr,
                              sorted_ids, list_capacity, offsets, workspace, workspace_bytes, info_host, flags, timer, &device_status, &tile_order, s);
    if (st) return st;
    timer.mark();                                                    // [4] start of "rasterization" (here: forward + backward)
    tg_host::set_tile_order(tile_order);
    st = tg_blend_step_l2(tri_geo, tri_attr, sorted_ids, offsets, V, W, H, tw, th, thr, max_layers, target, grad_scale,
                          loss_scale, loss_out, image, depthmap, final_weights, ends, grad_vertices, grad_colors,
                          grad_opacities, accumulate, scratch, scratch_bytes, stream);
    tg_host::set_tile_order(nullptr);
    if (st) return st;
    timer.mark();                                                    // [5] end
    if (device_status) TG_CUDA(cudaMemcpyAsync(&info_host[2], device_status, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    return finish_timing(timer, stage_ms_host, info_host, s);
}

}  // extern "C"
