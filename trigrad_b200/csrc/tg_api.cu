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
    uint32_t* long_list;       // work lists of the per-tile sort
    size_t total;

    ForwardWorkspace(void* base, int tiles, uint32_t cap) {
        size_t off = 0;
        auto take = [&](size_t bytes) {
            void* p = base ? (void*)((char*)base + off) : nullptr;
            off += align_up(bytes ? bytes : 1);
            return p;
        };
        const bool device_scan = tiles > tg::kTileScanByOneCta;
        // what outlives a call (TG_WORKSPACE_READY) lies first, at places that do not depend on the list capacity
        bin.tables = (float4*)take(sizeof(float4) * ((size_t)tiles + 1));     // tiles_x + tiles_y <= tiles + 1
        // everything from `status` up to the end of the tile counts must be zero when the kernels start
        bin.status = (uint32_t*)take(sizeof(uint32_t) * 4);
        bin.counters = (uint32_t*)take(sizeof(uint32_t) * 4);
        bin.tile_scan_scratch = take(device_scan ? tg_scan_scratch_bytes(tiles) : 0);
        bin.tile_counts = (uint32_t*)take(sizeof(uint32_t) * (size_t)tiles);
        bin.clear = bin.status;
        bin.clear_words = base ? (size_t)(bin.tile_counts + tiles - bin.clear) : 0;
        bin.info = (uint32_t*)take(sizeof(uint32_t) * 3);
        long_list = (uint32_t*)take(tg_host::tile_sort_scratch_bytes(tiles));
        bin.list_heads = long_list;
        bin.tile_order = (uint32_t*)take(sizeof(uint32_t) * (size_t)tiles);
        if (device_scan) bin.tile_order = nullptr;
        bin.entries = (uint64_t*)take(sizeof(uint64_t) * (size_t)cap);
        bin.pairs = (uint4*)take(sizeof(uint4) * (size_t)cap);
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

// Tile lists of a call, in two steps: start() launches everything up to the unsorted lists, wait() waits for K and checks
// it against the capacity (timer marks 0-2 and 3).
struct TileLists {
    ForwardWorkspace ws;
    int tiles;
    bool device_scan, mapped, no_count;
    bool in_place;                         // entries go straight to their lists, each with room for all triangles
    cudaEvent_t k_ready = nullptr;
    uint32_t* device_status;               // error word, null where no kernel of the path can raise it
    uint32_t K = 0, longest = 0;
    const uint32_t* order = nullptr;       // launch order of the compositing kernel, when one was written

    TileLists(void* workspace, int T, int W, int H, int tw, int th, uint32_t cap, unsigned flags)
        : ws(workspace, ((W + tw - 1) / tw) * ((H + th - 1) / th), cap), tiles(((W + tw - 1) / tw) * ((H + th - 1) / th)),
          device_scan(tiles > tg::kTileScanByOneCta), mapped((flags & TG_INFO_MAPPED) != 0 && T > 0), no_count((flags & TG_NO_COUNT) != 0),
          in_place(no_count && (flags & TG_LISTS_UNUSED) != 0),
          device_status(device_scan ? ws.bin.status : nullptr) {}       // only the scan waits

    int start(const float* vertices, const int32_t* indices, const float* colors, const float* opacities, int T, int W, int H,
              int tw, int th, float* tri_geo, float* tri_attr, int32_t* sorted_ids, uint32_t cap, int32_t* offsets,
              size_t workspace_bytes, uint32_t* info_host, unsigned flags, StageTimer& timer, cudaStream_t s) {
        if (workspace_bytes < ws.total) {
            tg_host::set_error("forward workspace: need %zu bytes, got %zu", ws.total, workspace_bytes);
            return TG_ERR_WORKSPACE;
        }
        TG_REQUIRE(cap == 0 || sorted_ids != nullptr, "null sorted_ids");
        if (!no_count) {
            info_host[0] = kNotArrived;     // K < 2^31, so this value means "K has not landed yet"
            info_host[1] = info_host[2] = info_host[3] = 0;
        }
        if (!mapped)
            if (int st = scratch_event(&k_ready)) return st;
        // beyond 65536 tiles the lists are the reference's
        const bool cull = (flags & TG_FORWARD_CULL_TILES) != 0 && !device_scan;
        timer.mark();                                                    // [0] start of "init"
        timer.mark();                                                    // [1] start of "bary_transforms"
        // per-triangle records, (triangle, tile) pairs with their depth keys
        if (int st = tg_host::bin_triangles(vertices, indices, colors, opacities, T, W, H, tw, th, tri_geo, tri_attr, ws.bin,
                                            offsets, cap, cull, (flags & TG_INPUT_PACKED) != 0,
                                            (flags & TG_WORKSPACE_READY) != 0, in_place, s))
            return st;
        timer.mark();                                                    // [2] start of "per_tile_lists"
        if (in_place) return TG_OK;
        if (int st = tg_host::place_entries(ws.bin, T, W, H, tw, th, offsets, cap, mapped && !no_count ? info_host : nullptr,
                                            no_count ? info_host + 1 : nullptr, s))
            return st;
        if (!mapped) {
            // [3] first: the host watches the word K arrives in
            TG_CUDA(cudaMemcpyAsync(&info_host[3], ws.bin.info + 2, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
            TG_CUDA(cudaMemcpyAsync(&info_host[0], ws.bin.info, 2 * sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
            TG_CUDA(cudaEventRecord(k_ready, s));
        }
        return TG_OK;
    }

    // K arrives in (preferably pinned) host memory.  Watching the word itself is quicker than waking up from
    // cudaEventSynchronize (unless the lists were expected to be short the compositing kernel cannot be launched before K
    // is known, so every microsecond here is an idle GPU); after a bounded while, or for pageable memory where the copy has
    // completed by now anyway, the event (the stream, without a copy) is waited for in the ordinary way, which also
    // surfaces any error of the kernels before it.
    int wait(uint32_t cap, uint32_t* info_host, cudaStream_t s) {
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
        if (info_host[0] == kNotArrived) {
            tg_host::set_error("the number of list entries never reached the host");
            return TG_ERR_CUDA;
        }
        K = info_host[0];
        // the longest-list word carries "a launch order of the tiles was written" in its top bit
        const bool have_order = (info_host[1] & tg::kOrderWrittenBit) != 0 && info_host[1] != UINT32_MAX;
        if (info_host[1] != UINT32_MAX) info_host[1] &= ~tg::kOrderWrittenBit;
        longest = info_host[1];
        if (have_order) order = ws.bin.tile_order;
        const uint32_t slots = info_host[3];            // K and the holes of culled pairs
        if (K >= tg::kTooManyPairs || slots >= tg::kTooManyPairs) {
            tg_host::set_error("the triangles' rectangles hold 2^31 or more (triangle, tile) pairs");
            return TG_ERR_BAD_ARG;
        }
        if (K > cap || slots > cap) {
            info_host[0] = K > slots ? K : slots;
            tg_host::set_error("%u entries and culled pairs exceed the list capacity %u", info_host[0], cap);
            return TG_ERR_CAPACITY;
        }
        return TG_OK;
    }

    // Before wait(): the lists are sorted while K travels to the host, where they turn out to be complete.
    int sort_short(int32_t* sorted_ids, const int32_t* offsets, uint32_t cap, int T, cudaStream_t s) {
        if (T == 0 || cap == 0) return TG_OK;
        return tg_host::sort_short_lists(ws.bin.entries, offsets, tiles, sorted_ids, ws.long_list, false, &ws.bin, cap, s);
    }
    int sort_long(int32_t* sorted_ids, const int32_t* offsets, cudaStream_t s) {
        if (K == 0) return TG_OK;
        return tg_host::sort_long_lists(ws.bin.entries, offsets, tiles, sorted_ids, ws.long_list, false, longest, s);
    }
};

static int check_forward_args(int T, int W, int H, int tw, int th, int max_layers, const void* workspace,
                              const void* info_host, const void* offsets, uint32_t list_capacity, unsigned flags) {
    TG_REQUIRE(T >= 0, "T < 0");
    if (int s = tg_host::check_sizes(W, H, tw, th)) return s;
    TG_REQUIRE(max_layers >= 1, "max_layers must be >= 1");
    TG_REQUIRE(workspace && info_host && offsets, "null pointer");
    TG_REQUIRE(((uintptr_t)workspace & 255) == 0, "workspace must be 256-byte aligned");
    TG_REQUIRE(list_capacity < 0x80000000u, "list capacity must stay below 2^31");
    TG_REQUIRE((flags & ~127u) == 0, "unknown flag");
    TG_REQUIRE(!(flags & TG_EXPECT_SHORT_LISTS) || (flags & TG_INFO_MAPPED), "TG_EXPECT_SHORT_LISTS needs TG_INFO_MAPPED");
    return TG_OK;
}

// Stage times from the timer's six marks (synchronises), then the device error word.
static int finish_timing(StageTimer& timer, float* stage_ms_host, const uint32_t* info_host, cudaStream_t s) {
    if (!stage_ms_host) return TG_OK;
    TG_CUDA(cudaStreamSynchronize(s));
    float ms[5];
    for (int i = 0; i < 5; i++) TG_CUDA(cudaEventElapsedTime(&ms[i], timer.ev[i], timer.ev[i + 1]));
    stage_ms_host[0] = ms[0];   // init
    stage_ms_host[1] = ms[2];   // per_tile_lists: tile offsets, entries to their places
    stage_ms_host[2] = ms[3];   // sorting: per-tile sort, K read-back meanwhile
    stage_ms_host[3] = ms[1];   // bary_transforms: records, pairs, tile counts
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
    if (int st = check_forward_args(T, W, H, tw, th, max_layers, workspace, info_host, offsets, list_capacity, flags)) return st;
    cudaStream_t s = (cudaStream_t)stream;
    StageTimer timer(stage_ms_host != nullptr, s);
    TileLists lists(workspace, T, W, H, tw, th, list_capacity, flags);
    if (lists.no_count) {
        cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
        TG_CUDA(cudaStreamIsCapturing(s, &capture));
        TG_REQUIRE(T > 0 && T <= tg::kNoCountTriangles && lists.tiles <= tg::kFusedTiles && (flags & TG_INFO_MAPPED) &&
                       (uint64_t)list_capacity >= (uint64_t)T * lists.tiles && stage_ms_host == nullptr &&
                       capture == cudaStreamCaptureStatusNone,
                   "TG_NO_COUNT is for small renders with room for every list, see the header");
    }
    if (int st = lists.start(vertices, indices, colors, opacities, T, W, H, tw, th, tri_geo, tri_attr, sorted_ids, list_capacity,
                             offsets, workspace_bytes, info_host, flags, timer, s))
        return st;
    // Lists of up to kFusedList entries are sorted by the compositing kernel itself in images of few tiles, where the caller
    // expects nothing longer: it checks on the device what the host is told afterwards.
    const bool early = lists.tiles <= tg::kFusedTiles && T > 0 && (flags & (TG_EXPECT_SHORT_LISTS | TG_NO_COUNT)) != 0 && stage_ms_host == nullptr;
    timer.mark();                                                    // [3] start of "sorting"
    int st = early ? tg_host::blend_forward_short(tri_geo, tri_attr, lists.ws.bin, list_capacity, lists.no_count, lists.in_place ? T : 0,
                                                  info_host + 1, sorted_ids, offsets, W, H, tw, th, thr, per_pixel_sort, max_layers, image, depthmap, final_weights, ends, selection, s)
                   : lists.sort_short(sorted_ids, offsets, list_capacity, T, s);
    if (st || lists.no_count) return st;
    if ((st = lists.wait(list_capacity, info_host, s))) return st;
    if (!early || lists.longest > tg::kFusedList) {
        if (early && (st = lists.sort_short(sorted_ids, offsets, list_capacity, T, s))) return st;
        if ((st = lists.sort_long(sorted_ids, offsets, s))) return st;
        timer.mark();                                                // [4] start of "rasterization"
        tg_host::set_tile_order(lists.order, lists.longest);         // with the longest list: long lists are streamed
        st = tg_blend_forward(tri_geo, tri_attr, sorted_ids, offsets, W, H, tw, th, thr, per_pixel_sort, max_layers, image,
                              depthmap, final_weights, ends, selection, stream);
        tg_host::set_tile_order(nullptr);
    }
    if (st) return st;
    timer.mark();                                                    // [5] end
    // device error word: valid on the host once the stream has been synchronised
    if (lists.device_status)
        TG_CUDA(cudaMemcpyAsync(&info_host[2], lists.device_status, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
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
    if (int st = check_forward_args(T, W, H, tw, th, max_layers, workspace, info_host, offsets, list_capacity, flags)) return st;
    TG_REQUIRE(!(flags & TG_NO_COUNT), "the one-kernel step waits for the number of entries");
    TG_REQUIRE(tw * th <= 256 && max_layers <= 32, "the one-kernel step needs tiles of at most 256 pixels and max_layers <= 32");
    cudaStream_t s = (cudaStream_t)stream;
    StageTimer timer(stage_ms_host != nullptr, s);
    TileLists lists(workspace, T, W, H, tw, th, list_capacity, flags);
    int st = lists.start(vertices, indices, colors, opacities, T, W, H, tw, th, tri_geo, tri_attr, sorted_ids, list_capacity,
                         offsets, workspace_bytes, info_host, flags, timer, s);
    if (st) return st;
    timer.mark();                                                    // [3] start of "sorting"
    if ((st = lists.sort_short(sorted_ids, offsets, list_capacity, T, s))) return st;
    if ((st = lists.wait(list_capacity, info_host, s))) return st;
    if ((st = lists.sort_long(sorted_ids, offsets, s))) return st;
    timer.mark();                                                    // [4] start of "rasterization" (here: forward + backward)
    tg_host::set_tile_order(lists.order);
    st = tg_blend_step_l2(tri_geo, tri_attr, sorted_ids, offsets, V, W, H, tw, th, thr, max_layers, target, grad_scale,
                          loss_scale, loss_out, image, depthmap, final_weights, ends, grad_vertices, grad_colors,
                          grad_opacities, accumulate, scratch, scratch_bytes, stream);
    tg_host::set_tile_order(nullptr);
    if (st) return st;
    timer.mark();                                                    // [5] end
    if (lists.device_status)
        TG_CUDA(cudaMemcpyAsync(&info_host[2], lists.device_status, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    return finish_timing(timer, stage_ms_host, info_host, s);
}

}  // extern "C"
