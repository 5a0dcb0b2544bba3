// Radix-sort constants and digit-histogram helpers, and the host functions that the .cu files share.
#pragma once
#include "tg_common.cuh"

namespace tg {

constexpr int kRadixBits = 8;
constexpr int kRadix = 1 << kRadixBits;
constexpr int kMaxPasses = 8;
constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;

// scratch layout (bytes): [0, 8 KB) digit histograms / offsets [kMaxPasses][256] uint32,
// [8 KB, 8 KB + 64) tickets[kMaxPasses] + histogram-done counter (word 8), then the look-back words
// [passes][parts][256] uint64.
constexpr size_t kHistBytes = (size_t)kMaxPasses * kRadix * sizeof(uint32_t);
constexpr size_t kCtrBytes = 64;
constexpr int kHistDoneWord = 8;
// Up to this many tiles one CTA scans the tile counts.
constexpr int kTileScanByOneCta = 65536;
// Up to this many every CTA that places entries does so for itself, in 220 KB of shared memory (64 KB up to the lower number).
constexpr int kPlaceTiles = 55 * 1024, kPlaceTilesSmall = 16384;
// Top bit of the longest-list word the binning kernel reports: a launch order of the tiles was written.
constexpr uint32_t kOrderWrittenBit = 0x80000000u;
// What it reports as K and as slots from this many (triangle, tile) pairs on: more than any list capacity.
constexpr uint32_t kTooManyPairs = 0x80000000u;
// Longest tile list that a warp sorts (tile_sort_kernel alone).
constexpr int kTileSortRank = 128;
// Longest tile list that the compositing kernel sorts itself, in images of at most kFusedTiles tiles: two waves of its
// CTAs.  There a launch and a trip through memory count (1280 triangles, 256x256: 36 -> 27 us with the early launch); with
// many waves the sort inside takes more of the SMs' time than the kernel of its own does (200k triangles, 1920x1080: 124 us
// against 110 + 6).
constexpr uint32_t kFusedList = TG_SHORT_LIST;
constexpr int kFusedTiles = 2 * 4 * 148;
// A call that does not wait for the number of entries (TG_NO_COUNT) has at most this many triangles, which is also the
// longest list that its compositing kernel can meet.
constexpr int kNoCountTriangles = TG_NO_COUNT_TRIANGLES;

// Exclusive scan of one value per thread over the first 256 threads of a CTA (all threads of the CTA
// must call it; threads beyond 256 pass 0 and ignore the result).
__device__ __forceinline__ uint32_t block_exclusive_scan_256(uint32_t v, uint32_t* s_warp_tot /*[8]*/) {
    uint32_t incl = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane_id() >= (unsigned)d) incl += y;
    }
    const int warp = threadIdx.x >> 5;
    __syncthreads();   // protect s_warp_tot from a previous use
    if (lane_id() == 31 && warp < kSortWarps) s_warp_tot[warp] = incl;
    __syncthreads();
    uint32_t off = 0;
#pragma unroll
    for (int w = 0; w < kSortWarps; w++) {
        uint32_t x = s_warp_tot[w];
        if (w < warp) off += x;
    }
    return off + incl - v;
}

struct HistArgs {
    uint32_t* hist;           // [kMaxPasses][256] global counts, zeroed by the host
    uint32_t* done_counter;   // zeroed by the host
    int begin_bit, end_bit, passes;
};

// Count the digits of one key into the CTA's shared histogram.
__device__ __forceinline__ void hist_count(uint32_t* s_hist, uint64_t key, const HistArgs& h) {
    for (int p = 0; p < h.passes; p++) {
        const int shift = h.begin_bit + p * kRadixBits;
        const int bits = min(kRadixBits, h.end_bit - shift);
        atomicAdd(&s_hist[p * kRadix + ((uint32_t)(key >> shift) & ((1u << bits) - 1u))], 1u);
    }
}

// Add the CTA's histogram to the global one; the last CTA to arrive turns the global counts into
// exclusive digit offsets, per pass.  Call with all 256 threads of every CTA, after a barrier.
__device__ __forceinline__ void hist_flush_and_finish(uint32_t* s_hist, uint32_t* s_warp_tot, bool* s_last,
                                                      const HistArgs& h) {
    for (int i = threadIdx.x; i < h.passes * kRadix; i += kSortThreads) {
        const uint32_t c = s_hist[i];
        if (c) atomicAdd(&h.hist[i], c);
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) *s_last = (atomicAdd(h.done_counter, 1u) == gridDim.x - 1);
    __syncthreads();
    if (!*s_last) return;
    __threadfence();
    for (int p = 0; p < h.passes; p++) {
        const uint32_t c = __ldcg(&h.hist[p * kRadix + threadIdx.x]);
        const uint32_t e = block_exclusive_scan_256(c, s_warp_tot);
        h.hist[p * kRadix + threadIdx.x] = e;
    }
}

// What a kernel behind the binning is told: whether the lists are complete, and counts and counters to zero for the next call.
struct AfterBinning {
    const uint32_t* info;         // K, longest list, slots; null: the lists are known to be complete
    uint32_t capacity;
    uint32_t* tile_counts;        // null: nothing to clear
    uint32_t* counters;           // [4]
    __device__ __forceinline__ bool incomplete() const { return info != nullptr && info[2] > capacity; }
    __device__ __forceinline__ void clear(int tile, bool one_thread) const {
        if (tile_counts == nullptr || !one_thread) return;
        tile_counts[tile] = 0;
        if (tile == 0) *reinterpret_cast<uint4*>(counters) = make_uint4(0, 0, 0, 0);
    }
};

}  // namespace tg

namespace tg_host {
// Internal (not part of the C ABI): the pieces tg_render_forward strings together.
void set_tile_order(const uint32_t* order, uint32_t longest_list = 0);
size_t tile_sort_scratch_bytes(int tiles);
// Workspace of the binning kernels (bin_triangles, place_entries).
struct BinBuffers {
    uint32_t* clear;             // zeroed by the first kernel: `clear_words` words that hold the next four
    size_t clear_words;
    uint32_t* status;            // device error word
    uint32_t* counters;          // [4], 8-byte aligned
    uint32_t* tile_counts;       // [tiles], 16-byte aligned
    void* tile_scan_scratch;     // device-wide scan of the tile counts, only beyond kTileScanByOneCta tiles; zeroed too
    float4* tables;              // [tiles_x + tiles_y]
    uint32_t* info;              // [3] K, longest list (UINT32_MAX: not known), slots of `pairs` in use
    uint4* pairs;                // [list capacity]
    uint64_t* entries;           // [list capacity]
    uint32_t* tile_order;        // [tiles] or null
    uint32_t* list_heads;        // [6] heads of the tile sort's work lists, zeroed by place_entries
};
// Records and pairs.  `ready`: the counters are zero and the tables valid from a call before.  `in_place`: no pairs, but every
// entry at once in `entries`, tile * T + rank (the caller has room for T * tiles; place_entries is not called).
int bin_triangles(const float* vertices, const int32_t* indices, const float* colors, const float* opacities, int T, int W,
                  int H, int tw, int th, float* tri_geo, float* tri_attr, const BinBuffers& b, int32_t* offsets,
                  uint32_t list_capacity, bool cull, bool packed, bool ready, bool in_place, cudaStream_t stream);
// Entries grouped by tile, offsets, info, launch order.  `info_host`: mapped host memory whose words 0, 1 and 3 receive the
// three info words (K last), or null; `long_host`: one that receives the longest list where it has more than kFusedList
// entries, or null.  Counts and counters of images of at most kPlaceTiles tiles are left to the kernel
// behind to clear (the sort's first one, or the compositing kernel that sorts short lists itself).
int place_entries(const BinBuffers& b, int T, int W, int H, int tw, int th, int32_t* offsets, uint32_t list_capacity,
                  uint32_t* info_host, uint32_t* long_host, cudaStream_t stream);
// The sort in two steps.  The first launch sorts lists of up to kTileSortRank entries and makes work lists of the others; it
// needs nothing from the host: given `b`, it does nothing where the slots exceed `capacity`, and clears the counts and
// counters (see above).  The second, when the longest list is known, launches what the other length classes need.
int sort_short_lists(uint64_t* entries, const int32_t* offsets, int tiles, int32_t* sorted_ids, uint32_t* lists, bool write_back,
                     const BinBuffers* b, uint32_t capacity, cudaStream_t stream);
inline tg::AfterBinning after_binning(const BinBuffers* b, int tiles, uint32_t capacity) {
    if (b == nullptr) return {};
    const bool clear = tiles <= tg::kPlaceTiles;
    return {b->info, capacity, clear ? b->tile_counts : nullptr, b->counters};
}
int sort_long_lists(uint64_t* entries, const int32_t* offsets, int tiles, int32_t* sorted_ids, uint32_t* lists, bool write_back,
                    uint32_t longest, cudaStream_t stream);
// Forward compositing with the sort of the tile lists (at most kFusedList entries each, `info` as the binning left it) in the
// same kernel, which does nothing when the slots exceed `capacity` or a list is longer; with `any_length` it sorts longer
// ones too (sort_words), and does not filter them.  `room` > 0: the lists lie `room` entries apart, as bin_triangles leaves them
// in place, complete; `long_host` as for place_entries, which is then not called.
int blend_forward_short(const float* tri_geo, const float* tri_attr, const BinBuffers& b, uint32_t capacity, bool any_length,
                        int room, uint32_t* long_host, int32_t* sorted_ids, const int32_t* offsets, int W, int H, int tw, int th, float thr,
                        int per_pixel_sort, int max_layers, float* image, float* depthmap, float* final_weights,
                        int32_t* ends, int32_t* selection, cudaStream_t stream);
}  // namespace tg_host
