// Binning stages: per-triangle preprocess, device-wide scan, key emission, tile ranges.
#include <stdarg.h>
#include <stdio.h>

#include <atomic>

#include "tg_radix.cuh"

namespace tg {

// ================================================================================================
// Stage 1: a triangle's gathers and its two packed records (64 and 96 bytes), which the compositing kernels stream.
struct TriInput {
    int ia, ib, ic;
    float4 a, b, c;         // vertices
    float4 ra, rb, rc;      // (r, g, b, opacity)
};

// packed inputs: faces as [T,4] int32 and colours as [V,4] (r, g, b, opacity), one 16-byte load each instead of the
// reference's 12-byte strides (util.h:457-573); the branch is uniform over the grid
__device__ __forceinline__ TriInput load_triangle(int t, const float4* __restrict__ vertices, const int* __restrict__ indices,
                                                  const float* __restrict__ colors, const float* __restrict__ opacities,
                                                  bool packed) {
    TriInput in;
    if (packed) {
        const int4 f = reinterpret_cast<const int4*>(indices)[t];
        in.ia = f.x; in.ib = f.y; in.ic = f.z;
    } else {
        in.ia = indices[3 * (size_t)t]; in.ib = indices[3 * (size_t)t + 1]; in.ic = indices[3 * (size_t)t + 2];
    }
    in.a = vertices[in.ia]; in.b = vertices[in.ib]; in.c = vertices[in.ic];
    if (packed) {
        const float4* rgba = reinterpret_cast<const float4*>(colors);
        in.ra = rgba[in.ia]; in.rb = rgba[in.ib]; in.rc = rgba[in.ic];
    } else {
        const float* ca = colors + 3 * (size_t)in.ia;
        const float* cb = colors + 3 * (size_t)in.ib;
        const float* cc = colors + 3 * (size_t)in.ic;
        in.ra = make_float4(ca[0], ca[1], ca[2], opacities[in.ia]);
        in.rb = make_float4(cb[0], cb[1], cb[2], opacities[in.ib]);
        in.rc = make_float4(cc[0], cc[1], cc[2], opacities[in.ic]);
    }
    return in;
}

__device__ __forceinline__ void make_attr(const TriInput& in, float4 (&q)[6]) {
    q[0] = make_float4(in.ra.w, in.rb.w, in.rc.w, in.ra.x);
    q[1] = make_float4(in.ra.y, in.ra.z, in.rb.x, in.rb.y);
    q[2] = make_float4(in.rb.z, in.rc.x, in.rc.y, in.rc.z);
    q[3] = make_float4(div(1.f, in.a.w), div(1.f, in.b.w), div(1.f, in.c.w), __int_as_float(in.ia));
    q[4] = make_float4(__int_as_float(in.ib), __int_as_float(in.ic), in.a.x, in.a.y);
    q[5] = make_float4(in.b.x, in.b.y, in.c.x, in.c.y);
}

__device__ __forceinline__ void make_geo(const TriInput& in, float4 (&g)[4]) {
    const float4 a = in.a, b = in.b, c = in.c;
    // barycentric matrix, reference render.cu:324-336: plain mul/sub/div
    float denom = add(add(mul(a.x, sub(b.y, c.y)), mul(b.x, sub(c.y, a.y))), mul(c.x, sub(a.y, b.y)));
    if (fabsf(denom) < kEffZero) denom = 1.0f;
    float m0 = div(sub(b.y, c.y), denom);
    float m1 = div(sub(c.x, b.x), denom);
    float m2 = div(sub(mul(b.x, c.y), mul(c.x, b.y)), denom);
    float m3 = div(sub(c.y, a.y), denom);
    float m4 = div(sub(a.x, c.x), denom);
    float m5 = div(sub(mul(c.x, a.y), mul(a.x, c.y)), denom);
    float m6 = div(sub(a.y, b.y), denom);
    float m7 = div(sub(b.x, a.x), denom);
    float m8 = div(sub(mul(a.x, b.y), mul(b.x, a.y)), denom);
    // Lower bound of the per-pixel sort depth: with weights of one sign the interpolated depth is
    // a convex combination of the vertex depths; a relative margin covers fp32 rounding.
    float zlow = -INFINITY;
    bool same_sign = (a.w > 0.f && b.w > 0.f && c.w > 0.f) || (a.w < 0.f && b.w < 0.f && c.w < 0.f);
    if (same_sign) {
        float zmin = fminf(fminf(a.z, b.z), c.z);
        float zabs = fmaxf(fmaxf(fabsf(a.z), fabsf(b.z)), fabsf(c.z));
        float lo = zmin - 4e-6f * zabs;
        if (isfinite(lo)) zlow = lo;
    }
    g[0] = make_float4(m0, m1, m2, m3);
    g[1] = make_float4(m4, m5, m6, m7);
    g[2] = make_float4(m8, a.z, b.z, c.z);
    g[3] = make_float4(a.w, b.w, c.w, zlow);
}

__global__ void __launch_bounds__(256) preprocess_kernel(const float4* __restrict__ vertices,
                                                         const int* __restrict__ indices,
                                                         const float* __restrict__ colors,
                                                         const float* __restrict__ opacities, int T, int W, int H,
                                                         int tw, int th, int tiles_x, int tiles_y,
                                                         uint32_t* __restrict__ tri_counts, int4* __restrict__ tri_rects,
                                                         float4* __restrict__ tri_geo, float4* __restrict__ tri_attr) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= T) return;
    const TriInput in = load_triangle(t, vertices, indices, colors, opacities, false);
    Rect r;
    const bool ok = tile_rect(in.a.x, in.a.y, in.b.x, in.b.y, in.c.x, in.c.y, W, H, tw, th, tiles_x, tiles_y, r);
    tri_counts[t] = ok ? (uint32_t)(r.x1 - r.x0 + 1) * (uint32_t)(r.y1 - r.y0 + 1) : 0u;
    if (tri_rects) tri_rects[t] = make_int4(r.x0, r.y0, r.x1, r.y1);
    float4 g[4], q[6];
    make_geo(in, g);
    make_attr(in, q);
#pragma unroll
    for (int k = 0; k < 4; k++) tri_geo[4 * (size_t)t + k] = g[k];
#pragma unroll
    for (int k = 0; k < 6; k++) tri_attr[6 * (size_t)t + k] = q[k];
}

// ================================================================================================
// Stage 2: single-pass exclusive scan with decoupled look-back.
// scratch: word 0 = ticket counter (uint32, padded to 8 bytes), then one uint64 per partition:
// (flag << 32) | value, flag 0 = nothing yet, 1 = partition aggregate, 2 = inclusive prefix.
constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;
constexpr uint32_t kSpinLimit = 1u << 22;   // bounded wait: ~ seconds with the nanosleep below

__device__ __forceinline__ uint64_t ld_volatile(const uint64_t* p) { return *(const volatile uint64_t*)p; }
__device__ __forceinline__ void st_volatile(uint64_t* p, uint64_t v) { *(volatile uint64_t*)p = v; }

// Wait (bounded) until the partition word has a non-zero flag.  Returns false if the wait ran out.
__device__ __forceinline__ bool wait_flag(const uint64_t* p, uint64_t& word, uint32_t spin_limit) {
    for (uint32_t it = 0; it < spin_limit; ++it) {
        word = ld_volatile(p);
        if ((word >> 32) != 0) return true;
        if (it > 64) __nanosleep(100);
    }
    return false;
}

// Decoupled look-back, executed by ONE WARP of partition p: publishes the partition's total, sums the
// totals of all earlier partitions (32 words per step) until one of them already carries an inclusive
// prefix, publishes its own inclusive prefix and returns the exclusive one.
__device__ __forceinline__ uint32_t lookback_exclusive(int p, uint32_t total, uint64_t* part_status, uint32_t* status,
                                                       uint32_t spin_limit = kSpinLimit) {
    uint32_t excl = 0;
    if (p == 0) {
        if (lane_id() == 0) st_volatile(&part_status[0], (2ull << 32) | total);
        return 0;
    }
    if (lane_id() == 0) st_volatile(&part_status[p], (1ull << 32) | total);
    int q = p - 1 - (int)lane_id();
    bool failed = false;
    while (true) {
        uint64_t word = 2ull << 32;   // virtual partitions before 0: inclusive prefix 0
        if (q >= 0 && !wait_flag(&part_status[q], word, spin_limit)) { failed = true; word = 2ull << 32; }
        const uint32_t flag = (uint32_t)(word >> 32), val = (uint32_t)word;
        const unsigned incl_mask = __ballot_sync(0xffffffffu, flag == 2u);
        uint32_t contrib = val;
        if (incl_mask) {
            const int first = __ffs(incl_mask) - 1;
            if ((int)lane_id() > first) contrib = 0;
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) contrib += __shfl_xor_sync(0xffffffffu, contrib, d);
        excl += contrib;
        if (incl_mask) break;
        q -= 32;
    }
    if (__any_sync(0xffffffffu, failed) && lane_id() == 0) atomicExch(status, 1u);
    if (lane_id() == 0) st_volatile(&part_status[p], (2ull << 32) | (uint64_t)(excl + total));
    return excl;
}

__global__ void __launch_bounds__(kScanThreads) scan_kernel(const uint32_t* __restrict__ in,
                                                            uint32_t* __restrict__ out, int n, int num_parts,
                                                            uint32_t* ticket, uint64_t* part_status,
                                                            uint32_t* status) {
    __shared__ uint32_t s_part;
    __shared__ uint32_t s_warp[kScanThreads / 32];
    __shared__ uint32_t s_excl;
    if (threadIdx.x == 0) s_part = atomicAdd(ticket, 1u);
    __syncthreads();
    const int p = (int)s_part;
    if (p >= num_parts) return;
    const int base = p * kScanTile + threadIdx.x * kScanItems;

    uint32_t v[kScanItems];
    uint32_t sum = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        v[i] = (base + i < n) ? in[base + i] : 0u;
        sum += v[i];
    }
    // block exclusive scan of `sum`
    uint32_t incl = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane_id() >= (unsigned)d) incl += y;
    }
    const int warp = threadIdx.x >> 5;
    if (lane_id() == 31) s_warp[warp] = incl;
    __syncthreads();
    uint32_t warp_off = 0, total = 0;
#pragma unroll
    for (int w = 0; w < kScanThreads / 32; w++) {
        uint32_t x = s_warp[w];
        if (w < warp) warp_off += x;
        total += x;
    }
    uint32_t thread_excl = warp_off + incl - sum;

    if (warp == 0) {
        const uint32_t excl = lookback_exclusive(p, total, part_status, status);
        if (lane_id() == 0) {
            s_excl = excl;
            if (p == num_parts - 1) out[n] = excl + total;
        }
    }
    __syncthreads();
    uint32_t run = s_excl + thread_excl;
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        if (base + i < n) out[base + i] = run;
        run += v[i];
    }
}

// Self-test of the bounded wait: ONE warp plays partition 1 of a scan whose partition 0 never publishes
// anything (its word stays zero), with a spin limit of a few polls.  The wait runs out, the warp raises the
// status word and returns; nothing waits for anything else, so the launch always ends.
__global__ void __launch_bounds__(32) bounded_wait_selftest_kernel(uint64_t* part_status /*[2], zero*/, uint32_t* status,
                                                                  uint32_t spin_limit, uint32_t* excl_out) {
    const uint32_t excl = lookback_exclusive(1, 7u, part_status, status, spin_limit);
    if (lane_id() == 0) *excl_out = excl;
}

// ---- the forward path's binning: shared pieces ------------------------------------------------------------------
// Pixel-centre extent and NDC borders of every tile column and row, in the exact arithmetic of the coverage test and of
// the clipper (double divisions): computed once per call instead of once per (triangle, tile) pair.
struct TileTables {
    const float4* cols;      // [tiles_x] (first centre, last centre, lower border, upper border)
    const float4* rows;      // [tiles_y]
};

__device__ __forceinline__ float4 tile_span(int i, int tile, int extent) {
    return make_float4(pixel_coord(i * tile, extent), pixel_coord(min((i + 1) * tile, extent) - 1, extent),
                       sub(mul(div((float)(i * tile), (float)extent), 2.f), 1.f),
                       sub(mul(div((float)((i + 1) * tile), (float)extent), 2.f), 1.f));
}

// Clears the counters of the binning kernel and fills the tile tables: first kernel of a forward.
__global__ void __launch_bounds__(256) bin_init_kernel(uint32_t* __restrict__ clear, size_t clear_words, float4* __restrict__ cols,
                                                       float4* __restrict__ rows, int tiles_x, int tiles_y, int W, int H,
                                                       int tw, int th) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < clear_words) clear[i] = 0;
    if (i < (size_t)tiles_x) cols[i] = tile_span((int)i, tw, W);
    else if (i < (size_t)tiles_x + tiles_y) rows[i - tiles_x] = tile_span((int)(i - tiles_x), th, H);
}

// Exclusive scan of counts[0..tiles) by one CTA into offsets[0..tiles] (global or shared memory); the sum in `total`.  Returns
// the largest count where `want_biggest` (uniform over the CTA).
// A warp takes 512 counts per round, four independent 16-byte loads per lane one round ahead: bound by the latency of those.
constexpr int kBinWarps = 4;         // warps of a CTA of the binning kernel (two and eight: 3 to 7 % slower)
constexpr int kFinishWarps = 16;     // of the kernel that scans the tile counts of images with very many tiles
__device__ __forceinline__ void load_counts(const uint32_t* counts, int first, int tiles, uint4 (&v)[4]) {
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int i = first + 128 * k;
        if (i + 3 < tiles) {
            v[k] = __ldcg(reinterpret_cast<const uint4*>(counts + i));
        } else {
            v[k].x = i < tiles ? __ldcg(counts + i) : 0u;
            v[k].y = i + 1 < tiles ? __ldcg(counts + i + 1) : 0u;
            v[k].z = i + 2 < tiles ? __ldcg(counts + i + 2) : 0u;
            v[k].w = 0u;
        }
    }
}
template <int WARPS>
__device__ __forceinline__ uint32_t tile_offsets_by_one_cta(const uint32_t* counts, int32_t* offsets, int tiles,
                                                            uint32_t* s_warp /*[WARPS]*/, bool want_biggest, uint32_t& total) {
    static_assert(WARPS <= 32, "a lane per warp");
    constexpr int kRound = 512 * WARPS;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, mine = 512 * warp + 4 * lane;
    const bool aligned = ((uintptr_t)offsets & 15) == 0;
    uint32_t carry = 0, biggest = 0;
    uint4 ahead[4];
    load_counts(counts, mine, tiles, ahead);
    for (int base = 0; base < tiles; base += kRound) {
        uint4 v[4];
        uint32_t excl[4], run = 0;              // of this lane's counts in the warp's 128; sum of the warp's 128s before
#pragma unroll
        for (int k = 0; k < 4; k++) v[k] = ahead[k];
        if (base + kRound < tiles) load_counts(counts, base + kRound + mine, tiles, ahead);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint32_t sum = v[k].x + v[k].y + v[k].z + v[k].w;
            biggest = max(max(biggest, max(v[k].x, v[k].y)), max(v[k].z, v[k].w));
            uint32_t incl = sum;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, incl, d);
                if (lane >= d) incl += y;
            }
            excl[k] = incl - sum + run;
            run += __shfl_sync(0xffffffffu, incl, 31);
        }
        __syncthreads();                      // s_warp free again
        if (lane == 0) s_warp[warp] = run;
        __syncthreads();
        uint32_t incl = lane < WARPS ? s_warp[lane] : 0u;
#pragma unroll
        for (int d = 1; d < WARPS; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += y;
        }
        const uint32_t before = carry + __shfl_sync(0xffffffffu, incl, warp) - run;
        carry += __shfl_sync(0xffffffffu, incl, WARPS - 1);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int i = base + mine + 128 * k;
            uint4 o;
            o.x = before + excl[k];
            o.y = o.x + v[k].x;
            o.z = o.y + v[k].y;
            o.w = o.z + v[k].z;
            if (i + 3 < tiles && aligned) {
                *reinterpret_cast<uint4*>(offsets + i) = o;
            } else {
                if (i < tiles) offsets[i] = (int32_t)o.x;
                if (i + 1 < tiles) offsets[i + 1] = (int32_t)o.y;
                if (i + 2 < tiles) offsets[i + 2] = (int32_t)o.z;
                if (i + 3 < tiles) offsets[i + 3] = (int32_t)o.w;
            }
        }
    }
    if (threadIdx.x == 0) offsets[tiles] = (int32_t)carry;
    total = carry;
    __syncthreads();                          // offsets visible to the CTA
    if (!want_biggest) return 0;
    biggest = __reduce_max_sync(0xffffffffu, biggest);
    if (lane == 0) s_warp[warp] = biggest;
    __syncthreads();
    return __reduce_max_sync(0xffffffffu, lane < WARPS ? s_warp[lane] : 0u);
}

// Launch order for the compositing kernel: tiles grouped by the length class of their lists, longest class first.  With one
// CTA per tile in scan order a tile whose list is as long as everything else an SM processes can start late and leave the
// other SMs idle (a view of a fine mesh: 28 % of the SM time); long lists first removes that tail.  Worth its passes over the
// offsets only when lists are long and uneven and the tiles are few enough for one CTA, which makes it while the others move
// the entries: every thread counts its tiles per class, eight 16-bit sums in four words, and a scan of the words over the CTA
// says where each thread's tiles of a class go (1920x1080, 8160 tiles: under 2 us; with an atomic per class and warp 10).
constexpr uint32_t kOrderMinLongest = 256;
constexpr uint32_t kOrderMinMean = 64;
constexpr int kOrderMaxTiles = kPlaceTilesSmall;
static_assert(kOrderMaxTiles < 65536, "16-bit sums");
// 7: empty, 6: below 64 entries, 5: below 128, ... 0: 2048 and more
__device__ __forceinline__ int length_class(int n) { return n <= 0 ? 7 : min(6, max(0, __clz(n) - 20)); }
template <int NT>
__device__ __forceinline__ void tile_order_by_one_cta(const int32_t* s_off, int tiles, uint32_t* order, uint4* s_sums /*[NT / 32]*/) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t c[4] = {0, 0, 0, 0};
    auto field = [](int cls) { return 1u << (16 * (cls & 1)); };
    for (int i = threadIdx.x; i < tiles; i += NT) {
        const int cls = length_class(s_off[i + 1] - s_off[i]);
#pragma unroll
        for (int k = 0; k < 4; k++) c[k] += (cls >> 1) == k ? field(cls) : 0u;
    }
    uint32_t incl[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        incl[k] = c[k];
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl[k], d);
            if (lane >= d) incl[k] += y;
        }
    }
    if (lane == 31) s_sums[warp] = make_uint4(incl[0], incl[1], incl[2], incl[3]);
    __syncthreads();
    uint32_t all[4] = {0, 0, 0, 0};
    for (int w = 0; w < NT / 32; w++) {
        const uint4 x = s_sums[w];
        const uint32_t y[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (w < warp) incl[k] += y[k];
            all[k] += y[k];
        }
    }
    uint32_t at[8], run = 0;            // where this thread's next tile of a class goes
#pragma unroll
    for (int cls = 0; cls < 8; cls++) {
        const int k = cls >> 1, shift = 16 * (cls & 1);
        at[cls] = run + (((incl[k] - c[k]) >> shift) & 0xffffu);
        run += (all[k] >> shift) & 0xffffu;
    }
    for (int i = threadIdx.x; i < tiles; i += NT) {
        const int cls = length_class(s_off[i + 1] - s_off[i]);
        uint32_t to = 0;
#pragma unroll
        for (int k = 0; k < 8; k++)
            if (cls == k) to = at[k]++;
        order[to] = (uint32_t)i;
    }
}

// ================================================================================================
// Stage 3: key emission.
struct Plane { float A, B, C; };

// reference render.cu:140-152, `1.0 / det` in double.
__device__ __forceinline__ Plane depth_plane(float ax, float ay, float az, float bx, float by, float bz, float cx,
                                             float cy, float cz) {
    float det = add(add(mul(ax, sub(by, cy)), mul(bx, sub(cy, ay))), mul(cx, sub(ay, by)));
    float id = (float)__drcp_rn((double)det);
    Plane p;
    p.A = mul(add(add(mul(az, sub(by, cy)), mul(bz, sub(cy, ay))), mul(cz, sub(ay, by))), id);
    p.B = mul(add(add(mul(ax, sub(bz, cz)), mul(bx, sub(cz, az))), mul(cx, sub(az, bz))), id);
    p.C = mul(add(add(mul(ax, sub(mul(by, cz), mul(cy, bz))), mul(bx, sub(mul(cy, az), mul(ay, cz)))),
                  mul(cx, sub(mul(ay, bz), mul(by, az)))),
              id);
    return p;
}

__device__ __forceinline__ float plane_depth(const Plane& p, float x, float y) { return fma_(p.A, x, fma_(p.B, y, p.C)); }

// One Sutherland-Hodgman pass against an axis-aligned half-plane (reference render.cu:159-189) over the `n_in` vertices
// poly[0], poly[stride], ...; `emit` receives the vertices of the clipped polygon in order and may write them back to
// the same places: two vertices are read ahead, and a pass over the at most six vertices of a polygon that is convex but
// for the rounding of its corners never gets further ahead of its reads.
template <int AXIS, class Emit>
__device__ __forceinline__ void clip_pass(const float2* poly, int stride, int n_in, float bound, Emit&& emit) {
    auto dist = [&](const float2& p) -> float {
        if (AXIS == 0) return sub(p.x, bound);
        if (AXIS == 1) return sub(bound, p.x);
        if (AXIS == 2) return sub(p.y, bound);
        return sub(bound, p.y);
    };
    float2 p0 = poly[(n_in - 1) * stride], p1 = poly[0], p2 = poly[min(1, n_in - 1) * stride];
    float d0 = dist(p0);
    bool in0 = d0 >= 0.f;
#pragma unroll 1
    for (int i = 0; i < n_in; i++) {
        const float2 p3 = poly[min(i + 2, n_in - 1) * stride];
        const float d1 = dist(p1);
        const bool in1 = d1 >= 0.f;
        if (in1 != in0) {
            const float t = div(d0, sub(d0, d1));
            emit(make_float2(fma_(t, sub(p1.x, p0.x), p0.x), fma_(t, sub(p1.y, p0.y), p0.y)));
        }
        if (in1) emit(p1);
        p0 = p1; d0 = d1; in0 = in1;
        p1 = p2; p2 = p3;
    }
}

struct TriXYZ { float ax, ay, bx, by, cx, cy; };

// Triangle entirely inside the tile: the clipper would return it unchanged.
__device__ __forceinline__ bool inside_tile(const TriXYZ& v, float xmin, float xmax, float ymin, float ymax) {
    const float lox = fminf(fminf(v.ax, v.bx), v.cx), hix = fmaxf(fmaxf(v.ax, v.bx), v.cx);
    const float loy = fminf(fminf(v.ay, v.by), v.cy), hiy = fmaxf(fmaxf(v.ay, v.by), v.cy);
    return sub(lox, xmin) >= 0.f && sub(xmax, hix) >= 0.f && sub(loy, ymin) >= 0.f && sub(ymax, hiy) >= 0.f;
}

// The polygon of a clip lives in shared memory, a column of kPolySlots float2 per thread of the CTA (no bank conflicts
// whatever slot a lane is at).  In local memory the two arrays of a thread made 131 KB of L1 working set per SM, more
// than L1 has beside the CTAs' shared memory (200k triangles, full HD: 55 us against 40).
constexpr int kPolySlots = 8;
__device__ __forceinline__ float tile_key(const TriXYZ& v, const Plane& pl, float xmin, float xmax, float ymin, float ymax,
                                          float2* poly, int stride) {
    if (inside_tile(v, xmin, xmax, ymin, ymax)) {
        float md0 = fminf(FLT_MAX, plane_depth(pl, v.ax, v.ay));
        md0 = fminf(md0, plane_depth(pl, v.bx, v.by));
        return fminf(md0, plane_depth(pl, v.cx, v.cy));
    }
    poly[0] = make_float2(v.ax, v.ay);
    poly[stride] = make_float2(v.bx, v.by);
    poly[2 * stride] = make_float2(v.cx, v.cy);
    int n = 3, m = 0;
    auto keep = [&](float2 p) { poly[min(m++, kPolySlots - 1) * stride] = p; };
    auto next = [&]() { n = min(m, kPolySlots); m = 0; return n > 0; };
    clip_pass<0>(poly, stride, n, xmin, keep);
    if (!next()) return 1e30f;
    clip_pass<1>(poly, stride, n, xmax, keep);
    if (!next()) return 1e30f;
    clip_pass<2>(poly, stride, n, ymin, keep);
    if (!next()) return 1e30f;
    float md = FLT_MAX;
    clip_pass<3>(poly, stride, n, ymax, [&](float2 p) { md = fminf(md, plane_depth(pl, p.x, p.y)); m++; });
    return m <= 0 ? 1e30f : md;
}

// Stage entry point: entries with their radix keys in emission order.  One CTA takes 256 consecutive triangles.  Phase 1
// (a thread per triangle) gathers the vertices and stages rectangle, depth plane and first output slot in shared memory.
// Phase 2 (a thread per OUTPUT entry) finds its triangle by binary search over the staged offsets, so that a triangle
// touching many tiles is spread over the whole CTA and no lane idles behind a long neighbour.
struct __align__(16) EmitTri {
    float ax, ay, bx, by, cx, cy;
    float A, B, C;
    int x0, y0, ny;
};
constexpr int kEmitThreads = 256;

__device__ __forceinline__ int find_segment(const uint32_t* first, int n, uint32_t e) {   // largest i with first[i] <= e
    int lo = 0, hi = n;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (first[mid] <= e) lo = mid; else hi = mid;
    }
    return lo;
}

__global__ void __launch_bounds__(kEmitThreads) emit_keys_kernel(const float4* __restrict__ vertices,
                                                                 const int* __restrict__ indices, int T, int W, int H,
                                                                 int tw, int th, int tiles_x, int tiles_y,
                                                                 const uint32_t* __restrict__ tri_offsets,
                                                                 uint64_t* __restrict__ keys, uint32_t* __restrict__ ids,
                                                                 uint32_t capacity) {
    __shared__ EmitTri s_tri[kEmitThreads];
    __shared__ uint32_t s_off[kEmitThreads + 1];
    __shared__ float2 s_poly[kPolySlots * kEmitThreads];
    const int tid = threadIdx.x;
    const int t0 = blockIdx.x * kEmitThreads;
    const int ntri = min(kEmitThreads, T - t0);
    if (tid < ntri) {
        const int t = t0 + tid;
        const float4 a = vertices[indices[3 * (size_t)t]], b = vertices[indices[3 * (size_t)t + 1]],
                     c = vertices[indices[3 * (size_t)t + 2]];
        EmitTri e;
        e.ax = a.x; e.ay = a.y; e.bx = b.x; e.by = b.y; e.cx = c.x; e.cy = c.y;
        Rect r;
        if (tile_rect(a.x, a.y, b.x, b.y, c.x, c.y, W, H, tw, th, tiles_x, tiles_y, r)) {
            const Plane pl = depth_plane(a.x, a.y, a.z, b.x, b.y, b.z, c.x, c.y, c.z);
            e.A = pl.A; e.B = pl.B; e.C = pl.C;
        } else {
            e.A = e.B = e.C = 0.f;
        }
        e.x0 = r.x0; e.y0 = r.y0; e.ny = r.y1 - r.y0 + 1;
        s_tri[tid] = e;
        s_off[tid] = tri_offsets[t];
    }
    if (tid == 0) s_off[ntri] = tri_offsets[t0 + ntri];
    __syncthreads();
    const uint32_t first = s_off[0], total = s_off[ntri] - first;
    for (uint32_t e = tid; e < total; e += kEmitThreads) {
        const uint32_t ge = first + e;
        const int lo = find_segment(s_off, ntri, ge);      // triangles without entries have equal offsets
        const EmitTri& tr = s_tri[lo];
        const uint32_t local = ge - s_off[lo];
        const int tx = tr.x0 + (int)(local / (uint32_t)tr.ny), ty = tr.y0 + (int)(local % (uint32_t)tr.ny);
        const float4 cx = tile_span(tx, tw, W), cy = tile_span(ty, th, H);
        const float depth = tile_key({tr.ax, tr.ay, tr.bx, tr.by, tr.cx, tr.cy}, {tr.A, tr.B, tr.C}, cx.z, cx.w, cy.z, cy.w,
                                     s_poly + tid, kEmitThreads);
        if (ge < capacity) {                       // the host guarantees K <= capacity before the result is used
            keys[ge] = ((uint64_t)(uint32_t)(ty * tiles_x + tx) << 32) | float_to_ordered(depth);
            ids[ge] = (uint32_t)(t0 + lo);
        }
    }
}

// ---- the forward path's binning ----------------------------------------------------------------------------------
// One pass over the triangles makes everything: the packed records, the (triangle, tile) pairs with their depth keys and
// the tile counts.  A CTA takes `per_cta` consecutive triangles, up to 32 per warp.  Phase 1, a lane per triangle: gathers,
// records, tile rectangle; matrix, corners and depth plane stay in shared memory.  Phase 2, a thread per pair of the
// CTA's rectangles: with CULL, pairs that cannot cover a pixel centre of their tile leave a hole (the exact test the
// reference leaves open, render.cu:110).  The others take their rank in the tile from one atomic on the tile's count
// (issued before the depth key, which hides its latency) and leave one 16-byte record (key, triangle, tile, rank).  Pairs
// that need the polygon clipper are put off to the end of the CTA when they are few in a warp, and run there with full
// warps.
// place_entries_kernel turns the counts into tile offsets and moves every entry to
// offset + rank.  Against counting and writing in two kernels, which gathered, tested and searched twice, B200, with the
// scatter: 1.3M triangles of a pixel each, full HD: 281 -> 170 us (this kernel 141); 200k triangles, full HD: 65 -> 36 (31);
// 2M triangles, 4K: 791 -> 477 (387).  Bound by latency: at 52 % of the issue slots, 38 % of L1 and 8 % of DRAM (200k
// triangles) its warps wait first for the gathers and for the rank atomics, then for one another at the barriers.
struct BinArgs {
    uint32_t* tile_counts;   // [tiles], zero on entry
    int32_t* offsets;        // [tiles + 1], written when scan_here
    uint32_t* counters;      // [4], zero on entry: -, -, slots handed out (64 bits)
    uint32_t* info;          // [3] K, when scan_here the longest list (kOrderWrittenBit: a launch order is wanted), slots;
                             // K and slots no larger than kTooManyPairs
    uint32_t* info_host;     // words 0, 1 and 3 of mapped host memory receive them too, or null
    uint32_t* long_host;     // mapped host memory that receives the longest list if it has more than kFusedList entries, or null
    uint4* pairs;            // [capacity]
    uint64_t* lists;         // [tiles][room], for entries that go straight to their lists, or null
    uint32_t room;
    uint32_t capacity;
    int tiles, tiles_x, tiles_y;
    int scan_here;           // 0: the host launches a device-wide scan of the tile counts
    int want_order;
    TileTables tables;
};

constexpr uint32_t kHole = 0xffffffffu;      // tile word of a pair that is not listed
__device__ __forceinline__ unsigned long long* slot_counter(const BinArgs& bin) {
    return reinterpret_cast<unsigned long long*>(bin.counters + 2);
}
// Clip queue of a CTA.  Twice as many took longer (1.3M triangles of a pixel 146 us against 143, 200k triangles 35.9 against 35.1,
// 2M piled up the same), with the clips later and 1.5 KB more of shared memory in each of the eight CTAs; half as many 143, 35.7.
constexpr int kBinQueue = 32 * kBinWarps;
// Shared memory of a warp, in words: first the staging area of its records (pitch 5 quads for the 4 of a geometry
// record, 7 for the 6 of half the warp's attribute records: 16-byte accesses of consecutive lanes then fall on different
// banks), then, component-major, what the pairs need of its triangles: matrix 9, corners 6, depth plane 3, tile
// rectangle (x0, y0, rows), first pair.
constexpr int kBinWarpWords = 22 * 32 + 4;
constexpr size_t kBinSmem = sizeof(float) * kBinWarps * kBinWarpWords + sizeof(float2) * kPolySlots * 32 * kBinWarps;
constexpr int kTriMatrix = 0, kTriCorners = 9, kTriPlane = 15, kTriX0 = 18, kTriY0 = 19, kTriRows = 20, kTriFirst = 21;
static_assert(32 * 20 <= kBinWarpWords && 16 * 28 <= kBinWarpWords, "the triangles' data replace the staging area");

// Key and record of one listed pair: triangle `lt` of the CTA with its data at `tri` (lane stride 32), tile (tx, ty).
__device__ __forceinline__ void write_pair(const BinArgs& bin, const float* tri, int t, uint32_t tx, uint32_t ty, uint32_t pos,
                                           const float4& cx, const float4& cy, float2* poly) {
    const uint32_t tile = ty * (uint32_t)bin.tiles_x + tx;
    const uint32_t rank = atomicAdd(bin.tile_counts + tile, 1u);     // travels while the key is computed
    const float* v = tri + 32 * kTriCorners;
    const float* p = tri + 32 * kTriPlane;
    const float depth = tile_key({v[0], v[32], v[64], v[96], v[128], v[160]}, {p[0], p[32], p[64]}, cx.z, cx.w, cy.z, cy.w,
                                 poly, 32 * kBinWarps);
    if (bin.lists != nullptr) {          // a triangle is in a tile's list once, so rank < room, which is T
        bin.lists[(size_t)tile * bin.room + rank] = ((uint64_t)float_to_ordered(depth) << 32) | (uint32_t)t;
        return;
    }
    if (pos < bin.capacity)              // the host checks K before anything that reads the entries is used
        bin.pairs[pos] = make_uint4((uint32_t)t, float_to_ordered(depth), tile, rank);
}

// K, the longest list and the number of slots, for the kernels behind and for the host.  By one thread.
__device__ __forceinline__ void publish_counts(const BinArgs& bin, uint32_t K, uint32_t longest, uint32_t slots) {
    bin.info[0] = K;
    bin.info[1] = longest;
    bin.info[2] = slots;
    if (bin.info_host) {                  // K last: the host watches that word
        volatile uint32_t* h = bin.info_host;
        h[1] = longest;
        h[3] = slots;
        __threadfence_system();
        h[0] = K;
    }
    if (bin.long_host && (longest & ~kOrderWrittenBit) > kFusedList) *(volatile uint32_t*)bin.long_host = longest & ~kOrderWrittenBit;
}
__device__ __forceinline__ uint32_t slots_used(const BinArgs& bin) {
    return (uint32_t)min(__ldcg(slot_counter(bin)), (unsigned long long)kTooManyPairs);
}
// Whether a launch order of the tiles is worth its two passes over the offsets: only for images of at most 16384 tiles
// whose lists are long on average and uneven (the longest one at least 256 entries).
__device__ __forceinline__ bool order_wanted(const BinArgs& bin, uint32_t K, uint32_t longest) {
    return bin.want_order && bin.tiles <= kOrderMaxTiles && K >= kOrderMinMean * (uint32_t)bin.tiles && longest >= kOrderMinLongest;
}

template <bool CULL>
__global__ void __launch_bounds__(32 * kBinWarps, 32 / kBinWarps) bin_kernel(const float4* __restrict__ vertices,
                                                                const int* __restrict__ indices,
                                                                const float* __restrict__ colors,
                                                                const float* __restrict__ opacities, int T, int per_cta,
                                                                int W, int H, int tw, int th, double inv_tw, double inv_th,
                                                                float4* __restrict__ tri_geo, float4* __restrict__ tri_attr,
                                                                BinArgs bin, int packed) {
    extern __shared__ __align__(16) char s_dynamic[];
    float (*s_tri)[kBinWarpWords] = reinterpret_cast<float (*)[kBinWarpWords]>(s_dynamic);
    float2* s_poly = reinterpret_cast<float2*>(s_dynamic + sizeof(float) * kBinWarps * kBinWarpWords);
    __shared__ uint32_t s_qx[kBinQueue], s_qy[kBinQueue], s_qe[kBinQueue];   // tile column, tile row << 8 | triangle, pair
    __shared__ uint32_t s_first[kBinWarps + 1];       // first pair of every warp's triangles
    __shared__ uint32_t s_queued, s_base;
    __shared__ uint32_t s_warp[kBinWarps];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const unsigned below = (1u << lane) - 1u;
    allow_dependents();
    await_prerequisites();
    const int per_warp = (per_cta + kBinWarps - 1) / kBinWarps;
    const int t_cta = blockIdx.x * per_cta, t0 = t_cta + warp * per_warp;
    const int ntri = min(min(per_warp, per_cta - warp * per_warp), T - t0);
    if (tid == 0) s_queued = 0;
    float* mine = s_tri[warp];
    float4* stage = reinterpret_cast<float4*>(mine);
    uint32_t total = 0;
    if (ntri > 0) {
        uint32_t count = 0;
        TriInput in = {};
        if (lane < ntri) in = load_triangle(t0 + lane, vertices, indices, colors, opacities, packed != 0);
        // the records leave through shared memory, so that the warp's stores are whole consecutive lines
        float4 q[6];
        make_attr(in, q);
#pragma unroll
        for (int half = 0; half < 2; half++) {
            const int n = min(16, ntri - 16 * half);
            if ((lane >> 4) == half) {
#pragma unroll
                for (int k = 0; k < 6; k++) stage[7 * (lane & 15) + k] = q[k];
            }
            __syncwarp();
            for (int i = lane; i < 6 * n; i += 32) tri_attr[6 * ((size_t)t0 + 16 * half) + i] = stage[7 * (i / 6) + i % 6];
            __syncwarp();
        }
        float4 g[4];
        if (lane < ntri) {
            make_geo(in, g);
#pragma unroll
            for (int k = 0; k < 4; k++) stage[5 * lane + k] = g[k];
        }
        __syncwarp();
        for (int i = lane; i < 4 * ntri; i += 32) tri_geo[4 * (size_t)t0 + i] = stage[5 * (i >> 2) + (i & 3)];
        __syncwarp();
        if (lane < ntri) {
            Rect r;
            float* d = mine + lane;
            if (tile_rect(in.a.x, in.a.y, in.b.x, in.b.y, in.c.x, in.c.y, W, H, tw, th, bin.tiles_x, bin.tiles_y, r, inv_tw, inv_th)) {
                count = (uint32_t)(r.x1 - r.x0 + 1) * (uint32_t)(r.y1 - r.y0 + 1);
                const Plane pl = depth_plane(in.a.x, in.a.y, in.a.z, in.b.x, in.b.y, in.b.z, in.c.x, in.c.y, in.c.z);
                const float m[9] = {g[0].x, g[0].y, g[0].z, g[0].w, g[1].x, g[1].y, g[1].z, g[1].w, g[2].x};
                const float rest[9] = {in.a.x, in.a.y, in.b.x, in.b.y, in.c.x, in.c.y, pl.A, pl.B, pl.C};
#pragma unroll
                for (int k = 0; k < 9; k++) { d[32 * (kTriMatrix + k)] = m[k]; d[32 * (kTriCorners + k)] = rest[k]; }
                d[32 * kTriX0] = __int_as_float(r.x0);
                d[32 * kTriY0] = __int_as_float(r.y0);
                d[32 * kTriRows] = __int_as_float(r.y1 - r.y0 + 1);
            }
        }
        uint32_t incl = count;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += y;
        }
        total = __shfl_sync(0xffffffffu, incl, 31);
        if (__any_sync(0xffffffffu, count >= 1u << 27)) {
            // A triangle has fewer than 2^31 pairs, but 32 of them can have more than 32 bits hold: the sum in halves, cut off
            const uint32_t low = __reduce_add_sync(0xffffffffu, count & 0xffffu), high = __reduce_add_sync(0xffffffffu, count >> 16);
            total = (uint32_t)min(((uint64_t)high << 16) + low, (uint64_t)UINT32_MAX);
        }
        mine[32 * kTriFirst + lane] = __uint_as_float(incl - count);
    }
    if (lane == 0) s_warp[warp] = total;
    __syncthreads();
    // Every pair of the rectangles has its slot; those that are not listed leave a hole there.  Slots are counted in 64 bits:
    // in 32 the count of a call with 2^32 pairs wraps to one that passes for fitting the list, while the tile offsets point
    // far behind it (3840x2160 in tiles of 4x4: 8300 triangles over the whole image).  Such a call is refused, so a CTA that
    // finds it lists nothing.
    if (tid == 0) {
        uint64_t sum = 0;
#pragma unroll
        for (int w = 0; w < kBinWarps; w++) { s_first[w] = (uint32_t)sum; sum += s_warp[w]; }
        const uint64_t at = bin.lists != nullptr ? 0 : atomicAdd(slot_counter(bin), (unsigned long long)sum);
        s_first[kBinWarps] = at + sum < kTooManyPairs ? (uint32_t)sum : 0u;
        s_base = (uint32_t)at;
    }
    __syncthreads();
    // The CTA's pairs in chunks of 32, whichever warp prepared the triangle
    const uint32_t all = s_first[kBinWarps], slot0 = s_base;
    for (uint32_t base = 32 * warp; base < all; base += 32 * kBinWarps) {
        const uint32_t e = base + lane;
        bool keep = false, inside = false;
        int ct = 0;                                  // triangle: warp << 5 | lane that prepared it
        uint32_t tx = 0, ty = 0;
        float4 cx, cy;
        if (e < all) {
            const int w = find_segment(s_first, kBinWarps, e);
            const uint32_t ew = e - s_first[w];
            const uint32_t* first_pair = reinterpret_cast<const uint32_t*>(s_tri[w] + 32 * kTriFirst);
            const int lt = find_segment(first_pair, 32, ew);
            ct = (w << 5) | lt;
            const float* d = s_tri[w] + lt;
            const uint32_t local = ew - first_pair[lt], rows = __float_as_uint(d[32 * kTriRows]);
            const uint32_t col = rows == 1 ? local : local / rows;
            tx = __float_as_uint(d[32 * kTriX0]) + col;
            ty = __float_as_uint(d[32 * kTriY0]) + (local - col * rows);
            cx = __ldg(bin.tables.cols + tx);
            cy = __ldg(bin.tables.rows + ty);
            keep = true;
            if (CULL) {
                float m[9];
#pragma unroll
                for (int k = 0; k < 9; k++) m[k] = d[32 * (kTriMatrix + k)];
                keep = rect_may_cover(m, {cx.x, cx.y, cy.x, cy.y});
                if (!keep && bin.lists == nullptr && slot0 + e < bin.capacity) bin.pairs[slot0 + e] = make_uint4(0, 0, kHole, 0);
            }
            const float* v = d + 32 * kTriCorners;
            inside = inside_tile({v[0], v[32], v[64], v[96], v[128], v[160]}, cx.z, cx.w, cy.z, cy.w);
        }
        // Pairs that need the clipper (a triangle across tile borders) wait for the CTA's queue and run there with full
        // warps, unless most lanes of this warp need it anyway or the queue is full.
        const unsigned clip = __ballot_sync(0xffffffffu, keep && !inside);
        bool now = keep;
        if (clip && __popc(clip) < 20) {
            uint32_t at = 0;
            if (lane == 0) at = atomicAdd(&s_queued, (uint32_t)__popc(clip));
            at = __shfl_sync(0xffffffffu, at, 0) + __popc(clip & below);
            if (keep && !inside && at < kBinQueue) {
                s_qx[at] = tx;
                s_qy[at] = (ty << 8) | (uint32_t)ct;
                s_qe[at] = e;
                now = false;
            }
        }
        if (now) write_pair(bin, s_tri[ct >> 5] + (ct & 31), t_cta + (ct >> 5) * per_warp + (ct & 31), tx, ty, slot0 + e, cx, cy,
                            s_poly + tid);
    }
    __syncthreads();
    const uint32_t queued = min(s_queued, (uint32_t)kBinQueue);
    for (uint32_t q = tid; q < queued; q += 32 * kBinWarps) {
        const uint32_t tx = s_qx[q], ty = s_qy[q] >> 8;
        const int ct = (int)(s_qy[q] & 255u);
        write_pair(bin, s_tri[ct >> 5] + (ct & 31), t_cta + (ct >> 5) * per_warp + (ct & 31), tx, ty, slot0 + s_qe[q],
                   __ldg(bin.tables.cols + tx), __ldg(bin.tables.rows + ty), s_poly + tid);
    }
}

// Images of more tiles than place_entries_kernel has shared memory for: one CTA turns the counts into tile offsets (unless a
// device-wide scan follows), and scatter_entries_kernel moves the entries.
__global__ void __launch_bounds__(32 * kFinishWarps) bin_finish_kernel(BinArgs bin) {
    __shared__ uint32_t s_warp[kFinishWarps];
    allow_dependents();
    await_prerequisites();
    const uint32_t slots = slots_used(bin);
    uint32_t K = slots, longest = UINT32_MAX;            // longest: not known
    if (bin.scan_here) {
        longest = tile_offsets_by_one_cta<kFinishWarps>(bin.tile_counts, bin.offsets, bin.tiles, s_warp, true, K);
        if (slots == kTooManyPairs) K = kTooManyPairs;   // the counts' sum is not the number of pairs then
    }
    if (threadIdx.x == 0) publish_counts(bin, K, longest, slots);
}

// Counts to tile offsets, and every entry to its place: offset of its tile plus its rank there.  Every CTA makes the offsets
// for itself, in shared memory, while its first pairs are on their way; the first one leaves them for the kernels behind, with K, the
// longest list and the launch order of the tiles, instead of moving entries.
// Against the scan by one CTA (the binning kernel's last, or a kernel of its own) and a scatter that looked the offsets up in
// memory, B200: 200k triangles, 1920x1080 13.4 -> 6.7 us; 1.3M triangles, the same image, with the launch order 39 -> 16;
// 2M triangles, 3840x2160 102 -> 92; 1280 triangles, 256x256, with the binning 15.6 -> 12.2.  Latency: half of the 6.7 us are
// the scan's loads and barriers; the large one is bound by the scattered stores of 8 bytes.
template <int NT>
__global__ void __launch_bounds__(NT) place_entries_kernel(BinArgs bin, uint64_t* __restrict__ entries, uint32_t* __restrict__ order,
                                                           uint32_t* __restrict__ list_heads) {
    extern __shared__ __align__(16) int32_t s_off[];            // [tiles + 1]
    __shared__ uint32_t s_warp[NT / 32];
    __shared__ uint4 s_sums[NT / 32];
    constexpr uint32_t kPer = 4;                                // pairs of a thread in flight
    const uint32_t tid = threadIdx.x, stride = (gridDim.x - 1) * kPer * NT;
    allow_dependents();
    await_prerequisites();
    const bool tables = blockIdx.x == 0;
    uint32_t first = (blockIdx.x - 1) * kPer * NT + tid;
    uint4 p[kPer];
#pragma unroll
    for (uint32_t k = 0; k < kPer; k++)
        if (!tables && first + NT * k < bin.capacity) p[k] = __ldcs(bin.pairs + first + NT * k);
    const uint32_t n = slots_used(bin);                         // holes included
    uint32_t K = 0;
    const uint32_t longest = tile_offsets_by_one_cta<NT / 32>(bin.tile_counts, s_off, bin.tiles, s_warp, tables, K);
    if (tables) {
        if (n == kTooManyPairs) K = kTooManyPairs;              // the counts' sum is not the number of pairs then
        const bool ordered = order_wanted(bin, K, longest);
        if (tid == 0) publish_counts(bin, K, ordered ? longest | kOrderWrittenBit : longest, n);
        if (tid < 6) list_heads[tid] = 0;
        for (int i = tid; i <= bin.tiles; i += NT) bin.offsets[i] = s_off[i];
        if (ordered) tile_order_by_one_cta<NT>(s_off, bin.tiles, order, s_sums);
        return;
    }
    if (n > bin.capacity) return;
    for (; first < n; first += stride) {
        uint32_t to[kPer];
#pragma unroll
        for (uint32_t k = 0; k < kPer; k++) {
            if (first + NT * k >= n) p[k].z = kHole;
            to[k] = p[k].z != kHole ? (uint32_t)s_off[p[k].z] + p[k].w : 0u;
        }
#pragma unroll
        for (uint32_t k = 0; k < kPer; k++) {
            if (p[k].z != kHole) entries[to[k]] = ((uint64_t)p[k].y << 32) | p[k].x;
            const uint32_t next = first + stride + NT * k;
            if (next < n) p[k] = __ldcs(bin.pairs + next);
        }
    }
}

// Every entry to its place.
__global__ void __launch_bounds__(256) scatter_entries_kernel(const uint4* __restrict__ pairs, const uint32_t* __restrict__ info,
                                                              uint32_t capacity, const int32_t* __restrict__ offsets,
                                                              uint64_t* __restrict__ entries,
                                                              int tiles, uint32_t* __restrict__ tile_counts,
                                                              uint32_t* __restrict__ counters, uint32_t* __restrict__ list_heads) {
    allow_dependents();
    await_prerequisites();
    // the binning kernel is done with its counters: zero for the next call
    const uint32_t me = blockIdx.x * 256 + threadIdx.x;
    for (uint32_t i = me; i < (uint32_t)tiles; i += gridDim.x * 256) tile_counts[i] = 0;
    if (me < 4) counters[me] = 0;
    if (me < 6) list_heads[me] = 0;
    const uint32_t n = info[2];               // slots, holes included
    if (n > capacity) return;
    // four entries per thread in flight: each is a chain of two loads and a scattered store
    const uint32_t stride = gridDim.x * 1024;
    for (uint32_t i = blockIdx.x * 1024 + threadIdx.x; i < n; i += stride) {
        uint4 p[4];
        uint32_t off[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            p[k].z = kHole;
            if (i + 256 * k < n) p[k] = __ldcs(pairs + i + 256 * k);
        }
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (p[k].z != kHole) off[k] = (uint32_t)__ldg(offsets + p[k].z);
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (p[k].z != kHole) entries[off[k] + p[k].w] = ((uint64_t)p[k].y << 32) | p[k].x;
    }
}

// Inputs in the packed layout: colours and opacities as one [V,4] array, faces as [T,4] (fourth word 0).
__global__ void __launch_bounds__(256) pack_inputs_kernel(const float* __restrict__ colors,
                                                          const float* __restrict__ opacities,
                                                          const int* __restrict__ indices, int V, int T,
                                                          float4* __restrict__ rgba, int4* __restrict__ faces) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < V) rgba[i] = make_float4(colors[3 * (size_t)i], colors[3 * (size_t)i + 1], colors[3 * (size_t)i + 2], opacities[i]);
    if (i < T) faces[i] = make_int4(indices[3 * (size_t)i], indices[3 * (size_t)i + 1], indices[3 * (size_t)i + 2], 0);
}

// ================================================================================================
// Stage 5: tile ranges from the sorted keys.  Thread i looks at the boundary before entry i.
__global__ void __launch_bounds__(256) tile_ranges_kernel(const uint64_t* __restrict__ keys, uint32_t n, int tiles,
                                                          int* __restrict__ offsets) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i > n) return;
    const int prev = (i == 0) ? -1 : (int)(keys[i - 1] >> 32);
    int cur = (i == n) ? tiles : (int)(keys[i] >> 32);
    if (cur > tiles) cur = tiles;
    for (int t = prev + 1; t <= cur; t++) offsets[t] = (int)i;
}

}  // namespace tg

// ================================================================================================
// host side
namespace tg_host {
static thread_local char g_err[512] = "";
void set_error(const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
}
int cuda_fail(cudaError_t e, const char* what) {
    set_error("CUDA error %d (%s) at %s", (int)e, cudaGetErrorString(e), what);
    return TG_ERR_CUDA;
}
const char* last_error() { return g_err; }

int check_sizes(int W, int H, int tw, int th) {
    TG_REQUIRE(W > 0 && H > 0, "image size must be positive");
    TG_REQUIRE(tw > 0 && th > 0, "tile size must be positive");
    TG_REQUIRE((int64_t)tw * th <= 1024, "tile_width * tile_height must be <= 1024");
    TG_REQUIRE(W <= INT32_MAX - tw && H <= INT32_MAX - th &&
                   (int64_t)((W + tw - 1) / tw) * ((H + th - 1) / th) < INT32_MAX,
               "too many tiles");
    return TG_OK;
}

int allow_smem(const void* kernel, size_t bytes, SmemAllowed& allowed) {
    int dev = 0;
    TG_CUDA(cudaGetDevice(&dev));
    TG_REQUIRE(dev >= 0 && dev < SmemAllowed::kMaxDevices, "device index outside the supported range");
    if (!allowed.set[dev].load(std::memory_order_acquire)) {
        TG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
        allowed.set[dev].store(true, std::memory_order_release);
    }
    return TG_OK;
}

int prefer_smem(const void* kernel, int kilobytes, SmemAllowed& preferred) {
    int dev = 0;
    TG_CUDA(cudaGetDevice(&dev));
    TG_REQUIRE(dev >= 0 && dev < SmemAllowed::kMaxDevices, "device index outside the supported range");
    if (!preferred.set[dev].load(std::memory_order_acquire)) {
        TG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, kilobytes * 100 / 228));
        preferred.set[dev].store(true, std::memory_order_release);
    }
    return TG_OK;
}

static tg::BinArgs bin_args(const BinBuffers& b, int W, int H, int tw, int th, int32_t* offsets, uint32_t list_capacity,
                            uint32_t* info_host, uint32_t* long_host) {
    const int tiles_x = (W + tw - 1) / tw, tiles_y = (H + th - 1) / th, tiles = tiles_x * tiles_y;
    return {b.tile_counts, offsets, b.counters, b.info, info_host, long_host, b.pairs, nullptr, 0, list_capacity, tiles, tiles_x, tiles_y,
            tiles <= tg::kTileScanByOneCta ? 1 : 0, b.tile_order ? 1 : 0, {b.tables, b.tables + tiles_x}};
}

// Per-triangle records and (triangle, tile) pairs: bin_init_kernel and bin_kernel (declared in tg_radix.cuh with what each
// argument is).
int bin_triangles(const float* vertices, const int32_t* indices, const float* colors, const float* opacities, int T, int W,
                  int H, int tw, int th, float* tri_geo, float* tri_attr, const BinBuffers& b, int32_t* offsets,
                  uint32_t list_capacity, bool cull, bool packed, bool ready, bool in_place, cudaStream_t stream) {
    TG_REQUIRE(T >= 0, "T < 0");
    if (int s = check_sizes(W, H, tw, th)) return s;
    TG_REQUIRE(offsets, "null pointer");
    const int tiles_x = (W + tw - 1) / tw, tiles_y = (H + th - 1) / th;
    const int tiles = tiles_x * tiles_y;
    TG_REQUIRE(T == 0 || (vertices && indices && colors && (packed || opacities) && tri_geo && tri_attr), "null pointer");
    TG_REQUIRE(((uintptr_t)vertices & 15) == 0 && ((uintptr_t)tri_geo & 15) == 0 && ((uintptr_t)tri_attr & 15) == 0,
               "vertices / tri_geo / tri_attr must be 16-byte aligned");
    TG_REQUIRE(!packed || ((((uintptr_t)indices | (uintptr_t)colors) & 15) == 0),
               "packed faces [T,4] and colours [V,4] must be 16-byte aligned");
    const bool by_one_cta = tiles <= tg::kTileScanByOneCta;
    TG_REQUIRE(!cull || by_one_cta, "tile culling is limited to 65536 tiles");
    float4* rows = b.tables + tiles_x;
    if (!ready || !by_one_cta) {
        const size_t init = b.clear_words > (size_t)tiles_x + tiles_y ? b.clear_words : (size_t)tiles_x + tiles_y;
        tg::bin_init_kernel<<<(unsigned)((init + 255) / 256), 256, 0, stream>>>(b.clear, b.clear_words, b.tables, rows, tiles_x,
                                                                              tiles_y, W, H, tw, th);
        TG_LAUNCH_CHECK("bin_init_kernel");
    }
    if (T == 0) {
        TG_CUDA(cudaMemsetAsync(b.info, 0, sizeof(uint32_t) * 3, stream));
        TG_CUDA(cudaMemsetAsync(offsets, 0, sizeof(int32_t) * ((size_t)tiles + 1), stream));
        return TG_OK;
    }
    // Triangles per CTA: 32 per warp where that fills the GPU; fewer below, so that a mesh of few triangles that cover many
    // tiles each still spreads over all SMs (eight CTAs on each).
    constexpr int kWave = 148 * 32 / tg::kBinWarps;
    const int per_cta = T >= 32 * tg::kBinWarps * kWave ? 32 * tg::kBinWarps : (T + kWave - 1) / kWave;
    const int grid = (T + per_cta - 1) / per_cta;
    tg::BinArgs bin = bin_args(b, W, H, tw, th, offsets, list_capacity, nullptr, nullptr);
    if (in_place) {
        TG_REQUIRE((uint64_t)T * tiles <= list_capacity, "no room for every pair");
        bin.lists = b.entries;
        bin.room = (uint32_t)T;
    }
    auto inverse = [](int n) { return (n & (n - 1)) == 0 ? 1.0 / n : 0.0; };
    auto kernel = cull ? tg::bin_kernel<true> : tg::bin_kernel<false>;
    static SmemAllowed bin_allowed[2];
    if (int st = allow_smem((const void*)kernel, tg::kBinSmem, bin_allowed[cull ? 1 : 0])) return st;
    TG_CUDA(launch_dependent(kernel, grid, 32 * tg::kBinWarps, tg::kBinSmem, stream, (const float4*)vertices, indices, colors,
                             opacities, T, per_cta, W, H, tw, th, inverse(tw), inverse(th), (float4*)tri_geo, (float4*)tri_attr,
                             bin, packed ? 1 : 0));
    TG_LAUNCH_CHECK("bin_kernel");
    return TG_OK;
}

int place_entries(const BinBuffers& b, int T, int W, int H, int tw, int th, int32_t* offsets, uint32_t list_capacity,
                  uint32_t* info_host, uint32_t* long_host, cudaStream_t stream) {
    if (T == 0) return TG_OK;
    const tg::BinArgs bin = bin_args(b, W, H, tw, th, offsets, list_capacity, info_host, long_host);
    const int tiles = bin.tiles;
    if (tiles <= tg::kPlaceTiles) {
        // One CTA per SM, and no more than the list capacity, which is what the host knows of the number of pairs, fills; the
        // first moves none.  More of them read the counts more often than the loop gains (two per SM: 8.0 us against 6.7,
        // 200k triangles, 1920x1080).  The offsets of very many tiles leave an SM room for one CTA, which then has 1024
        // threads (2M triangles, 3840x2160, 32400 tiles: 92 us; 8160 tiles with 1024 threads: 7.2 against 6.7).
        const bool big = tiles > tg::kPlaceTilesSmall;
        const int threads = big ? 1024 : 512;
        const uint32_t want = (list_capacity + 4 * threads - 1) / (4 * threads);
        const int ctas = (int)(want < 147 ? want + 1 : 148);
        const size_t smem = sizeof(int32_t) * ((size_t)tiles + 1);
        static SmemAllowed place_allowed[2];
        auto place = big ? tg::place_entries_kernel<1024> : tg::place_entries_kernel<512>;
        if (int st = allow_smem((const void*)place, sizeof(int32_t) * ((big ? tg::kPlaceTiles : tg::kPlaceTilesSmall) + 1), place_allowed[big]))
            return st;
        TG_CUDA(launch_dependent(place, ctas, threads, smem, stream, bin, b.entries, b.tile_order, b.list_heads));
        TG_LAUNCH_CHECK("place_entries_kernel");
        return TG_OK;
    }
    TG_CUDA(launch_dependent(tg::bin_finish_kernel, 1, 32 * tg::kFinishWarps, 0, stream, bin));
    TG_LAUNCH_CHECK("bin_finish_kernel");
    if (!bin.scan_here) {
        const int parts = (tiles + tg::kScanTile - 1) / tg::kScanTile;
        tg::scan_kernel<<<parts, tg::kScanThreads, 0, stream>>>(b.tile_counts, (uint32_t*)offsets, tiles, parts,
                                                                 (uint32_t*)b.tile_scan_scratch,
                                                                 (uint64_t*)((char*)b.tile_scan_scratch + 8), b.status);
        TG_LAUNCH_CHECK("scan_kernel");
    }
    // K is not known on the host yet: as many CTAs as its upper bound fills, at most eight per SM
    const uint32_t want = (list_capacity + 1023) / 1024;
    const int ctas = want < 1 ? 1 : (int)(want < 148 * 8 ? want : 148 * 8);
    TG_CUDA(launch_dependent(tg::scatter_entries_kernel, ctas, 256, 0, stream, b.pairs, b.info, list_capacity, offsets, b.entries,
                             tiles, b.tile_counts, b.counters, b.list_heads));
    TG_LAUNCH_CHECK("scatter_entries_kernel");
    return TG_OK;
}

static std::atomic<unsigned long long> g_launches{0};
void count_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }
}  // namespace tg_host

extern "C" {

int tg_version(void) { return 1; }

unsigned long long tg_launch_count(void) { return tg_host::g_launches.load(std::memory_order_relaxed); }

const char* tg_last_error(void) { return tg_host::last_error(); }

const char* tg_status_string(int s) {
    switch (s) {
        case TG_OK: return "ok";
        case TG_ERR_BAD_ARG: return "bad argument";
        case TG_ERR_WORKSPACE: return "workspace too small";
        case TG_ERR_CAPACITY: return "list capacity exceeded";
        case TG_ERR_DEVICE_FLAG: return "device error flag set (a bounded wait ran out)";
        case TG_ERR_CUDA: return "CUDA error";
        default: return "unknown status";
    }
}

static int check_dims(int T, int W, int H, int tw, int th) {
    TG_REQUIRE(T >= 0, "T < 0");
    return tg_host::check_sizes(W, H, tw, th);
}

int tg_preprocess(const float* vertices, const int32_t* indices, const float* colors, const float* opacities, int T,
                  int W, int H, int tw, int th, uint32_t* tri_counts, int32_t* tri_rects, float* tri_geo,
                  float* tri_attr, tg_stream_t stream) {
    if (int s = check_dims(T, W, H, tw, th)) return s;
    if (T == 0) return TG_OK;
    TG_REQUIRE(vertices && indices && colors && opacities && tri_counts && tri_geo && tri_attr, "null pointer");
    TG_REQUIRE(((uintptr_t)vertices & 15) == 0 && ((uintptr_t)tri_geo & 15) == 0 && ((uintptr_t)tri_attr & 15) == 0 &&
                   ((uintptr_t)tri_rects & 15) == 0,
               "vertices / tri_geo / tri_attr / tri_rects must be 16-byte aligned");
    const int tiles_x = (W + tw - 1) / tw, tiles_y = (H + th - 1) / th;
    tg::preprocess_kernel<<<(T + 255) / 256, 256, 0, (cudaStream_t)stream>>>(
        (const float4*)vertices, indices, colors, opacities, T, W, H, tw, th, tiles_x, tiles_y, tri_counts,
        (int4*)tri_rects, (float4*)tri_geo, (float4*)tri_attr);
    TG_LAUNCH_CHECK("preprocess_kernel");
    return TG_OK;
}

size_t tg_scan_scratch_bytes(int n) {
    size_t parts = (size_t)((n > 0 ? n : 0) + tg::kScanTile - 1) / tg::kScanTile;
    return 8 + 8 * (parts + 1);
}

int tg_scan(const uint32_t* in, uint32_t* out, int n, void* scratch, size_t scratch_bytes, uint32_t* status,
            tg_stream_t stream) {
    TG_REQUIRE(n >= 0, "n < 0");
    TG_REQUIRE(out && scratch && status, "null pointer");
    TG_REQUIRE(((uintptr_t)scratch & 7) == 0, "scratch must be 8-byte aligned");
    if (scratch_bytes < tg_scan_scratch_bytes(n)) {
        tg_host::set_error("scan scratch: need %zu bytes, got %zu", tg_scan_scratch_bytes(n), scratch_bytes);
        return TG_ERR_WORKSPACE;
    }
    cudaStream_t s = (cudaStream_t)stream;
    if (n == 0) {
        TG_CUDA(cudaMemsetAsync(out, 0, sizeof(uint32_t), s));
        return TG_OK;
    }
    TG_REQUIRE(in != nullptr, "null pointer");
    const int parts = (n + tg::kScanTile - 1) / tg::kScanTile;
    TG_CUDA(cudaMemsetAsync(scratch, 0, tg_scan_scratch_bytes(n), s));
    tg::scan_kernel<<<parts, tg::kScanThreads, 0, s>>>(in, out, n, parts, (uint32_t*)scratch,
                                                      (uint64_t*)((char*)scratch + 8), status);
    TG_LAUNCH_CHECK("scan_kernel");
    return TG_OK;
}

// ---- prefix scan without caller-provided scratch ------------------------------------------------
// Some hosts of this library may not allocate device memory at the point where they need a scan:
// code running under a fixed memory budget that was carved up at start-up, a real-time loop that
// must not touch the allocator, or a plugin whose embedding application owns every allocation.
// For them the partition words of the look-back scan live in a fixed array inside the library
// image.  Every GPU that loads the library holds these 64 KB + 256 B until the process exits.
constexpr int kStaticScanMaxN = 1 << 24;                                         // elements per call
constexpr int kStaticScanMaxParts = (kStaticScanMaxN + tg::kScanTile - 1) / tg::kScanTile;
constexpr size_t kStaticScanBytes = 256 + 8 * ((size_t)kStaticScanMaxParts + 1);  // ticket (padded) + words
static __device__ __align__(256) unsigned char g_static_scan_scratch[kStaticScanBytes];

// In host code the array's name is only a handle; the device address has to be asked for, once per
// device, with that device current.
static int static_scan_scratch_address(void** out) {
    constexpr int kMaxDevices = 64;
    static std::atomic<void*> cache[kMaxDevices];
    int dev = 0;
    TG_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) {
        tg_host::set_error("device index %d outside the supported range", dev);
        return TG_ERR_BAD_ARG;
    }
    void* p = cache[dev].load(std::memory_order_acquire);
    if (p == nullptr) {
        TG_CUDA(cudaGetSymbolAddress(&p, g_static_scan_scratch));
        cache[dev].store(p, std::memory_order_release);
    }
    *out = p;
    return TG_OK;
}

int tg_scan_static(const uint32_t* in, uint32_t* out, int n, uint32_t* status, tg_stream_t stream) {
    TG_REQUIRE(n >= 0, "n < 0");
    TG_REQUIRE(out && status, "null pointer");
    if (n > kStaticScanMaxN) {
        tg_host::set_error("tg_scan_static handles at most %d elements per call (got %d); use tg_scan with caller scratch",
                           kStaticScanMaxN, n);
        return TG_ERR_CAPACITY;
    }
    cudaStream_t s = (cudaStream_t)stream;
    if (n == 0) {
        TG_CUDA(cudaMemsetAsync(out, 0, sizeof(uint32_t), s));
        return TG_OK;
    }
    TG_REQUIRE(in != nullptr, "null pointer");
    void* scratch = nullptr;
    if (int st = static_scan_scratch_address(&scratch)) return st;
    const int parts = (n + tg::kScanTile - 1) / tg::kScanTile;
    // the array keeps what the previous call left: clear the ticket and the words this call uses
    TG_CUDA(cudaMemsetAsync(scratch, 0, 256 + 8 * ((size_t)parts + 1), s));
    tg::scan_kernel<<<parts, tg::kScanThreads, 0, s>>>(in, out, n, parts, (uint32_t*)scratch,
                                                      (uint64_t*)((char*)scratch + 256), status);
    TG_LAUNCH_CHECK("scan_kernel (static scratch)");
    return TG_OK;
}

int tg_pack_inputs(const float* colors, const float* opacities, const int32_t* indices, int V, int T, float* rgba,
                   int32_t* faces, tg_stream_t stream) {
    TG_REQUIRE(V >= 0 && T >= 0, "negative size");
    if (V == 0 && T == 0) return TG_OK;
    TG_REQUIRE((V == 0 || (colors && opacities && rgba)) && (T == 0 || (indices && faces)), "null pointer");
    TG_REQUIRE((((uintptr_t)rgba | (uintptr_t)faces) & 15) == 0, "rgba / faces must be 16-byte aligned");
    const int n = V > T ? V : T;
    tg::pack_inputs_kernel<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(colors, opacities, indices, V, T,
                                                                              (float4*)rgba, (int4*)faces);
    TG_LAUNCH_CHECK("pack_inputs_kernel");
    return TG_OK;
}

int tg_selftest_bounded_wait(void* scratch, size_t scratch_bytes, uint32_t* status, uint32_t spin_limit,
                             tg_stream_t stream) {
    TG_REQUIRE(scratch && status, "null pointer");
    TG_REQUIRE(((uintptr_t)scratch & 7) == 0 && scratch_bytes >= 32, "scratch: 32 bytes, 8-byte aligned");
    TG_REQUIRE(spin_limit >= 1 && spin_limit <= 4096, "spin_limit must be in 1..4096");
    cudaStream_t s = (cudaStream_t)stream;
    TG_CUDA(cudaMemsetAsync(scratch, 0, 32, s));
    tg::bounded_wait_selftest_kernel<<<1, 32, 0, s>>>((uint64_t*)scratch, status, spin_limit, (uint32_t*)scratch + 6);
    TG_LAUNCH_CHECK("bounded_wait_selftest_kernel");
    return TG_OK;
}

int tg_emit_keys(const float* vertices, const int32_t* indices, int T, int W, int H, int tw, int th,
                 const uint32_t* tri_offsets, uint64_t* keys, uint32_t* ids, uint32_t capacity, tg_stream_t stream) {
    if (int s = check_dims(T, W, H, tw, th)) return s;
    if (T == 0) return TG_OK;
    TG_REQUIRE(vertices && indices && tri_offsets && keys && ids, "null pointer");
    const int tiles_x = (W + tw - 1) / tw, tiles_y = (H + th - 1) / th;
    tg::emit_keys_kernel<<<(T + tg::kEmitThreads - 1) / tg::kEmitThreads, tg::kEmitThreads, 0, (cudaStream_t)stream>>>(
        (const float4*)vertices, indices, T, W, H, tw, th, tiles_x, tiles_y, tri_offsets, keys, ids, capacity);
    TG_LAUNCH_CHECK("emit_keys_kernel");
    return TG_OK;
}

int tg_tile_ranges(const uint64_t* sorted_keys, uint32_t n, int tiles, int32_t* offsets, tg_stream_t stream) {
    TG_REQUIRE(tiles > 0 && offsets, "bad tiles / offsets");
    TG_REQUIRE(n == 0 || sorted_keys, "null keys");
    TG_REQUIRE(n < 0x80000000u, "K must stay below 2^31");
    const uint32_t threads = n + 1;
    tg::tile_ranges_kernel<<<(threads + 255) / 256, 256, 0, (cudaStream_t)stream>>>(sorted_keys, n, tiles, offsets);
    TG_LAUNCH_CHECK("tile_ranges_kernel");
    return TG_OK;
}

}  // extern "C"
