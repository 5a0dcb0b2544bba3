// Stages 6 and 7: per-tile forward compositing and the backward (gradient) kernel.
//
// One CTA per tile, one thread per pixel (tile_w*tile_h threads rounded up to a warp multiple); a
// warp owns an 8x4 pixel block when the tile size allows it.  The tile's depth-sorted triangle
// list is streamed through shared memory in coalesced, vectorised chunks of packed 64-byte
// geometry records.  For every staged chunk each warp first rejects, with one lane per record, the
// records that cannot cover any of its 32 pixels (exact corner test on the same rounded
// arithmetic as the per-pixel test); only the survivors are tested per pixel.
//
// per_pixel_sort = true  (the reference default): each pixel keeps the nearest <= 32 covering
//     fragments by (interpolated depth, list position) and blends them in that order; further
//     batches of 32 follow while transmittance > threshold and blended < max_layers.  The ids of
//     the blended fragments can be saved per pixel so that the backward pass need not search again.
// per_pixel_sort = false: fragments are blended in list order; a pixel stops once its
//     transmittance is <= threshold, a warp skips chunks once all its lanes stopped (ballot) and
//     the CTA leaves the list as soon as every warp voted "done".
//
// Backward: per pixel the recorded fragments are walked last to first with the reference's
// recurrences; the contributions of a warp's lanes are summed per triangle, and the sums go to a packed
// per-vertex buffer (x, y, w, opacity | r, g, b, -), mostly with one 24-lane atomic addition per triangle
// (lanes of which too few share a triangle add for themselves, with red.global.add.v4.f32).  A small kernel
// unpacks the buffer into grad_vertices / grad_colors / grad_opacities.
#include "tg_radix.cuh"

namespace tg {

constexpr int kChunk = 64;   // records staged per step (64 bytes each, 80 bytes apart in shared memory)

struct BlendParams {
    const float4* geo;
    const float4* attr;
    const int* ids;
    const int* offsets;
    int W, H, tw, th, tiles_x;
    float thr;
    int max_layers;
    // Optional launch order of the tiles (longest lists first, so that no heavy tile starts late): CTA b handles tile
    // order[b], or tile b when there is none (the stage entry points; lists too short or too even to bother).
    const uint32_t* order;
};

__device__ __forceinline__ int tile_of_block(const BlendParams& P) {
    return P.order != nullptr ? (int)P.order[blockIdx.x] : (int)blockIdx.x;
}

struct PixelAcc {
    float alpha = 1.f, r = 0.f, g = 0.f, b = 0.f, depth = 0.f, weight = 0.f;
    int blended = 0;
};

// Load the geometry record of triangle `id` straight from global memory (L1/L2 resident).
__device__ __forceinline__ void load_geo(const float4* geo, int id, float* m, float* w) {
    const float4 g0 = __ldg(geo + 4 * (size_t)id), g1 = __ldg(geo + 4 * (size_t)id + 1);
    const float4 g2 = __ldg(geo + 4 * (size_t)id + 2), g3 = __ldg(geo + 4 * (size_t)id + 3);
    m[0] = g0.x; m[1] = g0.y; m[2] = g0.z; m[3] = g0.w; m[4] = g1.x; m[5] = g1.y; m[6] = g1.z; m[7] = g1.w; m[8] = g2.x;
    w[0] = g3.x; w[1] = g3.y; w[2] = g3.z;
}

constexpr int kAttrQuads = TG_ATTR_WORDS / 4;
// Brings a triangle's records towards L1: the backward knows the fragment after the current one (3 % of its time).
__device__ __forceinline__ void prefetch_record(const BlendParams& P, int id) {
    asm volatile("prefetch.global.L1 [%0];" ::"l"(P.geo + 4 * (size_t)id));
    asm volatile("prefetch.global.L1 [%0];" ::"l"(P.attr + kAttrQuads * (size_t)id));
}

struct AttrRec { float o[3]; float c[9]; float iw[3]; int vid[3]; float xy[6]; };

// FULL = false loads only what the forward pass needs (opacities, colours, 1/w).  `q`: global or shared memory.
template <bool FULL>
__device__ __forceinline__ AttrRec attr_from(const float4* q) {
    const float4 q0 = q[0], q1 = q[1], q2 = q[2], q3 = q[3];
    AttrRec a;
    a.o[0] = q0.x; a.o[1] = q0.y; a.o[2] = q0.z;
    a.c[0] = q0.w; a.c[1] = q1.x; a.c[2] = q1.y; a.c[3] = q1.z; a.c[4] = q1.w; a.c[5] = q2.x; a.c[6] = q2.y; a.c[7] = q2.z;
    a.c[8] = q2.w;
    a.iw[0] = q3.x; a.iw[1] = q3.y; a.iw[2] = q3.z;
    if (FULL) {
        const float4 q4 = q[4], q5 = q[5];
        a.vid[0] = __float_as_int(q3.w); a.vid[1] = __float_as_int(q4.x); a.vid[2] = __float_as_int(q4.y);
        a.xy[0] = q4.z; a.xy[1] = q4.w; a.xy[2] = q5.x; a.xy[3] = q5.y; a.xy[4] = q5.z; a.xy[5] = q5.w;
    }
    return a;
}
template <bool FULL>
__device__ __forceinline__ AttrRec load_attr(const float4* attr, int id) {
    const float4* g = attr + kAttrQuads * (size_t)id;
    float4 q[6];
#pragma unroll
    for (int k = 0; k < (FULL ? 6 : 4); k++) q[k] = __ldg(g + k);
    return attr_from<FULL>(q);
}

// process_forward of the reference (render.cu:417-453); every operation rounded separately, in the
// oracle's order, so that the image agrees bit for bit with it.  The four weighted interpolations
// share one correctly rounded reciprocal of their common denominator.
struct BlendedValues { float o_raw, cr, cg, cb, z, den; };

__device__ __forceinline__ BlendedValues blend_one(const Bary& b, const float* w, const AttrRec& a, PixelAcc& acc) {
    BlendedValues v;
    v.den = fma_(b.z, w[2], fma_(b.y, w[1], mul(b.x, w[0])));
    const float inv = __frcp_rn(v.den);
    auto weighted = [&](float a0, float a1, float a2) -> float {
        float nom = mul(mul(b.x, a0), w[0]);
        nom = fma_(mul(b.y, a1), w[1], nom);
        nom = fma_(mul(b.z, a2), w[2], nom);
        return mul(nom, inv);
    };
    v.o_raw = weighted(a.o[0], a.o[1], a.o[2]);
    const float o = fminf(fmaxf(v.o_raw, 0.f), kMaxOpacity);
    v.cr = weighted(a.c[0], a.c[3], a.c[6]);
    v.cg = weighted(a.c[1], a.c[4], a.c[7]);
    v.cb = weighted(a.c[2], a.c[5], a.c[8]);
    v.z = interp_rn(b, a.iw[0], a.iw[1], a.iw[2], 1.f, 1.f, 1.f);
    const float ao = mul(acc.alpha, o);
    acc.depth = add(acc.depth, mul(ao, v.z));
    acc.weight = add(acc.weight, ao);
    acc.r = add(acc.r, mul(ao, v.cr));
    acc.g = add(acc.g, mul(ao, v.cg));
    acc.b = add(acc.b, mul(ao, v.cb));
    acc.alpha = mul(acc.alpha, sub(1.f, o));
    acc.blended++;
    return v;
}

// NDC extent (pixel centres) of the active pixels of one warp.
using WarpRect = PixelRect;

struct TileCtx {
    int tile, start, end, ix, iy;
    bool active;
    float px, py;
    WarpRect rect;
    const float *s_x, *s_y;     // centres of the 8 columns and 4 rows of the warp's block, null without 8x4 blocks
};

// Pixel-centre coordinates need double arithmetic (one rounding, reference render.cu:561-562); the
// tile_w + tile_h distinct values of a tile are computed once by its first threads and shared.
constexpr int kMaxTileCoords = 1026;

__device__ __forceinline__ TileCtx tile_context(const BlendParams& P, float* s_coord) {
    TileCtx c;
    c.tile = tile_of_block(P);
    const int tx = c.tile % P.tiles_x, ty = c.tile / P.tiles_x;
    for (int i = threadIdx.x; i < P.tw + P.th; i += blockDim.x)
        s_coord[i] = (i < P.tw) ? pixel_coord(tx * P.tw + i, P.W) : pixel_coord(ty * P.th + (i - P.tw), P.H);
    int lx, ly;
    const bool blocks = (P.tw & 7) == 0 && (P.th & 3) == 0;
    int bx0 = 0, by0 = 0;
    if (blocks) {
        // a warp owns an 8x4 block of the tile: compact footprint, fewer records survive its cull
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, bpr = P.tw >> 3;
        bx0 = (warp % bpr) * 8;
        by0 = (warp / bpr) * 4;
        lx = bx0 + (lane & 7);
        ly = by0 + (lane >> 3);
    } else {
        lx = threadIdx.x % P.tw;
        ly = threadIdx.x / P.tw;
    }
    c.ix = tx * P.tw + lx;
    c.iy = ty * P.th + ly;
    c.active = (int)threadIdx.x < P.tw * P.th && c.ix < P.W && c.iy < P.H;
    // (a caller that walks no tile list - the queued backward, whose blocks need not be the forward's tiles - passes none)
    c.start = P.offsets ? P.offsets[c.tile] : 0;
    c.end = P.offsets ? P.offsets[c.tile + 1] : 0;
    __syncthreads();
    c.s_x = blocks ? s_coord + bx0 : nullptr;
    c.s_y = s_coord + P.tw + by0;
    c.px = s_coord[min(lx, P.tw - 1)];
    c.py = s_coord[P.tw + min(ly, P.th - 1)];
    if (blocks) {
        // the coordinates grow with the index, so the extent of the block's pixels inside the image is given by
        // its first and last valid column and row
        const int nx = min(8, P.W - tx * P.tw - bx0), ny = min(4, P.H - ty * P.th - by0);
        if (nx > 0 && ny > 0 && (int)threadIdx.x < P.tw * P.th)
            c.rect = {s_coord[bx0], s_coord[bx0 + nx - 1], s_coord[P.tw + by0], s_coord[P.tw + by0 + ny - 1]};
        else
            c.rect = {INFINITY, -INFINITY, INFINITY, -INFINITY};
        return c;
    }
    float x0 = c.active ? c.px : INFINITY, x1 = c.active ? c.px : -INFINITY;
    float y0 = c.active ? c.py : INFINITY, y1 = c.active ? c.py : -INFINITY;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        x0 = fminf(x0, __shfl_xor_sync(0xffffffffu, x0, d));
        x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, d));
        y0 = fminf(y0, __shfl_xor_sync(0xffffffffu, y0, d));
        y1 = fmaxf(y1, __shfl_xor_sync(0xffffffffu, y1, d));
    }
    c.rect = {x0, x1, y0, y1};
    return c;
}

// Stage `n` records of the list starting at `first` into shared memory (ids + geometry).
// Staged records are 80 bytes apart (64 bytes of record, 16 of padding): with that stride the 32 lanes of a warp can
// each read "their" record with 16-byte loads without shared-memory bank conflicts (a 64-byte stride puts every
// second lane on the same banks), and the words of a record keep constant offsets from its base.
constexpr int kStagedQuads = 5;
__device__ __forceinline__ int staged_quad(int r, int q) { return kStagedQuads * r + q; }

__device__ __forceinline__ void stage_chunk(const BlendParams& P, int first, int n, float4* s_geo, int* s_id) {
    for (int i = threadIdx.x; i < n * 4; i += blockDim.x) {
        const int rec = i >> 2, q = i & 3;
        const int id = P.ids[first + rec];
        if (q == 0) s_id[rec] = id;
        s_geo[staged_quad(rec, q)] = __ldg(P.geo + 4 * (size_t)id + q);
    }
}

// 16-byte asynchronous copy global -> shared (completion awaited with cp_async_wait_all by the issuing thread, then
// made visible to the CTA by a barrier).
__device__ __forceinline__ void cp_async16(float4* smem_dst, const float4* gmem_src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem_dst)),
                 "l"(gmem_src));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// The geometry of a whole list, asynchronously (see stage_list_async).
__device__ __forceinline__ void stage_geo_async(const BlendParams& P, int first, int n, float4* s_geo) {
    for (int i = threadIdx.x; i < n * 4; i += blockDim.x) {
        const int rec = i >> 2, q = i & 3;
        cp_async16(s_geo + staged_quad(rec, q), P.geo + 4 * (size_t)P.ids[first + rec] + q);
    }
    cp_async_commit();
}
// A whole list of at most one chunk, and with it the attribute quads the forward blend needs (opacities, colours, 1/w: the
// first four of the six): the blend of the selected fragments then reads its records from shared memory instead of
// gathering 128 bytes per fragment and lane through L1.  Asynchronous, started as soon as the list is known and awaited
// behind the set-up of the pixels: two load-then-store loops behind that and a barrier were up to four trips to L2 in a row
// in the life of a CTA of some ten (200k triangles, full HD: forward kernel 109 -> 99 us).  Same 80-byte pitch.
__device__ __forceinline__ void stage_list_async(const BlendParams& P, int first, int n, float4* s_geo, float4* s_attr, int* s_id) {
    for (int i = threadIdx.x; i < n * 4; i += blockDim.x) {
        const int rec = i >> 2, q = i & 3;
        const int id = P.ids[first + rec];
        if (q == 0) s_id[rec] = id;
        cp_async16(s_geo + staged_quad(rec, q), P.geo + 4 * (size_t)id + q);
        cp_async16(s_attr + staged_quad(rec, q), P.attr + kAttrQuads * (size_t)id + q);
    }
    cp_async_commit();
}
__device__ __forceinline__ AttrRec staged_attr(const float4* s_attr, int r) { return attr_from<false>(s_attr + kStagedQuads * r); }

// The walk of a CTA over its tile's list in list order, a chunk at a time: while one chunk of records is processed the next
// travels into the other half of `buf`, one barrier per chunk.  The attribute
// quads are staged with the geometry because a warp reads them record after record: fetched from L2 then, each would be a
// latency in a serial chain (20k triangles, 1001x777, forward kernel 40 -> 35 us).
struct ListPipe {
    static constexpr int kHalf = 2 * kChunk * kStagedQuads;
    float4* buf;                  // [2 * kHalf]
    __device__ __forceinline__ const float4* geo(int chunk, int r) const { return buf + (chunk & 1) * kHalf + kStagedQuads * r; }
    __device__ __forceinline__ const float4* attr(int chunk, int r) const {
        return buf + (chunk & 1) * kHalf + kChunk * kStagedQuads + kStagedQuads * r;
    }
    // chunk of n records, the first at list position `first`
    __device__ __forceinline__ void copy(const BlendParams& P, int chunk, int first, int n) const {
        float4* g = buf + (chunk & 1) * kHalf;
        float4* a = g + kChunk * kStagedQuads;
        for (int i = threadIdx.x; i < 4 * n; i += blockDim.x) {
            const int rec = i >> 2, q = i & 3;
            const int id = P.ids[first + rec];
            cp_async16(g + kStagedQuads * rec + q, P.geo + 4 * (size_t)id + q);
            cp_async16(a + kStagedQuads * rec + q, P.attr + kAttrQuads * (size_t)id + q);
        }
        cp_async_commit();
    }
};

// A staged geometry record in registers (only the parts a caller uses are actually loaded).
struct StagedGeo {
    float m[9];
    float z[3];
    float w[3];
    float zlow;
};
__device__ __forceinline__ StagedGeo load_staged(const float4* s_geo, int r) {
    const float4 a = s_geo[staged_quad(r, 0)], b = s_geo[staged_quad(r, 1)], c = s_geo[staged_quad(r, 2)],
                 d = s_geo[staged_quad(r, 3)];
    StagedGeo g;
    g.m[0] = a.x; g.m[1] = a.y; g.m[2] = a.z; g.m[3] = a.w; g.m[4] = b.x; g.m[5] = b.y; g.m[6] = b.z; g.m[7] = b.w;
    g.m[8] = c.x; g.z[0] = c.y; g.z[1] = c.z; g.z[2] = c.w; g.w[0] = d.x; g.w[1] = d.y; g.w[2] = d.z; g.zlow = d.w;
    return g;
}

__device__ __forceinline__ void load_geo_staged(const float4* s_geo, int r, float* m, float* w) {
    const StagedGeo g = load_staged(s_geo, r);
#pragma unroll
    for (int k = 0; k < 9; k++) m[k] = g.m[k];
#pragma unroll
    for (int k = 0; k < 3; k++) w[k] = g.w[k];
}

// Bit mask (64 records) of the staged records that may matter to this warp: the triangle may cover one
// of its pixels (corner test) and, when `depth_cut` is finite, its depth lower bound is below the cut
// (every lane already holds a full batch of nearer fragments otherwise).
__device__ __forceinline__ unsigned long long warp_cull(const float4* s_geo, int n, const WarpRect& R,
                                                        float depth_cut = INFINITY) {
    const int lane = lane_id();
    bool k0 = false, k1 = false;
    if (lane < n) {
        const StagedGeo g = load_staged(s_geo, lane);
        k0 = g.zlow < depth_cut && rect_may_cover(g.m, R);
    }
    if (lane + 32 < n) {
        const StagedGeo g = load_staged(s_geo, lane + 32);
        k1 = g.zlow < depth_cut && rect_may_cover(g.m, R);
    }
    const unsigned m0 = __ballot_sync(0xffffffffu, k0), m1 = __ballot_sync(0xffffffffu, k1);
    return (unsigned long long)m0 | ((unsigned long long)m1 << 32);
}

// The nearest fragments a pixel has collected in a sweep: at most `bs` words (ordered depth << 32 | list position),
// ascending.  One word per fragment, because the array lives in local memory.
struct Batch {
    uint64_t key[kBatchLayers];
    int found;
    float dfar;      // depth of the last one; -inf while the batch is empty, so the first fragment is appended
};
__device__ __forceinline__ float ordered_to_float(uint32_t u) {
    return __uint_as_float((u & 0x80000000u) ? u & 0x7fffffffu : ~u);
}

// Fragment of the covering record (list position j) into the batch, unless it does not lie behind `last`.
__device__ __forceinline__ void collect(Batch& s, int bs, uint64_t last, const Bary& b, const float4& q2, const float4& q3, int j) {
    const float d = interp_rn(b, q2.y, q2.z, q2.w, q3.x, q3.y, q3.z);
    const uint64_t key = ((uint64_t)float_to_ordered(d) << 32) | (uint32_t)j;
    if (key <= last) return;
    // the farthest kept depth stays in a register: lists come roughly front to back, so most
    // fragments go to the end of the batch (ties keep list order) or, once it is full, nowhere
    if (d >= s.dfar) {
        if (s.found == bs) return;
        s.key[s.found++] = key;
        s.dfar = d;
        return;
    }
    int pos = (s.found < bs) ? s.found : (bs - 1);
    while (pos > 0) {
        const uint64_t before = s.key[pos - 1];
        if (key >= before) break;
        s.key[pos--] = before;
    }
    s.key[pos] = key;
    if (s.found < bs) s.found++;
    s.dfar = ordered_to_float((uint32_t)(s.key[s.found - 1] >> 32));
}

// Two correctly rounded single-precision FMAs in one instruction.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("{ .reg .b64 a, b, c, d;\n\t"
        "mov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\t"
        "fma.rn.f32x2 d, a, b, c;\n\tmov.b64 {%0, %1}, d; }"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}

// Coverage of `rows` rows of the warp's 8x4 pixel block, from row `row` on, by the record whose matrix is in m: bit
// 8 * row + column, decided with the operations of apply_bary and covered().
__device__ __forceinline__ unsigned cover_rows(const float* m, const float* s_x /*[8], 16-byte aligned*/, const float* s_y,
                                               int row, int rows) {
    const float4 xa = *reinterpret_cast<const float4*>(s_x), xb = *reinterpret_cast<const float4*>(s_x + 4);
    const float2 x[4] = {{xa.x, xa.y}, {xa.z, xa.w}, {xb.x, xb.y}, {xb.z, xb.w}};
    unsigned cover = 0;
#pragma unroll 1
    for (int k = row; k < row + rows; k++) {
        const float py = s_y[k];
        const float c0 = fma_(m[1], py, m[2]), c1 = fma_(m[4], py, m[5]), c2 = fma_(m[7], py, m[8]);
        unsigned bits = 0;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float2 u = fma2({m[0], m[0]}, x[i], {c0, c0}), v = fma2({m[3], m[3]}, x[i], {c1, c1}),
                         t = fma2({m[6], m[6]}, x[i], {c2, c2});
            if (!(fminf(fminf(u.x, v.x), t.x) < kEffZero)) bits |= 1u << (2 * i);
            if (!(fminf(fminf(u.y, v.y), t.y) < kEffZero)) bits |= 2u << (2 * i);
        }
        cover |= bits << (8 * k);
    }
    return cover;
}

// 32x32 bit matrix, one row per lane, transposed: bit k of lane p becomes bit p of lane k.  The recursive exchange of
// blocks of H. S. Warren, Hacker's Delight, section 7-3, with the rows in lanes.
__device__ __forceinline__ unsigned transpose_bits(unsigned x) {
    const unsigned lane = lane_id();
    unsigned m = 0x0000ffffu;
#pragma unroll
    for (int j = 16; j > 0; j >>= 1) {
        const unsigned y = __shfl_xor_sync(0xffffffffu, x, j);
        x = (lane & j) ? ((x & ~m) | ((y & ~m) >> j)) : ((x & m) | ((y & m) << j));
        m ^= m << (j >> 1);
    }
    return x;
}

// One staged chunk of n <= 64 records: the warp's lanes with `go` collect the fragments that cover their pixels, in list
// order.  first: list position of record 0, or s_j: the records' list positions.
// The records that survive the warp's cull are tested against all 32 pixels by a lane each (two or four lanes when they
// are few), the bits are transposed, and every pixel then visits only the records that cover it: a triangle of a pixel
// or two costs a share of the warp's test instead of 20 instructions with one lane busy.  s_slot: 64 bytes per warp.
// Tiles without 8x4 blocks test one record at a time with the pixels in the lanes; so does a warp (from then on: `dense`)
// in which some pixel turned out to be covered by more than half of the records.
// Forward kernel, B200: 1.3M triangles of a pixel, full HD 272 -> 180 us; 1280 triangles 256x256 8.4 -> 6.2; 2M
// triangles, 4K 650 -> 617; 200k triangles, full HD 109 -> 110 (there a survivor covers a third of the lanes).
constexpr int kFewRecords = 3;      // up to this many survivors are tested one at a time in any case
__device__ __forceinline__ void process_chunk(const TileCtx& c, bool go, int bs, uint64_t last, Batch& s, bool& dense,
                                              const float4* geo, int n, int first, const int* s_j, uint8_t* s_slot) {
    // Once every collecting lane of the warp holds a full batch, a record whose depth lower bound is
    // not below the farthest kept depth of any lane cannot enter any lane's batch (ties lose).
    float cut = INFINITY;
    if (__all_sync(0xffffffffu, !go || s.found == bs)) {
        cut = go ? s.dfar : -INFINITY;
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) cut = fmaxf(cut, __shfl_xor_sync(0xffffffffu, cut, d));
    }
    const unsigned long long mask = warp_cull(geo, n, c.rect, cut);
    const unsigned m0 = (unsigned)mask, m1 = (unsigned)(mask >> 32);
    const int survivors = __popc(m0) + __popc(m1);
    if (c.s_x == nullptr || survivors <= kFewRecords || dense) {
        // the two 32-bit halves of the mask one after the other: bit scans on 32-bit words are cheaper
#pragma unroll 1
        for (int half = 0; half < 2; half++) {
            unsigned bits = half ? m1 : m0;
            while (bits) {
                const int r = __ffs((int)bits) - 1 + 32 * half;
                bits &= bits - 1;
                // all lanes read the same record: broadcast 16-byte loads
                const float4* rec = geo + kStagedQuads * r;
                const float4 q0 = rec[0], q1 = rec[1], q2 = rec[2];
                const float m[9] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w, q2.x};
                const Bary b = apply_bary(m, c.px, c.py);
                // one minimum instead of three comparisons: fminf skips NaN operands, so the result is below
                // kEffZero exactly when one of the three is (and NaN, i.e. "covered", when all three are NaN)
                if (!go || fminf(fminf(b.x, b.y), b.z) < kEffZero) continue;
                collect(s, bs, last, b, q2, rec[3], s_j ? s_j[r] : first + r);
            }
        }
        return;
    }
    const int lane = lane_id();
    const unsigned below = (1u << lane) - 1u;
    __syncwarp();                 // the slots of the chunk before have been read
    if ((m0 >> lane) & 1u) s_slot[__popc(m0 & below)] = (uint8_t)lane;
    if ((m1 >> lane) & 1u) s_slot[__popc(m0) + __popc(m1 & below)] = (uint8_t)(lane + 32);
    __syncwarp();
#pragma unroll 1
    for (int base = 0; base < survivors; base += 32) {
        const int count = min(32, survivors - base);
        const int shift = count <= 8 ? 2 : count <= 16 ? 1 : 0;      // log2 of the lanes per record
        const int k = lane & (31 >> shift), part = lane >> (5 - shift);
        unsigned cover = 0;
        if (k < count) {
            const float4* rec = geo + kStagedQuads * s_slot[base + k];
            const float4 q0 = rec[0], q1 = rec[1];
            const float m[9] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w, rec[2].x};
            cover = cover_rows(m, c.s_x, c.s_y, part * (4 >> shift), 4 >> shift);
        }
        __syncwarp();
        if (shift >= 1) cover |= __shfl_xor_sync(0xffffffffu, cover, 16);
        if (shift == 2) cover |= __shfl_xor_sync(0xffffffffu, cover, 8);
        unsigned mine = transpose_bits(lane < count ? cover : 0u);
        if (!go) mine = 0;
        dense = 2 * __reduce_max_sync(0xffffffffu, (unsigned)__popc(mine)) > (unsigned)count;
        while (mine) {
            const int r = s_slot[base + __ffs((int)mine) - 1];
            mine &= mine - 1;
            const float4* rec = geo + kStagedQuads * r;
            const float4 q0 = rec[0], q1 = rec[1], q2 = rec[2];
            const float m[9] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w, q2.x};
            collect(s, bs, last, apply_bary(m, c.px, c.py), q2, rec[3], s_j ? s_j[r] : first + r);
        }
        __syncwarp();
    }
}

// Shared memory of a sweep.  `staged`: the whole list is in `geo` already.
// `geo2` / `id2`, when given, are a second pair of staging buffers: a list of more than one chunk is then streamed
// (CTAs of 256 threads: one quad per thread and chunk) - the records of chunk k + 1 travel by asynchronous copies
// while chunk k is processed, their ids having been fetched one iteration earlier still, and one barrier per chunk
// replaces the two of the load-then-process loop.
constexpr int kFilterBatch = 1024;
struct SweepScratch {
    uint16_t keep[kFilterBatch];     // entries of a filtered batch, as offsets
    int j[kChunk];                   // list positions of a filtered chunk
    uint32_t count[33];              // per warp and quarter of a batch
};
struct SweepSmem {
    float4* geo;
    int* id;
    SweepScratch* scratch;     // of sweep_filtered
    uint8_t* slots;            // 64 per warp, see process_chunk
    bool staged;
    float4* geo2;
    int* id2;
};

// The rest of a tile list, from `pos` on, once every collecting pixel of the CTA holds a full batch: only entries whose
// depth lower bound is below the farthest kept depth of some pixel can still matter.  Lists are sorted by depth, so these
// are few: 1024 entries at a time the CTA reads just that word, and stages the ones that pass, 64 at a time (2M triangles
// piled up in the middle of a 4K image: most of a list of 5000 lies behind the 32 layers).
__device__ __forceinline__ void sweep_filtered(const BlendParams& P, const TileCtx& c, bool go, bool warp_go, int bs, uint64_t last,
                                            Batch& s, bool& dense, const SweepSmem& sm, int pos) {
    const int tid = threadIdx.x, warp = tid >> 5, nt = blockDim.x, warps = nt >> 5;
    const int per = nt <= 256 ? 4 : 1;          // per * warps <= 32 counts
    SweepScratch& x = *sm.scratch;
    const float* zlow = reinterpret_cast<const float*>(P.geo) + 15;
    for (; pos < c.end; pos += per * nt) {
        float cut = go ? s.dfar : -INFINITY;
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) cut = fmaxf(cut, __shfl_xor_sync(0xffffffffu, cut, d));
        __syncthreads();
        if (lane_id() == 0) x.count[warp] = __float_as_uint(cut);
        __syncthreads();
        cut = (int)lane_id() < warps ? __uint_as_float(x.count[lane_id()]) : -INFINITY;
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) cut = fmaxf(cut, __shfl_xor_sync(0xffffffffu, cut, d));
        __syncthreads();
        float z[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int j = pos + k * nt + tid;
            z[k] = (k < per && j < c.end) ? __ldg(zlow + 16 * (size_t)P.ids[j]) : INFINITY;
        }
        unsigned kept[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            kept[k] = __ballot_sync(0xffffffffu, z[k] < cut);
            if (k < per && lane_id() == 0) x.count[k * warps + warp] = (uint32_t)__popc(kept[k]);
        }
        __syncthreads();
        if (warp == 0) {
            const uint32_t mine = (int)lane_id() < per * warps ? x.count[lane_id()] : 0u;
            uint32_t incl = mine;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, incl, d);
                if ((int)lane_id() >= d) incl += y;
            }
            x.count[lane_id()] = incl - mine;
            if (lane_id() == 31) x.count[32] = incl;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (k < per && z[k] < cut)
                x.keep[x.count[k * warps + warp] + __popc(kept[k] & ((1u << lane_id()) - 1u))] = (uint16_t)(k * nt + tid);
        const int total = (int)x.count[32];
        __syncthreads();
        for (int c0 = 0; c0 < total; c0 += kChunk) {
            const int n = min(kChunk, total - c0);
            for (int i = tid; i < n * 4; i += nt) {
                const int rec = i >> 2, q = i & 3, j = pos + x.keep[c0 + rec];
                const int id = P.ids[j];
                if (q == 0) x.j[rec] = j;
                sm.geo[staged_quad(rec, q)] = __ldg(P.geo + 4 * (size_t)id + q);
            }
            __syncthreads();
            if (warp_go) process_chunk(c, go, bs, last, s, dense, sm.geo, n, 0, x.j, sm.slots + 64 * warp);
            __syncthreads();
        }
    }
}

// One selection sweep over the whole tile list (select_next_k_in_tile, reference render.cu:375-415):
// keeps the `bs` covered fragments smallest in (depth, j) among those behind `last` (a word of a batch, 0 for the first).
// All threads of the CTA must call it; `go` says whether this thread collects.
// (STREAM is a template parameter so that callers which never stream carry none of its state.)
template <bool STREAM = false, bool FILTER = true>
__device__ __forceinline__ void select_sweep(const BlendParams& P, const TileCtx& c, bool go, int bs, uint64_t last,
                                             Batch& s, const SweepSmem& sm) {
    s.found = 0;
    s.dfar = -INFINITY;
    bool dense = false;         // see process_chunk
    const bool warp_go = __any_sync(0xffffffffu, go);
    uint8_t* s_slot = sm.slots + 64 * (threadIdx.x >> 5);
    const bool streamed = STREAM && sm.geo2 != nullptr && c.end - c.start > kChunk && blockDim.x == 4 * kChunk;
    const int my_rec = threadIdx.x >> 2, my_q = threadIdx.x & 3;
    int id_ahead = -1;          // streamed: id of this thread's record in the chunk after the one being copied
    if (streamed) {
        __syncthreads();        // whoever read the buffers before (an earlier sweep) is done
        const int id = P.ids[c.start + my_rec];                       // chunk 0 is full: the list is longer
        if (my_q == 0) sm.id[my_rec] = id;
        cp_async16(sm.geo + staged_quad(my_rec, my_q), P.geo + 4 * (size_t)id + my_q);
        cp_async_commit();
        if (my_rec < c.end - c.start - kChunk) id_ahead = P.ids[c.start + kChunk + my_rec];
    }
    int chunk = 0;
    for (int first = c.start; first < c.end; first += kChunk, chunk++) {
        const int n = min(kChunk, c.end - first);
        const float4* geo_now = sm.geo;         // the staged records of this chunk
        const bool full = !go || s.found == bs;
        if (streamed) {
            float4* other_geo = sm.geo2;        // buffers the next chunk is copied into
            int* other_id = sm.id2;
            if (chunk & 1) { geo_now = sm.geo2; other_geo = sm.geo; other_id = sm.id; }
            cp_async_wait_all();
            // this chunk has landed for everyone, and everyone has left the chunk before
            if (__syncthreads_and(full) && c.end - first > kChunk) {
                sweep_filtered(P, c, go, warp_go, bs, last, s, dense, sm, first);
                break;
            }
            if (first + kChunk < c.end) {
                if (id_ahead >= 0) {
                    if (my_q == 0) other_id[my_rec] = id_ahead;
                    cp_async16(other_geo + staged_quad(my_rec, my_q), P.geo + 4 * (size_t)id_ahead + my_q);
                }
                cp_async_commit();
                const int first2 = first + 2 * kChunk;
                id_ahead = (first2 < c.end && my_rec < c.end - first2) ? P.ids[first2 + my_rec] : -1;
            }
        } else if (sm.staged) {
            geo_now = sm.geo + chunk * kChunk * kStagedQuads;
        } else {
            if (!FILTER) {
                __syncthreads();
            } else if (__syncthreads_and(full) && c.end - first > kChunk) {
                sweep_filtered(P, c, go, warp_go, bs, last, s, dense, sm, first);
                break;
            }
            stage_chunk(P, first, n, sm.geo, sm.id);
            __syncthreads();
        }
        if (warp_go) process_chunk(c, go, bs, last, s, dense, geo_now, n, first, nullptr, s_slot);
    }
}

__device__ __forceinline__ void store_pixel(const TileCtx& c, const BlendParams& P, PixelAcc& acc, float4* image,
                                            float* depthmap, float* final_w, int* ends) {
    if (!c.active) return;
    const size_t index = (size_t)c.iy * P.W + c.ix;
    float dm;
    if (acc.weight > kEffZero) dm = div(acc.depth, acc.weight);
    else { dm = INFINITY; acc.weight = 0.f; }
    depthmap[index] = dm;
    final_w[index] = acc.weight;
    ends[index] = acc.blended;
    image[index] = make_float4(acc.r, acc.g, acc.b, acc.alpha);
}

// Ascending sort of n words in memory by the CTA, with room for kSortRoom of them in shared memory: chunks of that size first, then
// merges whose steps of less than a chunk run in shared memory again.  In every comparator the smaller word goes first, so that
// words past the end, larger than any, would stay where they are and need not exist.  For the rare list that is longer than
// expected (see TG_NO_COUNT).  Every word counting the smaller ones of the whole list, in memory, took far longer: a call that meets
// lists of up to 3300 entries, 4096 triangles, B200: 160x160, tiles of 16x16 1434 -> 306 us; 64x64, tiles of 8x8 3377 -> 465 (205
// and 265 in a call that knows K and sorts and filters them as any others).  Bound by the barriers between the steps, 55 for a chunk.
constexpr int kSortRoom = 1024;
__device__ __noinline__ void sort_words(uint64_t* words, int n, uint64_t* s) {
    // pairs r and 2 half - 1 - r (first step of a merge) or r and r + half of every 2 half words
    auto step = [](uint64_t* p, int n, int half, bool mirrored) {
        const int pairs = (n + 2 * half - 1) / (2 * half) * half;
        for (int q = threadIdx.x; q < pairs; q += blockDim.x) {
            const int r = q & (half - 1), base = 2 * (q - r), low = base + r, high = mirrored ? base + 2 * half - 1 - r : low + half;
            if (high >= n) continue;
            const uint64_t a = p[low], b = p[high];
            if (a > b) {
                p[low] = b;
                p[high] = a;
            }
        }
        __syncthreads();
    };
    auto in_chunks = [&](auto steps) {
        for (int first = 0; first < n; first += kSortRoom) {
            const int m = min(kSortRoom, n - first);
            for (int i = threadIdx.x; i < m; i += blockDim.x) s[i] = words[first + i];
            __syncthreads();
            steps(m);
            for (int i = threadIdx.x; i < m; i += blockDim.x) words[first + i] = s[i];
            __syncthreads();
        }
    };
    in_chunks([&](int m) {
        for (int half = 1; half < m; half *= 2) {
            step(s, m, half, true);
            for (int h = half / 2; h >= 1; h /= 2) step(s, m, h, false);
        }
    });
    for (int half = kSortRoom; half < n; half *= 2) {
        step(words, n, half, true);
        for (int h = half / 2; h >= kSortRoom; h /= 2) step(words, n, h, false);
        in_chunks([&](int m) {
            for (int h = kSortRoom / 2; h >= 1; h /= 2) step(s, m, h, false);
        });
    }
}

// sel: optional [planes][H*W] int32; plane k of a pixel receives the triangle id of its k-th blended
// fragment (k < ends).  Only written when it is not null (per-pixel mode, max_layers <= 32).
// STREAM: lists of more than one chunk are streamed through two staging buffers (select_sweep); instantiated
// separately because the state it carries costs the one-chunk tiles a few spilled registers.
// FUSED: the lists (at most kFusedList entries) are still unsorted; the CTA sorts its own, by counting smaller words.  That
// is one launch and one trip through memory less, most of a small render's time.
// A call that does not count and whose caller reads no lists leaves out the kernel that moves them together as well: the
// binning writes every entry to its tile's list, `room` entries from the next, and this kernel takes the lengths from the
// tile counts (1280 triangles, 256x256, calls queued one behind another, 19.9 -> 16.5 us; waited for, 36.6 -> 31.9).
static_assert(kFusedList <= 2 * kChunk, "staged as a whole");
struct UnsortedLists {
    uint64_t* entries;            // ordered depth << 32 | triangle, grouped by tile; sorted in place where a list is long
    AfterBinning bin;
    int* sorted_ids;
    bool any_length;              // false: the host launches other kernels when a list is longer than kFusedList
    int room;                     // > 0: no offsets, the lists lie `room` entries apart, bin.tile_counts has their lengths
    uint32_t* long_host;          // then: mapped host memory that receives the length of a list of more than kFusedList, or null
};
template <bool SORT, int MAXT, bool STREAM = false, bool FUSED = false>
__global__ void __launch_bounds__(MAXT, MAXT <= 256 ? (SORT ? 4 : 5) : 1) blend_forward_kernel(BlendParams P, float4* __restrict__ image,
                                                             float* __restrict__ depthmap, float* __restrict__ final_w,
                                                             int* __restrict__ ends, int* __restrict__ sel,
                                                             UnsortedLists unsorted = {}) {
    __shared__ float4 s_geo[SORT ? 2 * kChunk * kStagedQuads : 2 * ListPipe::kHalf];
    float4* s_attr = s_geo + kChunk * kStagedQuads;      // lists of one chunk: attributes; of two: more geometry; longer: 2nd buffer
    __shared__ int s_id[kChunk];
    __shared__ int s_id2[STREAM ? kChunk : 1];
    constexpr bool kFilter = (STREAM || MAXT > 256) && !FUSED;
    __shared__ __align__(16) float s_coord[MAXT <= 256 ? 260 : kMaxTileCoords];      // tile_w + tile_h <= tile_w * tile_h + 1
    __shared__ SweepScratch s_scratch;
    __shared__ uint8_t s_slots[SORT ? 2 * MAXT : 1];
    __shared__ uint64_t s_key[FUSED ? kFusedList : 1];
    __shared__ int s_rank[FUSED ? kFusedList : 1];
    __shared__ int s_list[FUSED ? kFusedList : 1];
    allow_dependents();
    await_prerequisites();
    if (FUSED) {
        // launched before the host knows: nothing to do when the lists are too long or incomplete
        if (unsorted.room == 0) {
            unsorted.bin.clear((int)blockIdx.x, threadIdx.x == 0);
            const uint32_t longest = unsorted.bin.info[1] & ~kOrderWrittenBit;
            if (unsorted.bin.incomplete() || (longest > kFusedList && !unsorted.any_length)) return;
        }
    }
    const int this_tile = tile_of_block(P);
    const bool in_place = FUSED && unsorted.room > 0;
    const int list_first = in_place ? this_tile * unsorted.room : P.offsets[this_tile];
    const int list_n = in_place ? (int)__ldcg(unsorted.bin.tile_counts + this_tile) : P.offsets[this_tile + 1] - list_first;
    if (list_n == 0) {
        // a tile without entries: background, and no need for pixel-centre coordinates (any pixel order will do)
        const int tx = this_tile % P.tiles_x, ty = this_tile / P.tiles_x;
        const int ix = tx * P.tw + (int)threadIdx.x % P.tw, iy = ty * P.th + (int)threadIdx.x / P.tw;
        if ((int)threadIdx.x < P.tw * P.th && ix < P.W && iy < P.H) {
            const size_t index = (size_t)iy * P.W + ix;
            depthmap[index] = INFINITY;
            final_w[index] = 0.f;
            ends[index] = 0;
            image[index] = make_float4(0.f, 0.f, 0.f, 1.f);
        }
        return;
    }
    const bool one_chunk = SORT && list_n <= kChunk, two_chunks = SORT && !STREAM && !one_chunk && list_n <= 2 * kChunk;
    if (FUSED) {
        for (int i = threadIdx.x; i < min(list_n, (int)kFusedList); i += blockDim.x) {
            s_key[i] = unsorted.entries[list_first + i];
            s_rank[i] = 0;
        }
    } else if (!SORT) {
        ListPipe{s_geo}.copy(P, 0, list_first, min(kChunk, list_n));
    } else if (one_chunk) {
        stage_list_async(P, list_first, list_n, s_geo, s_attr, s_id);
    } else if (two_chunks) {
        stage_geo_async(P, list_first, list_n, s_geo);
    }
    TileCtx c = tile_context(P, s_coord);            // its barrier makes the words above visible
    if (FUSED) {
        c.start = list_first;
        c.end = list_first + list_n;
        if (in_place && threadIdx.x == 0) {          // everyone has the length
            unsorted.bin.tile_counts[this_tile] = 0;
            if (list_n > (int)kFusedList && unsorted.long_host) *(volatile uint32_t*)unsorted.long_host = (uint32_t)list_n;
        }
    }
    if (FUSED && list_n > (int)kFusedList) {
        uint64_t* words = unsorted.entries + c.start;
        static_assert(sizeof(s_geo) >= sizeof(uint64_t) * kSortRoom, "nothing is staged yet");
        sort_words(words, list_n, reinterpret_cast<uint64_t*>(s_geo));
        for (int i = threadIdx.x; i < list_n; i += blockDim.x) unsorted.sorted_ids[c.start + i] = (int)(uint32_t)words[i];
        P.ids = unsorted.sorted_ids;
        __syncthreads();
        if (!SORT) ListPipe{s_geo}.copy(P, 0, c.start, kChunk);
    } else if (FUSED) {
        const int n = c.end - c.start, nt = blockDim.x;
        // several threads per word where the CTA has them, each counting over a part of the list
        const int words = n <= 32 ? 32 : n <= 64 ? 64 : (int)kFusedList, parts = max(1, nt / words);
        const int step = (n + parts - 1) / parts, part = threadIdx.x / words;
        if (part < parts) {
            for (int i = threadIdx.x % words; i < n; i += (parts > 1 ? words : nt)) {
                const uint64_t mine = s_key[i];
                int below = 0;
                for (int j = part * step; j < min(n, (part + 1) * step); j++) below += s_key[j] < mine ? 1 : 0;
                if (below) atomicAdd(&s_rank[i], below);
            }
        }
        __syncthreads();
        for (int i = threadIdx.x; i < n; i += nt) {
            const int id = (int)(uint32_t)s_key[i], at = s_rank[i];
            s_list[at] = id;
            if (!in_place) unsorted.sorted_ids[c.start + at] = id;
        }
        P.ids = s_list - c.start;
        __syncthreads();
        if (!SORT) ListPipe{s_geo}.copy(P, 0, c.start, min(kChunk, n));
        else if (one_chunk) stage_list_async(P, c.start, n, s_geo, s_attr, s_id);
        else stage_geo_async(P, c.start, n, s_geo);          // kFusedList is two chunks
    }
    PixelAcc acc;

    if (SORT) {
        Batch batch;
        uint64_t last = 0;
        bool want = c.active;
        const size_t plane = (size_t)P.W * P.H, index = (size_t)c.iy * P.W + c.ix;
        while (true) {
            const bool go = want && acc.alpha > P.thr && acc.blended < P.max_layers;
            cp_async_wait_all();                       // a staged list; visible to all behind the barrier
            if (!__syncthreads_or(go)) break;
            const int bs = min(kBatchLayers, P.max_layers - acc.blended);
            select_sweep<STREAM, kFilter>(P, c, go, bs, last, batch,
                                 {s_geo, s_id, kFilter ? &s_scratch : nullptr, s_slots, one_chunk || two_chunks, one_chunk ? nullptr : s_attr, s_id2});
            const int found = batch.found;
            if (go) {
                const int n = min(found, P.max_layers - acc.blended);
                int id_ahead = STREAM && !one_chunk && n > 0 ? P.ids[(uint32_t)batch.key[0]] : 0;
                for (int i = 0; i < n; i++) {
                    if (one_chunk) {
                        const int r = (int)(uint32_t)batch.key[i] - c.start;
                        const StagedGeo g = load_staged(s_geo, r);
                        const Bary b = apply_bary(g.m, c.px, c.py);
                        const AttrRec a = staged_attr(s_attr, r);
                        if (sel) sel[(size_t)acc.blended * plane + index] = s_id[r];
                        blend_one(b, g.w, a, acc);
                        continue;
                    }
                    // Long lists: the id is fetched a fragment ahead (2M triangles piled up, 4K, kernel 586 -> 564 us; a
                    // prefetch of its records as well takes that back, and lists of two chunks lose 1 us of 102).
                    const int id = STREAM ? id_ahead : P.ids[(uint32_t)batch.key[i]];
                    float m[9], w[3];
                    load_geo(P.geo, id, m, w);
                    const Bary b = apply_bary(m, c.px, c.py);
                    const AttrRec a = load_attr<false>(P.attr, id);
                    if (STREAM && i + 1 < n) id_ahead = P.ids[(uint32_t)batch.key[i + 1]];
                    if (sel) sel[(size_t)acc.blended * plane + index] = id;
                    blend_one(b, w, a, acc);
                }
                if (n > 0) {
                    last = batch.key[n - 1];
                }
                // fewer than a full batch found: the sweep saw every remaining fragment, nothing is left
                if (found < bs) want = false;
            }
            if (P.max_layers <= kBatchLayers) break;   // a single batch is all there can be: no second vote
        }
    } else {
        bool done = !c.active;
        const ListPipe pipe = {s_geo};
        int chunk = 0;
        for (int first = c.start; first < c.end; first += kChunk, chunk++) {
            const int n = min(kChunk, c.end - first);
            cp_async_wait_all();
            if (__syncthreads_and(done)) break;
            if (first + kChunk < c.end) pipe.copy(P, chunk + 1, first + kChunk, min(kChunk, c.end - first - kChunk));
            // a warp whose lanes have all stopped skips the chunk
            if (!__all_sync(0xffffffffu, done)) {
                const unsigned long long mask = warp_cull(pipe.geo(chunk, 0), n, c.rect);
#pragma unroll 1
                for (int half = 0; half < 2; half++) {      // 32-bit bit scans, as in select_sweep
                    unsigned bits = half ? (unsigned)(mask >> 32) : (unsigned)mask;
                    while (bits) {
                        const int r = __ffs((int)bits) - 1 + 32 * half;
                        bits &= bits - 1;
                        if (done) continue;
                        if (!(acc.alpha > P.thr && acc.blended < P.max_layers)) { done = true; continue; }
                        const float* g = reinterpret_cast<const float*>(pipe.geo(chunk, r));
                        const Bary b = apply_bary(g, c.px, c.py);
                        if (!covered(b)) continue;
                        const AttrRec a = attr_from<false>(pipe.attr(chunk, r));
                        blend_one(b, g + 12, a, acc);
                    }
                }
                if (!(acc.alpha > P.thr && acc.blended < P.max_layers)) done = true;
            }
        }
    }
    store_pixel(c, P, acc, image, depthmap, final_w, ends);
}

// ------------------------------------------------------------------------------------------------
// Backward.

struct BackState { float alpha, sr = 0.f, sg = 0.f, sb = 0.f, oa = 0.f, zoa = 0.f; };

struct PixelGrad {
    float gr, gg, gb, ga, gd;          // upstream gradients of this pixel
    float final_alpha, final_weight, final_depth;
};

// Approximate reciprocal (1 ulp, one MUFU instruction): gradients carry a 1e-4 tolerance and float
// atomics already make their last bits run-dependent.
__device__ __forceinline__ float rcp_fast(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// One fragment's contribution to its triangle's three vertices: (x, y, w, opacity, r, g, b) each.
struct Contrib {
    float v[3][7];
    int vid[3];
};

// Packed per-vertex gradient accumulator: slot 0 = (d/dx, d/dy, d/dw, d/dopacity), slot 1 = (d/dr, d/dg, d/db, 0).
__device__ __forceinline__ void red_add_v4(float4* addr, float a, float b, float c, float d) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(addr), "f"(a), "f"(b), "f"(c), "f"(d));
}

__device__ __forceinline__ void emit_contrib(const Contrib& c, float4* __restrict__ gpack) {
#pragma unroll
    for (int k = 0; k < 3; k++) {
        red_add_v4(gpack + 2 * (size_t)c.vid[k], c.v[k][0], c.v[k][1], c.v[k][2], c.v[k][3]);
        red_add_v4(gpack + 2 * (size_t)c.vid[k] + 1, c.v[k][4], c.v[k][5], c.v[k][6], 0.f);
    }
}

// Sum of the contributions of the lanes with `in` (one triangle), added by 24 lanes with one instruction: a reduction by
// halves in which a lane keeps half of its 24 values and hands the other half to its partner (12 + 6 + 3 + 2 + 1
// exchanges instead of 5 x 21) and ends up with the total of one value of the triangle's three 32-byte slots.  All lanes
// of the warp must call; `leader` is one of those with `in`.
__device__ __forceinline__ void reduce_group(const Contrib& c, bool in, int leader, float4* __restrict__ gpack) {
    const int lane = lane_id();
    float v[24];
#pragma unroll
    for (int k = 0; k < 3; k++) {
#pragma unroll
        for (int q = 0; q < 7; q++) v[8 * k + q] = in ? c.v[k][q] : 0.f;
        v[8 * k + 7] = 0.f;
    }
    const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4, b1 = lane & 2, b0 = lane & 1;
#pragma unroll
    for (int i = 0; i < 12; i++) v[i] = (b4 ? v[i + 12] : v[i]) + __shfl_xor_sync(0xffffffffu, b4 ? v[i] : v[i + 12], 16);
#pragma unroll
    for (int i = 0; i < 6; i++) v[i] = (b3 ? v[i + 6] : v[i]) + __shfl_xor_sync(0xffffffffu, b3 ? v[i] : v[i + 6], 8);
#pragma unroll
    for (int i = 0; i < 3; i++) v[i] = (b2 ? v[i + 3] : v[i]) + __shfl_xor_sync(0xffffffffu, b2 ? v[i] : v[i + 3], 4);
    v[3] = 0.f;
#pragma unroll
    for (int i = 0; i < 2; i++) v[i] = (b1 ? v[i + 2] : v[i]) + __shfl_xor_sync(0xffffffffu, b1 ? v[i] : v[i + 2], 2);
    v[0] = (b0 ? v[1] : v[0]) + __shfl_xor_sync(0xffffffffu, b0 ? v[0] : v[1], 1);
    const int at = (lane >> 4) * 12 + ((lane >> 3) & 1) * 6 + ((lane >> 2) & 1) * 3 + (lane & 3);   // this lane's value
    const int v0 = __shfl_sync(0xffffffffu, c.vid[0], leader), v1 = __shfl_sync(0xffffffffu, c.vid[1], leader),
              v2 = __shfl_sync(0xffffffffu, c.vid[2], leader);
    const int vid = at < 8 ? v0 : at < 16 ? v1 : v2;
    if ((lane & 3) != 3 && (at & 7) != 7) atomicAdd(reinterpret_cast<float*>(gpack + 2 * (size_t)vid) + (at & 7), v[0]);
}

// From this many lanes on the reduction is cheaper than the lanes' own six vector reductions to the same three slots.
constexpr int kGroupMin = 6;

// Contributions of a warp whose lanes with `has` hold one and the same triangle.  All lanes must call.
__device__ __forceinline__ void emit_uniform(const Contrib& c, bool has, float4* __restrict__ gpack) {
    const unsigned group = __ballot_sync(0xffffffffu, has);
    if (__popc(group) >= kGroupMin) reduce_group(c, has, __ffs(group) - 1, gpack);
    else if (has) emit_contrib(c, gpack);
    __syncwarp();
}

// The same for lanes with triangles of their own (`id`): pixels next to each other under large triangles mostly blend the
// same triangle at the same place of their sequences.  All lanes must call.
__device__ __forceinline__ void emit_groups(const Contrib& c, bool has, int id, float4* __restrict__ gpack) {
    const unsigned peers = __match_any_sync(0xffffffffu, has ? id : -1 - (int)lane_id());
    const bool big = has && __popc(peers) >= kGroupMin;
    unsigned todo = __ballot_sync(0xffffffffu, big);
#pragma unroll 1
    for (int it = 0; it < 32 / kGroupMin && todo != 0; ++it) {
        const int leader = __ffs(todo) - 1;
        const unsigned group = __shfl_sync(0xffffffffu, peers, leader);
        todo &= ~group;
        reduce_group(c, (group >> lane_id()) & 1u, leader, gpack);
    }
    if (has && !big) emit_contrib(c, gpack);
    __syncwarp();
}

struct BackwardIn {
    const float4* gimage;
    const float* gdepth;
    const float4* image;
    const float* depthmap;
    const float* final_w;
    const int* ends;
    // fused mean-squared-error loss: when l2_target is set, the upstream gradient of the image is
    // l2_grad_scale * (image - target), the depth-map gradient is zero and the squared differences are
    // summed into l2_sums (add_loss; no gradient image is ever materialised)
    const float4* l2_target;
    float l2_grad_scale;
    float* l2_sums;
    // the same target as 8-bit RGBA (value / 255, correctly rounded division: what `u8.float() / 255` gives);
    // at most one of l2_target / l2_target_u8 is set
    const uchar4* l2_target_u8;
};

// DEPTH = false: no gradient flows into the depth map, so neither it nor the final weight is read.
template <bool DEPTH = true>
__device__ __forceinline__ int load_pixel_state(const TileCtx& c, const BlendParams& P, const BackwardIn& in,
                                                PixelGrad& pg, BackState& st, float* sq_diff = nullptr) {
    pg = PixelGrad{};
    st.alpha = 1.f;
    if (sq_diff) *sq_diff = 0.f;
    if (!c.active) return 0;
    const size_t index = (size_t)c.iy * P.W + c.ix;
    const float4 img = in.image[index];
    if (in.l2_target || in.l2_target_u8) {
        float4 t;
        if (in.l2_target_u8) {
            const uchar4 u = in.l2_target_u8[index];
            t = make_float4(__fdiv_rn((float)u.x, 255.f), __fdiv_rn((float)u.y, 255.f), __fdiv_rn((float)u.z, 255.f),
                            __fdiv_rn((float)u.w, 255.f));
        } else {
            t = in.l2_target[index];
        }
        const float dr = img.x - t.x, dg = img.y - t.y, db = img.z - t.z, da = img.w - t.w;
        pg.gr = in.l2_grad_scale * dr; pg.gg = in.l2_grad_scale * dg; pg.gb = in.l2_grad_scale * db;
        pg.ga = in.l2_grad_scale * da;
        pg.gd = 0.f;
        if (sq_diff) *sq_diff = dr * dr + dg * dg + db * db + da * da;
    } else {
        const float4 gi = in.gimage[index];
        pg.gr = gi.x; pg.gg = gi.y; pg.gb = gi.z; pg.ga = gi.w;
        pg.gd = DEPTH && in.gdepth ? in.gdepth[index] : 0.f;      // no depth-map gradient given: zero
    }
    pg.final_alpha = img.w;
    if (DEPTH) {
        pg.final_weight = in.final_w[index];
        pg.final_depth = in.depthmap[index];
    }
    st.alpha = pg.final_alpha;
    return min(in.ends[index], P.max_layers);
}

// ---- default mode, two-part gradient with a per-warp queue ------------------------------------------
// The pixels of a warp blend different numbers of fragments (on average fewer than half the lanes have
// one in a given round), and only the transmittance recurrence ties a pixel's fragments together.  So
// the work is split: part A (per pixel, back to front) runs the recurrence and produces the upstream
// gradients of the fragment's interpolations; these go into a queue in shared memory; part B (the
// expensive barycentric partials and the 21 per-vertex outputs) pops 32 queued fragments at a time and
// so runs with full warps.  A warp whose lanes are busy anyway (deep overlap, or one opaque layer everywhere) skips the
// queue.  (200k triangles, full HD: 146 us with L1 75 % busy and 63 % of the issue slots used; bound by the latency of the
// gathers, fourteen of 16 bytes per fragment, and by L1 together, which does shared memory's work too.)
// DEPTH = false (everywhere below): no gradient flows into the depth map, the terms that it feeds are left out.
struct QueuedFragment {
    float px, py;
    int id;
    float bx, by, bz;
    float o_raw, cr, cg, cb, z;
    float uo, ur, ug, ub, uz;
};
// A warp's queue: slots of 4 quads, rotated so that a quad of consecutive slots lies on different banks.  Up to kLeft fragments stay
// behind when a round ends; the slots above hold that round's, and, once these are in registers, the table of emit_lanes.  Every
// kilobyte of the seven or eight CTAs is L1 taken from the gathers: with kLeft = 26 and columns of 34 words eight CTAs take 163 KB
// and the SM is split at 164; with 31 slots and columns of 36, which are read four words at a time, it is split at 196, and fine
// meshes lose (kernel, 200k triangles 1920x1080 / 1.3M triangles of a pixel 1920x1080 / 2M piled up 3840x2160: 146 / 108 / 722
// us against 149 / 118 / 802; with 23 slots and 36 words, whose rounds end less full, 148 / 110 / 732).  Seven CTAs have room for both.
constexpr int kQueuePitch = 4;
template <bool DEPTH>
struct QueueShape {
    static constexpr int kLeft = DEPTH ? 31 : 26, kColumn = DEPTH ? 36 : 34;
    static constexpr int kTable = 24 * kColumn / 4;                       // quads
    static constexpr int kQuads = kLeft * kQueuePitch + (kTable > 32 * kQueuePitch ? kTable : 32 * kQueuePitch);
};

template <bool DEPTH>
__device__ __forceinline__ void queue_push(float4* q, int slot, const QueuedFragment& f) {
    q += kQueuePitch * slot;
    const int x = (slot >> 1) & 3;
    q[x] = make_float4(f.px, f.py, __int_as_float(f.id), f.bx);
    q[1 ^ x] = make_float4(f.by, f.bz, f.o_raw, f.cr);
    q[2 ^ x] = make_float4(f.cg, f.cb, f.uo, f.ur);
    if (DEPTH) q[3 ^ x] = make_float4(f.ug, f.ub, f.z, f.uz);
    else *reinterpret_cast<float2*>(q + (3 ^ x)) = make_float2(f.ug, f.ub);
}
template <bool DEPTH>
__device__ __forceinline__ QueuedFragment queue_pop(const float4* q, int slot) {
    QueuedFragment f;
    q += kQueuePitch * slot;
    const int x = (slot >> 1) & 3;
    const float4 a = q[x], b = q[1 ^ x], c = q[2 ^ x];
    f.px = a.x; f.py = a.y; f.id = __float_as_int(a.z); f.bx = a.w;
    f.by = b.x; f.bz = b.y; f.o_raw = b.z; f.cr = b.w;
    f.cg = c.x; f.cb = c.y; f.uo = c.z; f.ur = c.w;
    if (DEPTH) {
        const float4 d = q[3 ^ x];
        f.ug = d.x; f.ub = d.y; f.z = d.z; f.uz = d.w;
    } else {
        const float2 d = *reinterpret_cast<const float2*>(q + (3 ^ x));
        f.ug = d.x; f.ub = d.y; f.z = 0.f; f.uz = 0.f;
    }
    return f;
}

// Part A, second half: the transmittance recurrence of render.cu:455-538 for one fragment (back to
// front) and the upstream gradients of its interpolations.  inv_den / inv_denz are the reciprocals of
// the interpolation denominators, or 0 where the reference's guard returns zero gradients.
template <bool DEPTH>
__device__ __forceinline__ void backward_recurrence(float o_raw, float cr, float cg, float cb, float z, float inv_den,
                                                    float inv_denz, const PixelGrad& pg, BackState& st,
                                                    QueuedFragment& f) {
    const float o = fminf(fmaxf(o_raw, 0.f), kMaxOpacity);
    const float iom = rcp_fast(1.f - o);
    const float drgb_do = ((cr * st.alpha - st.sr) * pg.gr + (cg * st.alpha - st.sg) * pg.gg + (cb * st.alpha - st.sb) * pg.gb -
                           pg.ga * pg.final_alpha) * iom;
    st.alpha = st.alpha * iom;
    const float ao = st.alpha * o;
    st.sr += cr * ao;
    st.sg += cg * ao;
    st.sb += cb * ao;
    float d_do = drgb_do, uz = 0.f;
    if (DEPTH) {
        const float ddw_do = st.alpha - st.oa * iom;
        const float dud_do = st.alpha * z - st.zoa * iom;
        st.oa += ao;
        st.zoa += z * ao;
        const bool has_w = !(pg.final_weight < kEffZero);
        const float inv_fw = has_w ? rcp_fast(pg.final_weight) : 0.f;
        const float dd_do = (dud_do - pg.final_depth * ddw_do) * inv_fw * pg.gd;
        d_do = drgb_do + (has_w ? dd_do : 0.f);
        uz = has_w ? ao * pg.gd * inv_fw * inv_denz : 0.f;
    }
    f.o_raw = o_raw; f.cr = cr; f.cg = cg; f.cb = cb; f.z = z;
    f.uo = d_do * inv_den;
    f.ur = ao * pg.gr * inv_den;
    f.ug = ao * pg.gg * inv_den;
    f.ub = ao * pg.gb * inv_den;
    f.uz = uz;
}

// Part A: interpolations of the fragment (approximate reciprocals), then the recurrence.
template <bool DEPTH>
__device__ __forceinline__ void backward_state(const float* w, const AttrRec& a, const Bary& b, const PixelGrad& pg,
                                               BackState& st, QueuedFragment& f) {
    const float bw0 = b.x * w[0], bw1 = b.y * w[1], bw2 = b.z * w[2];
    const float den = bw0 + bw1 + bw2;
    const bool ok = !(den * den < kEffZero);
    const float inv = rcp_fast(den);
    const float o_raw = (bw0 * a.o[0] + bw1 * a.o[1] + bw2 * a.o[2]) * inv;
    const float cr = (bw0 * a.c[0] + bw1 * a.c[3] + bw2 * a.c[6]) * inv;
    const float cg = (bw0 * a.c[1] + bw1 * a.c[4] + bw2 * a.c[7]) * inv;
    const float cb = (bw0 * a.c[2] + bw1 * a.c[5] + bw2 * a.c[8]) * inv;
    float z = 0.f, inv_denz = 0.f;
    if (DEPTH) {
        const float denz = b.x + b.y + b.z;
        const bool okz = !(denz * denz < kEffZero);
        const float invz = rcp_fast(denz);
        z = (b.x * a.iw[0] + b.y * a.iw[1] + b.z * a.iw[2]) * invz;
        inv_denz = okz ? invz : 0.f;
    }
    f.bx = b.x; f.by = b.y; f.bz = b.z;
    backward_recurrence<DEPTH>(o_raw, cr, cg, cb, z, ok ? inv : 0.f, inv_denz, pg, st, f);
}

// Part B: from the upstream gradients to the contribution for the triangle's three vertices: process_backward of the
// reference (render.cu:455-538).  The interpolation VJPs (util.h:299-355) share 1/den; vertex-position gradients follow
// the reference's expanded partial derivatives (util.h:405-455) term by term: for small triangles their fp32
// cancellation is systematic and part of what "the same result" means.  EXPANDED = false, for gradients that are not meant to
// be the reference's: as p = l.(a, b, c), the eighteen terms are l_k times an edge, -c.y - l.y (b.y - c.y) + p.y = l.x (a.y - c.y)
// and so on, which is shorter and loses nothing to cancellation (3000 triangles about 90 layers deep, kernel 311 -> 306 us; distance to 64
// bits there 9.8e-7 -> 9.7e-7).
template <bool DEPTH, bool EXPANDED = true>
__device__ __forceinline__ void backward_outputs(const float* w, const AttrRec& a, const QueuedFragment& f, Contrib& out) {
    const float uo = f.uo, ur = f.ur, ug = f.ug, ub = f.ub;
    // e_k = sum over attributes of upstream * (a_k - value): d/d(b_k w_k) of the interpolated values
    const float e0 = uo * (a.o[0] - f.o_raw) + ur * (a.c[0] - f.cr) + ug * (a.c[1] - f.cg) + ub * (a.c[2] - f.cb);
    const float e1 = uo * (a.o[1] - f.o_raw) + ur * (a.c[3] - f.cr) + ug * (a.c[4] - f.cg) + ub * (a.c[5] - f.cb);
    const float e2 = uo * (a.o[2] - f.o_raw) + ur * (a.c[6] - f.cr) + ug * (a.c[7] - f.cg) + ub * (a.c[8] - f.cb);
    float g0 = w[0] * e0, g1 = w[1] * e1, g2 = w[2] * e2;                        // d/d bary
    float gw0 = f.bx * e0, gw1 = f.by * e1, gw2 = f.bz * e2;                     // d/dw
    if (DEPTH) {
        // depth interpolation (values 1/w, unit weights); d/dw as the reference does it (render.cu:530): also the gradient
        // w.r.t. the unit weights, plus the chain through the values 1/w
        const float uz = f.uz, iw0 = a.iw[0], iw1 = a.iw[1], iw2 = a.iw[2];
        const float z0 = uz * (iw0 - f.z), z1 = uz * (iw1 - f.z), z2 = uz * (iw2 - f.z);
        g0 += z0; g1 += z1; g2 += z2;
        gw0 = gw0 + f.bx * z0 - uz * f.bx * iw0 * iw0;
        gw1 = gw1 + f.by * z1 - uz * f.by * iw1 * iw1;
        gw2 = gw2 + f.bz * z2 - uz * f.bz * iw2 * iw2;
    }
    // barycentric_backward: l by cross products, then the expanded partials
    const float px = f.px, py = f.py;
    const float ax = a.xy[0], ay = a.xy[1], bx = a.xy[2], by = a.xy[3], cx = a.xy[4], cy = a.xy[5];
    float gxy[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    const float d = ax * (by - cy) + bx * (-ay + cy) + cx * (ay - by);
    if (!(fabsf(d) < kEffZero)) {
        const float iT = rcp_fast((bx - ax) * (cy - ay) - (by - ay) * (cx - ax));
        const float lx = ((bx - px) * (cy - py) - (by - py) * (cx - px)) * iT;
        const float ly = ((cx - px) * (ay - py) - (cy - py) * (ax - px)) * iT;
        const float lz = ((ax - px) * (by - py) - (ay - py) * (bx - px)) * iT;
        const float id = rcp_fast(d);
        if (!EXPANDED) {
            const float gx = (g0 * (cy - by) + g1 * (ay - cy) + g2 * (by - ay)) * id, gy = (g0 * (bx - cx) + g1 * (cx - ax) + g2 * (ax - bx)) * id;
            gxy[0] = lx * gx; gxy[1] = lx * gy;
            gxy[2] = ly * gx; gxy[3] = ly * gy;
            gxy[4] = lz * gx; gxy[5] = lz * gy;
        } else {
            gxy[0] = (g0 * (lx * (-by + cy)) + g1 * (-cy - ly * (by - cy) + py) + g2 * (by - lz * (by - cy) - py)) * id;
            gxy[1] = (g0 * (lx * (bx - cx)) + g1 * (cx + ly * (bx - cx) - px) + g2 * (-bx + lz * (bx - cx) + px)) * id;
            gxy[2] = (g0 * (cy + lx * (ay - cy) - py) + g1 * (ly * (ay - cy)) + g2 * (-ay + lz * (ay - cy) + py)) * id;
            gxy[3] = (g0 * (-cx - lx * (ax - cx) + px) + g1 * (ly * (-ax + cx)) + g2 * (ax - lz * (ax - cx) - px)) * id;
            gxy[4] = (g0 * (-by - lx * (ay - by) + py) + g1 * (ay - ly * (ay - by) - py) + g2 * (lz * (-ay + by))) * id;
            gxy[5] = (g0 * (bx + lx * (ax - bx) - px) + g1 * (-ax + ly * (ax - bx) + px) + g2 * (lz * (ax - bx))) * id;
        }
    }
    const float gw[3] = {gw0, gw1, gw2}, bwk[3] = {f.bx * w[0], f.by * w[1], f.bz * w[2]};
#pragma unroll
    for (int k = 0; k < 3; k++) {
        out.vid[k] = a.vid[k];
        out.v[k][0] = gxy[2 * k];
        out.v[k][1] = gxy[2 * k + 1];
        out.v[k][2] = gw[k];
        out.v[k][3] = uo * bwk[k];
        out.v[k][4] = ur * bwk[k];
        out.v[k][5] = ug * bwk[k];
        out.v[k][6] = ub * bwk[k];
    }
}

// Both parts for one fragment of one pixel.
template <bool DEPTH = true>
__device__ __forceinline__ void backward_one(const float* w, const AttrRec& a, const Bary& b, float px, float py,
                                             const PixelGrad& pg, BackState& st, Contrib& out) {
    QueuedFragment f;
    f.px = px; f.py = py; f.id = 0;
    backward_state<DEPTH>(w, a, b, pg, st, f);
    backward_outputs<DEPTH>(w, a, f, out);
}

// Contributions of a warp's lanes (triangles `id`) with as few atomics as their triangles allow.  All lanes must call.
// The lanes' outputs go to a table in shared memory, one column of 32 words per value, the lanes ordered by triangle; 24 lanes add the
// columns up and send each triangle's three 32-byte slots with one instruction.  The vertex ids ride in the unused eighth value
// of every slot.  Columns and not rows: a store then has the lanes in one column, 32 banks whatever their order, where rows, two
// times sixteen of them as there was less room, took 72 passes through shared memory instead of 24 and were most of what the
// kernel asked of L1, which it waits for where many triangles overlap (200k triangles, 1920x1080 154 -> 146 us; 1.3M
// triangles of a pixel, the same image 111 -> 106; 2M piled up, 3840x2160 807 -> 706; the three vertices' ids on one or two
// banks instead of three 146, 108, 715).
// (Adding up to four neighbouring lanes with 42 shuffles and six vector reductions per run took as long as rows where a triangle
// has one or two of the 32 fragments, and 17 % longer where a few triangles have them all: 2M overlapping triangles, 4K,
// 944 us against 804.  Sums of four values per lane, for five triangles at a time, which leave as vector reductions: 185 against
// 154 and 981 against 807 - reductions of 16 bytes to one 32-byte slot are not merged.)
// `rows`: 24 * COLUMN words of this warp.  COLUMN: 36, or 34, which is read two words at a time.  WHOLE: where all lanes have
// one and the same triangle the columns are read at once.
template <int COLUMN, bool WHOLE = false>
__device__ __forceinline__ void emit_lanes(const Contrib& c, bool valid, int id, float4* rows, float4* __restrict__ gpack) {
    const int lane = lane_id();
    const unsigned peers = __match_any_sync(0xffffffffu, valid ? id : -1 - lane);      // distinct negatives never match
    const unsigned below = (1u << lane) - 1u;
    const bool leads = valid && (peers & below) == 0;
    const int size = leads ? __popc(peers) : 0;
    int incl = size;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += y;
    }
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    const int place = __shfl_sync(0xffffffffu, incl - size, __ffs(peers) - 1) + __popc(peers & below);
    const unsigned ends = __reduce_or_sync(0xffffffffu, leads ? 1u << (incl - 1) : 0u);   // last row of every triangle
    float* table = reinterpret_cast<float*>(rows);
    const float* column = table + COLUMN * min(lane, 23);
    const int* ids = reinterpret_cast<const int*>(table) + COLUMN * (min(lane, 23) | 7) + (min(lane, 23) >> 3);    // on three banks
    const bool adds = lane < 24 && (lane & 7) != 7;
    static_assert(!WHOLE || COLUMN % 4 == 0, "read four words at a time");
    if (valid) {
        float* at = table + place;
#pragma unroll
        for (int k = 0; k < 3; k++) {
#pragma unroll
            for (int i = 0; i < 7; i++) at[COLUMN * (8 * k + i)] = c.v[k][i];
            at[COLUMN * (8 * k + 7) + k] = __int_as_float(c.vid[k]);
        }
    }
    __syncwarp();
    if (WHOLE && ends == 0x80000000u) {
        float4 even = make_float4(0.f, 0.f, 0.f, 0.f), odd = even;
#pragma unroll
        for (int j = 0; j < 32; j += 8) {
            const float4 q = *reinterpret_cast<const float4*>(column + j), r = *reinterpret_cast<const float4*>(column + j + 4);
            even.x += q.x; even.y += q.y; even.z += q.z; even.w += q.w;
            odd.x += r.x; odd.y += r.y; odd.z += r.z; odd.w += r.w;
        }
        if (adds) atomicAdd(reinterpret_cast<float*>(gpack + 2 * (size_t)ids[31]) + (lane & 7),
                            ((even.x + odd.x) + (even.y + odd.y)) + ((even.z + odd.z) + (even.w + odd.w)));
        __syncwarp();
        return;
    }
    float sum = 0.f;
#pragma unroll 1
    for (int j = 0; j < total; j += 4) {
        float x[4];                       // rows past `total` end no triangle
        if (COLUMN % 4 == 0) {
            const float4 q = *reinterpret_cast<const float4*>(column + j);
            x[0] = q.x; x[1] = q.y; x[2] = q.z; x[3] = q.w;
        } else {
            const float2 q = *reinterpret_cast<const float2*>(column + j), r = *reinterpret_cast<const float2*>(column + j + 2);
            x[0] = q.x; x[1] = q.y; x[2] = r.x; x[3] = r.y;
        }
#pragma unroll
        for (int k = 0; k < 4; k++) {
            sum += x[k];
            if ((ends >> (j + k)) & 1u) {
                const int vid = ids[j + k];
                if (adds) atomicAdd(reinterpret_cast<float*>(gpack + 2 * (size_t)vid) + (lane & 7), sum);
                sum = 0.f;
            }
        }
    }
    __syncwarp();
}

// Part B for the fragments in queue slots first .. first + count - 1 (count <= 32, first <= kLeft), one per lane.  The slots from
// `first` on are free once the fragments are in registers.
template <bool DEPTH>
__device__ __forceinline__ void drain_queue(const BlendParams& P, float4* q, int first, int count, float4* __restrict__ gpack) {
    const int lane = lane_id();
    const bool valid = lane < count;
    const QueuedFragment f = queue_pop<DEPTH>(q, first + (valid ? lane : 0));
    Contrib ct = {};
    if (valid) {
        const float4 g3 = __ldg(P.geo + 4 * (size_t)f.id + 3);
        const float w[3] = {g3.x, g3.y, g3.z};
        const AttrRec a = load_attr<true>(P.attr, f.id);
        backward_outputs<DEPTH>(w, a, f, ct);
    }
    __syncwarp();
    emit_lanes<QueueShape<DEPTH>::kColumn>(ct, valid, f.id, q + kQueuePitch * first, gpack);
}

// Whole fragments per round, for warps whose lanes are busy anyway.  Kept out of line so that it does not weigh on the
// register allocation of the queued path.
template <bool DEPTH>
__device__ __noinline__ void backward_rounds_direct(const BlendParams& P, float px, float py, PixelGrad pg, BackState st,
                                                    int n, int nmax, int id_next, const int* __restrict__ sel_pixel,
                                                    size_t plane, float4* rows, float4* __restrict__ gpack) {
    for (int s = 0; s < nmax; s++) {
        const int k = n - 1 - s;
        const bool has = k >= 0;
        const int id = id_next;
        if (k > 0) id_next = sel_pixel[(size_t)(k - 1) * plane];
        Contrib ct = {};
        if (has) {
            float m[9], w[3];
            load_geo(P.geo, id, m, w);
            const AttrRec a = load_attr<true>(P.attr, id);
            const Bary b = apply_bary(m, px, py);
            backward_one<DEPTH>(w, a, b, px, py, pg, st, ct);
        }
        emit_lanes<QueueShape<DEPTH>::kColumn>(ct, has, id, rows, gpack);
    }
}

// A CTA takes a block of kQueueCols x kQueueRows pixels, a warp 8x4 of them, and then PASSES - 1 blocks more, each the same
// number of rows further down; the queues go on through all of them.  What a warp does for 32 pixels of a layer or two is
// short against the start of a CTA and ends in a queue that is not full; against that, the last CTAs end later.  One and three
// passes, a fused step, B200, kernel as a trace has it: 200k triangles, 1920x1080 159, 146 us; 1.3M triangles of a pixel, the same
// image 107, 106; 2M piled up, 3840x2160 708, 699.  (With sums by rows instead of columns, one, two, three, four, six passes took 164,
// 154, 153, 154, 158; 111, 111, 116, 119, 136; 786, 814, 798, 799, 824, so three was the number.)  So three, and by
// the size of the image (backward_impl).  (Blocks next to each other: 3840x2160 850 with two, as the deep blocks all lie in
// the same CTAs and the last of them run alone.  In a loop of a number of passes known at run time the compiler spills.)
constexpr int kQueueCols = 16, kQueueRows = 8;

template <int PASSES, bool DEPTH>
__global__ void __launch_bounds__(kQueueCols * kQueueRows, DEPTH ? 7 : 8) blend_backward_queued_kernel(BlendParams P, BackwardIn in,
                                                                        const int* __restrict__ sel,
                                                                        float4* __restrict__ gpack) {
    constexpr int kWarps = kQueueCols * kQueueRows / 32;
    __shared__ __align__(16) float s_coord[kQueueCols + PASSES * kQueueRows];
    __shared__ float4 s_queue[kWarps][QueueShape<DEPTH>::kQuads];
    allow_dependents();
    const int lane = lane_id(), warp = threadIdx.x >> 5;
    const int x0 = ((int)blockIdx.x % P.tiles_x) * kQueueCols, y0 = ((int)blockIdx.x / P.tiles_x) * kQueueRows;
    const int apart = ((P.H + kQueueRows - 1) / kQueueRows + PASSES - 1) / PASSES * kQueueRows;      // rows between passes
    if ((int)threadIdx.x < kQueueCols) s_coord[threadIdx.x] = pixel_coord(x0 + threadIdx.x, P.W);
    else if ((int)threadIdx.x < kQueueCols + PASSES * kQueueRows) {
        const int r = (int)threadIdx.x - kQueueCols;
        s_coord[threadIdx.x] = pixel_coord(y0 + (r / kQueueRows) * apart + r % kQueueRows, P.H);
    }
    const int lx = 8 * (warp & 1) + (lane & 7);
    TileCtx c;
    c.ix = x0 + lx;
    const size_t plane = (size_t)P.W * P.H;
    float4* q = s_queue[warp];
    int queued = 0;                                    // uniform over the warp
    float sq_sum = 0.f;
    __syncthreads();
    c.px = s_coord[lx];
    await_prerequisites();
#pragma unroll 1
    for (int pass = 0; pass < PASSES; pass++) {
        const int ly = pass * kQueueRows + 4 * (warp >> 1) + (lane >> 3);
        c.iy = y0 + pass * apart + ly - pass * kQueueRows;
        c.active = c.ix < P.W && c.iy < P.H;
        c.py = s_coord[kQueueCols + ly];
        PixelGrad pg;
        BackState st;
        float sq = 0.f;
        const int n = load_pixel_state<DEPTH>(c, P, in, pg, st, &sq);
        sq_sum += sq;
        const size_t index = (size_t)c.iy * P.W + c.ix;
        int id_next = (n > 0) ? sel[(size_t)(n - 1) * plane + index] : 0;   // ids are fetched one fragment ahead
        const int nmax = __reduce_max_sync(0xffffffffu, n), nsum = __reduce_add_sync(0xffffffffu, n);
        if (nsum * 10 >= nmax * 32 * 9) {
            // Nearly all lanes have a fragment in every round (90 % or more): the queue would cost more than the idle
            // lanes do.
            backward_rounds_direct<DEPTH>(P, c.px, c.py, pg, st, n, nmax, id_next, sel + index, plane, q + kQueuePitch * queued, gpack);
            continue;
        }
        for (int s = 0; s < nmax; s++) {
            const int k = n - 1 - s;
            const bool has = k >= 0;
            const int id = id_next;
            if (k > 0) id_next = sel[(size_t)(k - 1) * plane + index];
            const unsigned pushing = __ballot_sync(0xffffffffu, has);
            if (has) {
                float m[9], w[3];
                load_geo(P.geo, id, m, w);
                const AttrRec a = load_attr<false>(P.attr, id);
                if (k > 0) prefetch_record(P, id_next);
                const Bary b = apply_bary(m, c.px, c.py);
                QueuedFragment f;
                f.px = c.px; f.py = c.py; f.id = id;
                backward_state<DEPTH>(w, a, b, pg, st, f);
                queue_push<DEPTH>(q, queued + __popc(pushing & ((1u << lane) - 1u)), f);
            }
            queued += __popc(pushing);
            __syncwarp();
            if (queued > QueueShape<DEPTH>::kLeft) {
                const int count = min(queued, 32);
                queued -= count;
                drain_queue<DEPTH>(P, q, queued, count, gpack);
                __syncwarp();
            }
        }
    }
    if (queued > 0) drain_queue<DEPTH>(P, q, 0, queued, gpack);
    if (in.l2_target || in.l2_target_u8) {
        // loss: warp sum, then one atomic per warp
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) sq_sum += __shfl_xor_sync(0xffffffffu, sq_sum, d);
        if (lane == 0 && sq_sum != 0.f) add_loss(in.l2_sums, blockIdx.x * kWarps + warp, sq_sum);
    }
}

// ---- one optimisation step of one view in a single kernel -------------------------------------------
// Forward compositing (default mode, max_layers <= 32: a single batch) followed, in the same thread, by
// the backward of mean((image - target)^2).  The values the forward interpolates for every blended
// fragment (opacity, colour, 1/w, barycentrics) are kept in local memory and feed the recurrence
// directly: no second pass over geometry and attributes for it, no selection planes, no re-read of the
// image; the per-vertex outputs go through the per-warp queue as in blend_backward_queued_kernel.
// Slower than the two kernels in most places by now, as it has none of their staging ahead of the pixel set-up, streamed
// lists and dependent launches, and its half for the forward runs with the registers of both (a step, B200: 200k triangles,
// full HD 300 us in two kernels against 335 in one; 2M triangles, 4K 1914 against 2165; 10k, 512x512 54 against 59; four
// streams of views, full HD 250 against 278 per view).  Nearly as fast where triangles are a pixel each and a pixel blends one
// fragment or none (1.3M triangles, full HD 502 against 508).  Used on request only.
template <int MAXT>
__global__ void __launch_bounds__(MAXT, 4) blend_step_l2_kernel(BlendParams P, float4* __restrict__ image,
                                                                float* __restrict__ depthmap, float* __restrict__ final_w,
                                                                int* __restrict__ ends, const float4* __restrict__ target,
                                                                float grad_scale, float* __restrict__ l2_sums,
                                                                float4* __restrict__ gpack) {
    static_assert(MAXT == 256, "the per-warp queues are sized for 8 warps");
    __shared__ float4 s_geo[kChunk * kStagedQuads];
    __shared__ int s_id[kChunk];
    __shared__ __align__(16) float s_coord[260];       // four CTAs take 195 KB, the SM is split at 196 (at 228: 2M triangles, 4K, a step 2242 -> 2423 us)
    __shared__ SweepScratch s_scratch;
    __shared__ uint8_t s_slots[2 * MAXT];
    extern __shared__ float4 s_step[];       // queues of the warps
    const TileCtx c = tile_context(P, s_coord);
    const int lane = lane_id();
    PixelAcc acc;
    float4 kept[kBatchLayers][3];   // per blended fragment: (b.x, b.y, b.z, o_raw), (cr, cg, cb, z), (1/den, 1/denz, id, -)
    int n = 0;
    {
        Batch batch;
        const bool go = c.active && acc.alpha > P.thr && P.max_layers > 0;
        if (__syncthreads_or(go)) {
            const int bs = min(kBatchLayers, P.max_layers);
            select_sweep(P, c, go, bs, 0, batch, {s_geo, s_id, &s_scratch, s_slots, false, nullptr, nullptr});
            if (go) {
                n = min(batch.found, P.max_layers);
                for (int i = 0; i < n; i++) {
                    const int id = P.ids[(uint32_t)batch.key[i]];
                    float m[9], w[3];
                    load_geo(P.geo, id, m, w);
                    const Bary b = apply_bary(m, c.px, c.py);
                    const AttrRec a = load_attr<false>(P.attr, id);
                    const BlendedValues v = blend_one(b, w, a, acc);
                    const float denz = b.x + b.y + b.z;
                    kept[i][0] = make_float4(b.x, b.y, b.z, v.o_raw);
                    kept[i][1] = make_float4(v.cr, v.cg, v.cb, v.z);
                    kept[i][2] = make_float4((v.den * v.den < kEffZero) ? 0.f : rcp_fast(v.den),
                                             (denz * denz < kEffZero) ? 0.f : rcp_fast(denz), __int_as_float(id), 0.f);
                }
            }
        }
    }
    const float final_alpha = acc.alpha, out_r = acc.r, out_g = acc.g, out_b = acc.b;
    store_pixel(c, P, acc, image, depthmap, final_w, ends);   // normalises acc.weight to 0 where no depth exists

    // upstream gradient of the image and the pixel's squared error
    PixelGrad pg = PixelGrad{};
    BackState st;
    st.alpha = final_alpha;
    float sq = 0.f;
    if (c.active) {
        const float4 t = target[(size_t)c.iy * P.W + c.ix];
        const float dr = out_r - t.x, dg = out_g - t.y, db = out_b - t.z, da = final_alpha - t.w;
        pg.gr = grad_scale * dr; pg.gg = grad_scale * dg; pg.gb = grad_scale * db; pg.ga = grad_scale * da;
        pg.gd = 0.f;
        pg.final_alpha = final_alpha;
        pg.final_weight = acc.weight;
        pg.final_depth = (acc.weight > kEffZero) ? div(acc.depth, acc.weight) : INFINITY;
        sq = dr * dr + dg * dg + db * db + da * da;
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, d);
    if (lane == 0 && sq != 0.f) add_loss(l2_sums, blockIdx.x * 8 + (threadIdx.x >> 5), sq);

    float4* q = s_step + QueueShape<false>::kQuads * (threadIdx.x >> 5);
    const int nmax = __reduce_max_sync(0xffffffffu, n);
    int queued = 0;                                    // uniform over the warp
    for (int s = 0; s < nmax; s++) {
        const int k = n - 1 - s;
        const bool has = k >= 0;
        const unsigned pushing = __ballot_sync(0xffffffffu, has);
        if (has) {
            const float4 k0 = kept[k][0], k1 = kept[k][1], k2 = kept[k][2];
            QueuedFragment f;
            f.px = c.px; f.py = c.py; f.id = __float_as_int(k2.z);
            f.bx = k0.x; f.by = k0.y; f.bz = k0.z;
            backward_recurrence<false>(k0.w, k1.x, k1.y, k1.z, k1.w, k2.x, k2.y, pg, st, f);
            queue_push<false>(q, queued + __popc(pushing & ((1u << lane) - 1u)), f);
        }
        queued += __popc(pushing);
        __syncwarp();
        if (queued > QueueShape<false>::kLeft) {
            const int count = min(queued, 32);
            queued -= count;
            drain_queue<false>(P, q, queued, count, gpack);
            __syncwarp();
        }
    }
    if (queued > 0) drain_queue<false>(P, q, 0, queued, gpack);
}

// General path (any max_layers, both modes): searches the list again as the reference does.
// Per-pixel mode, batch after batch sweeping the list: lists of up to kListRecords records are staged once for all sweeps, and for
// the gradients of the fragments found.  A warp's outputs leave as in the queued kernel, through a table of columns: its lanes
// hold a handful of triangles each round, and a reduction by halves for each (100 instructions, a lane's own six vector reductions
// where few lanes share one) took longer.  B200, corrected gradients, kernel: 3000 triangles about 90 layers deep, 637x421,
// tiles of 16 306 -> 266 us, of 32 367 -> 299, of 8 346 -> 288; 300 triangles, 480x360 102 -> 90; the reference's gradients 321 -> 267,
// 354 -> 285, 358 -> 287, 105 -> 92.  (Before the columns of a round with one triangle in all lanes were read at once, the table
// took 270, 314, 292, 94, 270, 304, 290, 95; 700 large triangles, 1280x720, 333, now 316, the reductions by halves 327.)  Bound
// by issue, 24 warps on an SM.  Where a pixel has a layer or two the table is the dearer one, corrected gradients above all: 200k
// triangles, 1920x1080, 199 -> 205 (the reference's 207 -> 205), 2000, the same image, 75 -> 79 (84 -> 79), in tiles of 32 124 -> 128
// (110 -> 113).  Not cured: both ways in one kernel, chosen by the number of rounds, take 290 for the 270, with the shorter one out
// of line all take longer; the groups of 6 or 8 lanes and more through the table instead of 12, 214 and 211 for the 205.
// 128 records in tiles of up to 256 pixels, 256 in larger ones.  With 256 in tiles of 8 the shared memory of small CTAs costs more
// than it gives, 291 -> 369; in tiles of 16, with a list of 33 records on average 93 -> 94, 71 231 -> 235, 142 270 -> 272, 192
// 279 -> 276, 239 285 -> 278, 287 293 -> 283.
// FEW: at most eight warps on an SM, where a round's latency counts and not its instructions: the lanes' own reductions, all the
// registers a thread wants and 256 records.  4000 triangles, 160x160 (100 tiles of 16) 99 -> 80 us, with the reductions alone
// 85; 3000, 96x96 90 -> 62; 400, 200x150 (130 tiles) 55 -> 51, in tiles of 8 (475 of two warps) 58 -> 43; 1500, 96x96 in tiles of 4
// 74 -> 50.  With more warps the table is ahead or much as fast: 400, 304x200 (247 tiles, two to an SM, whose registers are for one
// of FEW) 57 against 60, 200x200 in tiles of 8 (625, five) 60 against 61, the reference's gradients 58 against 56; and ahead
// with tiles of more than 256 pixels, whose CTA has more warps by itself (1500, 160x160 in tiles of 32 177 against 203).
constexpr int kFewWarps = 8;
template <bool SORT, int MAXT, bool FEW>
constexpr int kListRecords = !SORT ? kChunk : MAXT <= 256 && !FEW ? 2 * kChunk : 4 * kChunk;
constexpr int kListColumn = 36, kListTable = 24 * kListColumn / 4;      // quads per warp
constexpr size_t list_tables(int threads) { return sizeof(float4) * kListTable * (threads / 32); }
// A round's contributions.  From 12 lanes on the table is cheaper than the lanes' own vector reductions, below it a little dearer
// (100k small triangles in one or two layers 122 -> 114 us, deep stacks 1 % slower; 16 and 20 lanes: 300 triangles 95 -> 107, 119).
constexpr int kTableMin = 12;
template <bool FEW>
__device__ __forceinline__ void emit_round(const Contrib& c, bool has, int id, float4* rows, float4* __restrict__ gpack) {
    if (FEW) emit_groups(c, has, id, gpack);
    else if (__popc(__ballot_sync(0xffffffffu, has)) >= kTableMin) emit_lanes<kListColumn, true>(c, has, id, rows, gpack);
    else if (has) emit_contrib(c, gpack);
}
template <bool SORT, int MAXT, bool FEW = false>
__global__ void __launch_bounds__(MAXT, MAXT <= 256 && !FEW ? (SORT ? 3 : 4) : 1) blend_backward_kernel(BlendParams P, BackwardIn in, float4* __restrict__ gpack) {
    __shared__ float4 s_geo[kListRecords<SORT, MAXT, FEW> * kStagedQuads];
    __shared__ int s_id[kChunk];
    extern __shared__ float4 s_tables[];             // SORT and not FEW: kListTable quads per warp
    __shared__ __align__(16) float s_coord[MAXT <= 256 ? 260 : kMaxTileCoords];
    const TileCtx c = tile_context(P, s_coord);
    const bool resident = SORT && c.end - c.start <= kListRecords<SORT, MAXT, FEW>;
    if (resident) stage_geo_async(P, c.start, c.end - c.start, s_geo);
    PixelGrad pg;
    BackState st;
    allow_dependents();
    const int limit = load_pixel_state(c, P, in, pg, st);

    if (SORT) {
        __shared__ SweepScratch s_scratch;
        __shared__ uint8_t s_slots[2 * MAXT];
        Batch batch;
        uint64_t last = 0;
        int remaining = limit;
        while (true) {
            const bool go = remaining > 0;
            cp_async_wait_all();
            if (!__syncthreads_or(go)) break;
            const int bs = min(kBatchLayers, remaining);
            select_sweep(P, c, go, bs, last, batch, {s_geo, s_id, &s_scratch, s_slots, resident, nullptr, nullptr});
            const int n = go ? min(batch.found, remaining) : 0;
            const int rounds = __reduce_max_sync(0xffffffffu, n);
            // back to front inside the batch (reference render.cu:684-688); the first of the rounds starts at every lane's
            // last fragment
            int ahead = n > 0 ? (int)(uint32_t)batch.key[n - 1] : 0, id_ahead = n > 0 ? P.ids[ahead] : 0;
            for (int s = 0; s < rounds; ++s) {
                const int i = n - 1 - s;
                int id = -1;
                Contrib ct = {};
                if (i >= 0) {
                    const int j = ahead;
                    id = id_ahead;
                    if (i > 0) {
                        ahead = (int)(uint32_t)batch.key[i - 1];
                        id_ahead = P.ids[ahead];
                    }
                    float m[9], w[3];
                    if (resident) load_geo_staged(s_geo, j - c.start, m, w);
                    else load_geo(P.geo, id, m, w);
                    const Bary b = apply_bary(m, c.px, c.py);
                    const AttrRec a = load_attr<true>(P.attr, id);
                    backward_one(w, a, b, c.px, c.py, pg, st, ct);
                }
                emit_round<FEW>(ct, i >= 0, id, s_tables + kListTable * (threadIdx.x >> 5), gpack);
            }
            if (go) {
                if (n > 0) {
                    last = batch.key[n - 1];
                    remaining -= n;
                } else {
                    remaining = 0;
                }
            }
        }
    } else {
        // reference render.cu:659-666: the first `limit` list entries, front to back
        __shared__ int s_lim;
        if (threadIdx.x == 0) s_lim = 0;
        __syncthreads();
        if (limit > 0) atomicMax(&s_lim, limit);
        __syncthreads();
        const int cta_lim = min(s_lim, c.end - c.start);
        for (int first = 0; first < cta_lim; first += kChunk) {
            const int n = min(kChunk, cta_lim - first);
            __syncthreads();
            stage_chunk(P, c.start + first, n, s_geo, s_id);
            __syncthreads();
            if (!__any_sync(0xffffffffu, first < limit)) continue;
            unsigned long long mask = warp_cull(s_geo, n, c.rect);
            while (mask) {
                const int r = __ffsll((long long)mask) - 1;
                mask &= mask - 1;
                const float* g = reinterpret_cast<const float*>(s_geo + kStagedQuads * r);
                const Bary b = apply_bary(g, c.px, c.py);
                const bool has = first + r < limit && covered(b);
                Contrib ct = {};
                if (has) {
                    const AttrRec a = load_attr<true>(P.attr, s_id[r]);
                    backward_one(g + 12, a, b, c.px, c.py, pg, st, ct);
                }
                emit_uniform(ct, has, gpack);
            }
        }
    }
}

// ---- corrected gradients outside the default mode (an extension, not reference behaviour) -----------
// The reference's recurrences (render.cu:478-497) are written for a walk over a pixel's blended fragments from
// the last one to the first.  Its kernel does that only in the default mode: with per_pixel_sort = false it
// visits the first `ends` list entries front to back (render.cu:659-666), and beyond 32 layers it reverses the
// order inside each batch of 32 only (render.cu:673-693).  This kernel computes the gradient of what the forward
// pass actually blended, for any mode and any number of layers, without storing the sequence: it walks the
// fragments in FORWARD order and obtains the sums over the fragments behind the current one - the only thing
// the back-to-front walk is needed for - as (final value - running prefix), the final values being the forward
// outputs (image, final weight, depth map * final weight).
struct PrefixState { float alpha = 1.f, sr = 0.f, sg = 0.f, sb = 0.f, oa = 0.f, zoa = 0.f; };
struct PixelFinals { float r, g, b, depth_sum; };

__device__ __forceinline__ void backward_one_prefix(const float* w, const AttrRec& a, const Bary& b, float px, float py,
                                                    const PixelGrad& pg, const PixelFinals& fin, PrefixState& pf,
                                                    Contrib& out) {
    const float bw0 = b.x * w[0], bw1 = b.y * w[1], bw2 = b.z * w[2];
    const float den = bw0 + bw1 + bw2;
    const bool ok = !(den * den < kEffZero);
    const float inv = rcp_fast(den);
    QueuedFragment f;
    f.px = px; f.py = py; f.id = 0;
    f.bx = b.x; f.by = b.y; f.bz = b.z;
    f.o_raw = (bw0 * a.o[0] + bw1 * a.o[1] + bw2 * a.o[2]) * inv;
    f.cr = (bw0 * a.c[0] + bw1 * a.c[3] + bw2 * a.c[6]) * inv;
    f.cg = (bw0 * a.c[1] + bw1 * a.c[4] + bw2 * a.c[7]) * inv;
    f.cb = (bw0 * a.c[2] + bw1 * a.c[5] + bw2 * a.c[8]) * inv;
    const float denz = b.x + b.y + b.z;
    const bool okz = !(denz * denz < kEffZero);
    const float invz = rcp_fast(denz);
    f.z = (b.x * a.iw[0] + b.y * a.iw[1] + b.z * a.iw[2]) * invz;
    const float o = fminf(fmaxf(f.o_raw, 0.f), kMaxOpacity);
    const float iom = rcp_fast(1.f - o);
    const float alpha = pf.alpha;              // transmittance in front of this fragment
    const float ao = alpha * o;
    pf.sr += f.cr * ao; pf.sg += f.cg * ao; pf.sb += f.cb * ao;
    pf.oa += ao;
    pf.zoa += f.z * ao;
    pf.alpha = alpha * (1.f - o);
    // sums over the fragments behind this one
    const float sr = fin.r - pf.sr, sg = fin.g - pf.sg, sb = fin.b - pf.sb;
    const float oa = pg.final_weight - pf.oa, zoa = fin.depth_sum - pf.zoa;
    const float drgb_do = (f.cr * alpha - sr * iom) * pg.gr + (f.cg * alpha - sg * iom) * pg.gg +
                          (f.cb * alpha - sb * iom) * pg.gb - pg.ga * pg.final_alpha * iom;
    const float ddw_do = alpha - oa * iom;
    const float dud_do = alpha * f.z - zoa * iom;
    const bool has_w = !(pg.final_weight < kEffZero);
    const float inv_fw = has_w ? rcp_fast(pg.final_weight) : 0.f;
    const float d_do = drgb_do + (has_w ? (dud_do - pg.final_depth * ddw_do) * inv_fw * pg.gd : 0.f);
    const float inv_den = ok ? inv : 0.f;
    f.uo = d_do * inv_den;
    f.ur = ao * pg.gr * inv_den;
    f.ug = ao * pg.gg * inv_den;
    f.ub = ao * pg.gb * inv_den;
    f.uz = (has_w && okz) ? ao * pg.gd * inv_fw * invz : 0.f;
    backward_outputs<true, false>(w, a, f, out);
}

template <bool SORT, int MAXT, bool FEW = false>
__global__ void __launch_bounds__(MAXT, MAXT <= 256 && !FEW ? (SORT ? 3 : 4) : 1) blend_backward_corrected_kernel(BlendParams P, BackwardIn in,
                                                                        float4* __restrict__ gpack) {
    __shared__ float4 s_geo[kListRecords<SORT, MAXT, FEW> * kStagedQuads];
    __shared__ int s_id[kChunk];
    extern __shared__ float4 s_tables[];             // SORT and not FEW: kListTable quads per warp
    __shared__ __align__(16) float s_coord[MAXT <= 256 ? 260 : kMaxTileCoords];
    const TileCtx c = tile_context(P, s_coord);
    const bool resident = SORT && c.end - c.start <= kListRecords<SORT, MAXT, FEW>;
    if (resident) stage_geo_async(P, c.start, c.end - c.start, s_geo);
    PixelGrad pg;
    BackState unused;
    const int limit = load_pixel_state(c, P, in, pg, unused);
    PixelFinals fin = {0.f, 0.f, 0.f, 0.f};
    if (c.active) {
        const float4 img = in.image[(size_t)c.iy * P.W + c.ix];
        fin.r = img.x; fin.g = img.y; fin.b = img.z;
        fin.depth_sum = (pg.final_weight < kEffZero) ? 0.f : pg.final_depth * pg.final_weight;
    }
    PrefixState pf;

    if (SORT) {
        __shared__ SweepScratch s_scratch;
        __shared__ uint8_t s_slots[2 * MAXT];
        Batch batch;
        uint64_t last = 0;
        int remaining = limit;
        while (true) {
            const bool go = remaining > 0;
            cp_async_wait_all();
            if (!__syncthreads_or(go)) break;
            const int bs = min(kBatchLayers, remaining);
            select_sweep(P, c, go, bs, last, batch, {s_geo, s_id, &s_scratch, s_slots, resident, nullptr, nullptr});
            const int n = go ? min(batch.found, remaining) : 0;
            const int rounds = __reduce_max_sync(0xffffffffu, n);
            int ahead = n > 0 ? (int)(uint32_t)batch.key[0] : 0, id_ahead = n > 0 ? P.ids[ahead] : 0;
            for (int i = 0; i < rounds; ++i) {
                int id = -1;
                Contrib ct = {};
                if (i < n) {
                    const int j = ahead;
                    id = id_ahead;
                    if (i + 1 < n) {
                        ahead = (int)(uint32_t)batch.key[i + 1];
                        id_ahead = P.ids[ahead];
                    }
                    float m[9], w[3];
                    if (resident) load_geo_staged(s_geo, j - c.start, m, w);
                    else load_geo(P.geo, id, m, w);
                    const Bary b = apply_bary(m, c.px, c.py);
                    const AttrRec a = load_attr<true>(P.attr, id);
                    backward_one_prefix(w, a, b, c.px, c.py, pg, fin, pf, ct);
                }
                emit_round<FEW>(ct, i < n, id, s_tables + kListTable * (threadIdx.x >> 5), gpack);
            }
            if (go) {
                if (n > 0) {
                    last = batch.key[n - 1];
                    remaining -= n;
                } else {
                    remaining = 0;
                }
            }
        }
    } else {
        // the forward's walk (render.cu:578-581): list order, covered entries only, until `limit` are done
        int processed = 0;
        bool done = limit <= 0;
        for (int first = c.start; first < c.end; first += kChunk) {
            const int n = min(kChunk, c.end - first);
            __syncthreads();
            stage_chunk(P, first, n, s_geo, s_id);
            __syncthreads();
            if (!__all_sync(0xffffffffu, done)) {
                unsigned long long mask = warp_cull(s_geo, n, c.rect);
                while (mask) {
                    const int r = __ffsll((long long)mask) - 1;
                    mask &= mask - 1;
                    const float* g = reinterpret_cast<const float*>(s_geo + kStagedQuads * r);
                    const Bary b = apply_bary(g, c.px, c.py);
                    const bool has = !done && covered(b);
                    Contrib ct = {};
                    if (has) {
                        const AttrRec a = load_attr<true>(P.attr, s_id[r]);
                        backward_one_prefix(g + 12, a, b, c.px, c.py, pg, fin, pf, ct);
                        if (++processed >= limit) done = true;
                    }
                    emit_uniform(ct, has, gpack);
                }
            }
            if (__syncthreads_and(done)) break;
        }
    }
}

// One vertex of the packed accumulator; with `clear` its words are zeroed behind the read.  False: all zero.
__device__ __forceinline__ bool take_vertex(float4* gpack, int v, bool clear, float4& a, float4& b) {
    a = gpack[2 * (size_t)v];
    b = gpack[2 * (size_t)v + 1];
    const bool any = a.x != 0.f || a.y != 0.f || a.z != 0.f || a.w != 0.f || b.x != 0.f || b.y != 0.f || b.z != 0.f;
    if (clear && any) {
        gpack[2 * (size_t)v] = make_float4(0.f, 0.f, 0.f, 0.f);
        gpack[2 * (size_t)v + 1] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    return any;
}
__device__ __forceinline__ void unpack_loss(float* sums, float scale, float* loss_out, bool accumulate, bool clear) {
    if (blockIdx.x != 0 || threadIdx.x >= 32 || (!loss_out && !clear)) return;
    const float x = take_loss(sums, clear);
    if (threadIdx.x == 0 && loss_out) *loss_out = (accumulate ? *loss_out : 0.f) + x * scale;
}

// Packed accumulator -> the three gradient tensors of the reference (render.cu:789-791).  Bound by DRAM: 32 bytes read per
// vertex, and 32 written or, adding to the tensors, touched only for vertices that received something.
__global__ void __launch_bounds__(256) unpack_gradients_kernel(float4* __restrict__ gpack, int V, float4* __restrict__ gV,
                                                               float* __restrict__ gC, float* __restrict__ gO, int accumulate,
                                                               int clear, float* __restrict__ l2_sums,
                                                               float l2_loss_scale, float* __restrict__ l2_loss_out) {
    allow_dependents();
    await_prerequisites();
    unpack_loss(l2_sums, l2_loss_scale, l2_loss_out, accumulate != 0, clear != 0);
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= V) return;
    float4 a, b;
    if (!take_vertex(gpack, v, clear != 0, a, b) && accumulate) return;
    float4 ov = make_float4(a.x, a.y, 0.f, a.z);
    float c0 = b.x, c1 = b.y, c2 = b.z, o = a.w;
    if (accumulate) {
        const float4 old = gV[v];
        ov.x += old.x; ov.y += old.y; ov.z = old.z; ov.w += old.w;
        c0 += gC[3 * (size_t)v]; c1 += gC[3 * (size_t)v + 1]; c2 += gC[3 * (size_t)v + 2];
        o += gO[v];
    }
    gV[v] = ov;
    gC[3 * (size_t)v] = c0; gC[3 * (size_t)v + 1] = c1; gC[3 * (size_t)v + 2] = c2;
    gO[v] = o;
}

// The same for the packed input layout: colour and opacity gradients as one [V,4] array (dr, dg, db, dopacity).
__global__ void __launch_bounds__(256) unpack_gradients_rgba_kernel(float4* __restrict__ gpack, int V, float4* __restrict__ gV,
                                                                    float4* __restrict__ gRGBA, int accumulate, int clear,
                                                                    float* __restrict__ l2_sums, float l2_loss_scale,
                                                                    float* __restrict__ l2_loss_out) {
    allow_dependents();
    await_prerequisites();
    unpack_loss(l2_sums, l2_loss_scale, l2_loss_out, accumulate != 0, clear != 0);
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= V) return;
    float4 a, b;
    if (!take_vertex(gpack, v, clear != 0, a, b) && accumulate) return;
    float4 ov = make_float4(a.x, a.y, 0.f, a.z), oc = make_float4(b.x, b.y, b.z, a.w);
    if (accumulate) {
        const float4 pv = gV[v], pc = gRGBA[v];
        ov.x += pv.x; ov.y += pv.y; ov.z = pv.z; ov.w += pv.w;
        oc.x += pc.x; oc.y += pc.y; oc.z += pc.z; oc.w += pc.w;
    }
    gV[v] = ov;
    gRGBA[v] = oc;
}

}  // namespace tg

extern "C" {

static int blend_args(int W, int H, int tw, int th, int max_layers) {
    if (int s = tg_host::check_sizes(W, H, tw, th)) return s;
    TG_REQUIRE(max_layers >= 1, "max_layers must be >= 1");
    return TG_OK;
}

static tg::BlendParams make_params(const float* tri_geo, const float* tri_attr, const int32_t* sorted_ids,
                                   const int32_t* offsets, int W, int H, int tw, int th, float thr, int max_layers) {
    tg::BlendParams P;
    P.geo = (const float4*)tri_geo; P.attr = (const float4*)tri_attr; P.ids = sorted_ids; P.offsets = offsets;
    P.W = W; P.H = H; P.tw = tw; P.th = th; P.tiles_x = (W + tw - 1) / tw;
    P.thr = thr; P.max_layers = max_layers;
    P.order = nullptr;
    return P;
}

int tg_selection_planes(int per_pixel_sort, int max_layers) {
    return (per_pixel_sort && max_layers >= 1 && max_layers <= tg::kBatchLayers) ? max_layers : 0;
}

}  // extern "C"

namespace tg_host {
// Set by tg_render_forward / tg_render_step_l2 around their compositing call (same thread): the tile order the
// binning kernel left in the workspace.  The stage entry points run with the identity order.
static thread_local const uint32_t* g_tile_order = nullptr;
static thread_local uint32_t g_longest_list = 0;
void set_tile_order(const uint32_t* order, uint32_t longest_list) {
    g_tile_order = order;
    g_longest_list = longest_list;
}

int blend_forward_short(const float* tri_geo, const float* tri_attr, const BinBuffers& b, uint32_t capacity, bool any_length,
                        int room, uint32_t* long_host, int32_t* sorted_ids, const int32_t* offsets, int W, int H, int tw, int th, float thr,
                        int per_pixel_sort, int max_layers, float* image, float* depthmap, float* final_weights,
                        int32_t* ends, int32_t* selection, cudaStream_t s) {
    TG_REQUIRE(((uintptr_t)image & 15) == 0, "image must be 16-byte aligned");
    if (tg_selection_planes(per_pixel_sort, max_layers) == 0) selection = nullptr;
    const tg::BlendParams P = make_params(tri_geo, tri_attr, nullptr, room > 0 ? nullptr : offsets, W, H, tw, th, thr, max_layers);
    const int tiles = P.tiles_x * ((H + th - 1) / th);
    const tg::UnsortedLists lists = {b.entries, after_binning(&b, tiles, capacity), sorted_ids, any_length, room, long_host};
    const int threads = ((tw * th + 31) / 32) * 32;
    auto kernel = threads <= 256 ? (per_pixel_sort ? tg::blend_forward_kernel<true, 256, false, true>
                                                   : tg::blend_forward_kernel<false, 256, false, true>)
                                 : (per_pixel_sort ? tg::blend_forward_kernel<true, 1024, false, true>
                                                   : tg::blend_forward_kernel<false, 1024, false, true>);
    static SmemAllowed preferred;                 // L1 for the batches, as in tg_blend_forward
    if (per_pixel_sort && threads <= 256)
        if (int st = prefer_smem((const void*)kernel, 100, preferred)) return st;
    TG_CUDA(launch_dependent(kernel, tiles, threads, 0, s, P, (float4*)image, depthmap, final_weights, ends, selection, lists));
    TG_LAUNCH_CHECK("blend_forward_kernel (short lists)");
    return TG_OK;
}
}  // namespace tg_host

extern "C" {

int tg_blend_forward(const float* tri_geo, const float* tri_attr, const int32_t* sorted_ids, const int32_t* offsets,
                     int W, int H, int tw, int th, float thr, int per_pixel_sort, int max_layers, float* image,
                     float* depthmap, float* final_weights, int32_t* ends, int32_t* selection, tg_stream_t stream) {
    if (int s = blend_args(W, H, tw, th, max_layers)) return s;
    TG_REQUIRE(offsets && image && depthmap && final_weights && ends, "null pointer");
    TG_REQUIRE(((uintptr_t)image & 15) == 0 && ((uintptr_t)tri_geo & 15) == 0 && ((uintptr_t)tri_attr & 15) == 0,
               "image / tri_geo / tri_attr must be 16-byte aligned");
    if (tg_selection_planes(per_pixel_sort, max_layers) == 0) selection = nullptr;
    tg::BlendParams P = make_params(tri_geo, tri_attr, sorted_ids, offsets, W, H, tw, th, thr, max_layers);
    P.order = tg_host::g_tile_order;
    const int tiles = P.tiles_x * ((H + th - 1) / th);
    const int threads = ((tw * th + 31) / 32) * 32;
    cudaStream_t s = (cudaStream_t)stream;
    float4* img = (float4*)image;
    // Lists well beyond one staged chunk (the binning kernel of the same call reported the longest): stream them, and filter
    // them by depth once the batches are full.  Streaming moves a chunk with one quad per thread, which takes 256 threads.
    // The filter alone in smaller CTAs gains where almost all of a list lies behind the batches and loses elsewhere, with
    // its barriers over the few records that a small tile's chunk leaves to each warp (forward, 8x8 tiles: 2M triangles
    // piled up, 4K 1612 -> 1468 us, but 200k piled up, full HD 585 -> 700, 300k spread, 1001x777 748 -> 1124, 20k, 512x512,
    // lists of 375 205 -> 258; 4x4 tiles, 400k, full HD 4115 -> 6640); CTAs of more than 256 threads have it always.
    const bool stream_lists = threads == 256 && tg_host::g_longest_list > 2u * tg::kChunk;
    auto kernel = threads > 256 ? (per_pixel_sort ? tg::blend_forward_kernel<true, 1024> : tg::blend_forward_kernel<false, 1024>)
                  : !per_pixel_sort ? tg::blend_forward_kernel<false, 256>
                  : stream_lists ? tg::blend_forward_kernel<true, 256, true> : tg::blend_forward_kernel<true, 256>;
    // The batches live in local memory: what the CTAs leave of shared memory is L1 for them (2M triangles, 4K, a step:
    // 2112 -> 2083 us with 64 KB and CTAs that fit it; 196 KB for shared memory: 2404).
    static tg_host::SmemAllowed preferred[2];
    if (per_pixel_sort && threads <= 256)
        if (int st = tg_host::prefer_smem((const void*)kernel, 64, preferred[stream_lists])) return st;
    // Launched ahead of the end of the sort (200k triangles, full HD: a view 152 -> 146 us together with the sort's own early
    // launch), but only behind the kernel for short lists: CTAs that come to an SM while a sort kernel with much shared
    // memory is still there run with what L1 that leaves, and as the SM is never empty, to the end (2M triangles, 4K: 611 ->
    // 917 us; lists of up to 1024 entries, 400k triangles, full HD: 486 -> 537).
    TG_CUDA(tg_host::launch_early(tg_host::g_longest_list <= (uint32_t)tg::kTileSortRank, kernel, tiles, threads, 0, s, P, img, depthmap, final_weights, ends,
                                      per_pixel_sort ? selection : nullptr, tg::UnsortedLists{}));
    TG_LAUNCH_CHECK("blend_forward_kernel");
    return TG_OK;
}

size_t tg_backward_scratch_bytes(int V) { return (size_t)(V > 0 ? V : 0) * 32 + tg::kLossBytes; }

}  // extern "C"
// The kernels that walk the tile lists: the reference's backward or the corrected one.
template <bool CORRECTED>
static int launch_list_kernel(const tg::BlendParams& P, const tg::BackwardIn& in, float4* gpack, int tiles, int threads, bool sort, cudaStream_t s) {
    const bool large = threads > 256;
    const bool few = sort && !large && (tiles + 147) / 148 * (threads / 32) <= tg::kFewWarps;
    void (*kernel)(tg::BlendParams, tg::BackwardIn, float4*);
    if (CORRECTED)
        kernel = large ? (sort ? tg::blend_backward_corrected_kernel<true, 1024> : tg::blend_backward_corrected_kernel<false, 1024>)
                 : few ? tg::blend_backward_corrected_kernel<true, 256, true>
                       : (sort ? tg::blend_backward_corrected_kernel<true, 256> : tg::blend_backward_corrected_kernel<false, 256>);
    else
        kernel = large ? (sort ? tg::blend_backward_kernel<true, 1024> : tg::blend_backward_kernel<false, 1024>)
                 : few ? tg::blend_backward_kernel<true, 256, true>
                       : (sort ? tg::blend_backward_kernel<true, 256> : tg::blend_backward_kernel<false, 256>);
    const bool tables = sort && !few;
    static tg_host::SmemAllowed allowed[2];
    if (tables)
        if (int st = tg_host::allow_smem((const void*)kernel, tg::list_tables(large ? 1024 : 256), allowed[large])) return st;
    kernel<<<tiles, threads, tables ? tg::list_tables(threads) : 0, s>>>(P, in, gpack);
    return TG_OK;
}
extern "C" {

static int backward_impl(const float* tri_geo, const float* tri_attr, const int32_t* sorted_ids, const int32_t* offsets,
                         int V, int W, int H, int tw, int th, int per_pixel_sort, int max_layers,
                         const float* grad_image, const float* grad_depthmap, const void* l2_target, bool target_u8,
                         float l2_grad_scale,
                         float l2_loss_scale, float* l2_loss_out, const float* image, const float* depthmap,
                         const float* final_weights, const int32_t* ends, const int32_t* selection, float* grad_vertices,
                         float* grad_colors, float* grad_opacities, int accumulate, void* scratch, size_t scratch_bytes,
                         tg_stream_t stream) {
    if (int s = blend_args(W, H, tw, th, max_layers)) return s;
    TG_REQUIRE(V >= 0, "V < 0");
    TG_REQUIRE(offsets && image && depthmap && final_weights && ends, "null pointer");
    TG_REQUIRE(l2_target || grad_image, "null upstream gradient");
    if (V == 0) return TG_OK;
    const bool packed = accumulate == TG_ACCUMULATE_PACKED;   // gradients stay in the scratch, which keeps accumulating
    TG_REQUIRE(scratch && (packed || (grad_vertices && grad_colors && grad_opacities)), "null gradient / scratch pointer");
    TG_REQUIRE(((uintptr_t)image & 15) == 0 && ((uintptr_t)grad_image & 15) == 0 &&
                   ((uintptr_t)l2_target & (target_u8 ? 3 : 15)) == 0 &&
                   ((uintptr_t)tri_geo & 15) == 0 && ((uintptr_t)tri_attr & 15) == 0 &&
                   ((uintptr_t)grad_vertices & 15) == 0 && ((uintptr_t)scratch & 15) == 0,
               "image / grad_image / target / tri_geo / tri_attr / grad_vertices / scratch must be 16-byte aligned");
    if (scratch_bytes < tg_backward_scratch_bytes(V)) {
        tg_host::set_error("backward scratch: need %zu bytes, got %zu", tg_backward_scratch_bytes(V), scratch_bytes);
        return TG_ERR_WORKSPACE;
    }
    const bool saved = selection != nullptr && tg_selection_planes(per_pixel_sort, max_layers) > 0;
    TG_REQUIRE(!l2_target || saved, "the fused L2 backward needs the selection saved by the forward pass (default mode)");
    cudaStream_t s = (cudaStream_t)stream;
    float4* gpack = (float4*)scratch;
    float* loss_sums = (float*)((char*)scratch + (size_t)V * 32);
    if (!packed) TG_CUDA(cudaMemsetAsync(gpack, 0, (size_t)V * 32 + tg::kLossBytes, s));
    const tg::BlendParams P = make_params(tri_geo, tri_attr, sorted_ids, offsets, W, H, tw, th, 0.f, max_layers);
    const int tiles = P.tiles_x * ((H + th - 1) / th);
    const int threads = ((tw * th + 31) / 32) * 32;
    const tg::BackwardIn in = {(const float4*)grad_image, grad_depthmap, (const float4*)image, depthmap, final_weights,
                               ends, target_u8 ? nullptr : (const float4*)l2_target, l2_grad_scale, loss_sums,
                               target_u8 ? (const uchar4*)l2_target : nullptr};
    if (saved) {
        // The queued kernel walks the per-pixel selection, not the tile lists, so its blocks need not be the
        // forward's tiles: 16x8 pixels (four warps) finish more evenly than whole tiles do, and a block's
        // registers come free only when its slowest warp is done (200k triangles, full HD, when it was made: 179 -> 173
        // us; 64 threads the same, 32 threads slower again).
        tg::BlendParams Q = P;
        Q.tiles_x = (W + tg::kQueueCols - 1) / tg::kQueueCols;
        Q.offsets = nullptr; Q.ids = nullptr; Q.order = nullptr;
        // Three passes from the numbers of waves on that were measured to pay, B200, whole calls, one pass -> three, us.
        // No depth gradient, 8 CTAs per SM (fused steps; the same renders through autograd are alike): 2.0 waves (1280x720) 1.3M
        // triangles of a pixel 489 -> 494, 89k random triangles 156 -> 158, 100k piled up in the middle 362 -> 415; 3.2 (1600x900)
        // 502 -> 504, 225 -> 218, 364 -> 390; 3.8 (1760x990) 486 -> 487, 271 -> 257, 376 -> 387; 4.6 (1920x1080) 499 -> 500, 313 ->
        // 300, 384 -> 384; 8.1 (2560x1440) 599 -> 595, 530 -> 498, 425 -> 423; 18 (3840x2160) 878 -> 862, 1161 -> 1080, 686 -> 665.
        // With one, 7 per SM (through autograd; random, piled up, and 100k light triangles spread evenly): 3.6 waves (1600x900) 228 ->
        // 221, 366 -> 372, 170 -> 160; 5.2 (1920x1080) 319 -> 308, 381 -> 381, 222 -> 209; 9.3 (2560x1440) 543 -> 513, 434 -> 436,
        // 346 -> 313; 21 (3840x2160) 1193 -> 1115, 708 -> 688, 670 -> 594.  Between 3.6 and 5.2 one stands against the other.  Triangles piled up in the middle of a small image
        // lose: the passes of their CTAs hold what one pass spreads over all.
        constexpr int kPasses = 3;
        const int strips = (H + tg::kQueueRows - 1) / tg::kQueueRows;
        const int64_t wanted = grad_depthmap ? kPasses * 5 * 7 * 148 : kPasses * 7 * 8 * 148 / 2;      // 5 waves, 3.5 waves
        const bool many = (int64_t)Q.tiles_x * strips >= wanted;
        const int blocks = Q.tiles_x * (many ? (strips + kPasses - 1) / kPasses : strips);
        auto kernel = many ? (grad_depthmap ? tg::blend_backward_queued_kernel<kPasses, true> : tg::blend_backward_queued_kernel<kPasses, false>)
                           : (grad_depthmap ? tg::blend_backward_queued_kernel<1, true> : tg::blend_backward_queued_kernel<1, false>);
        TG_CUDA(tg_host::launch_dependent(kernel, blocks, tg::kQueueCols * tg::kQueueRows, 0, s, Q, in, selection, gpack));
    } else {
        if (int st = launch_list_kernel<false>(P, in, gpack, tiles, threads, per_pixel_sort, s)) return st;
    }
    TG_LAUNCH_CHECK("blend_backward_kernel");
    if (packed) return TG_OK;
    tg::unpack_gradients_kernel<<<(V + 255) / 256, 256, 0, s>>>(gpack, V, (float4*)grad_vertices, grad_colors,
                                                              grad_opacities, accumulate, 0, loss_sums, l2_loss_scale,
                                                              l2_target ? l2_loss_out : nullptr);
    TG_LAUNCH_CHECK("unpack_gradients_kernel");
    return TG_OK;
}

int tg_blend_step_l2(const float* tri_geo, const float* tri_attr, const int32_t* sorted_ids, const int32_t* offsets, int V,
                     int W, int H, int tw, int th, float thr, int max_layers, const float* target, float grad_scale,
                     float loss_scale, float* loss_out, float* image, float* depthmap, float* final_weights, int32_t* ends,
                     float* grad_vertices, float* grad_colors, float* grad_opacities, int accumulate, void* scratch,
                     size_t scratch_bytes, tg_stream_t stream) {
    if (int s = blend_args(W, H, tw, th, max_layers)) return s;
    TG_REQUIRE(tw * th <= 256 && max_layers <= tg::kBatchLayers,
               "the one-kernel step needs tiles of at most 256 pixels and max_layers <= 32 "
               "(otherwise: tg_blend_forward + tg_blend_backward_l2)");
    TG_REQUIRE(V > 0, "V must be positive");
    const bool packed = accumulate == TG_ACCUMULATE_PACKED;
    TG_REQUIRE(offsets && image && depthmap && final_weights && ends && target && (packed || loss_out), "null pointer");
    TG_REQUIRE(scratch && (packed || (grad_vertices && grad_colors && grad_opacities)), "null gradient / scratch pointer");
    TG_REQUIRE(((uintptr_t)image & 15) == 0 && ((uintptr_t)target & 15) == 0 && ((uintptr_t)tri_geo & 15) == 0 &&
                   ((uintptr_t)tri_attr & 15) == 0 && ((uintptr_t)grad_vertices & 15) == 0 && ((uintptr_t)scratch & 15) == 0,
               "image / target / tri_geo / tri_attr / grad_vertices / scratch must be 16-byte aligned");
    if (scratch_bytes < tg_backward_scratch_bytes(V)) {
        tg_host::set_error("backward scratch: need %zu bytes, got %zu", tg_backward_scratch_bytes(V), scratch_bytes);
        return TG_ERR_WORKSPACE;
    }
    cudaStream_t s = (cudaStream_t)stream;
    float4* gpack = (float4*)scratch;
    float* loss_sums = (float*)((char*)scratch + (size_t)V * 32);
    if (!packed) TG_CUDA(cudaMemsetAsync(gpack, 0, (size_t)V * 32 + tg::kLossBytes, s));
    tg::BlendParams P = make_params(tri_geo, tri_attr, sorted_ids, offsets, W, H, tw, th, thr, max_layers);
    P.order = tg_host::g_tile_order;
    const int tiles = P.tiles_x * ((H + th - 1) / th);
    const int threads = ((tw * th + 31) / 32) * 32;
    static tg_host::SmemAllowed allowed;
    constexpr size_t smem = 8 * sizeof(float4) * tg::QueueShape<false>::kQuads;
    if (int st = tg_host::allow_smem((const void*)tg::blend_step_l2_kernel<256>, smem, allowed)) return st;
    tg::blend_step_l2_kernel<256><<<tiles, threads, smem, s>>>(P, (float4*)image, depthmap, final_weights, ends,
                                                            (const float4*)target, grad_scale, loss_sums, gpack);
    TG_LAUNCH_CHECK("blend_step_l2_kernel");
    if (packed) return TG_OK;
    tg::unpack_gradients_kernel<<<(V + 255) / 256, 256, 0, s>>>(gpack, V, (float4*)grad_vertices, grad_colors,
                                                              grad_opacities, accumulate, 0, loss_sums, loss_scale, loss_out);
    TG_LAUNCH_CHECK("unpack_gradients_kernel");
    return TG_OK;
}

int tg_unpack_gradients(void* scratch, size_t scratch_bytes, int V, float loss_scale, float* loss_out,
                        float* grad_vertices, float* grad_colors, float* grad_opacities, int accumulate,
                        tg_stream_t stream) {
    TG_REQUIRE(V > 0, "V must be positive");
    TG_REQUIRE(scratch && grad_vertices && grad_colors && grad_opacities, "null pointer");
    const int clear = accumulate & TG_UNPACK_CLEAR;
    accumulate &= ~TG_UNPACK_CLEAR;
    TG_REQUIRE(accumulate == 0 || accumulate == 1, "accumulate must be 0 or 1 (+ TG_UNPACK_CLEAR)");
    TG_REQUIRE(((uintptr_t)grad_vertices & 15) == 0 && ((uintptr_t)scratch & 15) == 0,
               "grad_vertices / scratch must be 16-byte aligned");
    if (scratch_bytes < tg_backward_scratch_bytes(V)) {
        tg_host::set_error("backward scratch: need %zu bytes, got %zu", tg_backward_scratch_bytes(V), scratch_bytes);
        return TG_ERR_WORKSPACE;
    }
    float* loss_sums = (float*)((char*)scratch + (size_t)V * 32);
    TG_CUDA(tg_host::launch_dependent(tg::unpack_gradients_kernel, (V + 255) / 256, 256, 0, (cudaStream_t)stream, (float4*)scratch,
                                      V, (float4*)grad_vertices, grad_colors, grad_opacities, accumulate, clear, loss_sums,
                                      loss_scale, loss_out));
    TG_LAUNCH_CHECK("unpack_gradients_kernel");
    return TG_OK;
}

int tg_unpack_gradients_rgba(void* scratch, size_t scratch_bytes, int V, float loss_scale, float* loss_out,
                             float* grad_vertices, float* grad_rgba, int accumulate, tg_stream_t stream) {
    TG_REQUIRE(V > 0, "V must be positive");
    TG_REQUIRE(scratch && grad_vertices && grad_rgba, "null pointer");
    const int clear = accumulate & TG_UNPACK_CLEAR;
    accumulate &= ~TG_UNPACK_CLEAR;
    TG_REQUIRE(accumulate == 0 || accumulate == 1, "accumulate must be 0 or 1 (+ TG_UNPACK_CLEAR)");
    TG_REQUIRE((((uintptr_t)grad_vertices | (uintptr_t)grad_rgba | (uintptr_t)scratch) & 15) == 0,
               "grad_vertices / grad_rgba / scratch must be 16-byte aligned");
    if (scratch_bytes < tg_backward_scratch_bytes(V)) {
        tg_host::set_error("backward scratch: need %zu bytes, got %zu", tg_backward_scratch_bytes(V), scratch_bytes);
        return TG_ERR_WORKSPACE;
    }
    float* loss_sums = (float*)((char*)scratch + (size_t)V * 32);
    TG_CUDA(tg_host::launch_dependent(tg::unpack_gradients_rgba_kernel, (V + 255) / 256, 256, 0, (cudaStream_t)stream,
                                      (float4*)scratch, V, (float4*)grad_vertices, (float4*)grad_rgba, accumulate, clear,
                                      loss_sums, loss_scale, loss_out));
    TG_LAUNCH_CHECK("unpack_gradients_rgba_kernel");
    return TG_OK;
}

int tg_blend_backward(const float* tri_geo, const float* tri_attr, const int32_t* sorted_ids, const int32_t* offsets,
                      int V, int W, int H, int tw, int th, int per_pixel_sort, int max_layers, const float* grad_image,
                      const float* grad_depthmap, const float* image, const float* depthmap, const float* final_weights,
                      const int32_t* ends, const int32_t* selection, float* grad_vertices, float* grad_colors,
                      float* grad_opacities, int accumulate, void* scratch, size_t scratch_bytes, tg_stream_t stream) {
    TG_REQUIRE(grad_image, "null upstream gradient");
    return backward_impl(tri_geo, tri_attr, sorted_ids, offsets, V, W, H, tw, th, per_pixel_sort, max_layers, grad_image,
                         grad_depthmap, nullptr, false, 0.f, 0.f, nullptr, image, depthmap, final_weights, ends, selection,
                         grad_vertices, grad_colors, grad_opacities, accumulate, scratch, scratch_bytes, stream);
}

int tg_blend_backward_corrected(const float* tri_geo, const float* tri_attr, const int32_t* sorted_ids,
                                const int32_t* offsets, int V, int W, int H, int tw, int th, int per_pixel_sort,
                                int max_layers, const float* grad_image, const float* grad_depthmap, const float* image,
                                const float* depthmap, const float* final_weights, const int32_t* ends,
                                float* grad_vertices, float* grad_colors, float* grad_opacities, int accumulate,
                                void* scratch, size_t scratch_bytes, tg_stream_t stream) {
    if (int s = blend_args(W, H, tw, th, max_layers)) return s;
    TG_REQUIRE(V >= 0, "V < 0");
    TG_REQUIRE(offsets && image && depthmap && final_weights && ends && grad_image, "null pointer");
    if (V == 0) return TG_OK;
    TG_REQUIRE(accumulate == 0 || accumulate == 1, "accumulate must be 0 or 1");
    TG_REQUIRE(scratch && grad_vertices && grad_colors && grad_opacities, "null gradient / scratch pointer");
    TG_REQUIRE(((uintptr_t)image & 15) == 0 && ((uintptr_t)grad_image & 15) == 0 && ((uintptr_t)tri_geo & 15) == 0 &&
                   ((uintptr_t)tri_attr & 15) == 0 && ((uintptr_t)grad_vertices & 15) == 0 && ((uintptr_t)scratch & 15) == 0,
               "image / grad_image / tri_geo / tri_attr / grad_vertices / scratch must be 16-byte aligned");
    if (scratch_bytes < tg_backward_scratch_bytes(V)) {
        tg_host::set_error("backward scratch: need %zu bytes, got %zu", tg_backward_scratch_bytes(V), scratch_bytes);
        return TG_ERR_WORKSPACE;
    }
    cudaStream_t s = (cudaStream_t)stream;
    float4* gpack = (float4*)scratch;
    float* loss_sums = (float*)((char*)scratch + (size_t)V * 32);
    TG_CUDA(cudaMemsetAsync(gpack, 0, (size_t)V * 32 + tg::kLossBytes, s));
    const tg::BlendParams P = make_params(tri_geo, tri_attr, sorted_ids, offsets, W, H, tw, th, 0.f, max_layers);
    const int tiles = P.tiles_x * ((H + th - 1) / th);
    const int threads = ((tw * th + 31) / 32) * 32;
    const tg::BackwardIn in = {(const float4*)grad_image, grad_depthmap, (const float4*)image, depthmap, final_weights,
                               ends, nullptr, 0.f, loss_sums, nullptr};
    if (int st = launch_list_kernel<true>(P, in, gpack, tiles, threads, per_pixel_sort, s)) return st;
    TG_LAUNCH_CHECK("blend_backward_corrected_kernel");
    tg::unpack_gradients_kernel<<<(V + 255) / 256, 256, 0, s>>>(gpack, V, (float4*)grad_vertices, grad_colors,
                                                              grad_opacities, accumulate, 0, loss_sums, 0.f, nullptr);
    TG_LAUNCH_CHECK("unpack_gradients_kernel");
    return TG_OK;
}

int tg_blend_backward_l2(const float* tri_geo, const float* tri_attr, const int32_t* sorted_ids, const int32_t* offsets,
                         int V, int W, int H, int tw, int th, int per_pixel_sort, int max_layers, const float* target,
                         float grad_scale, float loss_scale, float* loss_out, const float* image, const float* depthmap,
                         const float* final_weights, const int32_t* ends, const int32_t* selection, float* grad_vertices,
                         float* grad_colors, float* grad_opacities, int accumulate, void* scratch, size_t scratch_bytes,
                         tg_stream_t stream) {
    TG_REQUIRE(target && (loss_out || accumulate == TG_ACCUMULATE_PACKED), "null target / loss pointer");
    return backward_impl(tri_geo, tri_attr, sorted_ids, offsets, V, W, H, tw, th, per_pixel_sort, max_layers, nullptr,
                         nullptr, target, false, grad_scale, loss_scale, loss_out, image, depthmap, final_weights, ends,
                         selection, grad_vertices, grad_colors, grad_opacities, accumulate, scratch, scratch_bytes, stream);
}

int tg_blend_backward_l2_u8(const float* tri_geo, const float* tri_attr, const int32_t* sorted_ids, const int32_t* offsets,
                            int V, int W, int H, int tw, int th, int per_pixel_sort, int max_layers,
                            const uint8_t* target_rgba8, float grad_scale, float loss_scale, float* loss_out,
                            const float* image, const float* depthmap, const float* final_weights, const int32_t* ends,
                            const int32_t* selection, float* grad_vertices, float* grad_colors, float* grad_opacities,
                            int accumulate, void* scratch, size_t scratch_bytes, tg_stream_t stream) {
    TG_REQUIRE(target_rgba8 && (loss_out || accumulate == TG_ACCUMULATE_PACKED), "null target / loss pointer");
    return backward_impl(tri_geo, tri_attr, sorted_ids, offsets, V, W, H, tw, th, per_pixel_sort, max_layers, nullptr,
                         nullptr, target_rgba8, true, grad_scale, loss_scale, loss_out, image, depthmap, final_weights, ends,
                         selection, grad_vertices, grad_colors, grad_opacities, accumulate, scratch, scratch_bytes, stream);
}

}  // extern "C"
