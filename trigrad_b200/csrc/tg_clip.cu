// Near-plane triangle splitter fused with the world -> render-space projection, and its vector-Jacobian
// product: the step before the rasteriser for cameras that sit inside or close to the mesh.
//
// The reference does this in its notebook with a Python loop over triangles (`split_clipped`,
// notebooks/renderer.ipynb cell "Clip Test"): clip-space vertices, signed distance d = z + w to the near plane,
// a triangle with all three vertices inside (d >= 0) is kept, one with none is dropped, one inside vertex gives
// one smaller triangle (in, new1, new2), two inside vertices give a quad split into (in1, in2, new1) and
// (new1, in2, new2); a new vertex is a + t (b - a) with t = d_a / (d_a - d_b) from the inside vertex a to the
// outside vertex b, and colours and opacities are interpolated with the same t.  The result is a triangle
// soup.  Here one thread handles one input triangle and owns two output slots (6 vertices), so the order of
// the reference's soup is kept and nothing has to be counted or compacted: slots that are not needed are
// filled with a degenerate triangle (all vertices (0,0,0,1)), which the rasteriser's preprocess drops.
// Output vertices are already divided: (x/w, y/w, z/w, 1/w), the render format (viewer.py:271-278).
#include "tg_common.cuh"

namespace tg {

struct ClipMat { float m[16]; };   // row-major projection * view

struct ClipVertex { float x, y, z, w; };

__device__ __forceinline__ ClipVertex to_clip(const float* __restrict__ points, int v, const ClipMat& pv) {
    const float x = points[3 * (size_t)v], y = points[3 * (size_t)v + 1], z = points[3 * (size_t)v + 2];
    float c[4];
#pragma unroll
    for (int r = 0; r < 4; r++) c[r] = fma_(pv.m[4 * r + 2], z, fma_(pv.m[4 * r + 1], y, fma_(pv.m[4 * r], x, pv.m[4 * r + 3])));
    return {c[0], c[1], c[2], c[3]};
}

// How many of a triangle's vertices are inside, and which vertex comes first in the reference's order: (in, out1, out2)
// with one inside, (out, in1, in2) with two, (0, 1, 2) otherwise.
struct ClipCase {
    int inside, first;
};
__device__ __forceinline__ ClipCase classify(float d0, float d1, float d2) {
    const bool i0 = d0 >= 0.f, i1 = d1 >= 0.f, i2 = d2 >= 0.f;
    ClipCase c;
    c.inside = (int)i0 + (int)i1 + (int)i2;
    c.first = 0;
    if (c.inside == 1) c.first = i0 ? 0 : i1 ? 1 : 2;
    if (c.inside == 2) c.first = !i0 ? 0 : !i1 ? 1 : 2;
    return c;
}
// (a, b, c) rotated so that element `first` comes first: selects, no indexed array (which would live in local memory).
template <class T>
__device__ __forceinline__ void rotate3(int first, T& a, T& b, T& c) {
    const T x = a, y = b, z = c;
    if (first == 1) { a = y; b = z; c = x; }
    if (first == 2) { a = z; b = x; c = y; }
}

struct SoupVertex { ClipVertex v; float r, g, b, o; };

// a + t (b - a), every operation rounded separately (what the tensor expression of the reference evaluates to)
__device__ __forceinline__ float lerp_rn(float a, float b, float t) { return add(a, mul(t, sub(b, a))); }

__device__ __forceinline__ SoupVertex lerp_vertex(const SoupVertex& a, const SoupVertex& b, float t) {
    SoupVertex n;
    n.v = {lerp_rn(a.v.x, b.v.x, t), lerp_rn(a.v.y, b.v.y, t), lerp_rn(a.v.z, b.v.z, t), lerp_rn(a.v.w, b.v.w, t)};
    n.r = lerp_rn(a.r, b.r, t); n.g = lerp_rn(a.g, b.g, t); n.b = lerp_rn(a.b, b.b, t);
    n.o = lerp_rn(a.o, b.o, t);
    return n;
}

// The triangle's vertices, rotated, with their signed distances to the near plane.
struct ClipTriangle {
    SoupVertex a, b, c;
    float da, db, dc;
    int va, vb, vc;
    int inside;
};
__device__ __forceinline__ SoupVertex load_soup(const float* points, const float* colors, const float* opacities, int v,
                                                const ClipMat& pv) {
    SoupVertex s;
    s.v = to_clip(points, v, pv);
    s.r = colors[3 * (size_t)v]; s.g = colors[3 * (size_t)v + 1]; s.b = colors[3 * (size_t)v + 2];
    s.o = opacities[v];
    return s;
}
__device__ __forceinline__ ClipTriangle load_clip_triangle(int t, const float* points, const int* indices, const float* colors,
                                                           const float* opacities, const ClipMat& pv) {
    ClipTriangle c;
    c.va = indices[3 * (size_t)t]; c.vb = indices[3 * (size_t)t + 1]; c.vc = indices[3 * (size_t)t + 2];
    c.a = load_soup(points, colors, opacities, c.va, pv);
    c.b = load_soup(points, colors, opacities, c.vb, pv);
    c.c = load_soup(points, colors, opacities, c.vc, pv);
    c.da = add(c.a.v.z, c.a.v.w); c.db = add(c.b.v.z, c.b.v.w); c.dc = add(c.c.v.z, c.c.v.w);
    const ClipCase cc = classify(c.da, c.db, c.dc);
    c.inside = cc.inside;
    rotate3(cc.first, c.a, c.b, c.c);
    rotate3(cc.first, c.da, c.db, c.dc);
    rotate3(cc.first, c.va, c.vb, c.vc);
    return c;
}

// One thread per input triangle; its six output vertices leave through shared memory, so that the CTA's stores are whole
// consecutive lines (stored by the threads themselves they were 16 bytes every 96, 4 bytes every 72 and every 24: 82k
// triangles 24 us).
constexpr int kClipThreads = 128;
__global__ void __launch_bounds__(kClipThreads) project_clip_kernel(const float* __restrict__ points,
                                                                    const int* __restrict__ indices,
                                                                    const float* __restrict__ colors,
                                                                    const float* __restrict__ opacities, int T, ClipMat pv,
                                                                    float4* __restrict__ out_vertices,
                                                                    int* __restrict__ out_indices,
                                                                    float* __restrict__ out_colors,
                                                                    float* __restrict__ out_opacities) {
    // odd pitches: 7 quads for 6 vertices, 19 words for 18 colour components, 7 words for 6 opacities
    __shared__ float4 s_v[kClipThreads * 7];
    __shared__ float s_c[kClipThreads * 19];
    __shared__ float s_o[kClipThreads * 7];
    allow_dependents();
    await_prerequisites();
    const int tid = threadIdx.x, t0 = blockIdx.x * kClipThreads, n = min(kClipThreads, T - t0);
    if (tid < n) {
        auto put = [&](int k, const SoupVertex& s) {
            s_v[7 * tid + k] = make_float4(div(s.v.x, s.v.w), div(s.v.y, s.v.w), div(s.v.z, s.v.w), div(1.f, s.v.w));
            s_c[19 * tid + 3 * k] = s.r; s_c[19 * tid + 3 * k + 1] = s.g; s_c[19 * tid + 3 * k + 2] = s.b;
            s_o[7 * tid + k] = s.o;
        };
        auto unused = [&](int k) {
            s_v[7 * tid + k] = make_float4(0.f, 0.f, 0.f, 1.f);
            s_c[19 * tid + 3 * k] = s_c[19 * tid + 3 * k + 1] = s_c[19 * tid + 3 * k + 2] = 0.f;
            s_o[7 * tid + k] = 0.f;
        };
        const ClipTriangle c = load_clip_triangle(t0 + tid, points, indices, colors, opacities, pv);
        if (c.inside == 2) {              // a outside
            const float t1 = div(c.db, sub(c.db, c.da)), t2 = div(c.dc, sub(c.dc, c.da));
            const SoupVertex n1 = lerp_vertex(c.b, c.a, t1), n2 = lerp_vertex(c.c, c.a, t2);
            put(0, c.b); put(1, c.c); put(2, n1);
            put(3, n1); put(4, c.c); put(5, n2);
        } else {
            if (c.inside == 3) {
                put(0, c.a); put(1, c.b); put(2, c.c);
            } else if (c.inside == 1) {   // a inside
                const float t1 = div(c.da, sub(c.da, c.db)), t2 = div(c.da, sub(c.da, c.dc));
                put(0, c.a); put(1, lerp_vertex(c.a, c.b, t1)); put(2, lerp_vertex(c.a, c.c, t2));
            } else {
                unused(0); unused(1); unused(2);
            }
            unused(3); unused(4); unused(5);
        }
    }
    __syncthreads();
    const size_t first = 6 * (size_t)t0;
    for (int i = tid; i < 6 * n; i += kClipThreads) {
        const int r = i / 6, k = i % 6;
        out_vertices[first + i] = s_v[7 * r + k];
        out_opacities[first + i] = s_o[7 * r + k];
        out_indices[first + i] = (int)first + i;
    }
    for (int i = tid; i < 18 * n; i += kClipThreads) out_colors[3 * first + i] = s_c[19 * (i / 18) + i % 18];
}

// ---- vector-Jacobian product ---------------------------------------------------------------------
// Gradient record of one ORIGINAL vertex of the triangle: clip-space position, colour, opacity.
struct VertexGrad { float x = 0.f, y = 0.f, z = 0.f, w = 0.f, r = 0.f, g = 0.f, b = 0.f, o = 0.f; };

struct SoupGrad { float x, y, z, w, r, g, b, o; };   // upstream gradient of one soup vertex, position already in clip space

// render-space gradient (of x/w, y/w, z/w, 1/w) -> clip-space gradient at clip vertex c
__device__ __forceinline__ SoupGrad load_soup_grad(const ClipVertex& c, int slot, const float4* __restrict__ gv,
                                                   const float* __restrict__ gc, const float* __restrict__ go) {
    const float4 g = gv[slot];
    const float iw = 1.f / c.w;
    SoupGrad s;
    s.x = g.x * iw; s.y = g.y * iw; s.z = g.z * iw;
    s.w = -(s.x * c.x + s.y * c.y + s.z * c.z + g.w * iw) * iw;
    s.r = gc[3 * (size_t)slot]; s.g = gc[3 * (size_t)slot + 1]; s.b = gc[3 * (size_t)slot + 2];
    s.o = go[slot];
    return s;
}

__device__ __forceinline__ void add_grad(VertexGrad& a, const SoupGrad& g, float f) {
    a.x += f * g.x; a.y += f * g.y; a.z += f * g.z; a.w += f * g.w;
    a.r += f * g.r; a.g += f * g.g; a.b += f * g.b; a.o += f * g.o;
}

// new = a + t (b - a), t = da / (da - db), d = z + w: the gradient g of `new` goes to a and b, also through t
__device__ __forceinline__ void lerp_backward(const SoupVertex& a, const SoupVertex& b, float da, float db, float t,
                                              const SoupGrad& g, VertexGrad& ga, VertexGrad& gb) {
    add_grad(ga, g, 1.f - t);
    add_grad(gb, g, t);
    const float gt = g.x * (b.v.x - a.v.x) + g.y * (b.v.y - a.v.y) + g.z * (b.v.z - a.v.z) + g.w * (b.v.w - a.v.w) +
                     g.r * (b.r - a.r) + g.g * (b.g - a.g) + g.b * (b.b - a.b) + g.o * (b.o - a.o);
    const float inv = 1.f / (da - db);
    const float gda = gt * (-db) * inv * inv, gdb = gt * da * inv * inv;
    ga.z += gda; ga.w += gda;
    gb.z += gdb; gb.w += gdb;
}

// Bound by latency: the gathers, then the atomics, 21 per triangle, of which those that would add nothing are left out (82k
// triangles around a camera that sees a fifth of them: 13.5 -> 11 us).
__global__ void __launch_bounds__(256) project_clip_backward_kernel(
    const float* __restrict__ points, const int* __restrict__ indices, const float* __restrict__ colors,
    const float* __restrict__ opacities, int T, ClipMat pv, const float4* __restrict__ grad_out_vertices,
    const float* __restrict__ grad_out_colors, const float* __restrict__ grad_out_opacities,
    float* __restrict__ grad_points, float* __restrict__ grad_colors, float* __restrict__ grad_opacities) {
    allow_dependents();
    await_prerequisites();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= T) return;
    const ClipTriangle c = load_clip_triangle(t, points, indices, colors, opacities, pv);
    if (c.inside == 0) return;
    const int base = 6 * t;
    VertexGrad ga, gb, gc;
    auto upstream = [&](const ClipVertex& v, int k) {
        return load_soup_grad(v, base + k, grad_out_vertices, grad_out_colors, grad_out_opacities);
    };
    if (c.inside == 3) {
        add_grad(ga, upstream(c.a.v, 0), 1.f);
        add_grad(gb, upstream(c.b.v, 1), 1.f);
        add_grad(gc, upstream(c.c.v, 2), 1.f);
    } else if (c.inside == 1) {           // a inside
        const float t1 = div(c.da, sub(c.da, c.db)), t2 = div(c.da, sub(c.da, c.dc));
        const SoupVertex n1 = lerp_vertex(c.a, c.b, t1), n2 = lerp_vertex(c.a, c.c, t2);
        add_grad(ga, upstream(c.a.v, 0), 1.f);
        lerp_backward(c.a, c.b, c.da, c.db, t1, upstream(n1.v, 1), ga, gb);
        lerp_backward(c.a, c.c, c.da, c.dc, t2, upstream(n2.v, 2), ga, gc);
    } else {                              // a outside; soup: (b, c, n1), (n1, c, n2)
        const float t1 = div(c.db, sub(c.db, c.da)), t2 = div(c.dc, sub(c.dc, c.da));
        const SoupVertex n1 = lerp_vertex(c.b, c.a, t1), n2 = lerp_vertex(c.c, c.a, t2);
        add_grad(gb, upstream(c.b.v, 0), 1.f);
        add_grad(gc, upstream(c.c.v, 1), 1.f);
        add_grad(gc, upstream(c.c.v, 4), 1.f);
        SoupGrad g1 = upstream(n1.v, 2);
        const SoupGrad g1b = upstream(n1.v, 3);
        g1.x += g1b.x; g1.y += g1b.y; g1.z += g1b.z; g1.w += g1b.w;
        g1.r += g1b.r; g1.g += g1b.g; g1.b += g1b.b; g1.o += g1b.o;
        lerp_backward(c.b, c.a, c.db, c.da, t1, g1, gb, ga);
        lerp_backward(c.c, c.a, c.dc, c.da, t2, upstream(n2.v, 5), gc, ga);
    }
    auto add_to = [&](int v, const VertexGrad& g) {
        // most triangles around a camera are out of its sight
        if (g.x == 0.f && g.y == 0.f && g.z == 0.f && g.w == 0.f && g.r == 0.f && g.g == 0.f && g.b == 0.f && g.o == 0.f) return;
        // clip -> world: clip = PV (p, 1)
#pragma unroll
        for (int j = 0; j < 3; j++)
            atomicAdd(grad_points + 3 * (size_t)v + j, g.x * pv.m[j] + g.y * pv.m[4 + j] + g.z * pv.m[8 + j] + g.w * pv.m[12 + j]);
        atomicAdd(grad_colors + 3 * (size_t)v, g.r);
        atomicAdd(grad_colors + 3 * (size_t)v + 1, g.g);
        atomicAdd(grad_colors + 3 * (size_t)v + 2, g.b);
        atomicAdd(grad_opacities + v, g.o);
    };
    add_to(c.va, ga);
    add_to(c.vb, gb);
    add_to(c.vc, gc);
}

// Zeroes the three gradient tensors of a backward with one launch, which starts before the kernel ahead has ended: with three
// fills it was 24 us from there to the end of the kernel above, now 12.
__global__ void __launch_bounds__(256) clear_gradients_kernel(float* __restrict__ points, float* __restrict__ colors,
                                                              float* __restrict__ opacities, size_t V) {
    allow_dependents();
    await_prerequisites();
    for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < 3 * V; i += (size_t)gridDim.x * 256) {
        points[i] = 0.f;
        colors[i] = 0.f;
        if (i < V) opacities[i] = 0.f;
    }
}

}  // namespace tg

extern "C" {

int tg_project_clip(const float* points, const int32_t* indices, const float* colors, const float* opacities, int T,
                    const float* pv_host, float* out_vertices, int32_t* out_indices, float* out_colors,
                    float* out_opacities, tg_stream_t stream) {
    TG_REQUIRE(T >= 0, "T < 0");
    if (T == 0) return TG_OK;
    TG_REQUIRE(T <= 0x7fffffff / 6, "T too large for 6 T soup vertices");
    TG_REQUIRE(points && indices && colors && opacities && pv_host && out_vertices && out_indices && out_colors &&
                   out_opacities, "null pointer");
    TG_REQUIRE(((uintptr_t)out_vertices & 15) == 0, "out_vertices must be 16-byte aligned");
    tg::ClipMat pv;
    for (int i = 0; i < 16; i++) pv.m[i] = pv_host[i];
    TG_CUDA(tg_host::launch_dependent(tg::project_clip_kernel, (T + tg::kClipThreads - 1) / tg::kClipThreads, tg::kClipThreads, 0,
                                      (cudaStream_t)stream, points, indices, colors, opacities, T, pv, (float4*)out_vertices,
                                      out_indices, out_colors, out_opacities));
    TG_LAUNCH_CHECK("project_clip_kernel");
    return TG_OK;
}

int tg_project_clip_backward(const float* points, const int32_t* indices, const float* colors, const float* opacities,
                             int T, const float* pv_host, const float* grad_out_vertices, const float* grad_out_colors,
                             const float* grad_out_opacities, float* grad_points, float* grad_colors,
                             float* grad_opacities, tg_stream_t stream) {
    TG_REQUIRE(T >= 0, "T < 0");
    if (T == 0) return TG_OK;
    TG_REQUIRE(points && indices && colors && opacities && pv_host && grad_out_vertices && grad_out_colors &&
                   grad_out_opacities && grad_points && grad_colors && grad_opacities, "null pointer");
    TG_REQUIRE(((uintptr_t)grad_out_vertices & 15) == 0, "grad_out_vertices must be 16-byte aligned");
    tg::ClipMat pv;
    for (int i = 0; i < 16; i++) pv.m[i] = pv_host[i];
    TG_CUDA(tg_host::launch_dependent(tg::project_clip_backward_kernel, (T + 255) / 256, 256, 0, (cudaStream_t)stream, points, indices,
                                      colors, opacities, T, pv, (const float4*)grad_out_vertices, grad_out_colors,
                                      grad_out_opacities, grad_points, grad_colors, grad_opacities));
    TG_LAUNCH_CHECK("project_clip_backward_kernel");
    return TG_OK;
}

int tg_clear_gradients(float* grad_points, float* grad_colors, float* grad_opacities, int V, tg_stream_t stream) {
    TG_REQUIRE(V >= 0, "V < 0");
    if (V == 0) return TG_OK;
    TG_REQUIRE(grad_points && grad_colors && grad_opacities, "null pointer");
    const int64_t want = (3 * (int64_t)V + 255) / 256;
    TG_CUDA(tg_host::launch_dependent(tg::clear_gradients_kernel, (int)(want < 148 * 8 ? want : 148 * 8), 256, 0, (cudaStream_t)stream,
                                      grad_points, grad_colors, grad_opacities, (size_t)V));
    TG_LAUNCH_CHECK("clear_gradients_kernel");
    return TG_OK;
}

}  // extern "C"
