// rast_device.cuh - per-vertex, per-triangle and per-fragment math of the raster pipeline.
//
// Every function restates one step of the reference renderer (NiklasJonsson/rusterizer,
// file:line cited) with the same binary32 operation order. The translation units that
// include this file are compiled with --fmad=false and IEEE division/sqrt, so each
// expression below rounds once per operation, like the reference's release build.
#pragma once

#include <cstdint>
#include <cfloat>
#include <cuda_runtime.h>

#include "rast_types.h"

namespace rast {

// ------------------------------------------------------------------ scalar rules

// Rust `f as u32` (truncate, saturate, NaN -> 0): cvt.rzi.u32.f32 saturates by definition.
__device__ __forceinline__ uint32_t sat_u32(float f) { return __float2uint_rz(f); }
// Rust `f as usize` on a 64-bit target.
__device__ __forceinline__ uint64_t sat_u64(float f) { return __float2ull_rz(f); }

// f32::clamp(0.0, 1.0) as used by clamp_bary (src/rasterizer/mod.rs:102-106):
// NaN and -0.0 pass through unchanged.
__device__ __forceinline__ float clamp01(float x) {
    if (x < 0.0f) x = 0.0f;
    if (x > 1.0f) x = 1.0f;
    return x;
}

// clamp01 that returns a NaN as a NaN of unspecified payload and may return +0.0 for -0.0
// (max.NaN / min.NaN: two instructions).
__device__ __forceinline__ float clamp01_nan(float x) {
    float r;
    asm("max.NaN.f32 %0, %1, 0f00000000;" : "=f"(r) : "f"(x));
    asm("min.NaN.f32 %0, %1, 0f3F800000;" : "=f"(r) : "f"(r));
    return r;
}

// ------------------------------------------------------------------ vertex stage

// Vector::dot (src/math/vector.rs:17-23): sum from 0.0, in order.
__device__ __forceinline__ float dot4(const float* r, float x, float y, float z, float w) {
    float s = 0.0f;
    s = s + r[0] * x;
    s = s + r[1] * y;
    s = s + r[2] * z;
    s = s + r[3] * w;
    return s;
}

// Rasterizer::perspective_divide (src/rasterizer/mod.rs:284-313): (x/w, y/w, z/w, w)
__device__ __forceinline__ float4 persp_divide(float4 c) {
    return make_float4(c.x / c.w, c.y / c.w, c.z / c.w, c.w);
}

// viewport_transform's per-vertex closure (src/rasterizer/mod.rs:318-331) on an NDC vertex;
// w passes through as depths_camera_space (mod.rs:338-342). Returns (sx, sy, sz, w).
__device__ __forceinline__ float4 viewport(float4 n, float fw, float fh) {
    const float zmin = 0.0f, zmax = 1.0f;
    float sx = fw * (n.x + 1.0f) / 2.0f;
    float sy = fh * (1.0f - (n.y + 1.0f) / 2.0f);
    float sz = (n.z + 1.0f) * 0.5f * (zmax - zmin) + zmin;
    return make_float4(sx, sy, sz, n.w);
}

__device__ __forceinline__ float4 to_screen(float4 c, float fw, float fh) {
    return viewport(persp_divide(c), fw, fh);
}

// Clip-plane predicates of try_clip's fast checks (src/rasterizer/clipping.rs:86-104):
// bits 0..5 "inside" (x >= -w, x <= w, y >= -w, y <= w, z >= -w, z <= w),
// bits 6..11 "outside" (x < -w, x > w, ...). NaN sets neither.
__device__ __forceinline__ uint32_t clip_code(float4 c) {
    uint32_t code = 0;
    const float v[3] = {c.x, c.y, c.z};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        code |= (uint32_t)(v[a] >= -c.w) << (2 * a);
        code |= (uint32_t)(v[a] <= c.w) << (2 * a + 1);
        code |= (uint32_t)(v[a] < -c.w) << (6 + 2 * a);
        code |= (uint32_t)(v[a] > c.w) << (6 + 2 * a + 1);
    }
    return code;
}
constexpr uint32_t kInsideAll = 0x3Fu;

// triangle_2x_area (src/rasterizer/mod.rs:15-21) with Vec2::cross (src/math/vector.rs:183-185)
__device__ __forceinline__ float tri2x_area(float x0, float y0, float x1, float y1, float x2,
                                            float y2) {
    float v10x = x1 - x0, v10y = y1 - y0;
    float v20x = x2 - x0, v20y = y2 - y0;
    return v10x * v20y - v20x * v10y;
}

// ------------------------------------------------------------------ clipping

struct ClipVert {
    float p[4];  // clip-space x, y, z, w
    float a[6];  // VertexAttribute colour r,g,b,a then uv (src/graphics_primitives.rs:9-13)
};

// distance_measure (src/rasterizer/clipping.rs:29-38), planes in CLIP_PLANES order (:53-60)
__device__ __forceinline__ float distance_measure(int plane, const float* p) {
    switch (plane) {
        case 0: return p[3] + p[0];
        case 1: return p[3] - p[0];
        case 2: return p[3] + p[1];
        case 3: return p[3] - p[1];
        case 4: return p[3] + p[2];
        default: return p[3] - p[2];
    }
}

// compute_intersection (clipping.rs:43-51) + the attribute lerp (clipping.rs:149, :161)
__device__ __forceinline__ void clip_intersect(const ClipVert& pv, float dp, const ClipVert& cv,
                                               float dc, ClipVert& out) {
    float alpha = dp / (dp - dc);
    float om = 1.0f - alpha;
#pragma unroll
    for (int k = 0; k < 4; ++k) out.p[k] = pv.p[k] * om + cv.p[k] * alpha;
#pragma unroll
    for (int k = 0; k < 6; ++k) out.a[k] = (cv.a[k] - pv.a[k]) * alpha + pv.a[k];
}

// Classification part of try_clip (src/rasterizer/clipping.rs:62-112): 0 Outside, 1 Inside,
// 2 needs Sutherland-Hodgman. area is triangle_2x_area of the clip-space xy.
__device__ __forceinline__ int clip_classify(float area, uint32_t c0, uint32_t c1, uint32_t c2) {
    if (fabsf(area) < kCullEps) return 0;
    uint32_t all = c0 & c1 & c2;
    if (all & 0xFC0u) return 0;
    if ((all & kInsideAll) == kInsideAll) return 1;
    return 2;
}

// ------------------------------------------------------------------ triangle setup

// RasterizerTriangle (src/rasterizer/mod.rs:177-222): edge points, inward normals, screen
// depths, camera-space w, 1 / (2 * area), attributes.
struct TriSetup {
    float px[3], py[3];
    float nx[3], ny[3];
    float z[3], w[3];
    float inv_area;
};

// RasterizerTriangle::new (src/rasterizer/mod.rs:186-222)
__device__ __forceinline__ void tri_setup(TriSetup& t, const float4 s[3]) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        t.px[k] = s[k].x;
        t.py[k] = s[k].y;
        t.z[k] = s[k].z;
        t.w[k] = s[k].w;
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        int n = (k + 1) % 3;
        float vx = s[n].x - s[k].x, vy = s[n].y - s[k].y;
        t.nx[k] = -vy;
        t.ny[k] = vx;
    }
    t.inv_area = 1.0f / tri2x_area(s[0].x, s[0].y, s[1].x, s[1].y, s[2].x, s[2].y);
}

// PixelBoundingBox::from (src/rasterizer/bounding_box.rs:13-41) clamped to the viewport
// (Rasterizer::bounding_box, src/rasterizer/mod.rs:347-361). Half-open [x0,x1) x [y0,y1).
// The reference converts with `as usize` (64-bit saturation) and then clamps to the viewport;
// converting with 32-bit saturation gives the same clamped result for any viewport below 2^32:
// both conversions agree below 2^32, and at or above it both results exceed the viewport and
// are clamped to it (NaN and negatives give 0 either way).
__device__ __forceinline__ void pixel_bbox(const float4 s[3], uint32_t width, uint32_t height,
                                           uint32_t& x0, uint32_t& x1, uint32_t& y0,
                                           uint32_t& y1) {
    float mnx = FLT_MAX, mxx = -FLT_MAX, mny = FLT_MAX, mxy = -FLT_MAX;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        mnx = fminf(mnx, s[k].x);
        mxx = fmaxf(mxx, s[k].x);
        mny = fminf(mny, s[k].y);
        mxy = fmaxf(mxy, s[k].y);
    }
    x0 = min(sat_u32(floorf(mnx)), width);
    x1 = min(sat_u32(ceilf(mxx)), width);
    y0 = min(sat_u32(floorf(mny)), height);
    y1 = min(sat_u32(ceilf(mxy)), height);
}

// EdgeFunctions::eval_single (src/rasterizer/mod.rs:125-132): normal . (p - point), dot
// accumulated from 0.0.
__device__ __forceinline__ float edge_eval(float nx, float ny, float px, float py, float x,
                                           float y) {
    float dx = x - px, dy = y - py;
    float s = 0.0f;
    s = s + nx * dx;
    s = s + ny * dy;
    return s;
}

// EdgeFunctions::inside for one edge (src/rasterizer/mod.rs:148-170) without branches: pass
// when the value is positive, or when it is zero (or NaN) and the tie rule holds; the tie rule
// keys off the normal: x > 0, or x not negative and y < 0 (edge_tie, once per triangle edge).
__device__ __forceinline__ bool edge_tie(float nx, float ny) { return (nx > 0.0f) | (!(nx < 0.0f) & (ny < 0.0f)); }
__device__ __forceinline__ bool edge_pass_t(float e, bool tie) { return (e > 0.0f) | (!(e < 0.0f) & tie); }

// RGSS_SAMPLE_PATTERN (src/rasterizer/mod.rs:109-114); 1 sample = pixel centre (extension).
template <int S>
__device__ __forceinline__ float sample_dx(int i) {
    if (S == 1) return 0.5f;
    return i == 0 ? 5.0f / 8.0f : i == 1 ? 7.0f / 8.0f : i == 2 ? 3.0f / 8.0f : 1.0f / 8.0f;
}
template <int S>
__device__ __forceinline__ float sample_dy(int i) {
    if (S == 1) return 0.5f;
    return i == 0 ? 1.0f / 8.0f : i == 1 ? 5.0f / 8.0f : i == 2 ? 7.0f / 8.0f : 3.0f / 8.0f;
}

// ------------------------------------------------------------------ coverage and sample depths

// Two binary32 values in one 64-bit register pair: the packed add and multiply round each half
// like the scalar instruction and take one issue slot for both.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// 1 / triangle_2x_area as cover_pixel takes it: NaN marks an item whose edge values or clamped
// barycentrics could be NaN (a coordinate of 2^30 or more, or an infinite or NaN reciprocal);
// its pixels take cover_exact. Below 2^30 every difference, product and sum of the edge
// functions stays finite.
__device__ __forceinline__ float cover_inv(const float4 s[3]) {
    const float inv = 1.0f / tri2x_area(s[0].x, s[0].y, s[1].x, s[1].y, s[2].x, s[2].y);
    float m = 0.0f;  // a NaN coordinate makes the reciprocal NaN
#pragma unroll
    for (int k = 0; k < 3; ++k) m = fmaxf(m, fmaxf(fabsf(s[k].x), fabsf(s[k].y)));
    return (m < 0x1p30f && fabsf(inv) <= FLT_MAX) ? inv : __int_as_float(0x7FC00000);
}

template <int S>
struct Cover {
    uint32_t mask;  // bit k: sample k covered
    float z[S];     // sample depths; meaningless where the sample is not covered
};

// Coverage (EdgeFunctions::eval, src/rasterizer/mod.rs:134-146) and sample depths
// (RasterizerTriangle::fragment, mod.rs:225-253) of one pixel in the reference's own steps: any
// input, including NaN and infinite ones. Kept out of line: cover_pixel calls it only for
// samples exactly on an edge and for items cover_inv marks.
template <int S>
__device__ __noinline__ Cover<S> cover_exact(float p0x, float p0y, float p1x, float p1y, float p2x, float p2y,
                                             float z0, float z1, float z2, float fx, float fy) {
    Cover<S> c;
    c.mask = 0;
    const float inv = 1.0f / tri2x_area(p0x, p0y, p1x, p1y, p2x, p2y);
    // inward normals (RasterizerTriangle::new, src/rasterizer/mod.rs:199-204)
    const float n0x = -(p1y - p0y), n0y = p1x - p0x;
    const float n1x = -(p2y - p1y), n1y = p2x - p1x;
    const float n2x = -(p0y - p2y), n2y = p0x - p2x;
    const bool t0 = edge_tie(n0x, n0y), t1 = edge_tie(n1x, n1y), t2 = edge_tie(n2x, n2y);
#pragma unroll
    for (int k = 0; k < S; ++k) {
        const float xs = fx + sample_dx<S>(k), ys = fy + sample_dy<S>(k);
        const float e0 = edge_eval(n0x, n0y, p0x, p0y, xs, ys);
        const float e1 = edge_eval(n1x, n1y, p1x, p1y, xs, ys);
        const float e2 = edge_eval(n2x, n2y, p2x, p2y, xs, ys);
        const bool in = edge_pass_t(e0, t0) & edge_pass_t(e1, t1) & edge_pass_t(e2, t2);
        const float b0 = clamp01(e1 * inv);
        const float b1 = clamp01(e2 * inv);
        const float b2 = clamp01(1.0f - b0 - b1);
        c.mask |= (uint32_t)in << k;
        c.z[k] = b0 * z0 + b1 * z1 + b2 * z2;
    }
    return c;
}

// The same coverage mask and depths, bit for bit where a sample is covered, in about half the
// issue slots. `inv` is cover_inv's.
//   - An edge's value (-vy) dx + vx dy, v = next point - point and d = sample - point, is
//     vx dy - vy dx: one packed add for both differences, one packed multiply, one subtraction.
//     Dropping the reference's leading 0 + can only turn +0 into -0.
//   - With no NaN among the three values, the smallest decides: above 0 every edge passes, below
//     0 one fails whatever the tie rule. Exactly 0 leaves it to the tie rule: cover_exact.
//   - Saturating multiplies and adds are clamp01 for values that are not NaN, except that a -0
//     comes out +0. A zero b0 or b1 of the other sign flips only the sign of a zero product
//     b z, and the sum can only change from +0 to -0 when another product is -0 too, which needs
//     a corner depth of -0; the viewport's final + zmin makes every screen depth +0 instead, and
//     clamp((1 - b0) - b1) is never -0.
// The raster kernels are bound by instruction issue (70-77% of slots). Against two compares per
// edge, two clamps per weight and scalar edge values: 3% off a frame of the 100k-triangle soup at
// 1080p, 4% off the 2M-triangle 4K terrain. Packing over pairs of samples instead, or the depth
// sums as well, gave no more (the latter is contracted to a fused multiply-add and is wrong).
template <int S>
__device__ __forceinline__ Cover<S> cover_pixel(float p0x, float p0y, float p1x, float p1y, float p2x, float p2y,
                                                float inv, float z0, float z1, float z2, float fx, float fy) {
    Cover<S> c;
    c.mask = 0;
    const f32x2 o = pack2(fy, fx);
    const f32x2 m0 = pack2(-p0y, -p0x), m1 = pack2(-p1y, -p1x), m2 = pack2(-p2y, -p2x);
    const f32x2 v0 = pack2(p1x - p0x, p1y - p0y), v1 = pack2(p2x - p1x, p2y - p1y), v2 = pack2(p0x - p2x, p0y - p2y);
    bool exact = !(fabsf(inv) <= FLT_MAX);
#pragma unroll
    for (int k = 0; k < S; ++k) {
        const f32x2 sp = add2(o, pack2(sample_dy<S>(k), sample_dx<S>(k)));  // exact
        float a, b, e0, e1, e2;
        unpack2(mul2(v0, add2(sp, m0)), a, b);
        e0 = a - b;
        unpack2(mul2(v1, add2(sp, m1)), a, b);
        e1 = a - b;
        unpack2(mul2(v2, add2(sp, m2)), a, b);
        e2 = a - b;
        const float e = fminf(fminf(e0, e1), e2);
        c.mask |= (e > 0.0f) ? 1u << k : 0u;
        exact |= e == 0.0f;
        const float b0 = __saturatef(e1 * inv), b1 = __saturatef(e2 * inv);
        const float b2 = __saturatef(1.0f - b0 - b1);
        c.z[k] = b0 * z0 + b1 * z1 + b2 * z2;
    }
    if (exact) c = cover_exact<S>(p0x, p0y, p1x, p1y, p2x, p2y, z0, z1, z2, fx, fy);
    return c;
}

// Fragment::interpolate's sample-point choice (src/rasterizer/mod.rs:70-83): pixel centre
// when every sample passed the depth test, else the first passed sample. The offsets, in eighths
// of a pixel, come from a nibble per depth mask; a float of 2^20 + n has steps of 1/8, so the
// position is exact for pixels below 2^20.
template <int S>
__device__ __forceinline__ void interp_point(uint32_t x, uint32_t y, uint32_t dm, float& xs,
                                             float& ys) {
    // nibble dm: 8 x the offset of sample ffs(dm) - 1 (5, 7, 3, 1 across and 1, 5, 7, 3 down),
    // 4 for dm = 15; one sample: always the centre
    const uint32_t dx = S == 1 ? 4u : (uint32_t)(0x4753575157535750ull >> (4 * dm)) & 0xFu;
    const uint32_t dy = S == 1 ? 4u : (uint32_t)(0x4517151315171510ull >> (4 * dm)) & 0xFu;
    xs = __uint_as_float(0x49800000u + 8u * x + dx) - 1048576.0f;
    ys = __uint_as_float(0x49800000u + 8u * y + dy) - 1048576.0f;
}

// Perspective-correct barycentrics of Fragment::interpolate (src/rasterizer/mod.rs:85-94) at
// (xs, ys). The edge values are cover_pixel's form, and clamp01_nan may turn a -0 weight into
// +0: the sign of a zero edge value or weight reaches no colour (a sum of zeros divides to NaN
// either way, and a zero product only changes the sign of a zero texture coordinate or channel).
__device__ __forceinline__ void persp_bary(float p0x, float p0y, float p1x, float p1y, float p2x, float p2y,
                                           float w0, float w1, float w2, float xs, float ys, float& u, float& v,
                                           float& w) {
    const f32x2 sp = pack2(ys, xs);
    float a, b;
    unpack2(mul2(pack2(p1x - p0x, p1y - p0y), add2(sp, pack2(-p0y, -p0x))), a, b);
    const float e0 = a - b;
    unpack2(mul2(pack2(p2x - p1x, p2y - p1y), add2(sp, pack2(-p1y, -p1x))), a, b);
    const float e1 = a - b;
    unpack2(mul2(pack2(p0x - p2x, p0y - p2y), add2(sp, pack2(-p2y, -p2x))), a, b);
    const float e2 = a - b;
    const float fu = e1 / w0;
    const float fv = e2 / w1;
    const float fw = e0 / w2;
    const float sum = fu + fv + fw;
    u = clamp01_nan(fu / sum);
    v = clamp01_nan(fv / sum);
    w = clamp01_nan(1.0f - u - v);
}

// ------------------------------------------------------------------ texture / colour

// Texture::read_texel (src/texture.rs:47-63) on a u32-per-texel RGBA8 image. The flat byte
// index wraps like a release build; a start past the buffer (where the reference panics)
// flags *oob and reads texel 0. Returns the texel word (byte 0 = red).
__device__ __forceinline__ uint32_t read_texel(const uint32_t* __restrict__ tex, uint32_t tw,
                                               uint32_t th, uint64_t x, uint64_t y, bool& oob) {
    uint64_t start = x * 4u + y * 4u * (uint64_t)tw;
    uint64_t len = (uint64_t)tw * (uint64_t)th * 4u;
    if (start >= len) {
        oob = true;
        start = 0;
    }
    return __ldg(tex + (start >> 2));
}

// Color::to_argb (src/color.rs:15-20): saturating casts, OR-combined u32 shifts.
__device__ __forceinline__ uint32_t to_argb(float r, float g, float b, float a) {
    return (sat_u32(a * 255.0f) << 24) | (sat_u32(r * 255.0f) << 16) |
           (sat_u32(g * 255.0f) << 8) | sat_u32(b * 255.0f);
}

// Texture::sample (src/texture.rs:65-83): manual f32 bilinear filter, for any texture
// coordinate. Color::from_rgba (src/color.rs:22-29) divides each byte by 255.
__device__ __forceinline__ void tex_sample(const uint32_t* __restrict__ tex, uint32_t tw,
                                           uint32_t th, float u, float v, float out[4], bool& oob) {
    const float x = u * (float)(uint64_t)(tw - 1);
    const float y = v * (float)(uint64_t)(th - 1);
    const uint64_t xf = sat_u64(floorf(x)), xc = sat_u64(ceilf(x));
    const uint64_t yf = sat_u64(floorf(y)), yc = sat_u64(ceilf(y));
    const uint32_t tl = read_texel(tex, tw, th, xf, yf, oob);
    const uint32_t tr = read_texel(tex, tw, th, xc, yf, oob);
    const uint32_t bl = read_texel(tex, tw, th, xf, yc, oob);
    const uint32_t br = read_texel(tex, tw, th, xc, yc, oob);
    const float x_f = x - truncf(x);
    const float y_f = y - truncf(y);
    const float omx = 1.0f - x_f, omy = 1.0f - y_f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float ctl = (float)((tl >> (8 * k)) & 0xFFu) / 255.0f;
        const float ctr = (float)((tr >> (8 * k)) & 0xFFu) / 255.0f;
        const float cbl = (float)((bl >> (8 * k)) & 0xFFu) / 255.0f;
        const float cbr = (float)((br >> (8 * k)) & 0xFFu) / 255.0f;
        const float y0 = ctl * omx + ctr * x_f;
        const float y1 = cbl * omx + cbr * x_f;
        out[k] = y0 * omy + y1 * y_f;
    }
}
// tex_sample and to_argb for a fragment outside tex_argb's range (out of line: rare).
__device__ __noinline__ uint32_t tex_argb_any(const uint32_t* __restrict__ tex, uint32_t tw, uint32_t th, float u,
                                              float v, uint32_t& oobc) {
    float c[4];
    bool oob = false;
    tex_sample(tex, tw, th, u, v, c, oob);
    if (oob) ++oobc;
    return to_argb(c[0], c[1], c[2], c[3]);
}

// One channel of two horizontally adjacent texels as binary32: a byte spliced under 2^23 by a
// byte permute, then b / 255 correctly rounded as b hi + RN(b lo), hi + lo = 1/255 to 2^-49
// (equal to the division for all 256 bytes; both channels per packed instruction).
__device__ __forceinline__ f32x2 texel_pair(uint32_t t0, uint32_t t1, uint32_t sel) {
    const f32x2 b = add2(pack2(__uint_as_float(__byte_perm(t0, 0x4B000000u, sel)),
                               __uint_as_float(__byte_perm(t1, 0x4B000000u, sel))),
                         pack2(-8388608.0f, -8388608.0f));
    return fma2(b, pack2(0x1.01p-8f, 0x1.01p-8f), mul2(b, pack2(0x1.010102p-24f, 0x1.010102p-24f)));
}

// Texture::sample and Color::to_argb of one fragment: ARGB with alpha computed only when `alpha`
// is set (the resolve ignores the samples' alpha; only a sample capture shows it), 255 otherwise.
// xmax, ymax = size - 1. Inside the texture (every in-range uv; `small`: both sides below 65536)
// floor and ceil stay below the size, so there is no row wrap or read past the end, and
//   - x + 2^23 rounded down holds floor(x) in its low bits (the coordinate is not negative);
//   - the channels lie in [0, 1 + 2^-21], so channel * 255 + 2^23 rounded down holds the byte;
// no conversion instruction is left, and no shared table is read.
__device__ __forceinline__ uint32_t tex_argb(const uint32_t* __restrict__ tex, uint32_t tw, uint32_t th, float xmax,
                                             float ymax, bool small, float u, float v, bool alpha, uint32_t& oobc) {
    const float x = u * xmax, y = v * ymax;
    if (!(small & (x >= 0.0f) & (y >= 0.0f) & (x <= xmax) & (y <= ymax)))
        return tex_argb_any(tex, tw, th, u, v, oobc);
    const float tx = __fadd_rz(x, 8388608.0f), ty = __fadd_rz(y, 8388608.0f);
    const float x_f = x - (tx - 8388608.0f), y_f = y - (ty - 8388608.0f);
    const uint32_t at = (__float_as_uint(tx) & 0x7FFFFFu) + (__float_as_uint(ty) & 0x7FFFFFu) * tw;
    const uint32_t right = x_f > 0.0f ? 1u : 0u, down = y_f > 0.0f ? tw : 0u;
    const uint32_t tl = __ldg(tex + at), tr = __ldg(tex + (at + right));
    const uint32_t bl = __ldg(tex + (at + down)), br = __ldg(tex + (at + down + right));
    const f32x2 fx = pack2(1.0f - x_f, x_f), fy = pack2(1.0f - y_f, y_f);
    auto channel = [&](uint32_t sel) {
        float a, b, c, d;
        unpack2(mul2(texel_pair(tl, tr, sel), fx), a, b);
        unpack2(mul2(texel_pair(bl, br, sel), fx), c, d);
        unpack2(mul2(pack2(a + b, c + d), fy), a, b);
        return __float_as_uint(__fadd_rz((a + b) * 255.0f, 8388608.0f));
    };
    const uint32_t r = channel(0x7650u), g = channel(0x7651u), b = channel(0x7652u);
    const uint32_t a = alpha ? channel(0x7653u) : 0xFFu;
    return __byte_perm(__byte_perm(b, g, 0x0040u), __byte_perm(r, a, 0x0040u), 0x5410u);
}

// ColorBuffer::box_filter_color (src/rasterizer/buffers.rs:111-125)
template <int S>
__device__ __forceinline__ uint32_t box_filter(const uint32_t* c) {
    uint32_t rs = 0, gs = 0, bs = 0;
#pragma unroll
    for (int i = 0; i < S; ++i) {
        rs += (c[i] & 0x00FF0000u) >> 16;
        gs += (c[i] & 0x0000FF00u) >> 8;
        bs += c[i] & 0x000000FFu;
    }
    return (0xFFu << 24) | (rs / (uint32_t)S) << 16 | (gs / (uint32_t)S) << 8 | (bs / (uint32_t)S);
}

}  // namespace rast
