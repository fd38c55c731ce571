// rast_kernels.cu - sm_103a kernels of the raster pipeline.
//
//   k_vertex       per vertex: MVP * v, divide, viewport; one word for binning  (HBM-bound)
//   k_bin_count    per chunk of triangles: classify, tile rectangle, per-chunk tile histogram
//                  in shared memory (band by band for frames of more than 16384 bins)
//   k_clip         one warp per triangle that straddles a clip plane: clip, fan boxes, counts
//   k_scan_cols    per tile: exclusive prefix of the histograms over chunks; per 32 tiles: their bin
//                  ranges, capacity check, and their places in the raster tile queue
//   k_bin_scatter  per chunk: order-preserving scatter of triangle ids into tile bins
//   k_front, k_bin_gather   in place of all these when every frame is small
//   k_bin_split    per 32-pixel bin: its entries split into four 16-pixel quadrant lists
//   k_raster<S,TS> per raster tile, a CTA of 4 warps: replays the tile's triangles in
//                  submission order with all colour/depth samples in shared memory; coverage,
//                  depth test, perspective-correct interpolation, fragment shader, resolve
//   k_raster_warp  the same with one warp per raster tile, for light tiles
//                  (rast_raster_warp.cuh)
//
// No kernel waits on another CTA; every loop is bounded by sizes read from descriptors.
#include <cuda_runtime.h>

#include <atomic>
#include <cstddef>
#include <cstdint>
#include <mutex>

#include "rast_device.cuh"
#include "rast_kernels.h"

namespace rast {

// ===================================================================== helpers

__device__ __forceinline__ unsigned long long pack_rect(uint32_t x0, uint32_t y0, uint32_t x1,
                                                        uint32_t y1) {
    return (unsigned long long)x0 | ((unsigned long long)y0 << 16) |
           ((unsigned long long)x1 << 32) | ((unsigned long long)y1 << 48);
}
__device__ __forceinline__ void unpack_rect(unsigned long long r, uint32_t& x0, uint32_t& y0,
                                            uint32_t& x1, uint32_t& y1) {
    x0 = (uint32_t)(r & 0xFFFFu);
    y0 = (uint32_t)((r >> 16) & 0xFFFFu);
    x1 = (uint32_t)((r >> 32) & 0xFFFFu);
    y1 = (uint32_t)((r >> 48) & 0xFFFFu);
}
// Tile rectangle (inclusive) of a pixel box (inclusive) for tiles of edge ts (a power of two).
__device__ __forceinline__ void tile_rect(unsigned long long r, uint32_t ts, uint32_t& x0, uint32_t& y0,
                                          uint32_t& x1, uint32_t& y1) {
    unpack_rect(r, x0, y0, x1, y1);
    const uint32_t sh = __ffs(ts) - 1;
    x0 >>= sh;
    y0 >>= sh;
    x1 >>= sh;
    y1 >>= sh;
}
__device__ __forceinline__ uint32_t rect_tiles(unsigned long long r, uint32_t ts) {
    if (r == kRectEmpty) return 0;
    uint32_t x0, y0, x1, y1;
    tile_rect(r, ts, x0, y0, x1, y1);
    return (x1 - x0 + 1) * (y1 - y0 + 1);
}
// Bin entry of a triangle for tile (tx, ty): triangle << 5 | clipped << 4 | the raster
// quadrants of the tile that the triangle's pixel box r touches (bit sy * nsx + sx; a single
// bit when nsx == 1).
__device__ __forceinline__ uint32_t bin_entry(uint32_t tri, bool clipped, unsigned long long r, uint32_t tx,
                                              uint32_t ty, uint32_t ts) {
    const uint32_t head = (tri << kEntShift) | (clipped ? kEntClipped : 0u);
    const uint32_t rs = (uint32_t)raster_edge((int)ts);
    if (rs == ts) return head | 1u;
    uint32_t px0, py0, px1, py1;
    unpack_rect(r, px0, py0, px1, py1);
    const uint32_t ox = tx * ts, oy = ty * ts, rsh = __ffs(rs) - 1, nsx = ts >> rsh;
    const uint32_t sx0 = (max(px0, ox) - ox) >> rsh, sx1 = (min(px1, ox + ts - 1) - ox) >> rsh;
    const uint32_t sy0 = (max(py0, oy) - oy) >> rsh, sy1 = (min(py1, oy + ts - 1) - oy) >> rsh;
    const uint32_t xm = (2u << sx1) - (1u << sx0);  // quadrant columns sx0 .. sx1
    uint32_t m = 0;
    for (uint32_t sy = sy0; sy <= sy1; ++sy) m |= xm << (sy * nsx);
    return head | m;
}

// Programmatic dependent launch: wait until the grid launched before this one in the stream has
// completed and its memory is visible (a no-op for a normal launch), then let the next grid's
// CTAs be scheduled once every CTA of this one is running. First statement of every pipeline
// kernel, so that no kernel finishes before its predecessor has.
__device__ __forceinline__ void pdl_enter() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

__device__ __forceinline__ uint32_t lane_id() { return threadIdx.x & 31u; }
__device__ __forceinline__ uint32_t lanemask_lt() { return (1u << lane_id()) - 1u; }

// Block-wide exclusive scan of one u32 per thread (blockDim.x <= 1024). `tmp` holds 33 words.
template <bool kTrailingBarrier = true>
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t* tmp, uint32_t& total) {
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    if (lane == 31) tmp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < nw ? tmp[lane] : 0u;
        uint32_t s = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xFFFFFFFFu, s, o);
            if (lane >= (uint32_t)o) s += y;
        }
        tmp[lane] = s - w;
        if (lane == 31) tmp[32] = s;
    }
    __syncthreads();
    uint32_t r = tmp[warp] + x - v;
    total = tmp[32];
    // without it, the caller must pass a barrier before tmp is written again
    if (kTrailingBarrier) __syncthreads();
    return r;
}

// ===================================================================== vertex stage

// vertex shader P*V*W*v (upstream src/main.rs:147-152) with MVP folded on the host in the
// same dot order; Mat4 * Vec4 is src/math/vector.rs:219-240
__device__ __forceinline__ float4 vertex_clip(const DrawDev& d, uint32_t v) {
    const float x = __ldg(d.pos + 3ull * v), y = __ldg(d.pos + 3ull * v + 1), z = __ldg(d.pos + 3ull * v + 2);
    return make_float4(dot4(d.mvp + 0, x, y, z, 1.0f), dot4(d.mvp + 4, x, y, z, 1.0f),
                       dot4(d.mvp + 8, x, y, z, 1.0f), dot4(d.mvp + 12, x, y, z, 1.0f));
}

// What binning reads of a vertex, one 16-byte word: clip-space x and y and the screen point. A vertex
// outside some clip plane (or with a NaN) carries its clip predicates in a NaN instead of clip x: a
// vertex inside all six planes never has a NaN there. Three loads per triangle instead of nine (clip
// position, screen point and predicates apart): on the 2M-triangle terrain k_bin_count 30.6 -> 24.5 us.
constexpr uint32_t kVbinTag = 0x7FC00000u;
__device__ __forceinline__ float4 vertex_bin(float4 c, float4 sc) {
    const uint32_t code = clip_code(c);
    return make_float4((code & kInsideAll) == kInsideAll ? c.x : __uint_as_float(kVbinTag | code), c.y, sc.x, sc.y);
}

__global__ void __launch_bounds__(256) k_vertex(const DrawDev* __restrict__ draws,
                                                const FrameDev* __restrict__ frames,
                                                const uint2* __restrict__ vblocks, Scratch s) {
    pdl_enter();
    const uint2 vb = vblocks[blockIdx.x];
    const DrawDev& d = draws[vb.x];
    const uint32_t v = vb.y + threadIdx.x;
    if (v >= d.nverts) return;
    const FrameDev& f = frames[d.frame];
    const float4 c = vertex_clip(d, v);
    const float4 sc = to_screen(c, (float)f.width, (float)f.height);
    s.vbin[d.vbase + v] = vertex_bin(c, sc);
    s.vscr[d.vbase + v] = sc;
}

// ===================================================================== triangle classify

// try_clip + divide + viewport + bounding box for one triangle (src/rasterizer/mod.rs:425-441).
// Returns its pixel box (kRectEmpty when nothing can be covered) and, for a clipped
// triangle, the offset of its polygon in the clip store.
__device__ void classify_triangle(const DrawDev& d, const FrameDev& f, uint32_t di, uint32_t tri, uint32_t row,
                                  const Scratch& s, unsigned long long& rect, uint32_t& aux) {
    rect = kRectEmpty;
    aux = kNone;
    const uint32_t i0 = __ldg(d.idx + 3ull * tri), i1 = __ldg(d.idx + 3ull * tri + 1),
                   i2 = __ldg(d.idx + 3ull * tri + 2);
    // primitive_assembly indexes the vertex list (src/render.rs:75-96) and panics past its end;
    // here the triangle is skipped and the frame reports an invalid argument
    if (i0 >= d.nverts || i1 >= d.nverts || i2 >= d.nverts) {
        atomicOr(s.status, ST_BAD_INDEX);
        return;
    }
    const float4 b0 = s.vbin[d.vbase + i0], b1 = s.vbin[d.vbase + i1], b2 = s.vbin[d.vbase + i2];
    if (isnan(b0.x) || isnan(b1.x) || isnan(b2.x)) {
        auto code = [](float4 b) { return isnan(b.x) ? __float_as_uint(b.x) & 0xFFFu : kInsideAll; };
        if (code(b0) & code(b1) & code(b2) & 0xFC0u) return;  // all outside one plane
        const float4 c0 = vertex_clip(d, i0), c1 = vertex_clip(d, i1), c2 = vertex_clip(d, i2);
        if (fabsf(tri2x_area(c0.x, c0.y, c1.x, c1.y, c2.x, c2.y)) < kCullEps) return;
        // straddles a clip plane: queued for k_clip, which clips it with one warp and adds its
        // tiles to this chunk's counts
        const uint32_t slot = atomicAdd(s.clip_n, 1u);
        if (slot < s.clip_list_cap) {
            uint32_t* L = s.clip_list + 3ull * slot;
            L[0] = di;
            L[1] = tri;
            L[2] = row;
        } else {
            atomicOr(s.status, ST_CLIP_STORE_OVERFLOW);
        }
        return;
    }
    // inside all planes (clip_classify)
    if (fabsf(tri2x_area(b0.x, b0.y, b1.x, b1.y, b2.x, b2.y)) < kCullEps) return;
    uint32_t bx0, bx1, by0, by1;
    const float4 sv[3] = {make_float4(b0.z, b0.w, 0.0f, 0.0f), make_float4(b1.z, b1.w, 0.0f, 0.0f),
                          make_float4(b2.z, b2.w, 0.0f, 0.0f)};
    pixel_bbox(sv, f.width, f.height, bx0, bx1, by0, by1);
    if (bx0 >= bx1 || by0 >= by1) return;
    rect = pack_rect(bx0, by0, bx1 - 1, by1 - 1);
}

// Sutherland-Hodgman against the six clip planes in CLIP_PLANES order
// (src/rasterizer/clipping.rs:113-177) with the polygon spread over a warp: lane i holds
// vertex i. Per plane every lane looks at its edge (previous vertex -> its vertex) and emits
// nothing, the intersection, its vertex, or both, in the reference's order; an exclusive scan
// of the emit counts places them. A plane every vertex is inside leaves the polygon as it is.
// Returns the new vertex count, or -1 past 32 vertices. Called by a whole warp.
__device__ __forceinline__ int warp_clip(ClipVert& v, int cn) {
    const uint32_t lane = lane_id();
    for (int plane = 0; plane < 6; ++plane) {
        const bool live = lane < (uint32_t)cn;
        const float dc = live ? distance_measure(plane, v.p) : 0.0f;
        const bool cin = dc >= 0.0f;
        if (__all_sync(0xFFFFFFFFu, !live || cin)) continue;
        const uint32_t prev = live ? (lane + (uint32_t)cn - 1u) % (uint32_t)cn : lane;
        ClipVert pv;
#pragma unroll
        for (int k = 0; k < 4; ++k) pv.p[k] = __shfl_sync(0xFFFFFFFFu, v.p[k], prev);
#pragma unroll
        for (int k = 0; k < 6; ++k) pv.a[k] = __shfl_sync(0xFFFFFFFFu, v.a[k], prev);
        const float dp = __shfl_sync(0xFFFFFFFFu, dc, prev);
        const bool pin = dp >= 0.0f;
        uint32_t emit = 0;
        if (live) emit = (pin && cin) ? 1u : (pin && !cin) ? 1u : (!pin && cin) ? 2u : 0u;
        ClipVert first = v;  // both inside: the vertex itself
        if (live && pin != cin) clip_intersect(pv, dp, v, dc, first);
        uint32_t incl = emit;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= (uint32_t)o) incl += y;
        }
        const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
        if (total > (uint32_t)kMaxPoly) return -1;
        // new vertex `lane`: emitted by the lane whose inclusive count first exceeds it
        uint32_t src = 0;
#pragma unroll
        for (int st = 16; st > 0; st >>= 1) {
            const uint32_t c = __shfl_sync(0xFFFFFFFFu, incl, src + st - 1);
            if (c <= lane) src += st;
        }
        src = min(src, 31u);
        const uint32_t second = lane - (__shfl_sync(0xFFFFFFFFu, incl, src) - __shfl_sync(0xFFFFFFFFu, emit, src));
        ClipVert nv;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float a = __shfl_sync(0xFFFFFFFFu, first.p[k], src), b = __shfl_sync(0xFFFFFFFFu, v.p[k], src);
            nv.p[k] = second ? b : a;
        }
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            const float a = __shfl_sync(0xFFFFFFFFu, first.a[k], src), b = __shfl_sync(0xFFFFFFFFu, v.a[k], src);
            nv.a[k] = second ? b : a;
        }
        v = nv;
        cn = (int)total;
        if (cn == 0) break;
    }
    return cn;
}

// Clips one straddling triangle with a whole warp: lane q < 3 holds vertex index vi and clip-space
// position c of corner q. The polygon goes to the clip store in screen space (to_screen per vertex, as
// the reference divides and maps the fan's triangles, src/rasterizer/mod.rs:425-441); the union
// of the fan's pixel boxes (clipping.rs:185-190) is the triangle's box. Returns the box
// (kRectEmpty when nothing can be covered) and the polygon's offset, the same in every lane.
__device__ __forceinline__ unsigned long long clip_triangle(const DrawDev& d, const FrameDev& f, const Scratch& s,
                                                            uint32_t vi, float4 c, uint32_t& off32) {
    const uint32_t lane = lane_id();
    ClipVert v;
    if (lane < 3) {
        v.p[0] = c.x;
        v.p[1] = c.y;
        v.p[2] = c.z;
        v.p[3] = c.w;
#pragma unroll
        for (int q = 0; q < 4; ++q) v.a[q] = d.rgba ? __ldg(d.rgba + 4ull * vi + q) : 0.0f;
        v.a[4] = __ldg(d.uv + 2ull * vi);
        v.a[5] = __ldg(d.uv + 2ull * vi + 1);
    } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) v.p[k] = 0.0f;
#pragma unroll
        for (int k = 0; k < 6; ++k) v.a[k] = 0.0f;
    }
    const int n = warp_clip(v, 3);
    if (n < 0) {
        if (lane == 0) atomicOr(s.status, ST_CLIP_OVERFLOW);
        return kRectEmpty;
    }
    if (n < 3) return kRectEmpty;
    const unsigned long long need = 1ull + 10ull * (unsigned long long)n;
    unsigned long long off = 0;
    if (lane == 0) off = atomicAdd(s.clip_used, need);
    off = __shfl_sync(0xFFFFFFFFu, off, 0);
    if (off + need > s.clip_cap) {
        if (lane == 0) atomicOr(s.status, ST_CLIP_STORE_OVERFLOW);
        return kRectEmpty;
    }
    float* st = s.clip_store + off;
    const float4 sc = to_screen(make_float4(v.p[0], v.p[1], v.p[2], v.p[3]), (float)f.width, (float)f.height);
    if (lane == 0) st[0] = __int_as_float(n);
    if (lane < (uint32_t)n) {
        float* o = st + 1 + 10 * lane;
        o[0] = sc.x;
        o[1] = sc.y;
        o[2] = sc.z;
        o[3] = sc.w;
#pragma unroll
        for (int q = 0; q < 6; ++q) o[4 + q] = v.a[q];
    }
    // fan triangle `lane`: vertices 0, lane + 1, lane + 2
    float4 tv[3];
    tv[0] = make_float4(__shfl_sync(0xFFFFFFFFu, sc.x, 0), __shfl_sync(0xFFFFFFFFu, sc.y, 0),
                        __shfl_sync(0xFFFFFFFFu, sc.z, 0), __shfl_sync(0xFFFFFFFFu, sc.w, 0));
    const uint32_t l1 = min(lane + 1, 31u), l2 = min(lane + 2, 31u);
    tv[1] = make_float4(__shfl_sync(0xFFFFFFFFu, sc.x, l1), __shfl_sync(0xFFFFFFFFu, sc.y, l1),
                        __shfl_sync(0xFFFFFFFFu, sc.z, l1), __shfl_sync(0xFFFFFFFFu, sc.w, l1));
    tv[2] = make_float4(__shfl_sync(0xFFFFFFFFu, sc.x, l2), __shfl_sync(0xFFFFFFFFu, sc.y, l2),
                        __shfl_sync(0xFFFFFFFFu, sc.z, l2), __shfl_sync(0xFFFFFFFFu, sc.w, l2));
    uint32_t a0 = 0xFFFFFFFFu, a1 = 0, b0 = 0xFFFFFFFFu, b1 = 0;
    if (lane + 2 < (uint32_t)n) {
        uint32_t x0, x1, y0, y1;
        pixel_bbox(tv, f.width, f.height, x0, x1, y0, y1);
        if (x0 < x1 && y0 < y1) {
            a0 = x0;
            a1 = x1;
            b0 = y0;
            b1 = y1;
        }
    }
    a0 = __reduce_min_sync(0xFFFFFFFFu, a0);
    a1 = __reduce_max_sync(0xFFFFFFFFu, a1);
    b0 = __reduce_min_sync(0xFFFFFFFFu, b0);
    b1 = __reduce_max_sync(0xFFFFFFFFu, b1);
    off32 = (uint32_t)off;
    return a0 < a1 && b0 < b1 ? pack_rect(a0, b0, a1 - 1, b1 - 1) : kRectEmpty;
}

// Clips the queued straddling triangles, one warp per triangle (grid-stride over the queue), and
// adds their tiles to their chunks' counts.
__global__ void __launch_bounds__(256) k_clip(const DrawDev* __restrict__ draws,
                                              const FrameDev* __restrict__ frames, Scratch s) {
    pdl_enter();
    const uint32_t lane = lane_id();
    const uint32_t nq = min(*(volatile unsigned int*)s.clip_n, (unsigned int)s.clip_list_cap);
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t e = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; e < nq; e += nwarps) {
        const uint32_t di = s.clip_list[3ull * e], tri = s.clip_list[3ull * e + 1], row = s.clip_list[3ull * e + 2];
        const DrawDev& d = draws[di];
        const FrameDev& f = frames[d.frame];
        uint32_t vi = 0, off = 0;
        float4 c = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (lane < 3) {
            vi = __ldg(d.idx + 3ull * tri + lane);
            c = vertex_clip(d, vi);
        }
        const unsigned long long rect = clip_triangle(d, f, s, vi, c, off);
        if (rect == kRectEmpty) continue;
        const uint32_t g = f.rect_base + d.tbase + tri;
        if (lane == 0) {
            s.tri_rect[g] = rect | kRectClippedBit;
            s.tri_aux[g] = off;
        }
        uint32_t x0, y0, x1, y1;
        tile_rect(rect, (uint32_t)f.ts, x0, y0, x1, y1);
        const uint32_t w = x1 - x0 + 1, nt = (y1 - y0 + 1) * w;
        uint32_t* crow = s.counts + f.count_base + (unsigned long long)row * f.ntiles;
        for (uint32_t k = lane; k < nt; k += 32) atomicAdd(&crow[(y0 + k / w) * f.tiles_x + x0 + k % w], 1u);
    }
}

// ===================================================================== binning: count

__global__ void __launch_bounds__(256, 6) k_bin_count(const ChunkDev* __restrict__ chunks,
                                                   const DrawDev* __restrict__ draws,
                                                   const FrameDev* __restrict__ frames,
                                                   Scratch s) {
    pdl_enter();
    // per-bin counts of the chunk, two 16-bit counters per word (bin t in half t & 1 of word
    // t / 2): a chunk holds at most 8192 triangles, so no counter carries into its neighbour,
    // and the histogram of kCountBandTiles = 16384 bins takes 32 KB (6 CTAs per SM by registers: with
    // 8 a frame of the 2M-triangle terrain takes 1% longer). Frames with more bins are counted band
    // by band: the first pass classifies the triangles and stores their boxes, later passes read the boxes back and
    // count the bins of their band (rows of the box outside the band are skipped).
    extern __shared__ uint32_t hist[];
    const ChunkDev ch = chunks[blockIdx.x];
    const DrawDev& d = draws[ch.draw];
    const FrameDev& f = frames[d.frame];
    const uint32_t nt = f.ntiles, tx = f.tiles_x;
    uint32_t* row = s.counts + f.count_base + (unsigned long long)ch.row * nt;
    for (uint32_t b0 = 0; b0 < nt; b0 += (uint32_t)kCountBandTiles) {
        const uint32_t b1 = min(nt, b0 + (uint32_t)kCountBandTiles);
        for (uint32_t t = threadIdx.x; t < (b1 - b0 + 1) / 2; t += blockDim.x) hist[t] = 0;
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < ch.tri_count; i += blockDim.x) {
            const uint32_t tri = ch.tri_begin + i;
            const uint32_t g = f.rect_base + d.tbase + tri;
            unsigned long long rect;
            if (b0 == 0) {
                uint32_t aux;
                classify_triangle(d, f, ch.draw, tri, ch.row, s, rect, aux);
                s.tri_rect[g] = rect;
                s.tri_aux[g] = aux;
            } else {
                rect = s.tri_rect[g];  // stored by this thread in the first pass
            }
            if (rect != kRectEmpty) {
                uint32_t x0, y0, x1, y1;
                tile_rect(rect, (uint32_t)f.ts, x0, y0, x1, y1);
                if (nt <= (uint32_t)kCountBandTiles) {  // one band: every bin of the box counts
                    for (uint32_t y = y0; y <= y1; ++y)
                        for (uint32_t x = x0; x <= x1; ++x) {
                            const uint32_t t = y * tx + x;
                            atomicAdd(&hist[t >> 1], (t & 1u) ? 0x10000u : 1u);
                        }
                } else {
                    // rows of the box whose bins can fall in [b0, b1)
                    const uint32_t ya = max(y0, b0 / tx), yb = min(y1, (b1 - 1) / tx);
                    for (uint32_t y = ya; y <= yb; ++y)
                        for (uint32_t x = x0; x <= x1; ++x) {
                            const uint32_t t = y * tx + x;
                            if (t >= b0 && t < b1) atomicAdd(&hist[(t - b0) >> 1], ((t - b0) & 1u) ? 0x10000u : 1u);
                        }
                }
            }
        }
        __syncthreads();
        for (uint32_t t = b0 + threadIdx.x; t < b1; t += blockDim.x)
            row[t] = (hist[(t - b0) >> 1] >> (((t - b0) & 1u) * 16u)) & 0xFFFFu;
        if (b1 < nt) __syncthreads();  // the histogram is cleared again for the next band
    }
}

// ===================================================================== binning: scans

// Place of the k-th bin of class c in the group's arrays of n tiles: two classes share an array and
// grow towards each other from its ends.
__device__ __forceinline__ unsigned long long order_slot(uint32_t c, uint32_t k, uint32_t n) {
    return (unsigned long long)(c >> 1) * n + ((c & 1u) ? k : n - 1 - k);
}

// Called by one warp whose lane holds bin t of frame f (live lanes) and its entry count; returns the
// bin's first entry. Allocates
// the bins' ranges in one step (the ranges of a frame lie in no particular order), checks the
// capacity and lists the bins in the raster queue. A prefix over a frame's tiles and a sort
// of them took two one-CTA kernels before (2M-triangle 4K terrain 13 us, 20 scenes 54 us).
__device__ __forceinline__ uint32_t place_bins(const FrameDev& f, uint32_t frame, const Scratch& s, uint32_t t,
                                               bool live, uint32_t count) {
    const uint32_t lane = lane_id();
    uint32_t incl = live ? count : 0u;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= (uint32_t)o) incl += y;
    }
    const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
    // the two allocations are independent: both in flight before either result is used
    const uint32_t c = !live            ? (uint32_t)kClasses
                       : f.order_coarse ? (count ? 1u : 0u)
                                        : order_class(count, f.heavy_bits);
    const uint32_t peers = __match_any_sync(0xFFFFFFFFu, c), leader = __ffs(peers) - 1;
    unsigned long long base = 0;
    uint32_t slot = 0;
    if (lane == 0 && total) base = atomicAdd(&s.frame_need[frame], (unsigned long long)total);
    if (live && lane == leader)
        slot = atomicAdd(&s.queues[kQueueSlots * f.queue + kQueueClass + c], (unsigned)__popc(peers));
    base = __shfl_sync(0xFFFFFFFFu, base, 0);
    slot = __shfl_sync(0xFFFFFFFFu, slot, leader) + __popc(peers & lanemask_lt());
    if (lane == 0 && base + total > f.bin_cap) atomicOr(s.status, ST_BIN_OVERFLOW);
    if (live) {
        const uint32_t gt = f.tile_begin + t;
        s.tile_count[gt] = count;
        s.tile_start[gt] = (uint32_t)base + incl - count;
        s.tile_order[(unsigned long long)kOrderArrays * f.order_begin + order_slot(c, slot, f.order_n)] = gt;
    }
    return (uint32_t)base + incl - count;
}

// One block per 32-tile group of a frame; 32 segments of chunks per tile: the exclusive prefix of
// each tile's counts over the chunks, then the tiles' bin ranges (place_bins).
__global__ void __launch_bounds__(1024) k_scan_cols(const FrameDev* __restrict__ frames,
                                                    int nframes, Scratch s) {
    pdl_enter();
    __shared__ uint32_t part[32][33];
    __shared__ int s_frame;
    if (threadIdx.x == 0) {
        int lo = 0, hi = nframes;
        while (hi - lo > 1) {
            int mid = (lo + hi) >> 1;
            if (frames[mid].group_begin <= blockIdx.x) lo = mid; else hi = mid;
        }
        s_frame = lo;
    }
    __syncthreads();
    const FrameDev& f = frames[s_frame];
    const uint32_t tl = threadIdx.x & 31u, seg = threadIdx.x >> 5;
    const uint32_t t = (blockIdx.x - f.group_begin) * 32u + tl;
    const uint32_t R = f.nchunks, nt = f.ntiles;
    const uint32_t r0 = (uint32_t)((unsigned long long)R * seg / 32u);
    const uint32_t r1 = (uint32_t)((unsigned long long)R * (seg + 1) / 32u);
    uint32_t* base = s.counts + f.count_base;
    uint32_t sum = 0;
    if (t < nt)
        for (uint32_t r = r0; r < r1; ++r) sum += base[(unsigned long long)r * nt + t];
    part[seg][tl] = sum;
    __syncthreads();
    uint32_t count = 0;
    if (seg == 0) {
        for (int k = 0; k < 32; ++k) {
            uint32_t c = part[k][tl];
            part[k][tl] = count;
            count += c;
        }
    }
    __syncthreads();
    if (seg == 0) place_bins(f, (uint32_t)s_frame, s, t, t < nt, count);
    if (t < nt) {
        uint32_t run = part[seg][tl];
        for (uint32_t r = r0; r < r1; ++r) {
            uint32_t* p = &base[(unsigned long long)r * nt + t];
            const uint32_t c = *p;
            // the scatter reads a chunk's offset only for bins the chunk has entries in: empty
            // cells keep their 0 (most of the matrix for dense meshes) and are not written
            if (c) *p = run;
            run += c;
        }
    }
}

// ===================================================================== binning: scatter

constexpr int kScatterThreads = 256;
constexpr int kScatterWarps = kScatterThreads / 32;
constexpr int kScatterTriPerThread = 2;
constexpr int kScatterWindow = kScatterThreads * kScatterTriPerThread;  // triangles per batch
constexpr int kPairsPerBatch = 512;  // (triangle, tile) pairs ranked per batch
constexpr uint32_t kBigTri = 32;     // triangles over more tiles are binned alone, tile-parallel
constexpr int kHashSlots = 1024;     // open-addressing table over tile ids, load <= 0.5
constexpr uint32_t kHashEmpty = 0xFFFFFFFFu;

__device__ __forceinline__ uint32_t hash_slot(uint32_t t) {
    return (t * 2654435761u) >> (32 - 10);
}

// Bins the (triangle, tile) pairs of a chunk in submission order. Per batch of up to
// kScatterWindow triangles (two consecutive ones per thread, so each warp holds a contiguous
// run) and kPairsPerBatch pairs, every warp walks its pairs 32 at a time: lanes with the same
// tile (match_any) take consecutive ranks from the warp's counter for that tile (wcnt, found
// through a small hash of the batch's tiles). A pair's position is then the tile's running
// offset + the counts of the earlier warps + its rank in its warp. A triangle over more than
// kBigTri tiles ends a batch and is binned alone, tile-parallel.
__global__ void __launch_bounds__(kScatterThreads) k_bin_scatter(
    const ChunkDev* __restrict__ chunks, const DrawDev* __restrict__ draws,
    const FrameDev* __restrict__ frames, Scratch s) {
    pdl_enter();
    __shared__ uint32_t hkey[kHashSlots];
    __shared__ uint16_t wcnt[kHashSlots][kScatterWarps];
    __shared__ uint16_t slot_list[kPairsPerBatch];
    __shared__ uint32_t pxy[kPairsPerBatch];  // tile x | tile y << 16
    __shared__ uint16_t pslot[kPairsPerBatch], prank[kPairsPerBatch];
    __shared__ uint16_t ptri[kPairsPerBatch];
    __shared__ unsigned long long trect[kScatterWindow];  // pixel box, bit 63: clipped
    __shared__ uint32_t sbase[kHashSlots];  // per slot: the tile's position before the batch
    __shared__ uint32_t nslots, take_s, npairs_s;
    __shared__ uint32_t tmp[33];
    if (*(volatile uint32_t*)s.status & ST_BIN_OVERFLOW) return;
    const ChunkDev ch = chunks[blockIdx.x];
    const DrawDev& d = draws[ch.draw];
    const FrameDev& f = frames[d.frame];
    const uint32_t nt = f.ntiles, tx = f.tiles_x, ts = (uint32_t)f.ts;
    // the chunk's row of scanned counts: its offset within each tile's list, advanced in place
    // as the chunk's entries are placed (the row is the chunk's own and dead after this
    // kernel); the chunk's next position in tile t is tile_start[t] + crow[t]
    uint32_t* crow = s.counts + f.count_base + (unsigned long long)ch.row * nt;
    const uint32_t* tstart = s.tile_start + f.tile_begin;
    for (uint32_t h = threadIdx.x; h < (uint32_t)kHashSlots; h += blockDim.x) {
        hkey[h] = kHashEmpty;
#pragma unroll
        for (int w = 0; w < kScatterWarps; ++w) wcnt[h][w] = 0;
    }
    if (threadIdx.x == 0) nslots = 0;
    __syncthreads();
    uint32_t* bins = s.bins + f.bin_base;
    const unsigned long long cap = f.bin_cap;
    const uint32_t gbase = f.rect_base + d.tbase + ch.tri_begin;
    const uint32_t fbase = d.tbase + ch.tri_begin;  // frame triangle index of the chunk's first
    const uint32_t warp = threadIdx.x >> 5, lane = lane_id();
    uint32_t base = 0;
    while (base < ch.tri_count) {
        // ---- this thread's two triangles: pixel boxes, clipped flags, tile counts
        unsigned long long r[kScatterTriPerThread];
        uint32_t n[kScatterTriPerThread];
        uint32_t mine = 0;
#pragma unroll
        for (int j = 0; j < kScatterTriPerThread; ++j) {
            const uint32_t v = threadIdx.x * kScatterTriPerThread + j;
            const uint32_t i = base + v;
            const bool live = i < ch.tri_count;
            r[j] = live ? s.tri_rect[gbase + i] : kRectEmpty;
            n[j] = r[j] == kRectEmpty ? 0u : rect_tiles(r[j] & ~kRectClippedBit, ts);
            trect[v] = r[j];
            mine += n[j];
        }
        if (threadIdx.x == 0) take_s = kScatterWindow;
        uint32_t total;
        const uint32_t excl = block_excl_scan(mine, tmp, total);  // its barriers order take_s
        // the batch: a prefix of the window within the pair budget
        {
            uint32_t run = excl;
#pragma unroll
            for (int j = 0; j < kScatterTriPerThread; ++j) {
                const uint32_t v = threadIdx.x * kScatterTriPerThread + j;
                run += n[j];
                if (run > (uint32_t)kPairsPerBatch || n[j] > kBigTri) {
                    atomicMin(&take_s, v);
                    break;
                }
            }
        }
        __syncthreads();
        uint32_t take = take_s;
        if (take == 0) {
            // a single triangle over more than kBigTri tiles: its tiles are distinct, each
            // takes the next position
            const bool c0 = (trect[0] & kRectClippedBit) != 0;
            const unsigned long long r0 = trect[0] & ~kRectClippedBit;
            uint32_t x0, y0, x1, y1;
            tile_rect(r0, ts, x0, y0, x1, y1);
            const uint32_t w = x1 - x0 + 1, n0 = rect_tiles(r0, ts);
            for (uint32_t k = threadIdx.x; k < n0; k += blockDim.x) {
                const uint32_t ttx = x0 + k % w, tty = y0 + k / w;
                const uint32_t t = tty * tx + ttx;
                const uint32_t pos = tstart[t] + crow[t];
                if (pos < cap) bins[pos] = bin_entry(fbase + base, c0, r0, ttx, tty, ts);
                crow[t] += 1;
            }
            __syncthreads();
            base += 1;
            continue;
        }
        take = min(take, ch.tri_count - base);
        // ---- per warp, its pairs in order, 32 at a time: rank within the warp per tile
        uint32_t pc = 0;  // this thread's pairs in the batch
#pragma unroll
        for (int j = 0; j < kScatterTriPerThread; ++j)
            if (threadIdx.x * kScatterTriPerThread + j < take) pc += n[j];
        uint32_t winc = pc;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, winc, o);
            if (lane >= (uint32_t)o) winc += y;
        }
        const uint32_t wtotal = __shfl_sync(0xFFFFFFFFu, winc, 31);
        const uint32_t wbase = __shfl_sync(0xFFFFFFFFu, excl, 0);  // block index of the warp's first pair
        for (uint32_t rb = 0; rb < wtotal; rb += 32) {
            const uint32_t pi = rb + lane;
            uint32_t sl = 0;
#pragma unroll
            for (int st = 16; st > 0; st >>= 1) {
                const uint32_t v = __shfl_sync(0xFFFFFFFFu, winc, sl + st - 1);
                if (v <= pi) sl += st;
            }
            const uint32_t src = min(sl, 31u);
            const uint32_t o = pi - __shfl_sync(0xFFFFFFFFu, winc - pc, src);
            const uint32_t n0 = __shfl_sync(0xFFFFFFFFu, n[0], src);
            uint32_t key = 0xFFFFFFFFu - lane, v = 0, xy = 0;
            if (pi < wtotal) {
                const uint32_t j = o < n0 ? 0u : 1u, k = o < n0 ? o : o - n0;
                v = (warp * 32 + src) * kScatterTriPerThread + j;
                uint32_t x0, y0, x1, y1;
                tile_rect(trect[v] & ~kRectClippedBit, ts, x0, y0, x1, y1);
                const uint32_t w = x1 - x0 + 1;
                const uint32_t ky = k < w ? 0u : k / w;
                const uint32_t ttx = x0 + (k - ky * w), tty = y0 + ky;
                key = tty * tx + ttx;
                xy = ttx | (tty << 16);
            }
            const uint32_t peers = __match_any_sync(0xFFFFFFFFu, key);
            const uint32_t leader = __ffs(peers) - 1;
            uint32_t slot = 0, old = 0;
            if (pi < wtotal && lane == leader) {
                uint32_t h = hash_slot(key);
                while (true) {
                    const uint32_t prev = atomicCAS(&hkey[h], kHashEmpty, key);
                    if (prev == kHashEmpty) {
                        slot_list[atomicAdd(&nslots, 1u)] = (uint16_t)h;
                        break;
                    }
                    if (prev == key) break;
                    h = (h + 1) & (kHashSlots - 1);
                }
                slot = h;
                old = wcnt[h][warp];
                wcnt[h][warp] = (uint16_t)(old + __popc(peers));
            }
            slot = __shfl_sync(0xFFFFFFFFu, slot, leader);
            old = __shfl_sync(0xFFFFFFFFu, old, leader);
            if (pi < wtotal) {
                const uint32_t bp = wbase + pi;
                pxy[bp] = xy;
                pslot[bp] = (uint16_t)slot;
                prank[bp] = (uint16_t)(old + __popc(peers & lanemask_lt()));
                ptri[bp] = (uint16_t)v;
            }
        }
        {
            const uint32_t t_last = take - 1;  // its thread holds the end of the batch's pairs
            if (threadIdx.x == t_last / kScatterTriPerThread) {
                uint32_t e = excl;
#pragma unroll
                for (int j = 0; j < kScatterTriPerThread; ++j)
                    if (threadIdx.x * kScatterTriPerThread + j < take) e += n[j];
                npairs_s = e;
            }
        }
        __syncthreads();
        // ---- per tile of the batch: its position before the batch, the warps' counts turned
        // into exclusive prefixes, and the chunk's offset advanced past the batch
        const uint32_t ns = nslots, npairs = npairs_s;
        for (uint32_t j = threadIdx.x; j < ns; j += blockDim.x) {
            const uint32_t h = slot_list[j], t = hkey[h];
            const uint32_t c = crow[t];
            const uint32_t b = tstart[t] + c;
            uint32_t tot = 0;
#pragma unroll
            for (int w2 = 0; w2 < kScatterWarps; ++w2) {
                const uint32_t c = wcnt[h][w2];
                wcnt[h][w2] = (uint16_t)tot;
                tot += c;
            }
            sbase[h] = b;
            crow[t] = c + tot;
        }
        __syncthreads();
        // ---- positions: the tile's position + earlier warps' counts + rank in the warp
        for (uint32_t bp = threadIdx.x; bp < npairs; bp += blockDim.x) {
            const uint32_t xy = pxy[bp], slot = pslot[bp], v = ptri[bp];
            const uint32_t pw = v / (32 * kScatterTriPerThread);
            const uint32_t pos = sbase[slot] + wcnt[slot][pw] + prank[bp];
            const unsigned long long rv = trect[v];
            const bool clipped = (rv & kRectClippedBit) != 0;
            if (pos < cap)
                bins[pos] = bin_entry(fbase + base + v, clipped, rv & ~kRectClippedBit, xy & 0xFFFFu, xy >> 16, ts);
        }
        __syncthreads();
        for (uint32_t j = threadIdx.x; j < ns; j += blockDim.x) {
            const uint32_t h = slot_list[j];
#pragma unroll
            for (int w2 = 0; w2 < kScatterWarps; ++w2) wcnt[h][w2] = 0;
            hkey[h] = kHashEmpty;
        }
        if (threadIdx.x == 0) nslots = 0;
        __syncthreads();
        base += take;
    }
}

// ===================================================================== small frames: front, gather
//
// Frames of at most kGatherTris triangles (every frame of the run) skip the chunk histograms, the
// column scan and the scatter: a chunk holds 256 triangles or more, so such a frame has a few chunks
// and the scatter's CTAs, each serial over its triangles, leave the GPU idle; triangles over many bins
// make it worse (12 chunks of large triangles at 1440p: 324 us in the scatter). Here vertices, classification and
// clipping are one launch over as many warps as there are triangles to clip, and the bins are
// filled from the tiles' side: each CTA owns a block of bins and looks at every triangle's box.
// us a frame among others, by chunks -> so: 3 000 triangles of 32-512 pixels at 1440p 724 -> 437, four demo
// objects at 720p 159 -> 42, the cube with readback 93 -> 69, soups (1-64 pixels) of 2 000 at 320x240 60 -> 46 and
// 1080p 84 -> 52, of 8 000 at 1080p 114 -> 92 and 4K 167 -> 161, 64 of them at 640x480 1821 -> 1783. Beyond 8 160
// triangles the boxes no longer fit shared memory, and the chunks begin to fill the GPU. (Thousands of
// triangles of a pixel or two on a small image are what the chunks do better: 7 938 of a terrain at 640x480 33
// against 35 us, at 320x240 43 against 47; of 16-256 pixels there, 505 against 284.)

// The first vertex_blocks CTAs transform 256 vertices each (what the raster reads: screen points); the
// others take a chunk of 8 `per` triangles, `per` (front_tris: 4, or 10 in a run of many) of them to a
// warp: lane 3 t + q transforms corner q of triangle t again from its position (no wait for the
// vertex CTAs), lane t classifies triangle t, and the whole warp clips the ones that straddle a plane, one
// after another. Few triangles per warp, from as many places of the mesh, keep that chain short: a mesh may hold all
// its straddlers in a row (2 000 triangles, 200 straddlers: 13 us with four neighbours per warp, 9 spread).
__global__ void __launch_bounds__(256) k_front(const ChunkDev* __restrict__ chunks,
                                               const DrawDev* __restrict__ draws,
                                               const FrameDev* __restrict__ frames,
                                               const uint2* __restrict__ vblocks, uint32_t vertex_blocks,
                                               uint32_t per, Scratch s) {
    pdl_enter();
    if (blockIdx.x < vertex_blocks) {
        const uint2 vb = vblocks[blockIdx.x];
        const DrawDev& d = draws[vb.x];
        const FrameDev& f = frames[d.frame];
        const uint32_t v = vb.y + threadIdx.x;
        if (v >= d.nverts) return;
        s.vscr[d.vbase + v] = to_screen(vertex_clip(d, v), (float)f.width, (float)f.height);
        return;
    }
    const ChunkDev ch = chunks[blockIdx.x - vertex_blocks];
    const DrawDev& d = draws[ch.draw];
    const FrameDev& f = frames[d.frame];
    const uint32_t lane = lane_id();
    // triangle t of this warp: tri0 + t * nw, nw warps in the draw
    const uint32_t nw = (d.ntris + per - 1) / per;
    const uint32_t tri0 = ch.tri_begin / per + (threadIdx.x >> 5);
    if (tri0 >= nw) return;  // whole warps
    const uint32_t nt = min(per, (d.ntris - tri0 + nw - 1) / nw);
    uint32_t vi = 0, code = 0;
    bool bad = false;
    float4 c = make_float4(0.0f, 0.0f, 0.0f, 0.0f), sc = c;
    if (lane < 3 * nt) {
        vi = __ldg(d.idx + 3ull * (tri0 + lane / 3 * nw) + lane % 3);
        bad = vi >= d.nverts;
        if (!bad) {
            c = vertex_clip(d, vi);
            code = clip_code(c);
            sc = to_screen(c, (float)f.width, (float)f.height);
        }
    }
    const uint32_t bads = __ballot_sync(0xFFFFFFFFu, bad);
    const uint32_t q0 = min(3 * lane, 29u);  // lane t: its corners are lanes 3 t .. 3 t + 2
    float cx[3], cy[3];
    float4 sv[3];
    uint32_t cd[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        cx[q] = __shfl_sync(0xFFFFFFFFu, c.x, q0 + q);
        cy[q] = __shfl_sync(0xFFFFFFFFu, c.y, q0 + q);
        cd[q] = __shfl_sync(0xFFFFFFFFu, code, q0 + q);
        sv[q] = make_float4(__shfl_sync(0xFFFFFFFFu, sc.x, q0 + q), __shfl_sync(0xFFFFFFFFu, sc.y, q0 + q), 0.0f, 0.0f);
    }
    const uint32_t g0 = f.rect_base + d.tbase + tri0;
    // each triangle's words have one writer: lane t here, or lane 0 for a straddler below (nothing in
    // between orders two lanes' stores to one address)
    bool straddles = false;
    if (lane < nt) {
        unsigned long long rect = kRectEmpty;
        if ((bads >> (3 * lane)) & 7u) {
            atomicOr(s.status, ST_BAD_INDEX);  // skipped, as in classify_triangle
        } else {
            const int cls = clip_classify(tri2x_area(cx[0], cy[0], cx[1], cy[1], cx[2], cy[2]), cd[0], cd[1], cd[2]);
            if (cls == 1) {
                uint32_t x0, x1, y0, y1;
                pixel_bbox(sv, f.width, f.height, x0, x1, y0, y1);
                if (x0 < x1 && y0 < y1) rect = pack_rect(x0, y0, x1 - 1, y1 - 1);
            }
            straddles = cls == 2;
        }
        if (!straddles) {
            s.tri_rect[g0 + lane * nw] = rect;
            s.tri_aux[g0 + lane * nw] = kNone;
        }
    }
    for (uint32_t m = __ballot_sync(0xFFFFFFFFu, straddles); m; m &= m - 1) {
        const uint32_t t = __ffs(m) - 1, src = min(3 * t + lane, 31u);
        const uint32_t cvi = __shfl_sync(0xFFFFFFFFu, vi, src);
        const float4 cc = make_float4(__shfl_sync(0xFFFFFFFFu, c.x, src), __shfl_sync(0xFFFFFFFFu, c.y, src),
                                      __shfl_sync(0xFFFFFFFFu, c.z, src), __shfl_sync(0xFFFFFFFFu, c.w, src));
        uint32_t off = 0;
        const unsigned long long rect = clip_triangle(d, f, s, cvi, cc, off);
        if (lane == 0) {
            const bool gone = rect == kRectEmpty;
            s.tri_rect[g0 + t * nw] = gone ? kRectEmpty : rect | kRectClippedBit;
            s.tri_aux[g0 + t * nw] = gone ? kNone : off;
        }
        __syncwarp();
    }
}

constexpr int kGatherThreads = 512;
constexpr int kGatherWarps = kGatherThreads / 32;
static_assert(kGatherWarps == 16, "16 warps share the block's 64 or 16 bins");
static_assert(kGatherTris % 32 == 0 && kGatherTris / 32 < 256, "a lane's entries of a bin fit a byte");

constexpr uint32_t kGatherLong = 256;  // entries of a 4 x 4 block's list from which its warps share it

// k_bin_gather for a block of 4 x 4 bins at (X, Y) with a long list: the warps share the list, each a
// contiguous part, 32 entries at a time. One pass counts per warp and bin (lane q: bin q), the bins'
// ranges are allocated (place_bins), a second pass writes each bin's entries in order; a step of
// either takes the bins that any of its 32 entries touches one after another.
__device__ __forceinline__ void gather_by_list(const FrameDev& f, uint32_t fi, const Scratch& s, uint32_t X, uint32_t Y,
                                               const uint16_t* ltri, const uint16_t* abox, uint32_t total,
                                               uint32_t (*wpos)[32]) {
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    const uint32_t groups = (total + 31) / 32, per = (groups + kGatherWarps - 1) / kGatherWarps;
    const uint32_t i0 = min(total, warp * per * 32), i1 = min(total, i0 + per * 32);
    auto mask = [](uint32_t b) {  // the bins of a box: bit 4 y + x
        const uint32_t x0 = b & 7u, x1 = (b >> 3) & 7u, y0 = (b >> 6) & 7u, y1 = (b >> 9) & 7u;
        return ((2u << x1) - (1u << x0)) * ((0x1111u << (4 * y0)) & (0xFFFFu >> (4 * (3 - y1))));
    };
    uint32_t pos = 0;  // this warp's entries of bin `lane`
    for (uint32_t ia = i0; ia < i1; ia += 32) {
        const uint32_t i = ia + lane, m = i < i1 ? mask(abox[ltri[i]]) : 0u;
        for (uint32_t u = __reduce_or_sync(0xFFFFFFFFu, m); u; u &= u - 1) {
            const uint32_t q = __ffs(u) - 1, c = __popc(__ballot_sync(0xFFFFFFFFu, (m >> q) & 1u));
            if (lane == q) pos += c;
        }
    }
    wpos[warp][lane] = pos;
    __syncthreads();
    if (warp == 0) {
        const uint32_t x = X + lane % 4, y = Y + lane / 4;
        const bool live = lane < 16 && x < f.tiles_x && y < f.tiles_y;
        uint32_t count = 0;
#pragma unroll
        for (int w = 0; w < kGatherWarps; ++w) {
            const uint32_t c = wpos[w][lane];
            wpos[w][lane] = count;
            count += c;
        }
        const uint32_t start = place_bins(f, fi, s, y * f.tiles_x + x, live, live ? count : 0u);
#pragma unroll
        for (int w = 0; w < kGatherWarps; ++w) wpos[w][lane] += start;
    }
    __syncthreads();
    uint32_t* bins = s.bins + f.bin_base;
    const uint32_t ts = (uint32_t)f.ts;
    const bool split = raster_edge((int)ts) != (int)ts;
    pos = wpos[warp][lane];  // now: this warp's next entry of bin `lane`
    for (uint32_t ia = i0; ia < i1; ia += 32) {
        const uint32_t i = ia + lane;
        uint32_t tri = 0, b = 0, m = 0;
        unsigned long long r = 0;
        if (i < i1) {
            tri = ltri[i];
            b = abox[tri];
            m = mask(b);
            if (split) r = s.tri_rect[f.rect_base + tri] & ~kRectClippedBit;  // for its quadrants
        }
        for (uint32_t u = __reduce_or_sync(0xFFFFFFFFu, m); u; u &= u - 1) {
            const uint32_t q = __ffs(u) - 1, bal = __ballot_sync(0xFFFFFFFFu, (m >> q) & 1u);
            const uint32_t p = __shfl_sync(0xFFFFFFFFu, pos, q) + __popc(bal & lanemask_lt());
            if (((m >> q) & 1u) && p < f.bin_cap)
                bins[p] = bin_entry(tri, (b & 0x8000u) != 0, r, X + q % 4, Y + q / 4, ts);
            if (lane == q) pos += __popc(bal);
        }
    }
}

// One CTA per block of B x B bins of a frame, B = 8 or 4 (gather_edge). It lists the triangles whose boxes
// touch the block (in submission order: every warp a contiguous part of the mesh, two passes), then
// each warp fills half a row of 8 bins (or one bin of 4 x 4) from the list: one pass counts (byte
// counters in the lanes), the bins' ranges are allocated (place_bins), a second pass writes each
// bin's entries in order. Blocks of 4 x 4 are those of images with few bins, where a block's list may be most of
// the mesh: from kGatherLong entries on the warps share it (gather_by_list) instead of each walking all of
// it. 7 938 triangles of a terrain, walked -> shared: at 64x64 149 -> 102 us a frame, at 320x240 64 -> 46, eight such
// frames at 64x64 235 -> 135; with 512 for kGatherLong 500 triangles at 64x64 take 124 us instead of 121. Blocks of
// 8 x 8 stay with the walk: their lists are short, and 64 bins one after another are a longer chain than a quarter
// row (shared, a 2 000-triangle soup at 1080p takes 60 us instead of 52).
__global__ void __launch_bounds__(kGatherThreads) k_bin_gather(const FrameDev* __restrict__ frames, int nframes,
                                                               Scratch s) {
    pdl_enter();
    __shared__ uint16_t abox[kGatherTris];  // by triangle: bins of the block x0 | x1 << 3 | y0 << 6 | y1 << 9 | clipped << 15
    __shared__ uint16_t ltri[kGatherTris];  // the block's triangles in order
    __shared__ uint32_t hit[kGatherTris / 32];
    __shared__ uint32_t wcount[kGatherWarps];
    __shared__ uint32_t bcount[64], bstart[64];
    __shared__ uint32_t wpos[kGatherWarps][32];  // gather_by_list: per warp and bin
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    int fi = 0;
    {
        int hi = nframes;
        while (hi - fi > 1) {
            const int mid = (fi + hi) >> 1;
            if (frames[mid].group_begin <= blockIdx.x) fi = mid; else hi = mid;
        }
    }
    const FrameDev& f = frames[fi];
    const uint32_t B = f.gather_bins;
    const uint32_t bx = (f.tiles_x + B - 1) / B;
    const uint32_t blk = blockIdx.x - f.group_begin;
    const uint32_t X = (blk % bx) * B, Y = (blk / bx) * B;  // the block's first bin
    // this warp's bins: nb from column col of row
    const uint32_t nb = B == 8 ? 4u : 1u, row = B == 8 ? warp >> 1 : warp >> 2, col = B == 8 ? 4 * (warp & 1u) : warp & 3u;
    const uint32_t T = f.ntris, ts = (uint32_t)f.ts;
    const uint32_t words = (T + 31) / 32, per = (words + kGatherWarps - 1) / kGatherWarps;
    const uint32_t w0 = min(words, warp * per), w1 = min(words, w0 + per);
    // ---- the block's triangles (kAhead boxes in flight per lane)
    uint32_t n = 0;
    constexpr uint32_t kAhead = 4;
    for (uint32_t wa = w0; wa < w1; wa += kAhead) {
        unsigned long long r[kAhead];
#pragma unroll
        for (uint32_t k = 0; k < kAhead; ++k) {
            const uint32_t i = (wa + k) * 32 + lane;
            r[k] = wa + k < w1 && i < T ? s.tri_rect[f.rect_base + i] : kRectEmpty;
        }
#pragma unroll
        for (uint32_t k = 0; k < kAhead; ++k) {
            if (wa + k >= w1) break;
            uint32_t x0, y0, x1, y1;
            tile_rect(r[k] & ~kRectClippedBit, ts, x0, y0, x1, y1);
            const bool in = r[k] != kRectEmpty && x0 < X + B && x1 >= X && y0 < Y + B && y1 >= Y;
            const uint32_t m = __ballot_sync(0xFFFFFFFFu, in);
            if (in)
                abox[(wa + k) * 32 + lane] =
                    (uint16_t)((max(x0, X) - X) | (min(x1 - X, B - 1) << 3) |
                               ((max(y0, Y) - Y) << 6) | (min(y1 - Y, B - 1) << 9) |
                               ((r[k] & kRectClippedBit) ? 0x8000u : 0u));
            if (lane == 0) hit[wa + k] = m;
            n += __popc(m);
        }
    }
    if (lane == 0) wcount[warp] = n;
    __syncthreads();
    uint32_t at = 0, total = 0;
#pragma unroll
    for (int k = 0; k < kGatherWarps; ++k) {
        const uint32_t c = wcount[k];
        if ((uint32_t)k < warp) at += c;
        total += c;
    }
    for (uint32_t w = w0; w < w1; ++w) {
        const uint32_t m = hit[w];
        if ((m >> lane) & 1u) {
            const uint32_t i = w * 32 + lane, k = at + __popc(m & lanemask_lt());
            ltri[k] = (uint16_t)i;
        }
        at += __popc(m);
    }
    __syncthreads();
    if (B == 4 && total >= kGatherLong) {
        gather_by_list(f, (uint32_t)fi, s, X, Y, ltri, abox, total, wpos);
        return;
    }
    // ---- entries per bin of the warp: bit k of the mask is bin k
    auto row_mask = [&](uint32_t b) {
        const uint32_t x0 = b & 7u, x1 = (b >> 3) & 7u, y0 = (b >> 6) & 7u, y1 = (b >> 9) & 7u;
        return row >= y0 && row <= y1 ? (((2u << x1) - (1u << x0)) >> col) & ((1u << nb) - 1u) : 0u;
    };
    uint32_t counts = 0;  // byte counters of the bins
    for (uint32_t i = lane; i < total; i += 32) {
        const uint32_t m = row_mask(abox[ltri[i]]);
        counts += (m * 0x00204081u) & 0x01010101u;
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if ((uint32_t)k >= nb) break;
        const uint32_t c = __reduce_add_sync(0xFFFFFFFFu, (counts >> (8 * k)) & 0xFFu);
        if (lane == 0) bcount[row * B + col + k] = c;
    }
    __syncthreads();
    if (warp * 32 < B * B) {
        const uint32_t b = warp * 32 + lane, x = X + b % B, y = Y + b / B;
        const bool live = b < B * B && x < f.tiles_x && y < f.tiles_y;
        bstart[b] = place_bins(f, (uint32_t)fi, s, y * f.tiles_x + x, live, live ? bcount[b] : 0u);
    }
    __syncthreads();
    // ---- the entries, in order
    uint32_t* bins = s.bins + f.bin_base;
    uint32_t pos = lane < nb ? bstart[row * B + col + lane] : 0u;  // lane k: next entry of bin k
    for (uint32_t i0 = 0; i0 < total; i0 += 32) {
        const uint32_t i = i0 + lane;
        uint32_t tri = 0, b = 0x40u;  // (an empty box: rows 1 .. 0)
        if (i < total) {
            tri = ltri[i];
            b = abox[tri];
        }
        const uint32_t m = row_mask(b);
        if (!__any_sync(0xFFFFFFFFu, m != 0)) continue;
        const bool clipped = (b & 0x8000u) != 0;
        unsigned long long r = 0;
        if (m) {
            if (raster_edge((int)ts) != (int)ts) r = s.tri_rect[f.rect_base + tri] & ~kRectClippedBit;  // its quadrants
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if ((uint32_t)k >= nb) break;
            const uint32_t bal = __ballot_sync(0xFFFFFFFFu, (m >> k) & 1u);
            const uint32_t p = __shfl_sync(0xFFFFFFFFu, pos, k) + __popc(bal & lanemask_lt());
            if (((m >> k) & 1u) && p < f.bin_cap) bins[p] = bin_entry(tri, clipped, r, X + col + k, Y + row, ts);
            if (lane == (uint32_t)k) pos += __popc(bal);
        }
    }
}

// ===================================================================== raster

constexpr int kRasterThreads = 128;
constexpr int kRasterWarps = kRasterThreads / 32;
constexpr int kRasterCtasPerSm = 7;  // occupancy the launch bounds aim at (shared memory allows 7)
constexpr int kEmptyRun = 8;  // bins without entries taken per queue update
constexpr uint32_t kTrimMin = 4;  // shortest box line that line_span trims

// A raster group's queue as its consumers read it: the classes' counts turned into ends (heaviest
// class first). After a bin overflow every tile counts as empty: each is cleared, and the host runs the
// frame again.
struct TileQueue {
    const uint32_t* order;  // the group's lists
    uint32_t n, first;      // tiles of the group, the first of them
    uint32_t end[kClasses - 1];  // bins of class 11, of 11 and 10, ...
    uint32_t busy, empty;
    bool overflow;
};
// The first warp fills it (one counter per lane, one trip to memory), then a block barrier.
__device__ __forceinline__ void load_queue(TileQueue& tq, const unsigned int* queue, const uint32_t* order, uint32_t n,
                                           const uint32_t* status, uint32_t first_tile) {
    if (threadIdx.x < 32) {
        const uint32_t lane = threadIdx.x;
        const uint32_t st = *(volatile const uint32_t*)status;
        const uint32_t own = lane < (uint32_t)kClasses
                                 ? ((volatile const unsigned int*)queue)[kQueueClass + kClasses - 1 - lane] : 0u;
        const bool overflow = (st & ST_BIN_OVERFLOW) != 0;
        uint32_t incl = lane < (uint32_t)(kClasses - 1) && !overflow ? own : 0u;
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= (uint32_t)o) incl += y;
        }
        if (lane < (uint32_t)(kClasses - 1)) tq.end[lane] = incl;
        if (lane == (uint32_t)(kClasses - 1)) {
            tq.order = order;
            tq.n = n;
            tq.first = first_tile;
            tq.busy = incl;
            tq.empty = overflow ? n : own;
            tq.overflow = overflow;
        }
    }
    __syncthreads();
}
// The i-th tile with entries (i < busy), heaviest class first.
__device__ __forceinline__ uint32_t busy_tile(const TileQueue& tq, uint32_t i) {
    uint32_t c = kClasses - 1, start = 0;
#pragma unroll
    for (int k = 0; k < kClasses - 2; ++k)
        if (i >= tq.end[k]) {
            c = kClasses - 2 - k;
            start = tq.end[k];
        }
    return tq.order[order_slot(c, i - start, tq.n)];
}
// The i-th tile without entries (i < empty).
__device__ __forceinline__ uint32_t empty_tile(const TileQueue& tq, uint32_t i) {
    return tq.overflow ? tq.first + i : tq.order[order_slot(0, i, tq.n)];
}
// Bins in the heavy classes: the first of the queue.
__device__ __forceinline__ uint32_t heavy_tiles(const TileQueue& tq, uint32_t heavy_bits) {
    const uint32_t h = heavy_class(heavy_bits);
    return h >= (uint32_t)kClasses ? 0u : tq.end[kClasses - 1 - h];
}

// Strips of rows that each raster unit is divided into, a CTA (or warp) each, when there are fewer units
// than places for them: every strip stages all of the unit's entries, so this pays only where the GPU
// would wait for a few units' serial batches. Returns log2 of their number. A 256-triangle sphere at
// 256x192 58 -> 49 us a frame, the cube at 800x600 with readback 74 -> 69.
__device__ __forceinline__ uint32_t strips_for(uint32_t nunits, uint32_t places) {
    return 4 * nunits <= places ? 2u : 2 * nunits <= places ? 1u : 0u;
}

// A raster CTA owns one TS x TS tile: a whole bin (bin edge == TS) or one quadrant of a bin
// twice as wide. Bin entries carry, in their low 4 bits, the quadrants the triangle's pixel box
// touches, so a quadrant CTA skips the other entries without loading them.
template <int S, int TS>
struct RasterCfg {
    static constexpr int NPIX = TS * TS;
    static constexpr int IC = kRasterThreads;  // items (triangles after clipping) per batch
    static constexpr int QC = 64;              // per-warp fragment ring
    static_assert(TS <= 16 && IC <= 256, "ring entries hold item and pixel in one byte each");
    static constexpr int LINES = (TS + kRasterWarps - 1) / kRasterWarps;  // lines of a tile per warp
    static_assert(LINES <= 7, "a warp's span counts are summed bit by bit, three bits each");
};

// One item (a triangle, or one fan triangle of a clipped polygon) as five 16-byte words, so that
// a candidate's lane gets it in three loads and a shaded fragment's in five: the items of a window are near
// neighbours, and a stride of five words keeps eight of them on different bank groups. k_raster is
// bound by instruction issue and next by shared-memory wavefronts. These records (22 loads before),
// the span list, the 16-byte depth rounds and the table-free texture filter (tex_argb) together
// took 12% off a frame of the 100k-triangle soup at 1080p, 6% off 3k large triangles at 1440p
// and 9% off a batch of 20 scenes.
struct RasterItem {
    float4 a;  // p0.x, p0.y, p1.x, p1.y (screen points)
    float4 b;  // p2.x, p2.y, cover_inv, z0
    float4 c;  // z1, z2, w0, w1
    float4 d;  // w2, u0, v0, u1
    float4 e;  // v1, u2, v2, draw << 8 | sub-triangle (bits)
};

template <int S, int TS>
struct alignas(16) RasterSmem {
    using C = RasterCfg<S, TS>;
    float zb[C::NPIX * S];     // pixel-major: the samples of pixel p at p * S (one 16-byte access)
    uint32_t cb[C::NPIX * S];  // sample-major: sample k of pixel p at k * NPIX + p
    RasterItem item[C::IC];    // items of the current batch
    float qz[kRasterWarps][C::QC][S];  // sample depths of the fragment ring, NaN where not covered
    uint32_t irect[C::IC];  // tile-local pixel box: x0 | y0 << 8 | x1 << 16 | y1 << 24
    uint32_t itri[C::IC];
    uint16_t span[kRasterWarps][C::IC * C::LINES];  // the warp's (item, line) pairs: item | line << 8
    uint2 run[kRasterWarps][32];                    // non-empty spans of a group: start, item | line << 8 | first << 16
    // per-warp ring of covered fragments, in submission order: item | pixel << 8 | mask << 16
    uint32_t q[kRasterWarps][C::QC];
    // per-warp ring of depth-passed fragments waiting for the fragment shader, in order:
    // item | pixel << 8 | depth mask << 16, and sample 0's depth
    uint32_t sq[kRasterWarps][C::QC];
    float sz0[kRasterWarps][C::QC];
    // candidate work of the batch by row (low half) and by column (high half), as differences; the
    // sums stay below 2^16 (at most 128 items of 16 pixels)
    uint32_t work[TS + 1];
    uint32_t tmp[40];
    uint32_t misc[8];  // [0] unit ticket, [1] items staged, [2..4] statistics, [5] the unit's bin, [6] log2 of the strips
    TileQueue tq;
    uint32_t zmaxw[kRasterWarps];  // per warp: largest stored depth of its share of the tile
};

// S consecutive floats of shared memory (16-byte aligned when S is 4).
template <int S>
__device__ __forceinline__ void load_samples(const float* p, float z[S]) {
    if (S == 4) {
        const float4 v = *reinterpret_cast<const float4*>(p);
        z[0] = v.x;
        z[1 % S] = v.y;
        z[2 % S] = v.z;
        z[3 % S] = v.w;
    } else {
#pragma unroll
        for (int k = 0; k < S; ++k) z[k] = p[k];
    }
}
template <int S>
__device__ __forceinline__ void store_samples(float* p, const float z[S]) {
    if (S == 4) {
        *reinterpret_cast<float4*>(p) = make_float4(z[0], z[1 % S], z[2 % S], z[3 % S]);
    } else {
#pragma unroll
        for (int k = 0; k < S; ++k) p[k] = z[k];
    }
}

__device__ __forceinline__ uint32_t find_draw(const DrawDev* __restrict__ draws,
                                              const FrameDev& f, uint32_t g) {
    uint32_t lo = f.draw_begin, hi = f.draw_begin + f.draw_count;
    while (hi - lo > 1) {
        uint32_t mid = (lo + hi) >> 1;
        if (draws[mid].tbase <= g) lo = mid; else hi = mid;
    }
    return lo;
}

__device__ __forceinline__ uint32_t frame_of_tile(const FrameDev* __restrict__ frames, int nframes,
                                                  uint32_t gt) {
    int lo = 0, hi = nframes;
    while (hi - lo > 1) {
        int mid = (lo + hi) >> 1;
        if (frames[mid].tile_begin <= gt) lo = mid; else hi = mid;
    }
    return (uint32_t)lo;
}

// Room added to edge k's value at a pixel centre so that it bounds the computed edge value at
// every sample of the pixel: s_k + m_k, derived at line_span.
template <int S>
__device__ __forceinline__ float edge_room(float nx, float ny, float Px, float Py) {
    const float sk = S == 1 ? 0.0f : 0.125f * fmaxf(fabsf(nx - 3.0f * ny), fabsf(3.0f * nx + ny));
    return sk + 1e-6f * (fabsf(nx) * (fabsf(Px) + 16400.0f) + fabsf(ny) * (fabsf(Py) + 16400.0f)) + 1e-37f;
}

// The pixels of one line of an item's box that can hold a covered sample: line lc (a tile-local
// row in mode 0, a column in mode 1), candidates [a0, a1) along it, trimmed in place. A pixel is
// dropped only where some edge k is negative at every sample with room to spare: with E_k the
// edge function in exact arithmetic over the stored f32 normal and point, the computed
// edge_eval value differs from E_k by at most 3 * 2^-24 * (|nx| |x - Px| + |ny| |y - Py|)
// (two subtractions, two products and one sum, each correctly rounded; the leading 0 + is
// exact). E_k is linear, so over the pixel's samples it is at most E_k(centre) + s_k, s_k the
// largest of nx ox + ny oy over the sample offsets (ox, oy) from the centre: for the 4-sample
// pattern (1/8, -3/8), (3/8, 1/8) and their negatives, s_k = max(|nx - 3 ny|, |3 nx + ny|) / 8;
// 0 for the single centre sample. So E_k(centre) + s_k + m_k < 0, m_k = 1e-6 (|nx| (|Px| +
// 16400) + |ny| (|Py| + 16400)) + 1e-37, makes every sample's computed value negative, and the
// edge test fails whatever the tie rule (screen coordinates stay below 16400; m_k also covers
// the f32 rounding of s_k and of the line offset below). Along the line the bound is linear in
// the pixel index, so the pixels that keep it are an interval [ceil(t), ...) or (..., t]; t is
// computed in f32 to within 0.03 pixel whenever it falls near the tile (|pal - gk / nal| below
// 2^16; farther out only its sign matters), and the interval is widened by 1/8 pixel.
// Items with non-finite points (cover_inv NaN) are not trimmed.
template <int S, int TS>
__device__ __forceinline__ void line_span_pts(const float px[3], const float py[3], uint32_t mode, uint32_t lc,
                                              uint32_t X0, uint32_t Y0, uint32_t& a0, uint32_t& a1) {
    // line centre across, and the pixel-centre origin along the line (global coordinates)
    const float cacross = (float)((mode == 0 ? Y0 : X0) + lc) + 0.5f;
    const float oalong = (float)(mode == 0 ? X0 : Y0) + 0.5f;
    int lo = (int)a0, hi = (int)a1;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int n = k == 2 ? 0 : k + 1;
        const float nx = -(py[n] - py[k]), ny = px[n] - px[k];
        const float R = edge_room<S>(nx, ny, px[k], py[k]);
        const float nal = mode == 0 ? nx : ny, nac = mode == 0 ? ny : nx;
        const float pal = mode == 0 ? px[k] : py[k], pac = mode == 0 ? py[k] : px[k];
        const float gk = nac * (cacross - pac) + R;  // E_k + R = nal * (c_along - pal) + gk
        if (fabsf(nal) <= 1e-20f) {
            // (almost) constant along the line
            if (gk + fabsf(nal) * (fabsf(pal) + 16400.0f) < 0.0f) hi = lo;
            continue;
        }
        // E_k + R >= 0  <=>  nal * (oalong + x - pal) >= -gk
        const float t = pal - __fdividef(gk, nal) - oalong;  // 2-ulp division is enough
        if (!isfinite(t)) continue;
        const float tc = fminf(fmaxf(t, -8.0f), (float)TS + 8.0f);
        if (nal > 0.0f) lo = max(lo, (int)ceilf(tc - 0.125f));
        else hi = min(hi, (int)floorf(tc + 0.125f) + 1);
    }
    if (hi < lo) hi = lo;
    a0 = (uint32_t)lo;
    a1 = (uint32_t)hi;
}

// Order-preserving map of floats to unsigned integers (NaN above +inf) and back.
__device__ __forceinline__ uint32_t float_to_ordered(float x) {
    const uint32_t b = __float_as_uint(x);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float ordered_to_float(uint32_t u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
}

// True when no sample of the triangle with screen depths z0..z2 can pass the strict depth
// test against a tile whose stored depths are all <= ztile. A sample depth is (b0 z0 + b1 z1)
// + b2 z2 with clamped b0, b1 in [0, 1] and b2 = clamp((1 - b0) - b1): a convex combination,
// or with b2 = 0 a combination with b0 + b1 >= 1, so for depths >= 0 it is at least
// min(z0, z1, z2) up to the rounding of the products and sums (well below 2^-20 relative).
// Never true with a negative or NaN corner depth or a NaN ztile.
__device__ __forceinline__ bool depth_cull(float z0, float z1, float z2, float ztile) {
    const float zmin = fminf(fminf(z0, z1), z2);
    const bool ok = z0 >= 0.0f && z1 >= 0.0f && z2 >= 0.0f;  // false for NaN
    return ok && zmin * (1.0f - 0x1p-20f) >= ztile;
}

// Stages the items of one bin entry (one triangle, or the fan of its clipped polygon) at
// positions first.. of the batch: screen points, depths, w, attributes, 1 / 2x area and the
// tile-local pixel box, and adds the box to the batch's row and column work.
template <int S, int TS>
__device__ __forceinline__ void stage_entry(RasterSmem<S, TS>& sm, const FrameDev& f,
                                            const DrawDev* __restrict__ draws, const Scratch& s,
                                            uint32_t g, uint32_t aux, uint32_t nitems, uint32_t first,
                                            uint32_t X0, uint32_t Y0, uint32_t row0, uint32_t row1, float ztile) {
    const uint32_t di = find_draw(draws, f, g);
    const DrawDev& d = draws[di];
    const int fs = d.fs;
    for (uint32_t k = 0; k < nitems; ++k) {
        const uint32_t it = first + k;
        float4 sv[3];
        float uv[3][2] = {{0.0f, 0.0f}, {0.0f, 0.0f}, {0.0f, 0.0f}};
        if (aux == kNone) {
            const uint32_t tri = g - d.tbase;
            const uint32_t ii[3] = {__ldg(d.idx + 3ull * tri), __ldg(d.idx + 3ull * tri + 1),
                                    __ldg(d.idx + 3ull * tri + 2)};
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                sv[q] = s.vscr[d.vbase + ii[q]];
                if (fs == 0) {
                    uv[q][0] = __ldg(d.uv + 2ull * ii[q]);
                    uv[q][1] = __ldg(d.uv + 2ull * ii[q] + 1);
                }
            }
        } else {
            const float* st = s.clip_store + aux + 1;
            const uint32_t vi[3] = {0u, k + 1, k + 2};
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const float* o = st + 10 * vi[q];
                sv[q] = make_float4(o[0], o[1], o[2], o[3]);
                uv[q][0] = o[8];
                uv[q][1] = o[9];
            }
        }
        RasterItem& m = sm.item[it];
        m.a = make_float4(sv[0].x, sv[0].y, sv[1].x, sv[1].y);
        m.b = make_float4(sv[2].x, sv[2].y, cover_inv(sv), sv[0].z);
        m.c = make_float4(sv[1].z, sv[2].z, sv[0].w, sv[1].w);
        m.d = make_float4(sv[2].w, uv[0][0], uv[0][1], uv[1][0]);
        m.e = make_float4(uv[1][1], uv[2][0], uv[2][1], __uint_as_float((di << 8) | k));
        uint32_t bx0, bx1, by0, by1;
        pixel_bbox(sv, f.width, f.height, bx0, bx1, by0, by1);
        const uint32_t cx0 = max(bx0, X0), cx1 = min(bx1, X0 + TS);
        const uint32_t cy0 = max(by0, Y0 + row0), cy1 = min(by1, Y0 + row1);
        // hidden: no sample depth can get below the largest depth stored in the tile
        // (depth_cull), so the strict depth test (mod.rs:363-378) fails everywhere
        const bool nonempty = bx0 < bx1 && by0 < by1 && cx0 < cx1 && cy0 < cy1 &&
                              !depth_cull(sv[0].z, sv[1].z, sv[2].z, ztile);
        uint32_t r = 0;
        if (nonempty) {
            const uint32_t lx0 = cx0 - X0, ly0 = cy0 - Y0, lx1 = cx1 - X0, ly1 = cy1 - Y0;
            r = lx0 | (ly0 << 8) | (lx1 << 16) | (ly1 << 24);
            const uint32_t cw = lx1 - lx0, ch = (ly1 - ly0) << 16;
            atomicAdd(&sm.work[ly0], cw);
            atomicAdd(&sm.work[ly1], 0u - cw);
            atomicAdd(&sm.work[lx0], ch);
            atomicAdd(&sm.work[lx1], 0u - ch);
        }
        sm.irect[it] = r;
        sm.itri[it] = g;
    }
}

// Chooses how the tile's pixels are divided among the warps for one batch: interleaved rows
// (row r to warp r % kRasterWarps; suits scattered triangles) or interleaved columns (suits
// runs of small triangles along a screen row, which crowd into a few rows), whichever gives
// the lighter heaviest warp by candidate-pixel work. Either way each warp owns its pixels for
// the batch, which keeps every pixel's fragments in one warp and in submission order, and an
// item meets each warp on at most TS / kRasterWarps lines. Returns 0 for rows, 1 for columns.
// Called by one warp.
template <int TS>
__device__ __forceinline__ uint32_t split_work(const uint32_t* work) {
    const uint32_t lane = lane_id();
    // per-line work from the differences (lane = line), rows and columns in one word
    uint32_t w = lane < (uint32_t)TS ? work[lane] : 0u;
#pragma unroll
    for (int o = 1; o < TS; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, w, o);
        if (lane >= (uint32_t)o) w += y;
    }
    if (lane >= (uint32_t)TS) w = 0;
    // each warp's load: the sum of its lines (lane % kRasterWarps), then the heaviest warp
#pragma unroll
    for (int o = kRasterWarps; o < TS; o <<= 1) w += __shfl_down_sync(0xFFFFFFFFu, w, o);
    uint32_t wr = w & 0xFFFFu, wc = w >> 16;
#pragma unroll
    for (int o = kRasterWarps / 2; o > 0; o >>= 1) {
        wr = max(wr, __shfl_xor_sync(0xFFFFFFFFu, wr, o));
        wc = max(wc, __shfl_xor_sync(0xFFFFFFFFu, wc, o));
    }
    return wc < wr ? 1u : 0u;  // lane 0's values cover lanes 0 .. kRasterWarps - 1
}

// Appends one fragment record to the debug log (rast_debug_log_enable); kept out of line.
__device__ __noinline__ void log_fragment(const Scratch& s, uint32_t tri, uint32_t sub, uint32_t yx,
                                          uint32_t masks) {
    const unsigned long long slot = atomicAdd(s.log_n, 1ull);
    if (slot < s.log_cap) {
        uint32_t* L = s.log + 4ull * slot;
        L[0] = tri;
        L[1] = sub;
        L[2] = yx;
        L[3] = masks;
    } else {
        atomicOr(s.status, ST_LOG_OVERFLOW);
    }
}

// FS::Color's input for an item: the vertex colours of its three corners (Color vertex
// attribute, src/graphics_primitives.rs:9-13), from the mesh or from the clipped polygon.
__device__ __noinline__ void item_colours(const DrawDev& d, const FrameDev& f, const Scratch& s, uint32_t g,
                                          uint32_t k, float col[3][4]) {
    const uint32_t aux = s.tri_aux[f.rect_base + g];
    if (aux == kNone) {
        const uint32_t tri = g - d.tbase;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const uint32_t vi = __ldg(d.idx + 3ull * tri + q);
#pragma unroll
            for (int c = 0; c < 4; ++c) col[q][c] = d.rgba ? __ldg(d.rgba + 4ull * vi + c) : 0.0f;
        }
    } else {
        const float* st = s.clip_store + aux + 1;
        const uint32_t vi[3] = {0u, k + 1, k + 2};
#pragma unroll
        for (int q = 0; q < 3; ++q)
#pragma unroll
            for (int c = 0; c < 4; ++c) col[q][c] = st[10 * vi[q] + 4 + c];
    }
}

// Depth test of up to 32 queued fragments of one warp (lane = one fragment, queue order =
// submission order). Fragments of the same pixel run in rounds of increasing rank, so the
// depth test (depth_coverage, src/rasterizer/mod.rs:363-378) happens in submission order; a
// sample that is not covered carries a NaN depth, which never passes.
// Fragments with samples that passed go, in the same order, to the warp's shade ring.
template <int S, int TS>
__device__ __forceinline__ void warp_depth(RasterSmem<S, TS>& sm, uint32_t w, uint32_t head, uint32_t n,
                                           uint32_t& stail, const Scratch& s, uint32_t X0, uint32_t Y0,
                                           uint32_t& shaded, uint32_t& fsinv) {
    using C = RasterCfg<S, TS>;
    const uint32_t lane = lane_id();
    const bool valid = lane < n;
    const uint32_t q = (head + lane) & (C::QC - 1);
    uint32_t fr = 0;
    float z[S];
#pragma unroll
    for (int k = 0; k < S; ++k) z[k] = 0.0f;
    if (valid) {
        fr = sm.q[w][q];
        load_samples<S>(sm.qz[w][q], z);
    }
    const uint32_t pix = (fr >> 8) & 0xFFu;
    // fragments of one item never share a pixel: most windows over large triangles need no match, whose
    // time grows with the distinct values (3 000 large triangles at 1440p 448 -> 433 us a frame; no
    // change on the 100k soup, 370 -> 371 on the 2M-triangle terrain, whose windows mix items)
    uint32_t rank = 0, maxr = 0;
    const uint32_t fr0 = __shfl_sync(0xFFFFFFFFu, fr, 0);  // every lane
    if (!__all_sync(0xFFFFFFFFu, (!valid) | (((fr ^ fr0) & 0xFFu) == 0))) {
        const uint32_t key = valid ? pix : 0x10000u + lane;
        rank = __popc(__match_any_sync(0xFFFFFFFFu, key) & lanemask_lt());
        maxr = __reduce_max_sync(0xFFFFFFFFu, rank);
    }
    uint32_t dm = 0;
    for (uint32_t r = 0; r <= maxr; ++r) {
        // this round's lanes: no two share a pixel
        if (valid && rank == r) {
            float old[S];
            load_samples<S>(&sm.zb[pix * S], old);
#pragma unroll
            for (int k = 0; k < S; ++k) {
                const bool pass = z[k] < old[k];
                old[k] = pass ? z[k] : old[k];
                dm |= pass ? 1u << k : 0u;
            }
            store_samples<S>(&sm.zb[pix * S], old);
            if (s.log)
                log_fragment(s, sm.itri[fr & 0xFFu], __float_as_uint(sm.item[fr & 0xFFu].e.w) & 0xFFu,
                             ((Y0 + pix / TS) << 16) | (X0 + pix % TS), (dm << 8) | (fr >> 16));
        }
        __syncwarp();
    }
    const uint32_t bal = __ballot_sync(0xFFFFFFFFu, dm != 0);
    if (dm) {
        const uint32_t sq = (stail + __popc(bal & lanemask_lt())) & (C::QC - 1);
        sm.sq[w][sq] = (fr & 0xFFFFu) | (dm << 16);
        sm.sz0[w][sq] = (fr & 0x10000u) ? z[0] : 0.0f;
        shaded += __popc(dm);
        fsinv += 1;
    }
    stail += __popc(bal);
    __syncwarp();
}

// What the fragment shader reads of its draw (DrawDev), two 16-byte loads.
struct ShadeDraw {
    const uint32_t* tex;
    uint32_t tex_w, tex_h;
    float xmax, ymax;
    int32_t fs;
    bool small;
};
__device__ __forceinline__ ShadeDraw shade_draw(const DrawDev* d) {
    static_assert(offsetof(DrawDev, tex) % 16 == 0 && offsetof(DrawDev, tex_xmax) == offsetof(DrawDev, tex) + 16 &&
                      sizeof(DrawDev) % 16 == 0,
                  "the shader's fields of a draw are two 16-byte words");
    const uint4 a = __ldg(reinterpret_cast<const uint4*>(&d->tex));
    const uint4 b = __ldg(reinterpret_cast<const uint4*>(&d->tex) + 1);
    ShadeDraw r;
    r.tex = reinterpret_cast<const uint32_t*>((unsigned long long)a.x | ((unsigned long long)a.y << 32));
    r.tex_w = a.z;
    r.tex_h = a.w;
    r.xmax = __uint_as_float(b.x);
    r.ymax = __uint_as_float(b.y);
    r.fs = (int32_t)b.z;
    r.small = b.w != 0;
    return r;
}

// Fragment shader and colour write of up to 32 fragments of the warp's shade ring (kept out of
// line: the coverage loop that calls it stays small enough for the instruction cache):
// Fragment::interpolate (src/rasterizer/mod.rs:69-100) at the point its depth-passed mask
// selects, the draw's shader by id, then write_pixel (mod.rs:380-397) to the passed samples,
// same-pixel fragments in rounds of increasing rank (submission order).
template <int S, int TS>
__device__ __noinline__ void warp_shade(RasterSmem<S, TS>& sm, uint32_t w, uint32_t head, uint32_t n,
                                           const DrawDev* __restrict__ draws, const FrameDev& f,
                                           const Scratch& s, uint32_t X0, uint32_t Y0, uint32_t& oobc) {
    using C = RasterCfg<S, TS>;
    const uint32_t lane = lane_id();
    const bool valid = lane < n;
    const uint32_t q = (head + lane) & (C::QC - 1);
    uint32_t argb = 0, pix = 0, dm = 0;
    if (valid) {
        const uint32_t fr = sm.sq[w][q];
        const uint32_t it = fr & 0xFFu;
        pix = (fr >> 8) & 0xFFu;
        dm = fr >> 16;
        const RasterItem& m = sm.item[it];
        const float4 a = m.a, b = m.b, c = m.c, d4 = m.d, e4 = m.e;
        const uint32_t meta = __float_as_uint(e4.w);
        const ShadeDraw d = shade_draw(&draws[meta >> 8]);
        float xs, ys;
        interp_point<S>(X0 + pix % TS, Y0 + pix / TS, dm, xs, ys);
        float u, v, ww;
        persp_bary(a.x, a.y, a.z, a.w, b.x, b.y, c.z, c.w, d4.x, xs, ys, u, v, ww);
        if (d.fs == 0) {
            // FS::Texture (upstream src/main.rs:214-216)
            const float tu = d4.y * u + d4.w * v + e4.y * ww;
            const float tv = d4.z * u + e4.x * v + e4.z * ww;
            argb = tex_argb(d.tex, d.tex_w, d.tex_h, d.xmax, d.ymax, d.small, tu, tv, f.dbg_color != nullptr, oobc);
        } else {
            float col[4];
            if (d.fs == 1) {
                // FS::Color (upstream src/main.rs:217)
                float vc[3][4];
                item_colours(draws[meta >> 8], f, s, sm.itri[it], meta & 0xFFu, vc);
#pragma unroll
                for (int k = 0; k < 4; ++k) col[k] = vc[0][k] * u + vc[1][k] * v + vc[2][k] * ww;
            } else {
                // FS::Debug (upstream src/main.rs:218-220): grayscale(frag_coords.depths[0])
                const float z0 = sm.sz0[w][q];
                col[0] = z0;
                col[1] = z0;
                col[2] = z0;
                col[3] = 1.0f;
            }
            argb = to_argb(col[0], col[1], col[2], col[3]);
        }
    }
    const uint32_t key = valid ? pix : 0x10000u + lane;
    const uint32_t grp = __match_any_sync(0xFFFFFFFFu, key);
    const uint32_t rank = __popc(grp & lanemask_lt());
    const uint32_t maxr = __reduce_max_sync(0xFFFFFFFFu, rank);
    for (uint32_t r = 0; r <= maxr; ++r) {
        const bool act = valid && rank == r;
#pragma unroll
        for (int k = 0; k < S; ++k)
            if (act & (((dm >> k) & 1u) != 0)) sm.cb[k * C::NPIX + pix] = argb;
        __syncwarp();
    }
}

// Writes the clear colour (and, when captured, clear samples) over one tile of a frame.
__device__ __forceinline__ void clear_tile_warp(const FrameDev& f, uint32_t x0, uint32_t y0,
                                                uint32_t edge, int S) {
    const uint32_t lane = lane_id();
    if (!f.dbg_depth && (f.width & 3u) == 0 && x0 + edge <= f.width &&
        (reinterpret_cast<uintptr_t>(f.out) & 15u) == 0) {
        // whole rows of 16-byte stores: the image starts on a 16-byte boundary (checked; batch
        // outputs can start anywhere), width % 4 == 0 and x0 is a multiple of the bin edge, so
        // every row segment does too
        const uint32_t q = edge / 4, sh = __ffs(q) - 1;  // uint4 per row (2, 4 or 8), its log2
        const uint4 c = make_uint4(kClearColor, kClearColor, kClearColor, kClearColor);
        for (uint32_t i = lane; i < edge * q; i += 32) {
            const uint32_t y = y0 + (i >> sh);
            if (y >= f.height) break;
            uint4* row = reinterpret_cast<uint4*>(f.out + (unsigned long long)y * f.width + x0);
            row[i & (q - 1)] = c;
        }
        return;
    }
    for (uint32_t i = lane; i < edge * edge; i += 32) {
        const uint32_t x = x0 + i % edge, y = y0 + i / edge;
        if (x >= f.width || y >= f.height) continue;
        const unsigned long long o = (unsigned long long)y * f.width + x;
        f.out[o] = kClearColor;
        if (f.dbg_depth) {
            for (int q = 0; q < S; ++q) {
                f.dbg_depth[o * S + q] = f.clear_depth;
                f.dbg_color[o * S + q] = kClearColor;
            }
        }
    }
}

// Persistent raster kernel for the heavy tiles. Units are (bin, quadrant) pairs of the first
// bins of the raster queue (those of the heavy classes; the others go one warp per
// tile to k_raster_warp), taken heaviest class first from queue[0]; per unit the CTA replays the
// bin in submission order in batches of up to IC items: stage the items (A), split the tile's rows or columns over the warps by work
// (B), then each warp walks the candidate pixels of its items inside its range — coverage
// (EdgeFunctions::eval, mod.rs:134-146) and sample depths (RasterizerTriangle::fragment,
// mod.rs:225-253) — and depth-tests, shades and writes the covered fragments in order (C).
// Bins without entries are then cleared by single warps from queue[1].
template <int S, int TS>
__global__ void __launch_bounds__(kRasterThreads, kRasterCtasPerSm) k_raster(const FrameDev* __restrict__ frames,
                                                           int nframes,
                                                           const uint32_t* __restrict__ order,
                                                           uint32_t ntotal, uint32_t first_tile, uint32_t nsx,
                                                           unsigned int* __restrict__ queue,
                                                           const DrawDev* __restrict__ draws,
                                                           Scratch s) {
    pdl_enter();
    using C = RasterCfg<S, TS>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    RasterSmem<S, TS>& sm = *reinterpret_cast<RasterSmem<S, TS>*>(smem_raw);
    const uint32_t warp = threadIdx.x >> 5, lane = lane_id();
    uint32_t shaded = 0, fsinv = 0, oobc = 0;
    const uint32_t nsub = nsx * nsx;
    load_queue(sm.tq, queue, order, ntotal, s.status, first_tile);

    // unit tickets (heaviest bins first); the next one is taken when the current unit starts its
    // resolve, so the queue update is in flight during the resolve. With no more units than CTAs, CTA
    // i takes unit i and no other: from the counter, the CTAs of the SMs nearest to it take up to
    // seven before the far ones get any (2 000-triangle soup with readback 86 -> 81 us a frame). With more
    // units the counter is the better one (a CTA that starts late would hold a heavy unit: 100k soup 10% slower).
    const uint32_t nwhole = heavy_tiles(sm.tq, frames[0].heavy_bits) * nsub;
    const uint32_t nunits = nwhole << strips_for(nwhole, gridDim.x);
    if (threadIdx.x == 0) sm.misc[6] = strips_for(nwhole, gridDim.x);
    if (threadIdx.x == 0) {
        const uint32_t qi = nunits <= gridDim.x ? blockIdx.x : atomicAdd(&queue[0], 1u);
        sm.misc[0] = qi;
        if (qi < nunits) sm.misc[5] = busy_tile(sm.tq, (qi >> sm.misc[6]) / nsub);
    }
    for (;;) {
    __syncthreads();
    // misc[0] and misc[5] are written again only after this unit's resolve, many barriers later
    const uint32_t qi = sm.misc[0];
    if (qi >= nunits) break;
    const uint32_t gt = sm.misc[5], ssh = sm.misc[6], sub = (qi >> ssh) % nsub;
    // the unit's rows of the tile, first | end << 8 (one register through the candidate loop)
    const uint32_t rows = (qi & ((1u << ssh) - 1u)) * (TS >> ssh) * 0x101u + ((TS >> ssh) << 8);
    const FrameDev& f = frames[frame_of_tile(frames, nframes, gt)];
    const uint32_t lt = gt - f.tile_begin;
    const uint32_t X0 = (lt % f.tiles_x) * (uint32_t)f.ts + (sub % nsx) * TS;
    const uint32_t Y0 = (lt / f.tiles_x) * (uint32_t)f.ts + (sub / nsx) * TS;
    const uint32_t W = f.width, H = f.height;
    {
        const float4 zc = make_float4(f.clear_depth, f.clear_depth, f.clear_depth, f.clear_depth);
        const uint4 cc = make_uint4(kClearColor, kClearColor, kClearColor, kClearColor);
        // the colours of other rows are not read, nor their depths
        for (uint32_t i = (rows & 0xFFu) * (TS * S / 4) + threadIdx.x; i < (rows >> 8) * (TS * S / 4); i += blockDim.x)
            reinterpret_cast<float4*>(sm.zb)[i] = zc;
        for (uint32_t i = threadIdx.x; i < (uint32_t)(C::NPIX * S / 4); i += blockDim.x)
            reinterpret_cast<uint4*>(sm.cb)[i] = cc;
    }
    // the bin's entries, or for a quadrant of a 32-pixel bin its own split list
    uint32_t nent;
    const uint32_t* bins;
    if (nsub > 1) {
        nent = s.qcount[4ull * gt + sub];
        bins = s.qbins + f.qbin_base + 4ull * s.tile_start[gt] + (unsigned long long)sub * s.tile_count[gt];
    } else {
        nent = s.tile_count[gt];
        bins = s.bins + f.bin_base + s.tile_start[gt];
    }
    const uint32_t mybit = 1u << sub;

    uint32_t pos = 0;  // next entry of the bin
    while (pos < nent) {
        // ---- A. fill a batch with the items of the next entries that touch this tile
        if (threadIdx.x <= (uint32_t)TS) {
            sm.work[threadIdx.x] = 0;
        }
        // largest depth stored in the tile before this batch, for depth_cull: the clear depth
        // for the unit's first batch; else reduced here and combined after the scan's barriers.
        // NaN (no culling) while the fragment log records depth-failed fragments too.
        float zt = s.log ? __int_as_float(0x7FC00000) : f.clear_depth;
        bool zt_ready = s.log || pos == 0;
        if (!zt_ready) {
            uint32_t zm = 0;
            for (uint32_t i = (rows & 0xFFu) * (TS * S) + threadIdx.x; i < (rows >> 8) * (TS * S); i += blockDim.x)
                zm = max(zm, float_to_ordered(sm.zb[i]));
            zm = __reduce_max_sync(0xFFFFFFFFu, zm);
            if (lane == 0) sm.zmaxw[warp] = zm;
        }
        uint32_t nit = 0;
        while (pos < nent) {
            const uint32_t e = pos + threadIdx.x;
            uint32_t g = 0, aux = kNone, nitems = 0;
            if (e < nent) {
                const uint32_t ent = bins[e];
                if (ent & mybit) {
                    g = ent >> kEntShift;
                    nitems = 1;
                    if (ent & kEntClipped) {
                        aux = s.tri_aux[f.rect_base + g];
                        nitems = (uint32_t)__float_as_int(s.clip_store[aux]) - 2u;
                    }
                }
            }
            if (threadIdx.x == 0) sm.misc[1] = nit;
            uint32_t itot;
            // the __syncthreads_count below orders the reads of tmp before its next use
            const uint32_t iex = block_excl_scan<false>(nitems, sm.tmp, itot);
            // entries fit while the running item count stays within the batch (a prefix)
            const bool part = (e < nent) && (nit + iex + nitems <= (uint32_t)C::IC);
            const uint32_t take = __syncthreads_count(part);
            if (part && threadIdx.x == take - 1) sm.misc[1] = nit + iex + nitems;
            if (part && nitems) {
                if (!zt_ready) {
                    uint32_t zm = sm.zmaxw[0];
#pragma unroll
                    for (int w = 1; w < kRasterWarps; ++w) zm = max(zm, sm.zmaxw[w]);
                    zt = ordered_to_float(zm);
                    zt_ready = true;
                }
                stage_entry<S, TS>(sm, f, draws, s, g, aux, nitems, nit + iex, X0, Y0, rows & 0xFFu, rows >> 8, zt);
            }
            __syncthreads();
            nit = sm.misc[1];
            const uint32_t window = min(nent - pos, (uint32_t)kRasterThreads);
            pos += take;
            if (take < window) break;  // the batch is full
        }
        // ---- B. divide the tile's pixels among the warps (every warp computes the same
        // choice from the batch's work histograms: no barrier to wait for one warp's), and list
        // this warp's spans in submission order: its lines of each item's box (rows, or columns
        // in column mode: line l belongs to warp l % kRasterWarps)
        const uint32_t mode = __shfl_sync(0xFFFFFFFFu, split_work<TS>(sm.work), 0);
        uint32_t nspan = 0;
        const uint32_t lsh = mode ? 0u : 8u;
        for (uint32_t i0 = 0; i0 < nit; i0 += 32) {
            const uint32_t it = i0 + lane;
            const uint32_t r = it < nit ? sm.irect[it] : 0u;
            const uint32_t l0 = (r >> lsh) & 0xFFu, l1 = (r >> (lsh + 16)) & 0xFFu;
            // the warp's first line at or past l0, and how many it has before l1 (0 for an empty box)
            const uint32_t first = l0 + ((warp - l0) & (kRasterWarps - 1));
            const uint32_t nl = (l1 + (uint32_t)kRasterWarps - 1 - first) / kRasterWarps;
            const uint32_t lt = lanemask_lt();
            const uint32_t n1 = __ballot_sync(0xFFFFFFFFu, nl & 1u);
            uint32_t at = nspan + __popc(n1 & lt);
            nspan += __popc(n1);
            if (C::LINES > 1) {
                const uint32_t n2 = __ballot_sync(0xFFFFFFFFu, nl & 2u);
                if (n2) {
                    at += 2 * __popc(n2 & lt);
                    nspan += 2 * __popc(n2);
                }
            }
            if (C::LINES > 3) {
                const uint32_t n4 = __ballot_sync(0xFFFFFFFFu, nl & 4u);
                if (n4) {
                    at += 4 * __popc(n4 & lt);
                    nspan += 4 * __popc(n4);
                }
            }
            const uint32_t e = it | (first << 8);
#pragma unroll
            for (uint32_t k = 0; k < (uint32_t)C::LINES; ++k)
                if (k < nl) sm.span[warp][at + k] = (uint16_t)(e + ((k * kRasterWarps) << 8));
        }
        __syncwarp();
        // ---- C. per warp, in submission order: its spans 32 at a time, one per lane, each
        // trimmed to the pixels that can hold a covered sample (line_span_pts); their pixels 32 at
        // a time: coverage and sample depths (cover_pixel); then ordered depth test and shading
        // of the covered fragments
        const uint32_t lstride = mode ? 1u : (uint32_t)TS, astride = mode ? (uint32_t)TS : 1u;
        uint32_t head = 0, tail = 0, shead = 0, stail = 0;
        for (uint32_t gb = 0; gb < nspan; gb += 32) {
            uint32_t c = 0, geo = 0;  // candidates; item | line << 8 | first candidate << 16
            if (gb + lane < nspan) {
                geo = sm.span[warp][gb + lane];
                const uint32_t it = geo & 0xFFu;
                const uint32_t r = sm.irect[it];
                uint32_t a0 = (mode ? r >> 8 : r) & 0xFFu, a1 = (mode ? r >> 24 : r >> 16) & 0xFFu;
                if (a1 - a0 >= kTrimMin) {  // shorter lines are cheaper to test whole than to trim
                    const float4 pa = sm.item[it].a, pb = sm.item[it].b;
                    const float px[3] = {pa.x, pa.z, pb.x}, py[3] = {pa.y, pa.w, pb.y};
                    if (fabsf(pb.z) <= FLT_MAX) line_span_pts<S, TS>(px, py, mode, geo >> 8, X0, Y0, a0, a1);
                }
                c = a1 - a0;
                geo |= a0 << 16;
            }
            uint32_t incl = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                if (lane >= (uint32_t)o) incl += y;
            }
            const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
            // the spans with candidates, compacted; each marks its first candidate, so a lane
            // finds its span by counting the marks up to its own candidate
            const uint32_t full = __ballot_sync(0xFFFFFFFFu, c != 0);
            const uint32_t start = c ? incl - c : 0xFFFFFFFFu;
            if (c) sm.run[warp][__popc(full & lanemask_lt())] = make_uint2(start, geo);
            __syncwarp();
            uint32_t before = 0xFFFFFFFFu;  // spans that start in earlier windows, less one
            for (uint32_t pb = 0; pb < total; pb += 32) {
                const uint32_t p = pb + lane;
                const uint32_t marks = __reduce_or_sync(0xFFFFFFFFu, start - pb < 32u ? 1u << (start - pb) : 0u);
                const uint2 sp = sm.run[warp][before + __popc(marks & (lanemask_lt() | (1u << lane)))];
                before += __popc(marks);
                const uint32_t it = sp.y & 0xFFu;
                uint32_t cov = 0, pix = 0;
                float z[S];
#pragma unroll
                for (int k = 0; k < S; ++k) z[k] = 0.0f;
                if (p < total) {
                    pix = ((sp.y >> 8) & 0xFFu) * lstride + ((sp.y >> 16) + (p - sp.x)) * astride;
                    const float fx = (float)(X0 + pix % TS), fy = (float)(Y0 + pix / TS);
                    const float4 a = sm.item[it].a, b = sm.item[it].b;
                    const float2 c2 = *reinterpret_cast<const float2*>(&sm.item[it].c);
                    const Cover<S> cv = cover_pixel<S>(a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, c2.x, c2.y, fx, fy);
                    cov = cv.mask;
#pragma unroll
                    for (int k = 0; k < S; ++k) z[k] = ((cov >> k) & 1u) ? cv.z[k] : __int_as_float(0x7FC00000);
                }
                const uint32_t bal = __ballot_sync(0xFFFFFFFFu, cov != 0);
                if (cov) {
                    const uint32_t q = (tail + __popc(bal & lanemask_lt())) & (C::QC - 1);
                    sm.q[warp][q] = it | (pix << 8) | (cov << 16);
                    store_samples<S>(sm.qz[warp][q], z);
                }
                tail += __popc(bal);
                __syncwarp();
                if (tail - head >= 32) {
                    warp_depth<S, TS>(sm, warp, head, 32, stail, s, X0, Y0, shaded, fsinv);
                    head += 32;
                    if (stail - shead >= 32) {
                        warp_shade<S, TS>(sm, warp, shead, 32, draws, f, s, X0, Y0, oobc);
                        shead += 32;
                    }
                }
            }
            __syncwarp();  // the runs are read before the next group's replace them
        }
        if (tail != head) warp_depth<S, TS>(sm, warp, head, tail - head, stail, s, X0, Y0, shaded, fsinv);
        while (stail != shead) {
            const uint32_t nsh = min(stail - shead, 32u);
            warp_shade<S, TS>(sm, warp, shead, nsh, draws, f, s, X0, Y0, oobc);
            shead += nsh;
        }
        __syncthreads();
    }

    // ---- resolve (resolve_and_clear + box_filter_color, mod.rs:478-518, buffers.rs:111-125)
    __syncthreads();
    uint32_t next_ticket = nunits;
    if (threadIdx.x == 0 && nunits > gridDim.x) next_ticket = atomicAdd(&queue[0], 1u);
    for (uint32_t p = (rows & 0xFFu) * TS + threadIdx.x; p < (rows >> 8) * TS; p += blockDim.x) {
        const uint32_t x = X0 + p % TS, y = Y0 + p / TS;
        if (x >= W || y >= H) continue;
        const unsigned long long o = (unsigned long long)y * W + x;
        uint32_t smp[S];
#pragma unroll
        for (int q = 0; q < S; ++q) smp[q] = sm.cb[q * C::NPIX + p];
        f.out[o] = box_filter<S>(smp);
        if (f.dbg_depth) {
#pragma unroll
            for (int q = 0; q < S; ++q) {
                f.dbg_depth[o * S + q] = sm.zb[p * S + q];
                f.dbg_color[o * S + q] = sm.cb[q * C::NPIX + p];
            }
        }
    }
    if (threadIdx.x == 0) {
        sm.misc[0] = next_ticket;
        if (next_ticket < nunits) sm.misc[5] = busy_tile(sm.tq, (next_ticket >> sm.misc[6]) / nsub);
    }
    }  // units with entries

    // ---- bins without entries: warps take runs of kEmptyRun bins (one counter update per run,
    // not per bin) and write the clear colour
    for (;;) {
        uint32_t q0 = 0;
        if (lane == 0) q0 = atomicAdd(&queue[1], (unsigned)kEmptyRun);
        q0 = __shfl_sync(0xFFFFFFFFu, q0, 0);
        if (q0 >= sm.tq.empty) break;
        const uint32_t q1 = min(q0 + (uint32_t)kEmptyRun, sm.tq.empty);
        for (uint32_t qi = q0; qi < q1; ++qi) {
            const uint32_t gt = empty_tile(sm.tq, qi);
            const FrameDev& f = frames[frame_of_tile(frames, nframes, gt)];
            const uint32_t lt = gt - f.tile_begin;
            const uint32_t edge = (uint32_t)f.ts;
            clear_tile_warp(f, (lt % f.tiles_x) * edge, (lt / f.tiles_x) * edge, edge, S);
        }
    }
    // per-block statistics
    __syncthreads();
    if (threadIdx.x == 0) {
        sm.misc[2] = 0;
        sm.misc[3] = 0;
        sm.misc[4] = 0;
    }
    __syncthreads();
    if (shaded) atomicAdd(&sm.misc[2], shaded);
    if (fsinv) atomicAdd(&sm.misc[3], fsinv);
    if (oobc) atomicAdd(&sm.misc[4], oobc);
    __syncthreads();
    if (threadIdx.x == 0) {
        if (sm.misc[2]) atomicAdd(&s.stats[STAT_SHADED], (unsigned long long)sm.misc[2]);
        if (sm.misc[3]) atomicAdd(&s.stats[STAT_FSINV], (unsigned long long)sm.misc[3]);
        if (sm.misc[4]) {
            atomicAdd(&s.stats[STAT_OOB], (unsigned long long)sm.misc[4]);
            atomicOr(s.status, ST_TEXTURE_OOB);
        }
    }
}

#include "rast_raster_warp.cuh"

// Splits each 32-pixel bin with entries into its four quadrant lists, keeping submission
// order within each (an entry goes to every quadrant its mask names). Persistent CTAs walk the
// bins with entries in the raster queue's order; the quadrant raster
// CTAs then read only their own entries. Windows of 4 consecutive entries per thread; the
// per-quadrant counts travel as 16-bit fields (two quadrants per word) through one block scan.
__global__ void __launch_bounds__(256) k_bin_split(const FrameDev* __restrict__ frames, int nframes,
                                                   const uint32_t* __restrict__ order, uint32_t ntotal,
                                                   uint32_t first_tile,
                                                   const unsigned int* __restrict__ queue, Scratch s) {
    pdl_enter();
    constexpr int kPer = 4;
    __shared__ TileQueue tq;
    load_queue(tq, queue, order, ntotal, s.status, first_tile);
    __shared__ uint32_t tmp[2][33];
    __shared__ uint32_t base[4];
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const uint32_t nbusy = tq.busy;
    for (uint32_t qi = blockIdx.x; qi < nbusy; qi += gridDim.x) {
        const uint32_t gt = busy_tile(tq, qi);
        const uint32_t n = s.tile_count[gt];
        const FrameDev& f = frames[frame_of_tile(frames, nframes, gt)];
        const unsigned long long start = s.tile_start[gt];
        const uint32_t* src = s.bins + f.bin_base + start;
        uint32_t* dst = s.qbins + f.qbin_base + 4ull * start;
        if (threadIdx.x < 4) base[threadIdx.x] = 0;
        for (uint32_t e0 = 0; e0 < n; e0 += blockDim.x * kPer) {
            uint32_t ent[kPer];
            uint32_t c01 = 0, c23 = 0;  // this thread's count per quadrant, 16 bits each
#pragma unroll
            for (int j = 0; j < kPer; ++j) {
                const uint32_t e = e0 + threadIdx.x * kPer + j;
                ent[j] = e < n ? src[e] : 0u;
                c01 += (ent[j] & 1u) + (((ent[j] >> 1) & 1u) << 16);
                c23 += ((ent[j] >> 2) & 1u) + (((ent[j] >> 3) & 1u) << 16);
            }
            // block-wide exclusive scan of both words at once
            uint32_t x01 = c01, x23 = c23;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y01 = __shfl_up_sync(0xFFFFFFFFu, x01, o), y23 = __shfl_up_sync(0xFFFFFFFFu, x23, o);
                if (lane >= (uint32_t)o) {
                    x01 += y01;
                    x23 += y23;
                }
            }
            if (lane == 31) {
                tmp[0][warp] = x01;
                tmp[1][warp] = x23;
            }
            __syncthreads();
            if (warp == 0) {
                const uint32_t w01 = lane < nw ? tmp[0][lane] : 0u, w23 = lane < nw ? tmp[1][lane] : 0u;
                uint32_t s01 = w01, s23 = w23;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t y01 = __shfl_up_sync(0xFFFFFFFFu, s01, o), y23 = __shfl_up_sync(0xFFFFFFFFu, s23, o);
                    if (lane >= (uint32_t)o) {
                        s01 += y01;
                        s23 += y23;
                    }
                }
                tmp[0][lane] = s01 - w01;
                tmp[1][lane] = s23 - w23;
                if (lane == 31) {
                    tmp[0][32] = s01;
                    tmp[1][32] = s23;
                }
            }
            __syncthreads();
            const uint32_t p01 = tmp[0][warp] + x01 - c01, p23 = tmp[1][warp] + x23 - c23;
            uint32_t o[4] = {base[0] + (p01 & 0xFFFFu), base[1] + (p01 >> 16), base[2] + (p23 & 0xFFFFu),
                             base[3] + (p23 >> 16)};
#pragma unroll
            for (int j = 0; j < kPer; ++j)
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if ((ent[j] >> q) & 1u) dst[(unsigned long long)q * n + o[q]++] = ent[j];
            __syncthreads();
            if (threadIdx.x < 4) {
                const uint32_t t = tmp[threadIdx.x >> 1][32];
                base[threadIdx.x] += (threadIdx.x & 1u) ? (t >> 16) : (t & 0xFFFFu);
            }
            __syncthreads();
        }
        if (threadIdx.x < 4) s.qcount[4ull * gt + threadIdx.x] = base[threadIdx.x];
        __syncthreads();
    }
}

// ===================================================================== launchers

// Launch with programmatic stream serialization (see pdl_enter): the kernel may be scheduled
// while its predecessor in the stream is still running and waits for it on entry.
// Pipeline kernels launched by this process (counted at enqueue, or at capture for graphs).
static std::atomic<unsigned long long> g_launches{0};
unsigned long long kernel_launches() { return g_launches.load(std::memory_order_relaxed); }

template <typename... KArgs, typename... Args>
static cudaError_t launch_pdl(void (*kernel)(KArgs...), unsigned grid, unsigned block, size_t smem,
                              cudaStream_t stream, Args... args) {
    g_launches.fetch_add(1, std::memory_order_relaxed);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

// Per-device launch set-up (multiprocessor count, raised shared-memory limits, persistent grid
// sizes), looked up once per device: a process may render on several GPUs, and
// cudaFuncSetAttribute applies to the current device only. Host threads may launch at once.
constexpr int kMaxDevices = 64;

static int current_device() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
        cudaGetLastError();
        return -1;
    }
    return dev;
}

// Multiprocessor count of the current device.
static int sm_count() {
    static std::atomic<int> sms[kMaxDevices];
    const int dev = current_device();
    if (dev < 0) return 1;
    int n = sms[dev].load(std::memory_order_relaxed);
    if (!n) {
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (n <= 0) n = 1;
        sms[dev].store(n, std::memory_order_relaxed);
    }
    return n;
}

// Persistent grid of a kernel on the current device: resident CTAs per SM x SMs, with its
// dynamic shared-memory limit raised to `bytes` (done once per device and kernel; every host
// thread computes the same).
template <typename K>
static cudaError_t persistent_grid(K kernel, int threads, size_t bytes, std::atomic<int>* cache, int& grid) {
    const int dev = current_device();
    if (dev < 0) return cudaErrorInvalidDevice;
    grid = cache[dev].load(std::memory_order_acquire);
    if (grid) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return e;
    int per = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, bytes);
    if (e != cudaSuccess) return e;
    grid = (per > 0 ? per : 1) * sm_count();
    cache[dev].store(grid, std::memory_order_release);
    return cudaSuccess;
}

template <int S, int TS>
static cudaError_t launch_raster_t(const LaunchArgs& a, uint32_t nsx) {
    const size_t bytes = sizeof(RasterSmem<S, TS>);
    const size_t wbytes = sizeof(WarpRasterSmem<S, TS>);
    static std::atomic<int> cta_cap[kMaxDevices], warp_cap[kMaxDevices];
    int grid_cap = 0, wgrid_cap = 0;
    cudaError_t e = persistent_grid(k_raster<S, TS>, kRasterThreads, bytes, cta_cap, grid_cap);
    if (e != cudaSuccess) return e;
    e = persistent_grid(k_raster_warp<S, TS>, 32 * kWarpUnitWarps, wbytes, warp_cap, wgrid_cap);
    if (e != cudaSuccess) return e;
    if (a.raster_ctas_per_sm > 0) {
        const int cap = a.raster_ctas_per_sm * sm_count();
        grid_cap = grid_cap < cap ? grid_cap : cap;
        wgrid_cap = wgrid_cap < cap ? wgrid_cap : cap;
    }
    if (a.raster_blocks == 0) return cudaSuccess;
    const uint32_t* order = a.scratch.tile_order + (unsigned long long)kOrderArrays * a.raster_tile_offset;
    // as many CTAs as there could be strips of units
    const unsigned long long units = 4ull * a.raster_blocks * nsx * nsx;
    // heavy tiles CTA-wide (none when every bin is below the threshold: the launch then only
    // helps with the bins without entries), then the light tiles one warp each
    if (a.raster_heavy_bits < 32) {
        const unsigned grid = units < (unsigned long long)grid_cap ? (unsigned)units : (unsigned)grid_cap;
        e = launch_pdl(k_raster<S, TS>, grid, kRasterThreads, bytes, a.stream, a.raster_frames, a.raster_nframes,
                       order, a.raster_blocks, a.raster_tile_offset, nsx, a.raster_queue, a.draws, a.scratch);
        if (e != cudaSuccess) return e;
    }
    if (a.raster_heavy_bits == 0) return cudaSuccess;  // every bin with entries is heavy
    const unsigned long long wunits = (units + kWarpUnitWarps - 1) / kWarpUnitWarps;
    const unsigned wgrid = wunits < (unsigned long long)wgrid_cap ? (unsigned)wunits : (unsigned)wgrid_cap;
    return launch_pdl(k_raster_warp<S, TS>, wgrid, 32 * kWarpUnitWarps, wbytes, a.stream, a.raster_frames,
                      a.raster_nframes, order, a.raster_blocks, a.raster_tile_offset, nsx, a.raster_queue, a.draws,
                      a.scratch);
}

cudaError_t launch_vertex(const LaunchArgs& a) {
    if (a.vertex_blocks == 0) return cudaSuccess;
    return launch_pdl(k_vertex, a.vertex_blocks, 256, 0, a.stream, a.draws, a.frames, a.vblocks, a.scratch);
}

cudaError_t launch_front(const LaunchArgs& a) {
    if (a.vertex_blocks + a.nchunks == 0) return cudaSuccess;
    return launch_pdl(k_front, a.vertex_blocks + a.nchunks, 256, 0, a.stream, a.chunks, a.draws, a.frames, a.vblocks,
                      a.vertex_blocks, a.front_tris, a.scratch);
}

cudaError_t launch_gather(const LaunchArgs& a) {
    if (a.scan_groups == 0) return cudaSuccess;
    return launch_pdl(k_bin_gather, a.scan_groups, kGatherThreads, 0, a.stream, a.frames, a.nframes, a.scratch);
}

cudaError_t launch_bin_count(const LaunchArgs& a) {
    if (a.nchunks == 0) return cudaSuccess;
    // the kernel's dynamic shared-memory limit (per device) only ever grows, under a lock: a
    // smaller value set by another host thread must not undercut a concurrent larger launch
    static std::mutex mu;
    static int configured[kMaxDevices] = {};
    const uint32_t band = a.max_tiles < (uint32_t)kCountBandTiles ? a.max_tiles : (uint32_t)kCountBandTiles;
    const int bytes = (int)(((band + 1) / 2) * sizeof(uint32_t));
    const int dev = current_device();
    if (dev < 0) return cudaErrorInvalidDevice;
    {
        std::lock_guard<std::mutex> lk(mu);
        if (bytes > configured[dev]) {
            cudaError_t e = cudaFuncSetAttribute(k_bin_count, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
            if (e != cudaSuccess) return e;
            configured[dev] = bytes;
        }
    }
    cudaError_t e = launch_pdl(k_bin_count, a.nchunks, 256, (size_t)bytes, a.stream, a.chunks, a.draws, a.frames,
                               a.scratch);
    if (e != cudaSuccess) return e;
    // the straddling triangles the count queued: a grid-stride pass, one warp per triangle
    const int sms = sm_count();
    // up to four resident CTAs per SM (57 registers a thread), 32 warps per chunk: a frame of
    // a few chunks spreads its straddlers over every SM, a tiny frame launches a few CTAs
    const uint32_t grid = a.nchunks < (uint32_t)sms ? 4u * a.nchunks : (uint32_t)(4 * sms);
    return launch_pdl(k_clip, grid, 256, 0, a.stream, a.draws, a.frames, a.scratch);
}

cudaError_t launch_scans(const LaunchArgs& a) {
    if (a.scan_groups == 0) return cudaSuccess;
    return launch_pdl(k_scan_cols, a.scan_groups, 1024, 0, a.stream, a.frames, a.nframes, a.scratch);
}

cudaError_t launch_bin_scatter(const LaunchArgs& a) {
    if (a.nchunks == 0) return cudaSuccess;
    return launch_pdl(k_bin_scatter, a.nchunks, kScatterThreads, 0, a.stream, a.chunks, a.draws, a.frames,
                      a.scratch);
}

cudaError_t launch_bin_split(const LaunchArgs& a, int ts) {
    if (raster_edge(ts) == ts || a.raster_blocks == 0) return cudaSuccess;
    const uint32_t cap = 8u * (uint32_t)sm_count();  // resident CTAs (2048 threads per SM)
    return launch_pdl(k_bin_split, a.raster_blocks < cap ? a.raster_blocks : cap, 256, 0, a.stream, a.raster_frames,
                      a.raster_nframes,
                      (const uint32_t*)(a.scratch.tile_order + (unsigned long long)kOrderArrays * a.raster_tile_offset),
                      a.raster_blocks, a.raster_tile_offset, (const unsigned int*)a.raster_queue, a.scratch);
}

cudaError_t launch_raster(const LaunchArgs& a, int msaa, int ts) {
    // bins of edge ts are rastered as tiles of edge raster_edge(ts) (quadrants of 32-pixel bins)
    if (ts != 8 && ts != 16 && ts != 32) return cudaErrorInvalidValue;
    const int rs = raster_edge(ts);
    const uint32_t nsx = (uint32_t)(ts / rs);
    if (msaa == 4) return rs == 8 ? launch_raster_t<4, 8>(a, nsx) : launch_raster_t<4, 16>(a, nsx);
    if (msaa == 1) return rs == 8 ? launch_raster_t<1, 8>(a, nsx) : launch_raster_t<1, 16>(a, nsx);
    return cudaErrorInvalidValue;
}

}  // namespace rast

// ===================================================================== known-answer kernel

namespace rast {

// Evaluates one pipeline device function on caller-supplied inputs (single thread). Layouts
// per op are documented beside rast_debug_kat in rast_api.cu.
__global__ void k_kat(int op, const unsigned char* __restrict__ in, unsigned char* __restrict__ out) {
    const float* fi = reinterpret_cast<const float*>(in);
    float* fo = reinterpret_cast<float*>(out);
    uint32_t* uo = reinterpret_cast<uint32_t*>(out);
    const int32_t* ii = reinterpret_cast<const int32_t*>(in);
    if (op != 5 && op != 11 && threadIdx.x != 0) return;
    switch (op) {
        case 0: {  // perspective divide of 3 clip vertices
            for (int v = 0; v < 3; ++v) {
                float4 n = persp_divide(make_float4(fi[4 * v], fi[4 * v + 1], fi[4 * v + 2], fi[4 * v + 3]));
                fo[4 * v] = n.x; fo[4 * v + 1] = n.y; fo[4 * v + 2] = n.z; fo[4 * v + 3] = n.w;
            }
            break;
        }
        case 1: {  // viewport + setup: in {i32 w, i32 h, f32 ndc[12]}
            const float* ndc = fi + 2;
            float4 sv[3];
            for (int v = 0; v < 3; ++v)
                sv[v] = viewport(make_float4(ndc[4 * v], ndc[4 * v + 1], ndc[4 * v + 2], ndc[4 * v + 3]),
                                 (float)ii[0], (float)ii[1]);
            TriSetup t;
            tri_setup(t, sv);
            for (int v = 0; v < 3; ++v) {
                fo[2 * v] = t.px[v]; fo[2 * v + 1] = t.py[v];
                fo[6 + v] = t.z[v]; fo[9 + v] = t.w[v];
                fo[13 + 2 * v] = t.nx[v]; fo[14 + 2 * v] = t.ny[v];
            }
            fo[12] = t.inv_area;
            break;
        }
        case 2:    // fragment at pixel: in {f32 screen[9], i32 x, i32 y}; out {u32 mask, f32 d[4]}
        case 4: {  // interpolate: in {screen[9], i32 x, i32 y, w[3], attrs[18]}; out attr[6]
            float4 sv[3];
            for (int v = 0; v < 3; ++v) sv[v] = make_float4(fi[3 * v], fi[3 * v + 1], fi[3 * v + 2], 1.0f);
            const uint32_t x = (uint32_t)ii[9], y = (uint32_t)ii[10];
            if (op == 4)
                for (int v = 0; v < 3; ++v) sv[v].w = fi[11 + v];
            TriSetup t;
            tri_setup(t, sv);
            // the raster kernel's coverage and sample-depth arithmetic
            const Cover<4> c = cover_pixel<4>(t.px[0], t.py[0], t.px[1], t.py[1], t.px[2], t.py[2], cover_inv(sv),
                                              t.z[0], t.z[1], t.z[2], (float)x, (float)y);
            const uint32_t cov = c.mask;
            float d[4];
            for (int q = 0; q < 4; ++q) d[q] = ((cov >> q) & 1u) ? c.z[q] : 0.0f;
            if (op == 2) {
                uo[0] = cov;
                for (int q = 0; q < 4; ++q) fo[1 + q] = d[q];
            } else {
                const float* at = fi + 14;
                float xs, ys;
                interp_point<4>(x, y, cov, xs, ys);
                float u, v, w;
                persp_bary(t.px[0], t.py[0], t.px[1], t.py[1], t.px[2], t.py[2], t.w[0], t.w[1], t.w[2], xs, ys, u, v,
                           w);
                for (int c = 0; c < 6; ++c) fo[c] = at[c] * u + at[6 + c] * v + at[12 + c] * w;
            }
            break;
        }
        case 3: {  // eval_single: in {screen[9], f32 x, f32 y}; out {e[3], u32 inside}
            float4 sv[3];
            for (int v = 0; v < 3; ++v) sv[v] = make_float4(fi[3 * v], fi[3 * v + 1], fi[3 * v + 2], 1.0f);
            TriSetup t;
            tri_setup(t, sv);
            bool in3 = true;
            for (int k = 0; k < 3; ++k) {
                fo[k] = edge_eval(t.nx[k], t.ny[k], t.px[k], t.py[k], fi[9], fi[10]);
                in3 = in3 && edge_pass_t(fo[k], edge_tie(t.nx[k], t.ny[k]));
            }
            uo[3] = in3;
            break;
        }
        case 5: {  // try_clip: in {verts[12], attrs[18]}; out {i32 result, i32 ntris, verts[ntris*12]}
            // the product path's warp clipper (k_clip): the whole warp runs this op
            const uint32_t lane = lane_id();
            ClipVert v;
            for (int k = 0; k < 4; ++k) v.p[k] = lane < 3 ? fi[4 * lane + k] : 0.0f;
            for (int k = 0; k < 6; ++k) v.a[k] = lane < 3 ? fi[12 + 6 * lane + k] : 0.0f;
            uint32_t codes[3];
            for (int q = 0; q < 3; ++q)
                codes[q] = clip_code(make_float4(fi[4 * q], fi[4 * q + 1], fi[4 * q + 2], fi[4 * q + 3]));
            int cls = clip_classify(tri2x_area(fi[0], fi[1], fi[4], fi[5], fi[8], fi[9]), codes[0], codes[1], codes[2]);
            int32_t* io = reinterpret_cast<int32_t*>(out);
            const int n = cls == 2 ? warp_clip(v, 3) : 0;
            // gather the polygon's positions to lane 0's view through shared memory
            __shared__ float poly[kMaxPoly][4];
            if (cls == 2 && n > 0 && lane < (uint32_t)n)
                for (int k = 0; k < 4; ++k) poly[lane][k] = v.p[k];
            __syncwarp();
            if (lane != 0) break;
            io[1] = 0;
            if (cls == 2) {
                if (n < 3) {
                    cls = 0;
                } else {
                    io[1] = n - 2;
                    for (int t = 0; t + 2 < n; ++t) {
                        const int vi[3] = {0, t + 1, t + 2};
                        for (int q = 0; q < 3; ++q)
                            for (int k = 0; k < 4; ++k) fo[2 + (3 * t + q) * 4 + k] = poly[vi[q]][k];
                    }
                }
            }
            io[0] = cls;
            break;
        }
        case 6: {  // bbox (unclamped viewport 65535): in points[6]; out u64[4]
            float4 sv[3];
            for (int v = 0; v < 3; ++v) sv[v] = make_float4(fi[2 * v], fi[2 * v + 1], 0.0f, 1.0f);
            uint32_t x0, x1, y0, y1;
            pixel_bbox(sv, 0xFFFFu, 0xFFFFu, x0, x1, y0, y1);
            unsigned long long* lo = reinterpret_cast<unsigned long long*>(out);
            lo[0] = x0; lo[1] = x1; lo[2] = y0; lo[3] = y1;
            break;
        }
        case 7: {  // box filter: in u32[4]; out u32
            uo[0] = box_filter<4>(reinterpret_cast<const uint32_t*>(in));
            break;
        }
        case 8: {  // to_argb: in rgba f32[4]; out u32
            uo[0] = to_argb(fi[0], fi[1], fi[2], fi[3]);
            break;
        }
        case 9: {  // texture sample (tex_argb's way for coordinates outside the texture): in {i32 w, i32 h, f32 u, f32 v, u32 texels[w*h]}; out {f32[4], u32 oob}
            bool oob = false;
            tex_sample(reinterpret_cast<const uint32_t*>(in) + 4, (uint32_t)ii[0], (uint32_t)ii[1], fi[2], fi[3],
                       fo, oob);
            uo[4] = oob;
            break;
        }
        case 10: {  // Mat4 * Vec4: in {m[16], v[4]}; out f32[4]
            for (int r = 0; r < 4; ++r) fo[r] = dot4(fi + 4 * r, fi[16], fi[17], fi[18], fi[19]);
            break;
        }
        case 11: {  // the shader's texture filter: in {u32 w, h, n, 0, f32 uv[2n], u32 texels[w*h]}; out {u32 argb[n], u32 oob[n]}
            const uint32_t* ui = reinterpret_cast<const uint32_t*>(in);
            const uint32_t n = ui[2];
            DrawDev d;
            d.set_texture(ui + 4 + 2ull * n, ui[0], ui[1]);
            for (uint32_t i = threadIdx.x; i < n; i += 32) {
                uint32_t oob = 0;
                uo[i] = tex_argb(d.tex, d.tex_w, d.tex_h, d.tex_xmax, d.tex_ymax, d.tex_small != 0, fi[4 + 2 * i],
                                 fi[5 + 2 * i], true, oob);
                uo[n + i] = oob;
            }
            break;
        }
        default:
            break;
    }
}

cudaError_t launch_kat(int op, const void* in, void* out, cudaStream_t stream) {
    // one warp: ops 5 (the warp clipper) and 11 use every lane, the others run on lane 0
    k_kat<<<1, 32, 0, stream>>>(op, static_cast<const unsigned char*>(in), static_cast<unsigned char*>(out));
    return cudaGetLastError();
}

}  // namespace rast
