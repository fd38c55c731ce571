// rast_raster_warp.cuh - warp-per-tile raster for light tiles (included by rast_kernels.cu).
//
// A raster tile with few bin entries leaves the warps of the CTA-wide kernel (k_raster) running
// partial warps between block barriers. Here one warp owns a whole tile: it stages the tile's
// items 32 at a time, one per lane and held in that lane's registers (other lanes read them
// with shuffles, which keeps shared memory for the samples and rings: 5 CTAs of 4 warps per
// SM), walks their candidate pixels 32 at a time, depth-tests the covered fragments in
// submission order and shades the passed ones, with full warps and no block barrier. The
// arithmetic is the same device functions as k_raster (coverage, sample depths, tie rule,
// interpolation, shaders, resolve), so results are bit-identical; only the work split differs.
//
// The persistent kernel takes light tiles (the bins of the raster queue below the heavy classes,
// heaviest class first) from their own counter, then helps clear the bins without entries. k_raster takes the heavy tiles.

constexpr int kWarpUnitWarps = 4;  // warps (independent tiles) per CTA of k_raster_warp
// CTAs per SM the launch bounds aim at: with 4 samples the shared sample tiles allow 5; with
// one sample registers do (6 would spill)
constexpr int kWarpUnitCtas = 5;

template <int S, int TS>
struct alignas(16) WarpUnitSmem {
    static constexpr int NPIX = TS * TS;
    static constexpr int IB = 32;  // items per batch (one per lane)
    static constexpr int QC = 64;  // ring entries
    float zb[NPIX * S];            // pixel-major: the samples of pixel p at p * S
    uint32_t cb[NPIX * S];         // sample-major: sample k of pixel p at k * NPIX + p
    float qz[QC][S];               // sample depths of the fragment ring, NaN where not covered
    uint2 run[32];                 // non-empty spans of a group: start, item | row << 8 | first column << 16
    uint32_t q[QC];   // ring of covered fragments, in submission order: item | pixel << 8 | mask << 16
    uint32_t sq[QC];  // ring of depth-passed fragments waiting for the shader: item | pixel << 8 | mask << 16
    uint8_t rowed[IB];  // items with rows, in order
};

template <int S, int TS>
struct WarpRasterSmem {
    TileQueue tq;
    WarpUnitSmem<S, TS> u[kWarpUnitWarps];
};

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v) {
    const uint32_t lane = lane_id();
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, v, o);
        if (lane >= (uint32_t)o) v += y;
    }
    return v;
}

// One item of a warp batch (a triangle, or one fan triangle of a clipped polygon), held by the
// lane of its slot: screen points, depths, w, texture coordinates, 1 / 2x area, tile-local box
// (x0 | y0 << 8 | x1 << 16 | y1 << 24, 0: nothing to do), frame triangle and draw << 8 | sub.
struct WItem {
    float px[3], py[3], z[3], w[3], inv;
    float uv[6];
    uint32_t rect, tri, meta;
};

// Stages item k of a bin entry (triangle g, clipped polygon at aux or kNone) into `it`, as
// stage_entry does for k_raster.
template <int TS>
__device__ __forceinline__ void wstage_item(WItem& it, const FrameDev& f, const DrawDev* __restrict__ draws,
                                            const Scratch& s, uint32_t g, uint32_t aux, uint32_t k, uint32_t X0,
                                            uint32_t Y0, uint32_t row0, uint32_t row1, float ztile) {
    const uint32_t di = find_draw(draws, f, g);
    const DrawDev& d = draws[di];
    float4 sv[3];
    float uv[3][2] = {{0.0f, 0.0f}, {0.0f, 0.0f}, {0.0f, 0.0f}};
    if (aux == kNone) {
        const uint32_t tri = g - d.tbase;
        const uint32_t ii[3] = {__ldg(d.idx + 3ull * tri), __ldg(d.idx + 3ull * tri + 1),
                                __ldg(d.idx + 3ull * tri + 2)};
        const bool tex = d.fs == 0;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            sv[q] = s.vscr[d.vbase + ii[q]];
            if (tex) {
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
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        it.px[q] = sv[q].x;
        it.py[q] = sv[q].y;
        it.z[q] = sv[q].z;
        it.w[q] = sv[q].w;
        it.uv[2 * q] = uv[q][0];
        it.uv[2 * q + 1] = uv[q][1];
    }
    // 1 / triangle_2x_area (RasterizerTriangle::new, src/rasterizer/mod.rs:206)
    it.inv = cover_inv(sv);
    uint32_t bx0, bx1, by0, by1;
    pixel_bbox(sv, f.width, f.height, bx0, bx1, by0, by1);
    const uint32_t cx0 = max(bx0, X0), cx1 = min(bx1, X0 + TS);
    const uint32_t cy0 = max(by0, Y0 + row0), cy1 = min(by1, Y0 + row1);
    // hidden items (depth_cull) cover nothing that could pass the strict depth test
    const bool nonempty = bx0 < bx1 && by0 < by1 && cx0 < cx1 && cy0 < cy1 &&
                          !depth_cull(sv[0].z, sv[1].z, sv[2].z, ztile);
    it.rect = nonempty ? ((cx0 - X0) | ((cy0 - Y0) << 8) | ((cx1 - X0) << 16) | ((cy1 - Y0) << 24)) : 0u;
    it.tri = g;
    it.meta = (di << 8) | k;
}

__device__ __forceinline__ float shfl_f(float v, uint32_t src) { return __shfl_sync(0xFFFFFFFFu, v, src); }
__device__ __forceinline__ uint32_t shfl_u(uint32_t v, uint32_t src) { return __shfl_sync(0xFFFFFFFFu, v, src); }

// Depth test of up to 32 queued fragments (lane = fragment, ring order = submission order):
// fragments of one pixel in rounds of increasing rank, as warp_depth does for k_raster.
template <int S, int TS>
__device__ __forceinline__ void wdepth(WarpUnitSmem<S, TS>& sm, const WItem& my, uint32_t head, uint32_t n,
                                       uint32_t& stail, const Scratch& s, uint32_t X0, uint32_t Y0,
                                       uint32_t& shaded, uint32_t& fsinv) {
    using U = WarpUnitSmem<S, TS>;
    const uint32_t lane = lane_id();
    const bool valid = lane < n;
    const uint32_t q = (head + lane) & (U::QC - 1);
    uint32_t fr = 0;
    float z[S];
#pragma unroll
    for (int k = 0; k < S; ++k) z[k] = 0.0f;
    if (valid) {
        fr = sm.q[q];
        load_samples<S>(sm.qz[q], z);
    }
    // the fragment log (debug) names the fragment's triangle: read from the item's lane
    uint32_t ltri = 0, lmeta = 0;
    if (s.log) {
        ltri = shfl_u(my.tri, fr & 31u);
        lmeta = shfl_u(my.meta, fr & 31u);
    }
    const uint32_t pix = (fr >> 8) & 0xFFu;
    // windows of one item need no match (see warp_depth): a captured batch of 20 scenes 1087 -> 1040 us,
    // with the same test in the shader
    uint32_t rank = 0, maxr = 0;
    const uint32_t fr0 = __shfl_sync(0xFFFFFFFFu, fr, 0);  // every lane
    if (!__all_sync(0xFFFFFFFFu, (!valid) | (((fr ^ fr0) & 0xFFu) == 0))) {
        const uint32_t key = valid ? pix : 0x10000u + lane;
        rank = __popc(__match_any_sync(0xFFFFFFFFu, key) & lanemask_lt());
        maxr = __reduce_max_sync(0xFFFFFFFFu, rank);
    }
    uint32_t dm = 0;
    for (uint32_t r = 0; r <= maxr; ++r) {
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
                log_fragment(s, ltri, lmeta & 0xFFu, ((Y0 + pix / TS) << 16) | (X0 + pix % TS),
                             (dm << 8) | (fr >> 16));
        }
        __syncwarp();
    }
    const uint32_t bal = __ballot_sync(0xFFFFFFFFu, dm != 0);
    if (dm) {
        sm.sq[(stail + __popc(bal & lanemask_lt())) & (U::QC - 1)] = (fr & 0xFFFFu) | (dm << 16);
        shaded += __popc(dm);
        fsinv += 1;
    }
    stail += __popc(bal);
    __syncwarp();
}

// Fragment shader and colour write of up to 32 fragments of the shade ring, as warp_shade does
// for k_raster; each lane reads its fragment's item from the item's lane.
template <int S, int TS>
__device__ __forceinline__ void wshade(WarpUnitSmem<S, TS>& sm, const WItem& my, uint32_t head, uint32_t n, const DrawDev* __restrict__ draws,
                                      const FrameDev& f, const Scratch& s, uint32_t X0, uint32_t Y0,
                                      uint32_t& oobc) {
    using U = WarpUnitSmem<S, TS>;
    const uint32_t lane = lane_id();
    const bool valid = lane < n;
    const uint32_t fr = valid ? sm.sq[(head + lane) & (U::QC - 1)] : 0u;
    const uint32_t it = fr & 31u;
    float px[3], py[3], w[3], tuv[6];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        px[k] = shfl_f(my.px[k], it);
        py[k] = shfl_f(my.py[k], it);
        w[k] = shfl_f(my.w[k], it);
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) tuv[k] = shfl_f(my.uv[k], it);
    const uint32_t meta = shfl_u(my.meta, it), tri = shfl_u(my.tri, it);
    const uint32_t pix = (fr >> 8) & 0xFFu, dm = fr >> 16;
    // FS::Debug reads sample 0's depth, computed again
    float z[3] = {0.0f, 0.0f, 0.0f}, inv = 0.0f;
    if (__any_sync(0xFFFFFFFFu, valid && draws[meta >> 8].fs == 2)) {
#pragma unroll
        for (int k = 0; k < 3; ++k) z[k] = shfl_f(my.z[k], it);
        inv = shfl_f(my.inv, it);
    }
    uint32_t argb = 0;
    if (valid) {
        float xs, ys;
        interp_point<S>(X0 + pix % TS, Y0 + pix / TS, dm, xs, ys);
        float u, v, ww;
        persp_bary(px[0], py[0], px[1], py[1], px[2], py[2], w[0], w[1], w[2], xs, ys, u, v, ww);
        const ShadeDraw d = shade_draw(&draws[meta >> 8]);
        if (d.fs == 0) {
            // FS::Texture (upstream src/main.rs:214-216)
            const float tu = tuv[0] * u + tuv[2] * v + tuv[4] * ww;
            const float tv = tuv[1] * u + tuv[3] * v + tuv[5] * ww;
            argb = tex_argb(d.tex, d.tex_w, d.tex_h, d.xmax, d.ymax, d.small, tu, tv, f.dbg_color != nullptr, oobc);
        } else {
            float col[4];
            if (d.fs == 1) {
                // FS::Color (upstream src/main.rs:217)
                float vc[3][4];
                item_colours(draws[meta >> 8], f, s, tri, meta & 0xFFu, vc);
#pragma unroll
                for (int c = 0; c < 4; ++c) col[c] = vc[0][c] * u + vc[1][c] * v + vc[2][c] * ww;
            } else {
                // FS::Debug (upstream src/main.rs:218-220): grayscale(frag_coords.depths[0]), 0 where
                // sample 0 is not covered
                const Cover<S> cv = cover_pixel<S>(px[0], py[0], px[1], py[1], px[2], py[2], inv, z[0], z[1], z[2],
                                                   (float)(X0 + pix % TS), (float)(Y0 + pix / TS));
                const float z0 = (cv.mask & 1u) ? cv.z[0] : 0.0f;
                col[0] = z0;
                col[1] = z0;
                col[2] = z0;
                col[3] = 1.0f;
            }
            argb = to_argb(col[0], col[1], col[2], col[3]);
        }
    }
    uint32_t rank = 0, maxr = 0;  // windows of one item need no match, as in wdepth
    const uint32_t it0 = __shfl_sync(0xFFFFFFFFu, it, 0);  // every lane
    if (!__all_sync(0xFFFFFFFFu, (!valid) | (it == it0))) {
        const uint32_t key = valid ? pix : 0x10000u + lane;
        rank = __popc(__match_any_sync(0xFFFFFFFFu, key) & lanemask_lt());
        maxr = __reduce_max_sync(0xFFFFFFFFu, rank);
    }
    for (uint32_t r = 0; r <= maxr; ++r) {
        const bool act = valid && rank == r;
#pragma unroll
        for (int k = 0; k < S; ++k)
            if (act & (((dm >> k) & 1u) != 0)) sm.cb[k * U::NPIX + pix] = argb;
        __syncwarp();
    }
}

// Resolve (resolve_and_clear + box_filter_color, mod.rs:478-518, buffers.rs:111-125) of the
// warp's tile: four consecutive pixels of a row per lane with 16-byte stores where the image
// row allows them, one pixel per lane otherwise (image edges, unaligned outputs, sample capture).
template <int S, int TS>
__device__ __forceinline__ void wresolve(const WarpUnitSmem<S, TS>& sm, const FrameDev& f, uint32_t X0, uint32_t Y0,
                                         uint32_t row0, uint32_t row1) {
    using U = WarpUnitSmem<S, TS>;
    const uint32_t lane = lane_id();
    const uint32_t W = f.width, H = f.height;
    const bool vec = !f.dbg_depth && (W & 3u) == 0 && X0 + TS <= W &&
                     (reinterpret_cast<uintptr_t>(f.out) & 15u) == 0;
    if (vec) {
        for (uint32_t p = row0 * TS + 4 * lane; p < row1 * TS; p += 128) {
            const uint32_t y = Y0 + p / TS;
            if (y >= H) break;  // rows go down with p
            uint4 c[S];
#pragma unroll
            for (int k = 0; k < S; ++k) c[k] = *reinterpret_cast<const uint4*>(&sm.cb[k * U::NPIX + p]);
            uint32_t px[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                uint32_t smp[S];
#pragma unroll
                for (int k = 0; k < S; ++k) smp[k] = j == 0 ? c[k].x : j == 1 ? c[k].y : j == 2 ? c[k].z : c[k].w;
                px[j] = box_filter<S>(smp);
            }
            *reinterpret_cast<uint4*>(f.out + (unsigned long long)y * W + X0 + p % TS) =
                make_uint4(px[0], px[1], px[2], px[3]);
        }
        return;
    }
    for (uint32_t p = row0 * TS + lane; p < row1 * TS; p += 32) {
        const uint32_t x = X0 + p % TS, y = Y0 + p / TS;
        if (x >= W || y >= H) continue;
        const unsigned long long o = (unsigned long long)y * W + x;
        uint32_t smp[S];
#pragma unroll
        for (int k = 0; k < S; ++k) smp[k] = sm.cb[k * U::NPIX + p];
        f.out[o] = box_filter<S>(smp);
        if (f.dbg_depth) {
#pragma unroll
            for (int k = 0; k < S; ++k) {
                f.dbg_depth[o * S + k] = sm.zb[p * S + k];
                f.dbg_color[o * S + k] = sm.cb[k * U::NPIX + p];
            }
        }
    }
}

// One light tile (or strip of its rows) by one warp: the entries in submission order, 32 items at a time.
// (A) the items of the next entries, one per lane (a lane finds its entry and fan triangle
// from the entries' running item counts); (B) per item (lane) its candidate pixels: the whole
// tile-local box, or for boxes of kTrimMin+ columns each row trimmed by line_span; (C) the
// candidates 32 at a time - coverage (EdgeFunctions::eval, mod.rs:134-146) and sample depths
// (RasterizerTriangle::fragment, mod.rs:225-253) - into the fragment ring, ordered depth test
// into the shade ring, shading; both rings are drained before the next batch replaces the items
// they refer to. Then the resolve.
template <int S, int TS>
__device__ __forceinline__ void warp_unit(WarpUnitSmem<S, TS>& sm, const FrameDev& f,
                                          const DrawDev* __restrict__ draws, const Scratch& s,
                                          const uint32_t* __restrict__ bins, uint32_t nent, uint32_t mybit,
                                          uint32_t X0, uint32_t Y0, uint32_t row0, uint32_t row1,
                                          uint32_t& shaded, uint32_t& fsinv, uint32_t& oobc) {
    using U = WarpUnitSmem<S, TS>;
    const uint32_t lane = lane_id();
    {
        const float4 zc = make_float4(f.clear_depth, f.clear_depth, f.clear_depth, f.clear_depth);
        const uint4 cc = make_uint4(kClearColor, kClearColor, kClearColor, kClearColor);
        float4* z4 = reinterpret_cast<float4*>(sm.zb);
        uint4* c4 = reinterpret_cast<uint4*>(sm.cb);
        for (uint32_t i = lane; i < (uint32_t)(U::NPIX * S / 4); i += 32) {
            z4[i] = zc;
            c4[i] = cc;
        }
    }
    __syncwarp();
    WItem my;  // the item of this lane's slot in the current batch
    uint32_t pos = 0, batch = 0;
    // depth_cull bound: the clear depth at first; NaN (no culling) while the fragment log
    // records depth-failed fragments too
    float zt = s.log ? __int_as_float(0x7FC00000) : f.clear_depth;
    while (pos < nent) {
        // the largest stored depth, refreshed before batches 1, 2, 4, 8, ...
        if (!s.log && batch > 0 && (batch & (batch - 1)) == 0) {
            uint32_t zm = 0;
            for (uint32_t i = row0 * (TS * S) + lane; i < row1 * (TS * S); i += 32)
                zm = max(zm, float_to_ordered(sm.zb[i]));
            zt = ordered_to_float(__reduce_max_sync(0xFFFFFFFFu, zm));
        }
        ++batch;
        // ---- A. items of the next entries that touch this tile, while they fit the batch
        uint32_t nit = 0;
        my.rect = 0;
        while (pos < nent) {
            const uint32_t e = pos + lane;
            uint32_t g = 0, aux = kNone, nitems = 0;
            if (e < nent) {
                const uint32_t ent = bins[e];
                if (ent & mybit) {
                    g = ent >> kEntShift;
                    nitems = 1;
                    if (ent & kEntClipped) {
                        aux = s.tri_aux[f.rect_base + g];
                        // a fan of at most kMaxPoly - 2 <= IB triangles (k_clip stores 3..kMaxPoly
                        // vertices); the bound keeps every entry within one batch
                        nitems = min((uint32_t)__float_as_int(s.clip_store[aux]) - 2u, (uint32_t)U::IB);
                    }
                }
            }
            const uint32_t incl = warp_incl_scan(nitems);
            // running item counts only grow along the lanes, so the entries that fit are a prefix
            const bool fits = e < nent && nit + incl <= (uint32_t)U::IB;
            const uint32_t take = __popc(__ballot_sync(0xFFFFFFFFu, fits));
            const uint32_t win = take ? __shfl_sync(0xFFFFFFFFu, incl, take - 1) : 0u;  // items taken
            // slot lane gets item q = lane - nit of this window: entry src, fan triangle k
            const uint32_t qi = lane - nit;  // wraps for lanes below nit (not staged)
            uint32_t src = 0;
#pragma unroll
            for (int st = 16; st > 0; st >>= 1) {
                const uint32_t v = __shfl_sync(0xFFFFFFFFu, incl, src + st - 1);
                if (v <= qi) src += st;
            }
            src = min(src, 31u);
            const uint32_t sg = __shfl_sync(0xFFFFFFFFu, g, src), saux = __shfl_sync(0xFFFFFFFFu, aux, src);
            const uint32_t sk = qi - (__shfl_sync(0xFFFFFFFFu, incl, src) - __shfl_sync(0xFFFFFFFFu, nitems, src));
            if (lane >= nit && lane < nit + win) wstage_item<TS>(my, f, draws, s, sg, saux, sk, X0, Y0, row0, row1, zt);
            nit += win;
            pos += take;
            if (take < 32) break;  // the batch is full, or the entries ran out
        }
        // ---- B. the rows of the items' boxes in submission order, 32 at a time, one span per lane (a
        // lane finds its item by counting the marks of the items that start up to its row): boxes of
        // kTrimMin+ columns trimmed by line_span_pts; the non-empty spans go to `run`
        uint32_t geo = 0, nrows = 0;  // x0 | y0 << 8 | x1 << 16
        if (lane < nit) {
            geo = my.rect & 0xFFFFFFu;
            nrows = (my.rect >> 24) - ((my.rect >> 8) & 0xFFu);
        }
        const uint32_t rincl = warp_incl_scan(nrows);
        const uint32_t rtot = __shfl_sync(0xFFFFFFFFu, rincl, 31);
        const uint32_t rowed = __ballot_sync(0xFFFFFFFFu, nrows != 0);
        const uint32_t rstart = nrows ? rincl - nrows : 0xFFFFFFFFu;
        if (nrows) sm.rowed[__popc(rowed & lanemask_lt())] = (uint8_t)lane;
        __syncwarp();
        const uint32_t upto = lanemask_lt() | (1u << lane);
        uint32_t rbefore = 0xFFFFFFFFu;  // items that start in earlier groups, less one
        // ---- C. the spans' candidates, 32 at a time, in submission order. One loop takes the groups, their
        // windows and, after the last, the rings' rests, so that the depth test and the shader are
        // inlined once each: with a second copy of both for the rests the kernel waited for
        // instructions (2.2 of 9 cycles per issue with four samples).
        uint32_t head = 0, tail = 0, shead = 0, stail = 0;
        uint32_t gb = 0, pb = 0, total = 0, start = 0xFFFFFFFFu;
        uint32_t before = 0xFFFFFFFFu;  // spans that start in earlier windows, less one
        for (;;) {
            while (pb >= total && gb < rtot) {  // the next group with candidates
                uint32_t c = 0, sp = 0;
                {
                    const uint32_t marks = __reduce_or_sync(0xFFFFFFFFu, rstart - gb < 32u ? 1u << (rstart - gb) : 0u);
                    const uint32_t j = sm.rowed[rbefore + __popc(marks & upto)];
                    rbefore += __popc(marks);
                    const float px[3] = {shfl_f(my.px[0], j), shfl_f(my.px[1], j), shfl_f(my.px[2], j)};
                    const float py[3] = {shfl_f(my.py[0], j), shfl_f(my.py[1], j), shfl_f(my.py[2], j)};
                    const bool finite = fabsf(shfl_f(my.inv, j)) <= FLT_MAX;
                    const uint32_t gj = shfl_u(geo, j), rj = shfl_u(rstart, j);
                    if (gb + lane < rtot) {
                        const uint32_t ly = ((gj >> 8) & 0xFFu) + (gb + lane - rj);
                        uint32_t a0 = gj & 0xFFu, a1 = gj >> 16;
                        if (a1 - a0 >= kTrimMin && finite) line_span_pts<S, TS>(px, py, 0u, ly, X0, Y0, a0, a1);
                        c = a1 - a0;
                        sp = j | (ly << 8) | (a0 << 16);
                    }
                }
                const uint32_t incl = warp_incl_scan(c);
                total = __shfl_sync(0xFFFFFFFFu, incl, 31);
                const uint32_t full = __ballot_sync(0xFFFFFFFFu, c != 0);
                start = c ? incl - c : 0xFFFFFFFFu;
                if (c) sm.run[__popc(full & lanemask_lt())] = make_uint2(start, sp);
                __syncwarp();
                gb += 32;
                pb = 0;
                before = 0xFFFFFFFFu;
            }
            const bool more = pb < total;
            if (more) {
                const uint32_t p = pb + lane;
                const uint32_t marks = __reduce_or_sync(0xFFFFFFFFu, start - pb < 32u ? 1u << (start - pb) : 0u);
                const uint2 r = sm.run[before + __popc(marks & upto)];
                before += __popc(marks);
                const uint32_t it = r.y & 31u;
                // the item's points, depths and 1 / 2x area from its lane
                const float p0x = shfl_f(my.px[0], it), p0y = shfl_f(my.py[0], it);
                const float p1x = shfl_f(my.px[1], it), p1y = shfl_f(my.py[1], it);
                const float p2x = shfl_f(my.px[2], it), p2y = shfl_f(my.py[2], it);
                const float z0 = shfl_f(my.z[0], it), z1 = shfl_f(my.z[1], it), z2 = shfl_f(my.z[2], it);
                const float inv = shfl_f(my.inv, it);
                uint32_t cov = 0, pix = 0;
                float z[S];
#pragma unroll
                for (int k = 0; k < S; ++k) z[k] = 0.0f;
                if (p < total) {
                    const uint32_t ly = (r.y >> 8) & 0xFFu, lx = (r.y >> 16) + (p - r.x);
                    pix = ly * TS + lx;
                    const float fx = (float)(X0 + lx), fy = (float)(Y0 + ly);
                    const Cover<S> cv = cover_pixel<S>(p0x, p0y, p1x, p1y, p2x, p2y, inv, z0, z1, z2, fx, fy);
                    cov = cv.mask;
#pragma unroll
                    for (int k = 0; k < S; ++k) z[k] = ((cov >> k) & 1u) ? cv.z[k] : __int_as_float(0x7FC00000);
                }
                const uint32_t bal = __ballot_sync(0xFFFFFFFFu, cov != 0);
                if (cov) {
                    const uint32_t q = (tail + __popc(bal & lanemask_lt())) & (U::QC - 1);
                    sm.q[q] = it | (pix << 8) | (cov << 16);
                    store_samples<S>(sm.qz[q], z);
                }
                tail += __popc(bal);
                __syncwarp();
                pb += 32;
            }
            if (tail - head >= (more ? 32u : 1u)) {
                const uint32_t n = min(tail - head, 32u);
                wdepth<S, TS>(sm, my, head, n, stail, s, X0, Y0, shaded, fsinv);
                head += n;
            }
            if (stail - shead >= (more ? 32u : 1u)) {
                const uint32_t n = min(stail - shead, 32u);
                wshade<S, TS>(sm, my, shead, n, draws, f, s, X0, Y0, oobc);
                shead += n;
            }
            if (!more && tail == head && stail == shead) break;
        }
        __syncwarp();
    }
    __syncwarp();
    wresolve<S, TS>(sm, f, X0, Y0, row0, row1);
    __syncwarp();
}

// Persistent warp-per-tile raster kernel over the light tiles of one raster launch: the bins
// past the heavy classes, times nsx * nsx quadrants, taken one tile per warp from queue[2]; then bins
// without entries from queue[1], like k_raster.
template <int S, int TS>
__global__ void __launch_bounds__(32 * kWarpUnitWarps, kWarpUnitCtas) k_raster_warp(const FrameDev* __restrict__ frames,
                                                                     int nframes,
                                                                     const uint32_t* __restrict__ order,
                                                                     uint32_t ntotal, uint32_t first_tile,
                                                                     uint32_t nsx,
                                                                     unsigned int* __restrict__ queue,
                                                                     const DrawDev* __restrict__ draws,
                                                                     Scratch s) {
    pdl_enter();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    WarpRasterSmem<S, TS>& sh = *reinterpret_cast<WarpRasterSmem<S, TS>*>(smem_raw);
    const uint32_t warp = threadIdx.x >> 5, lane = lane_id();
    WarpUnitSmem<S, TS>& sm = sh.u[warp];
    load_queue(sh.tq, queue, order, ntotal, s.status, first_tile);
    const uint32_t nheavy = heavy_tiles(sh.tq, frames[0].heavy_bits);
    const uint32_t nsub = nsx * nsx;
    // units of the light bins, in strips where they are few. (Strips of the deepest bins, whose length sets
    // a launch's when it runs alone - 17% less for the one-sample scenes of a batch of 20 - cost
    // 1% where the batch's other launch fills the tail, which a mixed batch always has.)
    const uint32_t nwhole = (sh.tq.busy - nheavy) * nsub;
    const uint32_t places = gridDim.x * kWarpUnitWarps;
    const uint32_t ssh = strips_for(nwhole, places), nlight = nwhole << ssh;
    uint32_t shaded = 0, fsinv = 0, oobc = 0;
    // with no more units than warps, one unit per warp by its place, SMs first (see k_raster)
    const bool few = nlight <= places;
    for (bool more = true; more; more = !few) {
        uint32_t qi = warp * gridDim.x + blockIdx.x;
        if (!few) {
            if (lane == 0) qi = atomicAdd(&queue[2], 1u);
            qi = __shfl_sync(0xFFFFFFFFu, qi, 0);
        }
        if (qi >= nlight) break;
        const uint32_t row0 = (qi & ((1u << ssh) - 1u)) * (TS >> ssh), row1 = row0 + (TS >> ssh);
        const uint32_t sub = (qi >> ssh) % nsub, gt = busy_tile(sh.tq, nheavy + (qi >> ssh) / nsub);
        const FrameDev& f = frames[frame_of_tile(frames, nframes, gt)];
        const uint32_t lt = gt - f.tile_begin;
        const uint32_t X0 = (lt % f.tiles_x) * (uint32_t)f.ts + (sub % nsx) * TS;
        const uint32_t Y0 = (lt / f.tiles_x) * (uint32_t)f.ts + (sub / nsx) * TS;
        uint32_t nent;
        const uint32_t* bins;
        if (nsub > 1) {
            nent = s.qcount[4ull * gt + sub];
            bins = s.qbins + f.qbin_base + 4ull * s.tile_start[gt] + (unsigned long long)sub * s.tile_count[gt];
        } else {
            nent = s.tile_count[gt];
            bins = s.bins + f.bin_base + s.tile_start[gt];
        }
        warp_unit<S, TS>(sm, f, draws, s, bins, nent, 1u << sub, X0, Y0, row0, row1, shaded, fsinv, oobc);
    }
    // bins without entries: runs of kEmptyRun bins per counter update, the clear colour
    for (;;) {
        uint32_t q0 = 0;
        if (lane == 0) q0 = atomicAdd(&queue[1], (unsigned)kEmptyRun);
        q0 = __shfl_sync(0xFFFFFFFFu, q0, 0);
        if (q0 >= sh.tq.empty) break;
        const uint32_t q1 = min(q0 + (uint32_t)kEmptyRun, sh.tq.empty);
        for (uint32_t qi = q0; qi < q1; ++qi) {
            const uint32_t gt = empty_tile(sh.tq, qi);
            const FrameDev& f = frames[frame_of_tile(frames, nframes, gt)];
            const uint32_t lt = gt - f.tile_begin;
            const uint32_t edge = (uint32_t)f.ts;
            clear_tile_warp(f, (lt % f.tiles_x) * edge, (lt / f.tiles_x) * edge, edge, S);
        }
    }
    shaded = __reduce_add_sync(0xFFFFFFFFu, shaded);
    fsinv = __reduce_add_sync(0xFFFFFFFFu, fsinv);
    oobc = __reduce_add_sync(0xFFFFFFFFu, oobc);
    if (lane == 0) {
        if (shaded) atomicAdd(&s.stats[STAT_SHADED], (unsigned long long)shaded);
        if (fsinv) atomicAdd(&s.stats[STAT_FSINV], (unsigned long long)fsinv);
        if (oobc) {
            atomicAdd(&s.stats[STAT_OOB], (unsigned long long)oobc);
            atomicOr(s.status, ST_TEXTURE_OOB);
        }
    }
}
