// rast_types.h - device-side descriptors and scratch layout of the raster pipeline.
//
// One launch sequence renders a list of frames (scenes); each frame holds an ordered list of
// draws. Plain rendering is one frame; the batched and serving paths pass many.
//
// HBM layout (all scratch owned by the context, grown on demand, never per frame):
//   vbin[v]   float4  what binning reads of vertex v: clip x, y and screen x, y, or the clip predicates
//                     in place of clip x (rast_kernels.cu vertex_bin)
//   vscr[v]   float4  (screen x, screen y, screen z, w) after divide + viewport
//   tri_rect[t] u64   pixel box of triangle t (x0,y0,x1,y1 inclusive, 16 bits each),
//                     kRectEmpty when culled; bit 63: clipped
//   tri_aux[t]  u32   offset of the clipped polygon in clip_store, kNone when unclipped
//   clip_list[] u32×3 triangles that straddle a clip plane (draw, triangle, chunk row), clipped
//                     afterwards by one warp each (k_clip)
//   counts[frame][chunk][tile] u32  per-chunk tile histograms, then exclusive prefixes
//   tile_start / tile_count [tile]  each tile's bin range
//   bins[]    u32     per-tile lists in submission order: triangle << 5 | clipped << 4 |
//                     mask of the raster quadrants of the bin that its pixel box touches
//   qbins[]   u32     32-pixel bins only: each bin's entries split into its four 16-pixel
//                     quadrants (stable), quadrant q of bin t at 4 * start(t) + q * count(t)
// Per-sample colour and depth never touch HBM: they live in shared memory of the tile CTA.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define RAST_HD __host__ __device__
#else
#define RAST_HD
#endif

namespace rast {

constexpr uint32_t kClearColor = 0xFF191919u;  // src/rasterizer/buffers.rs:5
constexpr float kCullEps = 0.000001f;          // src/rasterizer/clipping.rs:12
constexpr int kMaxPoly = 32;                   // clip polygon capacity (a convex clip needs 9)
constexpr uint32_t kNone = 0xFFFFFFFFu;
constexpr unsigned long long kRectEmpty = ~0ull;
constexpr unsigned long long kRectClippedBit = 1ull << 63;  // pixel boxes stay below 2^15
// bins of one frame: up to kCountBandTiles are counted in one pass over a chunk's triangles
// (a 32 KB shared histogram); larger frames (any 16384 x 16384 frame fits) take one pass per
// band of kCountBandTiles bins, so the automatic bin size avoids them where it can
constexpr int kCountBandTiles = 16384;
constexpr int kMaxTilesPerFrame = 1 << 22;
// Raster tile queue of one (msaa, tile) launch group: counters [0] heavy-tile tickets, [1] empty-bin
// tickets, [2] light-tile tickets, [4 + c] bins of class c. Classes order the bins roughly heaviest
// first (0: no entries; see order_class); the bins of each class are listed by the kernel that
// counts them, in no particular order, at order_slot.
constexpr int kQueueSlots = 16;
constexpr int kQueueClass = 4;
constexpr int kClasses = 12;
constexpr int kOrderArrays = kClasses / 2;  // arrays of tiles per raster group
constexpr int kMaxRasterGroups = 8;
// Class of a bin in its raster queue by the bit length of its entry count: 0 without entries, then
// steps at 1, 4, 16, 32, 64, ... 4096 entries; the step nearest to the heavy limit 2^heavy_bits is
// moved onto it where none lies there, so that the heavy bins are whole classes (heavy_class and up).
// Steps of 2 where most bins lie: the queue's end is then filled with small tiles (steps of 4 made the
// 100k-triangle soup at 1080p 3% slower).
RAST_HD inline uint32_t order_class(uint32_t count, uint32_t heavy_bits) {
#ifdef __CUDA_ARCH__
    const uint32_t b = 32 - __clz(count), h = heavy_bits + 1;
#else
    const uint32_t b = count ? 32u - (uint32_t)__builtin_clz(count) : 0u, h = heavy_bits + 1;
#endif
    const uint32_t s2 = h == 2 ? 2u : 3u, s3 = h == 4 ? 4u : 5u, s11 = h >= 13 && h <= 31 ? h : 13u;
    if (b >= 5) return b >= s11 ? 11u : (b < 12u ? b : 12u) - 2u;
    return (b >= 1) + (b >= s2) + (b >= s3);
}
// Lowest class whose bins are rastered CTA-wide.
RAST_HD inline uint32_t heavy_class(uint32_t heavy_bits) {
    const uint32_t h = heavy_bits + 1;
    return h >= 32 ? (uint32_t)kClasses : h >= 13 ? 11u : h >= 5 ? h - 2u : h >= 4 ? 3u : h >= 2 ? 2u : 1u;
}
// Bins with at least 2^kDefaultHeavyBits entries are rastered CTA-wide, the others one warp per
// raster tile (rast_set_heavy_tile_entries)
constexpr uint32_t kDefaultHeavyBits = 0;
// bin entries: triangle << 5 | clipped << 4 | mask of the raster quadrants the box touches
constexpr int kEntShift = 5;
constexpr uint32_t kEntClipped = 1u << 4;
constexpr uint32_t kMaxFrameTris = 1u << (32 - kEntShift);

// Edge of the raster tile that one CTA owns for bins of edge ts: 32-pixel bins are rastered as
// four 16-pixel quadrants (more, smaller units balance the persistent raster kernel better).
RAST_HD constexpr int raster_edge(int ts) { return ts > 16 ? 16 : ts; }

// Triangles per binning chunk (one CTA of the count and scatter kernels; one row of per-tile
// counts): about 900 chunks for large meshes, a multiple of 256 in [256, 8192].
inline uint32_t chunk_size_for(uint32_t ntris) {
    uint32_t c = (ntris + 899u) / 900u;
    c = (c + 255u) & ~255u;
    return c < 256u ? 256u : (c > 8192u ? 8192u : c);
}

// Runs whose frames all have at most kGatherTris triangles take k_front and k_bin_gather: chunks of
// 8 front_tris triangles, scan groups of gather_edge^2 bins.
constexpr uint32_t kGatherTris = 8160;
// Triangles per warp of k_front for a run of `tris` triangles: four keep a warp's chain of clipped triangles
// short while one round of warps takes the run; a larger run fills the GPU either way, and four
// triangles then leave 20 of a warp's lanes without a corner to transform: 64 frames of 7 938 triangles at
// 320x240 214 -> 185 us a run with ten (k_front 69 -> 34 us; with eight 189). With 65 536 for kFrontFew eight
// frames of 8 000 at 640x480 take 258 us instead of 248.
constexpr uint64_t kFrontFew = 16384;
constexpr uint32_t front_tris(uint64_t tris) { return tris <= kFrontFew ? 4u : 10u; }
inline uint32_t gather_groups(uint32_t tiles_x, uint32_t tiles_y, uint32_t edge) {
    return ((tiles_x + edge - 1) / edge) * ((tiles_y + edge - 1) / edge);
}
// Blocks of 8 x 8 bins where there are enough of them for the GPU, else 4 x 4: more CTAs, each with a
// shorter list.
inline uint32_t gather_edge(uint32_t tiles_x, uint32_t tiles_y) {
    return gather_groups(tiles_x, tiles_y, 8) >= 100 ? 8 : 4;
}

// Device bytes that a one-draw frame of width x height with bins of edge ts takes while in flight (what
// run_frames reserves for it, and its image): vertex records, per-triangle boxes and straddler list, chunk
// histograms, bin tables and raster queue, bins (and quadrant lists for 32-pixel bins), clip store. `bins`:
// entries that an earlier such frame needed.
inline uint64_t frame_bytes(uint64_t nverts, uint32_t ntris, uint64_t width, uint64_t height, int ts, uint64_t bins) {
    const uint64_t tiles = ((width + ts - 1) / ts) * ((height + ts - 1) / ts);
    const uint64_t cs = chunk_size_for(ntris), chunks = (ntris + cs - 1) / cs;
    const uint64_t first = 4ull * ntris + tiles + 1024ull, cap = bins > first ? bins : first;
    const uint64_t split = raster_edge(ts) < ts ? 16ull * (cap + tiles) : 0ull;       // qbins, qcount
    return 2ull * 16 * nverts                                                          // vbin, vscr
           + (8ull + 4 + 12) * ntris                                                   // tri_rect, tri_aux, clip_list
           + 4ull * chunks * tiles + 4ull * (2 + kOrderArrays) * tiles                 // counts; start, count, order
           + 4ull * cap + split + 4ull * (32ull * ntris + 4096) + 4ull * width * height + 65536ull;
}

enum StatusBits : uint32_t {
    ST_TEXTURE_OOB = 1u << 0,
    ST_BIN_OVERFLOW = 1u << 1,
    ST_CLIP_OVERFLOW = 1u << 2,
    ST_CLIP_STORE_OVERFLOW = 1u << 3,
    ST_LOG_OVERFLOW = 1u << 4,
    ST_BAD_INDEX = 1u << 5,  // a vertex index >= the mesh's vertex count (triangle skipped)
};

enum StatSlots : int {
    STAT_SHADED = 0,
    STAT_FSINV = 1,
    STAT_OOB = 2,
    STAT_CLIP_NEED = 3,
    STAT_COUNT = 4,
};

struct alignas(16) DrawDev {
    const float* pos;      // nverts * 3
    const float* uv;       // nverts * 2
    const float* rgba;     // nverts * 4 or null
    const uint32_t* idx;   // ntris * 3
    // what the fragment shader reads, 32 bytes (two 16-byte loads)
    const uint32_t* tex;   // texture 0 (RGBA8 packed in u32), may be null unless fs == 0
    uint32_t tex_w, tex_h;
    float tex_xmax, tex_ymax;  // tex_w - 1, tex_h - 1
    int32_t fs;
    uint32_t tex_small;    // both sides below 65536: texel indices fit 32 bits (tex_argb)
    uint32_t nverts, ntris;
    uint32_t vbase;        // first vertex record of this draw
    uint32_t tbase;        // first triangle index of this draw within its frame
    uint32_t frame;
    float mvp[16];         // (P * V) * W, row-major

    RAST_HD void set_texture(const uint32_t* data, uint32_t w, uint32_t h) {
        tex = data;
        tex_w = w;
        tex_h = h;
        tex_xmax = (float)(uint64_t)(w - 1u);
        tex_ymax = (float)(uint64_t)(h - 1u);
        tex_small = w < 65536u && h < 65536u;
    }
};

struct FrameDev {
    uint32_t width, height;
    int32_t msaa;
    int32_t ts;            // tile edge in pixels
    uint32_t tiles_x, tiles_y, ntiles;
    uint32_t draw_begin, draw_count;
    uint32_t ntris;
    uint32_t nchunks;
    uint32_t tile_begin;   // global index of this frame's first tile
    uint32_t group_begin;  // first scan group of this frame (32 tiles, or gather_bins^2 in a small run)
    uint32_t rect_base;    // global index of this frame's first triangle in tri_rect/tri_aux
    unsigned long long count_base;  // offset of counts[frame]
    unsigned long long bin_base;    // offset of this frame's bins
    unsigned long long bin_cap;     // bins reserved for this frame
    unsigned long long qbin_base;   // offset of this frame's quadrant lists (32-pixel bins)
    uint32_t queue;        // raster group (its counters: Scratch::queues + kQueueSlots * queue)
    uint32_t order_begin;  // the group's first tile; its lists start at kOrderArrays * order_begin
    uint32_t order_n;      // tiles of the group
    uint32_t heavy_bits;   // bins of >= 2^heavy_bits entries are rastered CTA-wide (32: none)
    uint32_t gather_bins;  // block edge of k_bin_gather
    uint32_t order_coarse; // only classes 0 and 1 are used: the group's lists need one array
    float clear_depth;
    uint32_t* out;         // width * height ARGB (device)
    float* dbg_depth;      // optional [y][x][s]
    uint32_t* dbg_color;
};

struct ChunkDev {
    uint32_t draw;
    uint32_t tri_begin;    // first triangle within the draw
    uint32_t tri_count;
    uint32_t row;          // chunk index within the frame
};

struct Scratch {
    float4* vbin;
    float4* vscr;
    unsigned long long* tri_rect;
    uint32_t* tri_aux;
    uint32_t* counts;
    uint32_t* tile_start;
    uint32_t* tile_count;
    uint32_t* tile_order;               // raster queues: kOrderArrays arrays of tiles per raster group
    unsigned int* queues;               // raster queue counters
    uint32_t* bins;
    uint32_t* qbins;                    // per 32-pixel bin: its entries split by raster quadrant
    uint32_t* qcount;                   // [4 * tile + quadrant] entries in each quadrant list
    float* clip_store;
    unsigned long long clip_cap;        // floats
    uint32_t* clip_list;                // triangles needing Sutherland-Hodgman: draw, triangle, chunk row
    unsigned long long clip_list_cap;   // entries
    unsigned int* clip_n;
    unsigned long long* clip_used;      // floats allocated this frame
    uint32_t* status;
    unsigned long long* stats;          // StatSlots
    unsigned long long* frame_need;     // per frame: bin entries allocated so far, then needed
    uint32_t* log;
    unsigned long long* log_n;
    unsigned long long log_cap;
};

}  // namespace rast
