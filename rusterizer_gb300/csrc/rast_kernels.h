// rast_kernels.h - launch interface between the host runtime and the kernels.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

#include "rast_types.h"

namespace rast {

struct LaunchArgs {
    cudaStream_t stream;
    const DrawDev* draws;
    const FrameDev* frames;
    int nframes;
    const ChunkDev* chunks;
    uint32_t nchunks;
    const uint2* vblocks;  // (draw, first vertex) per 256-vertex block
    uint32_t vertex_blocks;
    uint32_t front_tris;   // small runs: triangles per warp of k_front (a chunk holds 8 times that)
    uint32_t scan_groups;  // scan groups over all frames
    uint32_t max_tiles;    // largest per-frame tile count
    // raster launch over one (msaa, tile) group of consecutive frames
    const FrameDev* raster_frames;
    int raster_nframes;
    uint32_t raster_tile_offset;
    uint32_t raster_blocks;        // tiles in the group
    unsigned int* raster_queue;    // the group's kQueueSlots tile-queue counters (zeroed per frame)
    uint32_t raster_heavy_bits;    // bins of >= 2^bits entries are rastered CTA-wide (32: none)
    int raster_ctas_per_sm;        // persistent raster CTAs per SM (0: as many as fit)
    Scratch scratch;
};

// small runs: launch_front and launch_gather instead of launch_vertex .. launch_bin_scatter
cudaError_t launch_front(const LaunchArgs& a);
cudaError_t launch_gather(const LaunchArgs& a);
cudaError_t launch_vertex(const LaunchArgs& a);
cudaError_t launch_bin_count(const LaunchArgs& a);
cudaError_t launch_scans(const LaunchArgs& a);
cudaError_t launch_bin_scatter(const LaunchArgs& a);
cudaError_t launch_bin_split(const LaunchArgs& a, int ts);  // 32-pixel bins: before launch_raster
cudaError_t launch_raster(const LaunchArgs& a, int msaa, int ts);
unsigned long long kernel_launches();

}  // namespace rast

namespace rast {
cudaError_t launch_kat(int op, const void* in, void* out, cudaStream_t stream);
}
