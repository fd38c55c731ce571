// Prints figures of rast_types.h that the CPU tests check: for every line of standard input
// "nverts ntris width height ts bins", the device bytes of such a frame (frame_bytes).
#include <cstdio>

struct float4;  // rast_types.h names it in pointers only
#include "rast_types.h"

int main() {
    unsigned long long nverts, ntris, w, h, bins;
    int ts;
    while (std::scanf("%llu %llu %llu %llu %d %llu", &nverts, &ntris, &w, &h, &ts, &bins) == 6)
        std::printf("%llu\n", (unsigned long long)rast::frame_bytes(nverts, (uint32_t)ntris, w, h, ts, bins));
    return 0;
}
