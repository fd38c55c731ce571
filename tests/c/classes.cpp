// Checks the raster queue's classes (rast_types.h) for every heavy limit and the counts around every
// power of two: class 0 is the empty bins, classes never fall as counts grow, and a class is heavy exactly when its counts
// reach the limit. Prints "ok" or the first mismatches.
#include <cstdint>
#include <cstdio>

struct float4;  // rast_types.h names it in pointers only
#include "rast_types.h"

int main() {
    int bad = 0;
    for (uint32_t bits = 0; bits <= 32; ++bits) {
        const uint32_t heavy = rast::heavy_class(bits);
        uint32_t last = 0, seen = 0;
        for (int k = 0; (1u << k) < rast::kMaxFrameTris; ++k)  // a bin holds a triangle once
            for (int d = -1; d <= 1; ++d) {
                const uint32_t count = (1u << k) + (uint32_t)d;
                if (count < seen) continue;  // 2^1 - 1 and 2^2 - 1 come after larger ones
                seen = count;
                const uint32_t c = rast::order_class(count, bits);
                const bool is = (uint64_t)count >= (1ull << bits);
                if (c >= (uint32_t)rast::kClasses || (c == 0) != (count == 0) || (count && (c >= heavy) != is) ||
                    c < last) {
                    if (bad++ < 10) std::printf("limit 2^%u count %u class %u heavy from %u\n", bits, count, c, heavy);
                }
                last = c;
            }
    }
    if (!bad) std::printf("ok\n");
    return 0;
}
