// csrc/unit_runs.cuh: over every number of CTAs, tiles and units that is tried, the runs of a launch hold every unit of every tile once,
// in order, whichever of the three ways deals them.
#include "unit_runs.cuh"

#include <cstdio>
#include <initializer_list>

using namespace sxb;

int main() {
    const uint32_t tiles_of[] = {0, 1, 2, 3, 7, 10, 36, 37, 73, 74, 75, 147, 148, 149, 296, 1000, 8000, 131072};
    const uint32_t units_of[] = {1, 2, 3, 15, 16, 17, 31, 64, 95, 96, 97, 128, 255, 256, 1000, 1776, 1777, 14208, 14209, 300000, 134217728};
    int bad = 0, inside = 0, narrow = 0, wide = 0;
    for (uint32_t ctas : {1u, 2u, 132u, 148u, 160u})
        for (uint32_t tiles : tiles_of)
            for (uint32_t units : units_of) {
                const uint64_t total = (uint64_t)tiles * units;
                if (total > 0x7fffffffffffull / ctas || tiles > (1u << 17) + 1024) continue;
                uint64_t at = 0;
                bool one_tile = tiles > 0;
                for (uint32_t c = 0; c < ctas; ++c) {
                    const UnitRun r = unit_run(tiles, units, c, ctas, 16);
                    if (r.tile0 > r.tile1) continue;
                    const uint64_t begin = (uint64_t)r.tile0 * units + (uint32_t)r.u0, end = (uint64_t)r.tile1 * units + (uint32_t)r.u1;
                    if (begin != at || end <= begin || (uint32_t)r.u1 > units || r.u1 < 1) ++bad, std::printf("FAIL ctas %u tiles %u units %u cta %u\n", ctas, tiles, units, c);
                    at = end, one_tile = one_tile && r.tile0 == r.tile1;
                }
                if (at != total) ++bad, std::printf("FAIL ctas %u tiles %u units %u: %llu of %llu\n", ctas, tiles, units, (unsigned long long)at, (unsigned long long)total);
                if (one_tile && tiles > 1 && tiles < ctas) ++inside;
                else if (total * ctas <= 0xffffffffu) ++narrow;
                else ++wide;
            }
    if (inside < 20 || narrow < 20 || wide < 20) ++bad, std::printf("FAIL: ways %d %d %d\n", inside, narrow, wide);
    return bad != 0;
}
