// How the streaming kernel of the routed experts deals the units of its tiles to CTAs.  Plain integers, for host and device.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define SXB_HD __host__ __device__
#else
#define SXB_HD
#endif

namespace sxb {

// From unit u0 of tile0 to before unit u1 of tile1; tile0 > tile1: none.
struct UnitRun {
    int tile0, u0, tile1, u1;
};

// Whether runs that lie in one tile each, of at most `run` units, suit the launch better than even ones, which cost a CTA the staging of another
// tile by half its warps, about a third of a unit's time: where a warp has one unit at most anyway, or where the runs fill their warps' rounds and leave
// less than a seventh of the CTAs' time idle.  Above six rounds even runs were better whatever the rounds.  us, even -> inside
// tiles: gate/up, 512 experts, 4096 x 2048 Q4, 1 token 22.2 -> 18.3, 8 75 -> 68; 16 experts, 4096 x 3072 Q8, 64 tokens 64 -> 56, 255 162 -> 136;
// 8 experts, 6144 x 1024 Q8, 255 tokens 161 -> 118; against it, 16 experts' Q4 down of 1536, 150 tokens, 35.8 -> 37.4 (5.4 rounds).
SXB_HD inline bool runs_inside_tiles(uint32_t run, uint32_t tiles, uint32_t units, uint32_t ctas, uint32_t warps) {
    const uint32_t rounds = (run + warps - 1) / warps;
    return run <= warps || (run <= 6 * warps && 4 * run >= 3 * warps * rounds && (uint64_t)run * ctas * 100 <= (uint64_t)tiles * units * 116);
}

// The run of CTA `cta` of `ctas`, each of `warps` warps, over `tiles` tiles of `units` units (at least one).  In 32 bits where that
// is enough: four 64-bit divisions were half a microsecond of every launch.
SXB_HD inline UnitRun unit_run(uint32_t tiles, uint32_t units, uint32_t cta, uint32_t ctas, uint32_t warps) {
    const UnitRun none{0, 0, -1, 0};
    if (tiles > 0 && tiles <= ctas) {
        const uint32_t per = ctas / tiles, run = (units + per - 1) / per;
        if (runs_inside_tiles(run, tiles, units, ctas, warps)) {  // units <= 6 warps * ctas: no overflow below
            const uint32_t tile = cta / per, part = cta - tile * per, u0 = units * part / per, u1 = units * (part + 1) / per;
            return tile < tiles && u0 < u1 ? UnitRun{(int)tile, (int)u0, (int)tile, (int)u1} : none;
        }
    }
    const uint64_t total = (uint64_t)tiles * units;
    if (total * ctas <= 0xffffffffu) {
        const uint32_t t = (uint32_t)total, begin = t * cta / ctas, end = t * (cta + 1) / ctas;
        if (begin >= end) return none;
        const uint32_t tile0 = begin / units, tile1 = (end - 1) / units;
        return UnitRun{(int)tile0, (int)(begin - tile0 * units), (int)tile1, (int)(end - tile1 * units)};
    }
    const uint64_t begin = total * cta / ctas, end = total * (cta + 1) / ctas, tile0 = begin / units, tile1 = (end - 1) / units;
    return UnitRun{(int)tile0, (int)(begin - tile0 * units), (int)tile1, (int)(end - tile1 * units)};
}

}  // namespace sxb
