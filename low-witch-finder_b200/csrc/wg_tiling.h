// How a rect of regions is cut into units (tiles, wg_phase1.cuh).  Host code without CUDA.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdint>

namespace wg {

struct Tiling {
    uint32_t tw = 1, th = 1, ntx = 1;
    uint64_t n_win = 1;           // tiles per seed
    uint64_t win() const { return (uint64_t)tw * th; }   // regions per tile at most
};
inline Tiling tiling_of(uint64_t rw, uint64_t rh, uint64_t tw, uint64_t th) {
    Tiling t;
    t.tw = (uint32_t)tw;
    t.th = (uint32_t)th;
    t.ntx = (uint32_t)((rw + tw - 1) / tw);
    t.n_win = t.ntx * ((rh + th - 1) / th);
    return t;
}

// Regions along a tile's side at most in the unit and list kernels: a hut's chunk offset stays below 2^15.
constexpr uint64_t kTileSide = 1023;
// Regions per unit of the one-CTA kernel at most.
constexpr uint64_t kUnitCtaMax = 1ull << 16;

// Tiles of at most `target` regions (at least one), near square, of equal size up to rounding.
inline Tiling tile_rect(uint64_t rw, uint64_t rh, uint64_t target, uint64_t max_side = kTileSide) {
    target = std::max<uint64_t>(target, 1);
    uint64_t tw = rw, th = rh;
    if (rw > target / rh || rw > max_side || rh > max_side) {
        const uint64_t side = std::max<uint64_t>(1, (uint64_t)std::sqrt((double)target));
        tw = std::min<uint64_t>({rw, side, max_side});
        th = std::min<uint64_t>({rh, std::max<uint64_t>(1, target / tw), max_side});
        tw = std::min<uint64_t>({rw, std::max<uint64_t>(1, target / th), max_side});   // a low rect: wider tiles
        tw = (rw + (rw + tw - 1) / tw - 1) / ((rw + tw - 1) / tw);                     // of equal size
        th = (rh + (rh + th - 1) / th - 1) / ((rh + th - 1) / th);
    }
    return tiling_of(rw, rh, tw, th);
}

// Tiles of the one-CTA kernel that fill whole waves of its resident CTAs (slots).  A wave lasts as long as its
// tiles' regions and about 2,000 more (the table builds, the last gates), and a part of a wave, whose CTAs have
// the SM to themselves, not as long.  The tilings of one to four waves are compared by that, by their tiles
// along the rect's short side (nx), so that a rect and its transpose get the same.  Against tiles of an
// eighth of a slot's share (2,048 regions at least), one seed: 400 x 400 regions 100 -> 88 us, 2000 x 2000
// 429 -> 249 us (3 units a slot, then 1), 6000 x 6000 1.87 -> 1.44 ms; 40 seeds x 600 x 600 1.01 -> 0.59 ms.
// Requests past four waves of the largest tiles take those, and those of more seeds than four waves one a seed.
inline Tiling wave_tiles(uint64_t rw, uint64_t rh, uint64_t n_seeds, uint64_t slots) {
    constexpr uint64_t kWaveRegions = 2000;
    const uint64_t sw = std::min(rw, rh), sh = std::max(rw, rh);
    uint64_t best = ~0ull, btw = 0, bth = 0;
    for (uint64_t waves = 1; waves <= 4; waves++) {
        const uint64_t m = std::min(waves * slots / n_seeds, (rw * rh + 31) / 32);   // tiles per seed
        if (m == 0) continue;
        const double square = std::sqrt((double)m * (double)sw / (double)sh);
        const uint64_t lo = std::max<uint64_t>(1, (uint64_t)(square * 0.6)), hi = std::min<uint64_t>({sw, m, (uint64_t)(square * 1.7) + 1});
        for (uint64_t nx = lo; nx <= hi; nx++) {
            const uint64_t tw = (sw + nx - 1) / nx, nz = std::min(sh, m / ((sw + tw - 1) / tw)), th = (sh + nz - 1) / nz;
            if (tw > kTileSide || th > kTileSide || tw * th > kUnitCtaMax) continue;
            const uint64_t units = n_seeds * ((sw + tw - 1) / tw) * ((sh + th - 1) / th), part = units % slots;
            const uint64_t cost = (units / slots) * (tw * th + kWaveRegions) +
                                  (part ? kWaveRegions + tw * th * (2 * slots + 3 * part) / (5 * slots) : 0);
            if (cost < best) {
                best = cost;
                btw = tw;
                bth = th;
            }
        }
    }
    if (best == ~0ull) return tile_rect(rw, rh, kUnitCtaMax);
    return rw <= rh ? tiling_of(rw, rh, btw, bth) : tiling_of(rw, rh, bth, btw);
}

}  // namespace wg
