// Shape, cost and cutting of the temporal tiles: host arithmetic only, no CUDA.  Times are of one
// half-sweep on one B200, in microseconds.
#pragma once

#include <cmath>
#include <cstddef>
#include <cstdint>

#include "lane_plan.h"

namespace ising {

constexpr int kTileMaxSmem = 200 * 1024;
constexpr int kTileMaxDepth = 16;
constexpr int kTileMinDepth = 3;

// A 2D lattice as the plan sees it: rows of `units` 16-site chunks (int8) or 64-spin words (msc).
struct TileRows {
    bool msc;
    int ly, units;
    size_t row_bytes;  // of one colour
    int sms;
};

// Rows that a CTA writes back and half-sweeps per launch; depth 0: the rows do not fit.
struct TileShape {
    int band, depth;
};

// The depth rule: the cost of a launch beside its steps, and of one row on one SM per chunk and
// word, with which it gives the measured best depths (int8 256^2 8, 1024^2 4, 2048^2 3; msc 512^2
// 8, 1152^2 5, 2048^2 4, 4096^2 3).
constexpr double kLaunchUs = 1.0, kDepthChunkUs = 2.0e-3, kDepthWordUs = 4.1e-3;

inline TileShape tile_shape(const TileRows& r)
{
    TileShape s;
    s.band = (r.ly + r.sms - 1) / r.sms;
    if (s.band < 2) s.band = 2;
    const double row_us = (r.msc ? kDepthWordUs : kDepthChunkUs) * r.units;
    int d = (int)(std::sqrt(kLaunchUs / row_us) + 0.5);
    d = d < kTileMinDepth ? kTileMinDepth : (d > kTileMaxDepth ? kTileMaxDepth : d);
    if (d > r.ly / 2) d = r.ly / 2;
    while (d > 0 && 2 * (size_t)(s.band + 2 * d) * r.row_bytes > (size_t)kTileMaxSmem) --d;
    s.depth = d;
    return s;
}

// A step on tiles: a chain of latencies, its share of the launch, and the rows that a CTA updates
// (band + depth - 1 on average).  A lattice of few rows has few CTAs, each of which recomputes
// nearly as many rows as it keeps.
constexpr double kTileChunkUs = 2.2e-3, kTileWordUs = 3.35e-3;

inline double tile_half_us(const TileRows& r, const TileShape& s, double depth)
{
    const double row_us = (r.msc ? kTileWordUs : kTileChunkUs) * r.units;
    return (r.msc ? 0.5 : 0.4) + kLaunchUs / depth + row_us * (s.band + depth - 1);
}

// A half-sweep of its own, spread over all SMs.  int8: one chunk per thread.  msc: word ranges up to
// kLaneWords words per SM, then the lane walk, whose lanes (two blocks of 256 per SM) take an even
// number of rows each.
inline double single_half_us(const TileRows& r)
{
    const double units = (double)r.ly * r.units;
    if (!r.msc) return 1.45 + kTileChunkUs * units / r.sms;
    const double fill = units / ((double)kLaneWords * r.sms);
    if (fill < 1) return 2.55 + 0.4 * fill;
    const double rows = 2 * std::ceil(units / (512.0 * r.sms) / 2);
    return (units / rows / 256 > r.sms ? 2.35 : 1.15) + 1.07 * rows;
}

// A run of `halves` half-sweeps in an even number of launches of about the same depth, at most
// `depth` each.
struct TileCuts {
    int64_t launches, base, longer;  // the first `longer` launches have base + 1 half-sweeps

    TileCuts(int64_t halves, int depth)
    {
        launches = 2 * (halves / (2 * (int64_t)depth) + (halves % (2 * (int64_t)depth) != 0));
        base = launches ? halves / launches : 0;
        longer = launches ? halves % launches : 0;
    }
    int64_t depth(int64_t i) const { return base + (i < longer); }
};

// Whether tiles beat single half-sweeps.  Measured, flips/ns, tiles / single half-sweeps (and the
// two times of the model): int8 1024^2 391 / 300 (1.35, 1.94), 64x1024 34 / 26 (1.00, 1.48), 512x4096
// 451 / 431 (2.42, 2.42), 64x4096 77 / 91 (1.86, 1.57), 64x16384 102 / 265 (5.24, 1.94), 1024x8192
// 713 / 789 (5.80, 5.35); msc 1152^2 571 / 239 (1.06, 2.66), 4096^2 2116 / 1861 (4.05, 4.49), 6000x5248
// 2282 / 2364 (6.74, 6.63), 64x8192 169 / 99 (1.69, 2.59), 64x65536 285 / 724 (7.69, 2.90), 128x32768
// 523 / 731 (4.26, 2.90).
//
// Measured every `every` sweeps, a run on tiles is cut at each measurement, and single half-sweeps are
// replayed as a graph per measurement, whose last kernel, which advances its counters, and next start
// cost about 4 us more (us per sweep, tiles / graphs: int8 256x8192 measured every sweep 7.4 / 9.5, msc
// 64x32768 every two 7.2 / 8.4).
constexpr double kMeasuredGraphUs = 4.0;

inline bool tiles_pay(const TileRows& r, int64_t every)
{
    const TileShape s = tile_shape(r);
    if (s.depth <= 0) return false;
    if (every <= 0) return tile_half_us(r, s, s.depth) <= single_half_us(r);
    const TileCuts cuts(2 * every, s.depth);
    const double halves = 2.0 * every;
    return halves * tile_half_us(r, s, halves / cuts.launches) <=
           halves * single_half_us(r) + kMeasuredGraphUs;
}

}  // namespace ising
