// Which packed half-sweeps take the lane walk, and with which bands: host arithmetic only, no CUDA.
#pragma once

namespace ising {

// Words per SM from which a half-sweep takes the lane walk; a smaller one is mostly latency, and
// the ranges put every word on a lane of its own.  Measured ranges / lanes (flips/ns): 1152^2
// (10,368 words) 234 / 208, 2000x1920 (30,000) 584 / 590, 3072^2 (73,728) 1267 / 1438.  (Strips, for
// rows of whole 32-word strips, are slower still on few words: 64x8192 99 / 83, 64x65536 724 / 618.)
constexpr int kLaneWords = 256;

// Rows per lane of the lane walk (an even number) on `lanes` resident lanes; 0: word ranges.
//
// A band height that just fits the words may need more lanes than are resident, by the lanes that
// a last short band leaves unused; the few blocks over would run alone after the others, so the
// band grows until all fit (505172x384, 75777 lanes: 2912 -> 3602 flips/ns).  With one word per row a
// band of 16 rows is 128 bytes: the lanes of a warp then read lines at a multiple of 128 bytes, and
// bands of 16, 32 or 48 rows were slower than the next larger ones (1076018x128 2698, word ranges
// 2994).
//
// Bands come in pairs of rows, so short bands may leave many lanes without one, where word ranges,
// in steps of 32 words per warp, waste less.  With one wave of either, a half-sweep takes about 2.45 us
// + 1.09 per row of a band, or 2.2 us + 1.4 per word of a lane's share (flips/ns, ranges / lanes): bands
// of 4 rows for 2.03 words per lane 1549 / 1506 (2402x8192), for 3 2256 / 2177 (3552x8192), for 3.1 1896
// / 2172 (58726x512), for 3.9 2435 / 2812; bands of 6 for 4.05 2143 / 2211 (4794x8192).  Bands of 2 are
// always faster (650x8192 737 / 824, 1242x8192 1024 / 1143).  Rows of more words than lanes leave no
// band height at all.
inline long long lane_band(long long rows, long long nw, long long lanes, long long sms)
{
    const long long words = rows * nw;
    if (rows % 2 || words > 0xFFFFFFFFll || words < kLaneWords * sms) return 0;
    long long band = (words + lanes - 1) / lanes;
    band += band & 1;
    if (band > rows) band = rows;
    while (band < rows && (rows + band - 1) / band * nw > lanes) band += 2;
    if (nw == 1 && band % 16 == 0 && band < rows) band += 2;
    const long long share = (words + lanes - 1) / lanes;
    if (band > 2 && (nw > lanes || 220 + 140 * share < 245 + 109 * band)) return 0;
    return band;
}

}  // namespace ising
