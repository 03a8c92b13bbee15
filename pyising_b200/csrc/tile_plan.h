// How a run of sweeps is cut into tile launches: host arithmetic only, no CUDA.
#pragma once

#include <cstdint>

namespace ising {

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

}  // namespace ising
