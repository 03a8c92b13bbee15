// Bounded walks in the union-find forest of one tile of a cluster update (shared memory), plain
// enough to compile for the host.
#pragma once

#ifdef __CUDACC__
#define ISING_TILE_FN __host__ __device__ __forceinline__
#else
#define ISING_TILE_FN inline
#endif

namespace ising {

// One union (its finds and retries) or one root walk in a tile may take at most kTileSteps steps, a
// few milliseconds in shared memory; a tile has at most 12288 sites, so no walk of a forest comes
// near it.  A walk that runs out leaves `left` negative, and its caller sets the error word.
// (Reading that word on the way, as the walks in global memory do, made whole updates 4-8% slower.)
constexpr int kTileSteps = 1 << 16;

ISING_TILE_FN int tile_find(volatile int* lab, int x, int& left)
{
    while (--left >= 0) {
        const int p = lab[x];
        if (p == x) return x;
        const int gp = lab[p];
        if (gp == p) return p;
        lab[x] = gp;  // path halving
        x = gp;
    }
    return x;
}

ISING_TILE_FN int tile_root(const volatile int* lab, int x, int& left)
{
    while (--left >= 0) {
        const int p = lab[x];
        if (p == x) return x;
        x = p;
    }
    return x;
}

}  // namespace ising
