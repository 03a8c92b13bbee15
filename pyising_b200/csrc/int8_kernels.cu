// int8 compressed-checkerboard half-sweep kernel (2D/3D, Metropolis/heat bath) with the fused
// integer (M, E) reduction; the per-chunk update is int8_update in int8_core.cuh.
//
// Band schedule: the work of one launch is a list of slots (band, chunk column), band-major; a
// band is `band` consecutive rows of one plane.  A thread takes slots grid-stride and walks its
// band's rows top to bottom (int8_band), so consecutive threads of a warp read consecutive
// 16-byte chunks of the same rows.  Longer bands reuse more opposite-colour rows but leave fewer
// slots to fill the GPU; the launcher's default (band_plan.h) weighs the two, and a tuned value can
// replace it.
//
// The band walk is bound by the logic (ALU) pipe: two cycles per warp and SM quarter for each
// logic, compare, permute or shift instruction, and two more for each wide multiply of the random
// numbers (which also takes four of the multiplier pipe).  A 16-site chunk takes about 205 such
// slots (258 before the decisions became lookups), by that count 86% of the time; byte cuts (dp4a),
// predicated adds and sums run on the multiplier pipe (busy 77% in ncu).  Measured on one B200, flips/ns before -> after:
// 2D 16384^2 1030 -> 1211, 3D 512^3 heat bath 818 -> 1062, 3D 256^3 heat bath 710 -> 858.
//
// Lattices below kOneChunkRows chunks run one chunk per thread instead (int8_one_kernel).
#include "band_plan.h"
#include "int8_core.cuh"

namespace ising {

template <int V, int NDIM, int RULE, bool MIXED, bool MEAS>
__global__ void __launch_bounds__(256, 4) int8_half_kernel(const Int8Half p_in)
{
    Int8Half p = p_in;
    __shared__ u32 rt[kLookupWords];  // the lookup table of the decisions
    if (threadIdx.x == 0) fill_lookup<NDIM, RULE>(rt, p.table);
    pdl_wait();  // the previous half-sweep has completed
    pdl_trigger();
    resolve_ctl(p);
    __syncthreads();
    long long m_acc = 0, e_acc = 0;
    const u32 cpr = (u32)p.cpr, bpp = (u32)p.bpp;
    const u32 nslots = (u32)p.lz * bpp * cpr;
    for (u32 slot = blockIdx.x * blockDim.x + threadIdx.x; slot < nslots;
         slot += gridDim.x * blockDim.x) {
        const u32 band = fast_div(slot, cpr, p.cpr_magic);
        const int j0 = (int)(slot - band * cpr) * V;
        int z = 0, yb = (int)band;
        if constexpr (NDIM == 3) {
            z = (int)fast_div(band, bpp, p.bpp_magic);
            yb = (int)(band - (u32)z * bpp);
        }
        const int y0 = yb * p.band;
        const int y1 = y0 + p.band < p.ly ? y0 + p.band : p.ly;
        int8_band<V, NDIM, RULE, MIXED, MEAS>(p, z, y0, y1, j0, rt, m_acc, e_acc);
    }
    if constexpr (MEAS) block_accumulate2(m_acc, e_acc, p.meas);
}

// One chunk per thread: the schedule of lattices with too few chunks to give every thread a band.
// A half-sweep is then a chain of latencies (launch, loads, random numbers, decisions, store), and
// the random numbers, most of its instructions, depend on no spin: they are drawn before
// griddepcontrol.wait, while the previous half-sweep runs.  Measured on one B200 against the band
// schedule (flips/ns): 3D 64^3 58 -> 97, 3D 70x90x120 166 -> 209, 3D 160^3 519 -> 639, 2D 2048^2
// 582 -> 640, 2D 1500x2488 heat bath 481 -> 593.  Letting the next grid launch before the wait
// instead of after it was slower (3D 160^3 550, 2D 1536^2 376 against 494).
constexpr int kOneThreads = 128;

template <int V, int NDIM, int RULE, bool MIXED, bool MEAS>
__global__ void __launch_bounds__(kOneThreads) int8_one_kernel(const Int8Half p_in)
{
    constexpr int W = V / 4;
    Int8Half p = p_in;
    __shared__ u32 rt[kLookupWords];  // the lookup table of the decisions
    if (threadIdx.x == 0) fill_lookup<NDIM, RULE>(rt, p.table);
    // The control block is written between graph replays only, by kernels that have completed
    // before the first half-sweep of a replay starts: it can be read before the wait.
    resolve_ctl(p);
    const u32 slot = blockIdx.x * kOneThreads + threadIdx.x;
    const u32 row = fast_div(slot, (u32)p.cpr, p.cpr_magic);
    const int j0 = (int)(slot - row * (u32)p.cpr) * V;
    int z = 0, y = (int)row;
    if constexpr (NDIM == 3) {
        z = (int)fast_div(row, (u32)p.bpp, p.bpp_magic);
        y = (int)(row - (u32)z * (u32)p.bpp);
    }
    const DrawSites<NDIM> sites{p, site_counter(p, row, j0)};
    u32x4 r[W];
#pragma unroll
    for (int k = 0; k < W; ++k) {
        r[k] = sites(k);
        // drawn here, not where it is used
        asm volatile("" : "+r"(r[k].x), "+r"(r[k].y), "+r"(r[k].z), "+r"(r[k].w));
    }
    __syncthreads();
    pdl_wait();  // the previous half-sweep has completed
    pdl_trigger();
    long long m_acc = 0, e_acc = 0;
    if (row < (u32)p.rows)
        int8_chunk<V, NDIM, RULE, false, MIXED, MEAS>(
            p, [&](int k) { return r[k]; }, row, y, z, j0, rt, m_acc, e_acc);
    if constexpr (MEAS) block_accumulate2(m_acc, e_acc, p.meas);
}

// ------------------------------------------------------------------------- host side ---
// How a half-sweep is launched: the band schedule on `grid` blocks, or one chunk per thread.
struct Int8Plan {
    unsigned grid;
    bool one;
};

template <int V, int NDIM, int RULE, bool MIXED, bool MEAS>
static cudaError_t launch_plan(const Int8Plan& plan, const Int8Half& p, cudaStream_t st)
{
    if (plan.one)
        return launch_pdl(int8_one_kernel<V, NDIM, RULE, MIXED, MEAS>, plan.grid, kOneThreads, st, p);
    return launch_pdl(int8_half_kernel<V, NDIM, RULE, MIXED, MEAS>, plan.grid, 256, st, p);
}

template <int V, int NDIM, bool MIXED, bool MEAS>
static cudaError_t launch_rule(int rule, const Int8Plan& plan, const Int8Half& p, cudaStream_t st)
{
    switch (rule) {
    case kMetroFast: return launch_plan<V, NDIM, kMetroFast, MIXED, MEAS>(plan, p, st);
    case kHeat: return launch_plan<V, NDIM, kHeat, MIXED, MEAS>(plan, p, st);
    case kMetroGeneric: return launch_plan<V, NDIM, kMetroGeneric, MIXED, MEAS>(plan, p, st);
    default:
        return launch_pdl(int8_half_kernel<V, NDIM, kObserve, MIXED, true>, plan.grid, 256, st, p);
    }
}

template <int V, bool MIXED = false>
static cudaError_t launch_v(int ndim, int rule, const Int8Plan& plan, const Int8Half& p,
                            cudaStream_t st)
{
    const bool meas = p.meas != nullptr;
    if (ndim == 3)
        return meas ? launch_rule<V, 3, MIXED, true>(rule, plan, p, st)
                    : launch_rule<V, 3, MIXED, false>(rule, plan, p, st);
    return meas ? launch_rule<V, 2, MIXED, true>(rule, plan, p, st)
                : launch_rule<V, 2, MIXED, false>(rule, plan, p, st);
}

// Chunk width used for a row of lh bytes: the widest of 16/8/4 that divides it.
int int8_chunk_width(int lh) { return lh % 16 == 0 ? 16 : (lh % 8 == 0 ? 8 : 4); }

// Fills in the band fields of p (band from p.band, or the default when p.band <= 0) and
// returns the grid: one block per 256 slots, at most max_blocks.
unsigned int8_band_geometry(Int8Half& p, int max_blocks, int sm_count)
{
    if (p.band <= 0) p.band = int8_default_band(p.rows, p.ly, p.cpr, sm_count);
    if (p.band > p.ly) p.band = p.ly;
    p.bpp = (p.ly + p.band - 1) / p.band;
    const unsigned long long nslots = (unsigned long long)p.lz * p.bpp * p.cpr;
    p.cpr_magic = fast_div_magic((u32)p.cpr, nslots);
    p.bpp_magic = fast_div_magic((u32)p.bpp, (unsigned long long)p.lz * p.bpp);
    unsigned long long g = (nslots + 255) / 256;
    if (g > (unsigned long long)max_blocks) g = (unsigned long long)max_blocks;
    return (unsigned)(g < 1 ? 1 : g);
}

// Chunks (per SM) below which the default is one chunk per thread.  Measured one chunk / bands of
// two rows (flips/ns): 460,800 chunks (3D 240^3) 759 / 707, 392,000 (2D 3500x3584) 839 / 802,
// 524,288 (3D 256^3) 851 / 856 and (2D 4096^2) 884 / 938.
constexpr long long kOneChunkRows = 3400;
// Words (of four sites, per SM) up to which a thread of that schedule takes one word instead of
// four: 3D 64^3 (32,768 words) 98 / 88, 3D 96^3 (110,592) 219 / 264.
constexpr long long kOneWordRows = 512;

cudaError_t launch_int8_half(int ndim, int rule, const Int8Half& p_in, int max_blocks, int sm_count,
                             cudaStream_t st)
{
    Int8Half p = p_in;
    Int8Plan plan{0, false};
    if (rule != kObserve && p.band <= 0 && p.rows * p.cpr < kOneChunkRows * sm_count) {
        if (p.vw == 16 && p.rows * (long long)(p.lh / 4) <= kOneWordRows * sm_count) {
            p.vw = 4;
            p.cpr = p.lh / 4;
        }
        p.band = 1;
        plan.one = true;
    }
    plan.grid = int8_band_geometry(p, max_blocks, sm_count);
    if (plan.one) plan.grid = (unsigned)((p.rows * p.cpr + kOneThreads - 1) / kOneThreads);
    const int v = p.vw;
    if (v == 16) {  // padded rows (lh % 16 != 0) need the partial-chunk code
        return (p.lh % 16) ? launch_v<16, true>(ndim, rule, plan, p, st)
                           : launch_v<16, false>(ndim, rule, plan, p, st);
    }
    if (v == 8) return launch_v<8>(ndim, rule, plan, p, st);
    return launch_v<4>(ndim, rule, plan, p, st);
}

}  // namespace ising
