// Temporally blocked 2D half-sweeps (int8 and msc): several half-sweeps per launch on tiles of rows
// held in shared memory.
//
// A small lattice's half-sweep takes less time than starting a kernel and fetching its operands
// (about 2 us on B200 even with graphs and programmatic dependent launch).  Here one launch does H
// half-sweeps: a CTA loads a band of B rows plus H halo rows on each side (periodic in y) of both
// colours into shared memory, runs the half-sweeps there on a row range that shrinks by one row
// per half-sweep (half-sweep k updates tile rows [k+1, rows-1-k): exactly what the band's rows
// need after the last one, since each half-sweep reads the opposite colour one row further out),
// and writes back only the band.  Halo rows are updated by several CTAs with the same random
// numbers, keyed by (site, sweep, colour) as everywhere else, so every result is bit-identical to
// H single half-sweeps.  The last half-sweep updates the band's rows only; if it ends a measured
// sweep, their (M, E) are summed there.
//
// Every thread draws the random numbers of its (first) item of a half-sweep before the barrier
// that starts it, and those of the first half-sweep before the previous launch has finished.
//
// Depth: with row_us the time of one row on one SM and kLaunchUs the cost of a launch, a
// half-sweep costs kLaunchUs / H + row_us (B + H - 1), least at H = sqrt(kLaunchUs / row_us).
//
// A step is bound by the latency of one warp's chain of instructions (draws, barrier, neighbour
// loads, decisions, store), not by a pipe: about 0.5 us (int8) to 0.8 us (msc) on lattices whose
// rows are a few words.  Measured on one B200, flips/ns, single half-sweeps -> tiles: int8 256^2
// 26 -> 51, 1024^2 300 -> 391, 2048^2 646 -> 700; msc 512^2 52 -> 156, 1152^2 239 -> 570, 2048^2
// 742 -> 1267, 4096^2 1861 -> 2116.  tile_plan.h: bands, depths and where tiles pay.
#include <cstring>

#include "capi_internal.h"
#include "int8_core.cuh"
#include "msc_core.cuh"
#include "tile_plan.h"

namespace ising {

// One CTA of 16 warps per SM and 128 registers a thread: with two CTAs' worth of registers (64) the
// pre-drawn random numbers spilled, and a step took up to 1.5 times as long.
constexpr int kTileThreads = 512;

// Where a tile launch is: half-sweeps h0 .. h0 + depth - 1, counted from colour 0 of sweep p.t.
struct TileRun {
    int h0, depth;
    int band;         // rows a CTA writes back (the last CTA's may be fewer)
    u32 items_magic;  // fast_div magic of the items per row
};

// Tile geometry of this CTA: rows of the tile and the global row of tile row 0.
struct Tile {
    int r0, nb, rows, base;
    __device__ __forceinline__ Tile(const TileRun& run, int ly)
    {
        r0 = (int)blockIdx.x * run.band;
        nb = r0 + run.band < ly ? run.band : ly - r0;
        rows = nb + 2 * run.depth;
        base = r0 - run.depth;
        if (base < 0) base += ly;  // the depth is at most ly / 2
    }
    __device__ __forceinline__ int global_row(int tr, int ly) const
    {
        int g = base + tr;
        if (g >= ly) g -= ly;
        if (g >= ly) g -= ly;
        return g;
    }
};

// Reads both colours from in0/in1 and writes the band to out0/out1: separate arrays, since a
// CTA's halo rows are other CTAs' bands, which those write back in the same launch.
template <int V, int RULE, bool MIXED, bool MEAS>
__global__ void __launch_bounds__(kTileThreads, 1)
    int8_tile_kernel(const Int8Half p_in, const TileRun run, const int8_t* in0, const int8_t* in1,
                     int8_t* out0, int8_t* out1)
{
    constexpr int W = V / 4;
    extern __shared__ __align__(16) int8_t tile[];  // [colour][rows][pitch]
    __shared__ u32 rt[kLookupWords];                // the lookup table of the decisions
    Int8Half p = p_in;
    if (threadIdx.x == 0) fill_lookup<2, RULE>(rt, p.table);
    const int ly = p.ly, pitch = p.pitch, cpr = p.cpr;
    const Tile T(run, ly);
    const int stride = T.rows * pitch;
    long long m_acc = 0, e_acc = 0;
    for (int k = 0; k < run.depth; ++k) {
        const int half = run.h0 + k, color = half & 1;
        Int8Half q = p;
        q.t = p.t + (u32)(half >> 1);
        q.color = (u32)color;
        const int n = (T.rows - 2 - 2 * k) * cpr;
        // item i of the half-sweep: chunk column jc of tile row tr
        auto place = [&](int i, int& tr, int& j0, int& gr) {
            const int ir = (int)fast_div((u32)i, (u32)cpr, run.items_magic);
            tr = k + 1 + ir;
            j0 = (i - ir * cpr) * V;
            gr = T.global_row(tr, ly);
        };
        u32x4 r[W];
        auto draw = [&](int gr, int j0) {
            const DrawSites<2> sites{q, site_counter(q, gr, j0)};
#pragma unroll
            for (int w = 0; w < W; ++w) {
                r[w] = sites(w);
                asm volatile("" : "+r"(r[w].x), "+r"(r[w].y), "+r"(r[w].z), "+r"(r[w].w));
            }
        };
        int i = (int)threadIdx.x, tr = 0, j0 = 0, gr = 0;
        if (i < n) {
            place(i, tr, j0, gr);
            draw(gr, j0);
        }
        if (k == 0) {
            pdl_wait();  // the previous launch of the stream has completed
            pdl_trigger();
            // the tile's rows are contiguous in memory but for the wrap
            const long long first = (long long)T.base * pitch, end = (long long)ly * pitch;
            for (int c = 16 * (int)threadIdx.x; c < stride; c += 16 * kTileThreads) {
                long long off = first + c;
                off -= off >= end ? end : 0;
                off -= off >= end ? end : 0;
                const uint4 a = __ldcg(reinterpret_cast<const uint4*>(in0 + off));
                const uint4 b = __ldcg(reinterpret_cast<const uint4*>(in1 + off));
                *reinterpret_cast<uint4*>(tile + c) = a;
                *reinterpret_cast<uint4*>(tile + stride + c) = b;
            }
        }
        __syncthreads();
        int8_t* own = tile + color * stride;
        const int8_t* oth = tile + (color ^ 1) * stride;
        const bool last = k + 1 == run.depth;
        int8_t* out = color ? out1 : out0;
        while (i < n) {
            const int par = (gr + color) & 1;
            const int wv = valid_words<MIXED, W>(p, j0);
            const int8_t* orow = oth + tr * pitch;
            const Words<W> s = load_words<W>(own + tr * pitch + j0);
            const Words<W> c = downs(load_words<W>(orow + j0));
            const Words<W> nu = downs(load_words<W>(orow + pitch + j0));
            const Words<W> nd = downs(load_words<W>(orow - pitch + j0));
            const u32 edge = (u32)(uint8_t)orow[edge_index(p, par, j0, wv)] & kBit2;
            auto drawn = [&](int w) { return r[w]; };
            Words<W> ns;
            if (MEAS && last)
                ns = int8_update<V, 2, RULE, MIXED, true>(drawn, par, wv, s, c, nu, nd, nu, nd,
                                                          edge, rt, m_acc, e_acc);
            else
                ns = int8_update<V, 2, RULE, MIXED, false>(drawn, par, wv, s, c, nu, nd, nu, nd,
                                                           edge, rt, m_acc, e_acc);
            if (last) store_words<W>(out + (long long)gr * pitch + j0, ns);
            else store_words<W>(own + tr * pitch + j0, ns);
            i += kTileThreads;
            if (i < n) {
                place(i, tr, j0, gr);
                draw(gr, j0);
            }
        }
        if (last) {  // the other colour's band rows are final
            int8_t* o = color ? out0 : out1;
            const int chunks = T.nb * (pitch >> 4);
            for (int c = (int)threadIdx.x; c < chunks; c += kTileThreads)
                *reinterpret_cast<uint4*>(o + (long long)T.r0 * pitch + 16 * c) =
                    *reinterpret_cast<const uint4*>(oth + run.depth * pitch + 16 * c);
        }
    }
    if constexpr (MEAS) block_accumulate2(m_acc, e_acc, p.meas);
}

// The msc tile.  G lanes share a word: lane g draws blocks KB g .. KB g + KB - 1 before the barrier
// and evaluates them by itself, and the lanes' partial decisions are composed by shuffles.  With
// few words per CTA a step is one warp's chain of dependent instructions, which G shortens; with
// many, one lane per word wastes the least.
template <int G, int KB, bool MEAS>
__global__ void __launch_bounds__(kTileThreads, 1)
    msc_tile_kernel(const MscHalf p_in, const TileRun run, const u64* in0, const u64* in1,
                    u64* out0, u64* out1)
{
    constexpr int kWords = kTileThreads / G;  // words per pass
    extern __shared__ __align__(16) u64 wtile[];  // [colour][rows][nw]
    __shared__ uint4 lvmask[16];
    MscHalf p = p_in;
    if (threadIdx.x < 16) lvmask[threadIdx.x] = level_masks(p.thr4, p.thr8, threadIdx.x);
    const int ly = p.rows, nw = p.nw;
    const Tile T(run, ly);
    const int stride = T.rows * nw;
    const u32 g = threadIdx.x & (u32)(G - 1);
    const int first_word = (int)(threadIdx.x / G);
    const int warp_word = (int)((threadIdx.x & ~31u) / G);  // first word of the warp
    long long m_acc = 0, e_acc = 0;
    for (int k = 0; k < run.depth; ++k) {
        const int half = run.h0 + k, color = half & 1;
        const u32 t = p.t + (u32)(half >> 1);
        const int n = (T.rows - 2 - 2 * k) * nw;
        u32x4 r[KB];
        auto place = [&](int i, int& tr, int& x, int& gr) {
            const int ir = (int)fast_div((u32)i, (u32)nw, run.items_magic);
            tr = k + 1 + ir;
            x = i - ir * nw;
            gr = T.global_row(tr, ly);
        };
        auto draw = [&](u32 w) {
#pragma unroll
            for (int b = 0; b < KB; ++b) {
                r[b] = philox4x32_10<true>(w, t, (u32)color, 1u + g * KB + (u32)b, p.k0, p.k1);
                asm volatile("" : "+r"(r[b].x), "+r"(r[b].y), "+r"(r[b].z), "+r"(r[b].w));
            }
        };
        int i = first_word, tr = 0, x = 0, gr = 0;
        if (i < n) {
            place(i, tr, x, gr);
            draw((u32)gr * (u32)nw + (u32)x);
        }
        if (k == 0) {
            pdl_wait();  // the previous launch of the stream has completed
            pdl_trigger();
            // the tile's rows are contiguous in memory but for the wrap
            const long long first = (long long)T.base * nw, end = (long long)ly * nw;
            for (int c = (int)threadIdx.x; c < stride; c += kTileThreads) {
                long long off = first + c;
                off -= off >= end ? end : 0;
                off -= off >= end ? end : 0;
                const u64 a = __ldcg(in0 + off), b = __ldcg(in1 + off);
                wtile[c] = a;
                wtile[stride + c] = b;
            }
        }
        __syncthreads();
        u64* own = wtile + color * stride;
        const u64* oth = wtile + (color ^ 1) * stride;
        const bool last = k + 1 == run.depth;
        u64* out = color ? out1 : out0;
        for (int iw = warp_word; iw < n; iw += kWords) {  // whole warps
            const bool valid = i < n;
            u64 o = 0, c = 0, up = 0, dn = 0, hz = 0;
            if (valid) {
                const u64* orow = oth + tr * nw;
                o = own[tr * nw + x];
                c = orow[x];
                up = orow[x - nw];
                dn = orow[x + nw];
                const bool par = ((gr + color) & 1) != 0;
                const u64 side = orow[par ? (x + 1 == nw ? 0 : x + 1) : (x == 0 ? nw - 1 : x - 1)];
                hz = par ? ((c >> 1) | (side << 63)) : ((c << 1) | (side >> 63));
            }
            const HalfSlices al = slice_half((u32)o, (u32)c, (u32)hz, (u32)up, (u32)dn);
            const HalfSlices ah = slice_half((u32)(o >> 32), (u32)(c >> 32), (u32)(hz >> 32),
                                             (u32)(up >> 32), (u32)(dn >> 32));
            u32 ul = valid ? ~al.a2 : 0u, uh = valid ? ~ah.a2 : 0u, accl = 0, acch = 0;
            const u32 w = (u32)gr * (u32)nw + (u32)x;
            if constexpr (G == 1) {
#pragma unroll
                for (int b = 0; b < KB; ++b)
                    block_levels(r[b], lvmask[b], al.a1, ah.a1, ul, uh, accl, acch);
                for (u32 lp = KB; lp < 16u && (ul | uh) != 0; ++lp) {
                    const u32x4 more = philox4x32_10<true>(w, t, (u32)color, 1u + lp, p.k0, p.k1);
                    block_levels(more, lvmask[lp], al.a1, ah.a1, ul, uh, accl, acch);
                }
            } else {
                HalfBlock l{~0u, 0u}, h{~0u, 0u};
#pragma unroll
                for (int b = 0; b < KB; ++b) {
                    const uint4 m = lvmask[g * KB + b];
                    const HalfBlock bl = half_block(r[b].x, r[b].z, m, al.a1);
                    const HalfBlock bh = half_block(r[b].y, r[b].w, m, ah.a1);
                    l.lt |= l.eq & bl.lt;
                    l.eq &= bl.eq;
                    h.lt |= h.eq & bh.lt;
                    h.eq &= bh.eq;
                }
                compose_lanes<G>(l);
                compose_lanes<G>(h);
                accl = ul & l.lt;
                acch = uh & h.lt;
                ul &= l.eq;
                uh &= h.eq;
                for (u32 lp = G * KB; lp < 16u && __any_sync(0xFFFFFFFFu, (ul | uh) != 0); lp += G) {
                    const u32x4 more =
                        philox4x32_10<true>(w, t, (u32)color, 1u + lp + g, p.k0, p.k1);
                    const uint4 m = lvmask[lp + g];
                    HalfBlock ml = half_block(more.x, more.z, m, al.a1);
                    HalfBlock mh = half_block(more.y, more.w, m, ah.a1);
                    compose_lanes<G>(ml);
                    compose_lanes<G>(mh);
                    accl |= ul & ml.lt;
                    acch |= uh & mh.lt;
                    ul &= ml.eq;
                    uh &= mh.eq;
                }
            }
            const u64 ns = o ^ ((u64)(al.a2 | accl) | ((u64)(ah.a2 | acch) << 32));
            if (valid && g == 0) {
                if (MEAS && last) {
                    const int anti = __popcll(ns ^ c) + __popcll(ns ^ hz) + __popcll(ns ^ up) +
                                     __popcll(ns ^ dn);
                    m_acc += 2 * (__popcll(ns) + __popcll(c)) - 128;
                    e_acc += 2 * anti - 256;
                }
                if (last) out[(long long)gr * nw + x] = ns;
                else own[tr * nw + x] = ns;
            }
            i += kWords;
            if (i < n) {
                place(i, tr, x, gr);
                draw((u32)gr * (u32)nw + (u32)x);
            }
        }
        if (last) {  // the other colour's band rows are final
            u64* o = color ? out0 : out1;
            for (int c = (int)threadIdx.x; c < T.nb * nw; c += kTileThreads)
                o[(long long)T.r0 * nw + c] = oth[run.depth * nw + c];
        }
    }
    if constexpr (MEAS) block_accumulate2(m_acc, e_acc, p.meas);
}

// ------------------------------------------------------------------------- host side ---

static size_t tile_row_bytes(const ising_sim* h)
{
    return h->variant == ISING_VARIANT_MSC ? (size_t)h->nw * 8 : (size_t)h->pitch;
}

// Tile words (of four int8 sites) up to which an int8 item is one word instead of four: 256^2
// 44 / 38 flips/ns, 128^2 13 / 10; 1024^2 (above it) 287 / 355.
constexpr int kTileWordItems = 1024;

static TileRows tile_rows(const ising_sim* h)
{
    const bool msc = h->variant == ISING_VARIANT_MSC;
    return TileRows{msc, h->ly, msc ? h->nw : (h->lh + 15) / 16, tile_row_bytes(h),
                    h->sm_count > 0 ? h->sm_count : 1};
}

bool temporal_ok(const ising_sim* h)
{
    return h->ndim == 2 && tile_shape(tile_rows(h)).depth > 0;
}

bool temporal_pays(const ising_sim* h, int64_t every)
{
    return h->ndim == 2 && tiles_pay(tile_rows(h), every);
}

template <class Kernel, class... Args>
static cudaError_t launch_tile(Kernel kernel, unsigned blocks, size_t smem, cudaStream_t st,
                               const Args&... args)
{
    // Above 48 KiB with the static arrays the limit must be raised.  It belongs to the function,
    // not to the launch: always the same value, so that no thread lowers it between another
    // thread's call and its launch.
    if (smem > 32 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(
            kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kTileMaxSmem);
        if (e != cudaSuccess) return e;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(kTileThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

template <bool MEAS>
static cudaError_t launch_int8_tile(int rule, const Int8Half& p, const TileRun& run,
                                    unsigned blocks, size_t smem, cudaStream_t st,
                                    const int8_t* i0, const int8_t* i1, int8_t* o0, int8_t* o1)
{
    auto go = [&](auto V, auto mixed) {
        constexpr int v = decltype(V)::value;
        constexpr bool mx = decltype(mixed)::value;
        switch (rule) {
        case kMetroFast:
            return launch_tile(int8_tile_kernel<v, kMetroFast, mx, MEAS>, blocks, smem, st, p, run,
                               i0, i1, o0, o1);
        case kHeat:
            return launch_tile(int8_tile_kernel<v, kHeat, mx, MEAS>, blocks, smem, st, p, run, i0,
                               i1, o0, o1);
        default:
            return launch_tile(int8_tile_kernel<v, kMetroGeneric, mx, MEAS>, blocks, smem, st, p,
                               run, i0, i1, o0, o1);
        }
    };
    if (p.vw == 4) return go(std::integral_constant<int, 4>{}, std::false_type{});
    return p.lh % 16 ? go(std::integral_constant<int, 16>{}, std::true_type{})
                     : go(std::integral_constant<int, 16>{}, std::false_type{});
}

// One launch: half-sweeps h0 .. h0 + depth - 1 from sweep t, from the handle's arrays into its
// scratch pair (to_scratch) or back; meas: the (M, E) accumulators of its last half-sweep.
static cudaError_t launch_tiles(const ising_sim* h, u32 t, int h0, int depth, int band,
                                unsigned long long* meas, bool to_scratch)
{
    TileRun run{h0, depth, band, 0};
    const unsigned blocks = (unsigned)((h->ly + band - 1) / band);
    const size_t smem = 2 * (size_t)(band + 2 * depth) * tile_row_bytes(h);
    void* const* in = to_scratch ? h->c : h->tb_scratch;
    void* const* out = to_scratch ? h->tb_scratch : h->c;
    const unsigned long long rows = (unsigned long long)band + 2 * depth;
    if (h->variant == ISING_VARIANT_MSC) {
        MscHalf p;
        memset(&p, 0, sizeof p);
        p.rows = (int)h->rows;
        p.nw = h->nw;
        p.t = t;
        p.k0 = (u32)h->seed;
        p.k1 = (u32)(h->seed >> 32);
        p.thr4 = h->table[3];
        p.thr8 = h->table[4];
        p.meas = meas;
        run.items_magic = fast_div_magic((u32)p.nw, rows * p.nw);
        const u64 *i0 = (const u64*)in[0], *i1 = (const u64*)in[1];
        u64 *o0 = (u64*)out[0], *o1 = (u64*)out[1];
        auto go = [&](auto G, auto KB) {
            constexpr int g = decltype(G)::value, kb = decltype(KB)::value;
            return meas ? launch_tile(msc_tile_kernel<g, kb, true>, blocks, smem, h->stream, p, run,
                                      i0, i1, o0, o1)
                        : launch_tile(msc_tile_kernel<g, kb, false>, blocks, smem, h->stream, p,
                                      run, i0, i1, o0, o1);
        };
        // Lanes per word and blocks per lane, by the words of the first step.  Measured (flips/ns)
        // with (4, 2) / (2, 4) / (1, 6): 256^2 41 / 35 / 31, 512^2 148 / 140 / 119, 1024^2
        // 429 / 441 / 425, 1152^2 481 / 530 / 516, 2048^2 829 / 991 / 1212, 4096^2 1149 / 1491 /
        // 2043; (1, 4), which draws the least, 1160 at 2048^2 and 1933 at 4096^2.
        const int first = (band + 2 * depth - 2) * h->nw;
        if (first <= 96)
            return go(std::integral_constant<int, 4>{}, std::integral_constant<int, 2>{});
        if (first <= 256)
            return go(std::integral_constant<int, 2>{}, std::integral_constant<int, 4>{});
        return go(std::integral_constant<int, 1>{}, std::integral_constant<int, 6>{});
    }
    Int8Half p;
    memset(&p, 0, sizeof p);
    p.rows = h->rows;
    p.lh = h->lh;
    p.ly = h->ly;
    p.lz = 1;
    p.pitch = h->pitch;
    p.vw = 16;
    p.cpr = (h->lh + 15) / 16;
    if (rows * (unsigned)(h->lh / 4) <= (unsigned long long)kTileWordItems) {
        p.vw = 4;
        p.cpr = h->lh / 4;
    }
    p.t = t;
    p.k0 = (u32)h->seed;
    p.k1 = (u32)(h->seed >> 32);
    for (int i = 0; i < 7; ++i) p.table[i] = h->table[i];
    p.meas = meas;
    run.items_magic = fast_div_magic((u32)p.cpr, rows * p.cpr);
    const int8_t *i0 = (const int8_t*)in[0], *i1 = (const int8_t*)in[1];
    int8_t *o0 = (int8_t*)out[0], *o1 = (int8_t*)out[1];
    return meas ? launch_int8_tile<true>(h->rule, p, run, blocks, smem, h->stream, i0, i1, o0, o1)
                : launch_int8_tile<false>(h->rule, p, run, blocks, smem, h->stream, i0, i1, o0, o1);
}

int temporal_scratch(ising_sim* h)
{
    // Another stream may be under capture in a mode that forbids waiting for a stream: the
    // allocation has nothing to do with it, so this thread does it in the relaxed mode.
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaThreadExchangeStreamCaptureMode(&mode);
    int rc = ISING_OK;
    for (int c = 0; c < 2 && rc == ISING_OK; ++c) {
        if (h->tb_scratch[c]) continue;
        // on a stream that is then waited for: usable from any stream the handle is given later
        cudaError_t e =
            pool_alloc(h->device, &h->tb_scratch[c], h->colour_bytes, h->own_stream_handle);
        if (e == cudaSuccess) e = cudaStreamSynchronize(h->own_stream_handle);
        if (e != cudaSuccess) {
            cudaGetLastError();
            h->tb_scratch[c] = nullptr;
            rc = fail(ISING_ERR_NOMEM, "allocation of the temporal schedule's second arrays");
        }
    }
    cudaThreadExchangeStreamCaptureMode(&mode);
    return rc;
}

// `sweeps` sweeps from sweep t, (M, E) of the last one into meas (unless null): an even number of
// launches of about the same depth, alternating between the handle's arrays and the scratch pair,
// so that the lattice ends in the handle's arrays.
cudaError_t launch_temporal_run(const ising_sim* h, u32 t, int64_t sweeps,
                                unsigned long long* meas)
{
    const TileShape shape = tile_shape(tile_rows(h));
    const TileCuts cuts(2 * sweeps, shape.depth);
    int64_t done = 0;
    for (int64_t i = 0; i < cuts.launches; ++i) {
        const int d = (int)cuts.depth(i);
        const cudaError_t e =
            launch_tiles(h, t + (u32)(done >> 1), (int)(done & 1), d, shape.band,
                         i + 1 == cuts.launches ? meas : nullptr, (i & 1) == 0);
        if (e != cudaSuccess) return e;
        done += d;
    }
    return cudaSuccess;
}

}  // namespace ising
