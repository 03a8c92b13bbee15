// Batched ensembles and continuous-batching serving: many independent lattices of uneven size,
// dimension, variant and temperature advanced together, one grouped launch per half-sweep
// "epoch" over a (lattice, tile) work list.
//
// Every lattice keeps its own seed, table, sweep counter and measurement interval.  Its sweep
// counter at epoch e is t0 + (e - join) / 2 (lattices join at even epochs, so every launch
// updates one colour, e % 2, of every active lattice); its (M, E) after sweep s lands in its
// own series slot.  The random numbers depend only on (site, sweep, colour, seed), so each
// lattice is bit-identical to running it alone with the single-lattice kernels.
//
// Lattices of one kernel class (variant, dims, decision rule, padded or not) share a launch, and
// classes run side by side on streams of their own (measured on one B200, 21 served jobs of five
// classes: 21.4 ms one after another, 15.9 side by side, 11.7 with small classes on one chunk or
// word per thread).  The host engine decides membership deterministically from sweep counts, so
// it never waits for the device except to hand results back (events) and to bound how far it runs
// ahead.
#include <algorithm>
#include <climits>
#include <chrono>
#include <condition_variable>
#include <cstring>
#include <deque>
#include <map>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

#include "band_plan.h"
#include "capi_internal.h"
#include "int8_core.cuh"
#include "msc_core.cuh"

namespace ising {

// One msc lattice of a batch (read from global memory by the msc kernel).
struct BatchLattice {
    void* c[2];
    long long* series;     // (M, E) pairs, or nullptr
    long long join_epoch;  // even epoch of the first half-sweep
    int rows, nw, nw_shift;
    u64 nw_magic;          // ceil(2^64 / nw)
    int every;             // measurement interval in sweeps (0 = none)
    u32 t0;
    u32 k0, k1;
    u32 table[7];
};

// Work-item sizes follow the work of each kernel class: about kItemsPerSlot items per resident
// block of the class's kernel (so a launch has no long tail and small lattices still fill the
// GPU), within these bounds; both are multiples of 256 chunks or words.
constexpr long long kInt8ItemMin = 512, kInt8ItemMax = 4096;    // band slots
constexpr long long kMscItemMin = 2048, kMscItemMax = 16384;    // words
constexpr long long kItemsPerSlot = 6;  // default of the ISING_KNOB_ITEMS_PER_SLOT knob
// Chunk-rows (2D, 3D) and msc words per SM below which a class runs one chunk or word per thread.
// Measured on one B200 against bands and word ranges (flips/ns of a batch): 64 x 256^2 398 / 353,
// 8 x 1000x1048 640 / 524, 12 x 64^3 heat bath 409 / 303, 3D heat bath 56^3..248^3 (707,000
// chunks) 656 / 607, msc 128^2..2688^2 1541 / 690, 6 x msc 4096^2 (786,000 words) 2328 / 2278.
// (16 x 1024^2, 524,288 chunks: 709 / 670; 32 lattices of 755,000 chunks: 633 / 653.)
constexpr long long kOneUnits2 = 4000, kOneUnits3 = 6000, kOneWords = 6000;
// Blocks of 256 band slots per resident block that the band height of a class leaves: two keep the
// bands two rows high (which fixes the row parity in the code) where six, as for the work items,
// gave bands of one row: 32 lattices of 755,000 chunks 602 -> 653, 2 x 4096^2 851 -> 974.
constexpr long long kBandBlocks = 2;
constexpr int kBandCap = 8;             // default of the ISING_KNOB_BAND knob (batch)

// Item size for `total` units of work over `slots` resident blocks, `per_slot` items each.
inline long long item_size(long long total, long long slots, long long per_slot, long long lo,
                           long long hi)
{
    long long want = (total + per_slot * slots - 1) / (per_slot * slots);
    return want < lo ? lo : (want > hi ? hi : want);
}

// ----------------------------------------------------------------------------- int8 -------
// An int8 launch covers up to kInt8PerLaunch lattices of one kernel class; their descriptors are
// the launch's parameter block (constant memory), so every field a block reads is uniform, as
// in the single-lattice kernel.  Block b belongs to the last lattice whose block_begin <= b (a
// uniform binary search) and updates its slots [(b - block_begin) * per, ...), a slot being a
// band of L.band rows of one plane in one chunk column (int8_band), band-major.
struct Int8Desc {
    void* c[2];
    long long* series;     // (M, E) pairs, or nullptr
    long long join_epoch;  // even epoch of the first half-sweep
    int every;             // measurement interval in sweeps (0 = none)
    u32 t0, k0, k1;
    u32 table[7];
    int rows, lh, ly, lz, pitch, cpr, band, bpp;
    u32 cpr_magic, bpp_magic;  // fast_div magics of cpr and bpp
    int block_begin;           // first block of this lattice in the launch
    int per_block;             // band slots per block (a multiple of 256)
    int nslots;                // band slots of the lattice: lz * bpp * cpr
};

// Parameter blocks come in three capacities; a launch passes the smallest that holds its
// lattices, since the host cost of a launch grows with the size of its parameters.
constexpr int kInt8PerLaunch = 240;

template <int N>
struct Int8LaunchN {
    long long epoch;               // the launch's epoch, relative to *epoch_base when set
    const long long* epoch_base;   // replayed graph chunks: device epoch counter, else nullptr
    int n;  // lattices
    int pad;
    Int8Desc lat[N];
};
using Int8Launch = Int8LaunchN<kInt8PerLaunch>;
static_assert(sizeof(Int8Launch) <= 32764, "kernel parameter block over the 32 KB limit");

// The lattice of this block: the last one whose block_begin is not beyond it.
template <class Desc>
__device__ __forceinline__ int find_lattice(const Desc* lat, int n)
{
    const int b = (int)blockIdx.x;
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (lat[mid].block_begin <= b) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// The half-sweep of lattice L at `epoch`; meas: it ends a measured sweep.
__device__ __forceinline__ Int8Half lattice_half(const Int8Desc& L, long long epoch, int v, bool& meas)
{
    const u32 color = (u32)(epoch & 1);
    const u32 s = (u32)((epoch - L.join_epoch) >> 1);  // sweeps done (< 2^31)
    meas = color == 1 && L.every > 0 && ((s + 1u) % (u32)L.every) == 0;
    Int8Half p;
    p.own = static_cast<int8_t*>(L.c[color]);
    p.other = static_cast<const int8_t*>(L.c[color ^ 1]);
    p.rows = L.rows;
    p.lh = L.lh;
    p.ly = L.ly;
    p.lz = L.lz;
    p.cpr = L.cpr;
    p.pitch = L.pitch;
    p.vw = v;
    p.t = L.t0 + s;
    p.color = color;
    p.k0 = L.k0;
    p.k1 = L.k1;
    p.meas = meas ? reinterpret_cast<unsigned long long*>(
                        L.series + 2 * ((s + 1u) / (u32)L.every - 1u))
                  : nullptr;
    p.ctl = nullptr;
    return p;
}

template <int V, int NDIM, int RULE, bool MIXED, bool MEAS>
__device__ __forceinline__ void batch_int8_slots(const Int8Half& p, const Int8Desc& L, u32 s0,
                                                 u32 s1, const u32* rt, long long& m_acc,
                                                 long long& e_acc)
{
    const u32 cpr = (u32)L.cpr, bpp = (u32)L.bpp;
    for (u32 slot = s0 + threadIdx.x; slot < s1; slot += 256u) {
        const u32 band = fast_div(slot, cpr, L.cpr_magic);
        const int j0 = (int)(slot - band * cpr) * V;
        int z = 0, yb = (int)band;
        if constexpr (NDIM == 3) {
            z = (int)fast_div(band, bpp, L.bpp_magic);
            yb = (int)(band - (u32)z * bpp);
        }
        const int y0 = yb * L.band;
        const int y1 = y0 + L.band < L.ly ? y0 + L.band : L.ly;
        int8_band<V, NDIM, RULE, MIXED, MEAS, NDIM == 2 || kRowPairs<RULE, MIXED, MEAS>>(
            p, z, y0, y1, j0, rt, m_acc, e_acc);
    }
}

#ifndef ISING_BATCH_MIN_BLOCKS
#define ISING_BATCH_MIN_BLOCKS 4
#endif
template <int V, int NDIM, int RULE, bool MIXED, int N>
__global__ void __launch_bounds__(256, ISING_BATCH_MIN_BLOCKS)
    batch_int8_kernel(const __grid_constant__ Int8LaunchN<N> P)
{
    __shared__ u32 rt[kLookupWords];  // the lookup table of the decisions
    // The lattice, its table and epoch come from the launch's parameters (whose first reads are
    // slow) and a counter that changes between graph replays only: all before the wait.
    const Int8Desc& L = P.lat[find_lattice(P.lat, P.n)];
    if (threadIdx.x == 0) fill_lookup<NDIM, RULE>(rt, L.table);
    const long long epoch = P.epoch + (P.epoch_base ? *P.epoch_base : 0);
    bool meas;
    const Int8Half p = lattice_half(L, epoch, V, meas);
    const int b = (int)blockIdx.x;
    __syncthreads();
    // launched with programmatic stream serialization: wait for the class's previous half-sweep,
    // then let the next launch start
    pdl_wait();
    pdl_trigger();
    const u32 s0 = (u32)(b - L.block_begin) * (u32)L.per_block;
    const u32 s1 = s0 + (u32)L.per_block < (u32)L.nslots ? s0 + (u32)L.per_block : (u32)L.nslots;
    long long m_acc = 0, e_acc = 0;
    if (meas) {
        batch_int8_slots<V, NDIM, RULE, MIXED, true>(p, L, s0, s1, rt, m_acc, e_acc);
        block_accumulate2(m_acc, e_acc, p.meas);
    } else {
        batch_int8_slots<V, NDIM, RULE, MIXED, false>(p, L, s0, s1, rt, m_acc, e_acc);
    }
}

// One chunk per thread, for classes with too few chunks to give every thread a band: as
// int8_one_kernel, the random numbers are drawn before the class's previous half-sweep is done.
constexpr int kOneThreads = 128;

template <int NDIM, int RULE, bool MIXED, int N>
__global__ void __launch_bounds__(kOneThreads)
    batch_int8_one_kernel(const __grid_constant__ Int8LaunchN<N> P)
{
    constexpr int V = 16, W = 4;
    __shared__ u32 rt[kLookupWords];  // the lookup table of the decisions
    const Int8Desc& L = P.lat[find_lattice(P.lat, P.n)];
    if (threadIdx.x == 0) fill_lookup<NDIM, RULE>(rt, L.table);
    // (the device epoch counter changes between graph replays only)
    const long long epoch = P.epoch + (P.epoch_base ? *P.epoch_base : 0);
    bool meas;
    const Int8Half p = lattice_half(L, epoch, V, meas);
    const u32 slot = (u32)((int)blockIdx.x - L.block_begin) * kOneThreads + threadIdx.x;
    const u32 row = fast_div(slot, (u32)L.cpr, L.cpr_magic);
    const int j0 = (int)(slot - row * (u32)L.cpr) * V;
    int z = 0, y = (int)row;
    if constexpr (NDIM == 3) {
        z = (int)fast_div(row, (u32)L.bpp, L.bpp_magic);
        y = (int)(row - (u32)z * (u32)L.bpp);
    }
    const DrawSites<NDIM> sites{p, site_counter(p, row, j0)};
    u32x4 r[W];
#pragma unroll
    for (int k = 0; k < W; ++k) {
        r[k] = sites(k);
        asm volatile("" : "+r"(r[k].x), "+r"(r[k].y), "+r"(r[k].z), "+r"(r[k].w));
    }
    __syncthreads();
    pdl_wait();
    pdl_trigger();
    auto drawn = [&](int k) { return r[k]; };
    long long m_acc = 0, e_acc = 0;
    const bool valid = slot < (u32)L.nslots;
    if (meas) {
        if (valid)
            int8_chunk<V, NDIM, RULE, false, MIXED, true>(p, drawn, row, y, z, j0, rt, m_acc, e_acc);
        block_accumulate2(m_acc, e_acc, p.meas);
    } else if (valid) {
        int8_chunk<V, NDIM, RULE, false, MIXED, false>(p, drawn, row, y, z, j0, rt, m_acc, e_acc);
    }
}

// ------------------------------------------------------------------------------ msc -------
// Small msc classes run one word per thread, the lattice descriptors in the launch's parameters
// as for int8 and kOneCalls Philox blocks per word drawn before the class's previous half-sweep is
// done; larger ones walk word ranges with a work stack (batch_msc_kernel).
struct MscDesc {
    u64* c[2];
    long long* series;     // (M, E) pairs, or nullptr
    long long join_epoch;  // even epoch of the first half-sweep
    u64 nw_magic;          // ceil(2^64 / nw)
    int every;             // measurement interval in sweeps (0 = none)
    int rows, nw, nw_shift;
    u32 t0, k0, k1, thr4, thr8;
    int block_begin;       // first block of this lattice in the launch
};

template <int N>
struct MscLaunchN {
    long long epoch;
    const long long* epoch_base;
    int n;
    int pad;
    MscDesc lat[N];
};
using MscLaunch = MscLaunchN<kInt8PerLaunch>;
static_assert(sizeof(MscLaunch) <= 32764, "kernel parameter block over the 32 KB limit");

constexpr int kOneCalls = 6;

template <int N>
__global__ void __launch_bounds__(kOneThreads)
    batch_msc_one_kernel(const __grid_constant__ MscLaunchN<N> P)
{
    __shared__ uint4 lvmask[16];
    const MscDesc& L = P.lat[find_lattice(P.lat, P.n)];
    if (threadIdx.x < 16) lvmask[threadIdx.x] = level_masks(L.thr4, L.thr8, threadIdx.x);
    const long long epoch = P.epoch + (P.epoch_base ? *P.epoch_base : 0);
    const u32 color = (u32)(epoch & 1);
    const u32 s = (u32)((epoch - L.join_epoch) >> 1);  // sweeps done (< 2^31)
    const bool meas = color == 1 && L.every > 0 && ((s + 1u) % (u32)L.every) == 0;
    MscHalf p;
    p.own = L.c[color];
    p.other = L.c[color ^ 1];
    p.rows = L.rows;
    p.nw = L.nw;
    p.t = L.t0 + s;
    p.color = color;
    p.k0 = L.k0;
    p.k1 = L.k1;
    p.nw_magic = L.nw_magic;
    const u32 w = (u32)((int)blockIdx.x - L.block_begin) * kOneThreads + threadIdx.x;
    u32x4 r[kOneCalls];
#pragma unroll
    for (int b = 0; b < kOneCalls; ++b) {
        r[b] = philox4x32_10<true>(w, p.t, color, 1u + (u32)b, p.k0, p.k1);
        asm volatile("" : "+r"(r[b].x), "+r"(r[b].y), "+r"(r[b].z), "+r"(r[b].w));
    }
    __syncthreads();
    pdl_wait();
    pdl_trigger();
    long long m_acc = 0, e_acc = 0;
    const bool valid = w < (u32)L.rows * (u32)L.nw;
    if (valid) {
        IntakeLoads I;
        intake_load(p, w, true, L.nw, L.nw_shift, I);
        const bool par = ((I.y + (int)color) & 1) != 0;
        const u64 hz = par ? ((I.c >> 1) | (I.side << 63)) : ((I.c << 1) | (I.side >> 63));
        const HalfSlices al = slice_half((u32)I.o, (u32)I.c, (u32)hz, (u32)I.up, (u32)I.dn);
        const HalfSlices ah = slice_half((u32)(I.o >> 32), (u32)(I.c >> 32), (u32)(hz >> 32),
                                         (u32)(I.up >> 32), (u32)(I.dn >> 32));
        u32 ul = ~al.a2, uh = ~ah.a2, accl = 0, acch = 0;
#pragma unroll
        for (int b = 0; b < kOneCalls; ++b)
            block_levels(r[b], lvmask[b], al.a1, ah.a1, ul, uh, accl, acch);
        for (u32 lp = kOneCalls; lp < 16u && (ul | uh) != 0; ++lp) {
            const u32x4 more = philox4x32_10<true>(w, p.t, color, 1u + lp, p.k0, p.k1);
            block_levels(more, lvmask[lp], al.a1, ah.a1, ul, uh, accl, acch);
        }
        const u64 ns = I.o ^ ((u64)(al.a2 | accl) | ((u64)(ah.a2 | acch) << 32));
        p.own[w] = ns;
        if (meas) {
            const int anti = __popcll(ns ^ I.c) + __popcll(ns ^ hz) + __popcll(ns ^ I.up) +
                             __popcll(ns ^ I.dn);
            m_acc = 2 * (__popcll(ns) + __popcll(I.c)) - 128;
            e_acc = 2 * anti - 256;
        }
    }
    if (meas)
        block_accumulate2(m_acc, e_acc, reinterpret_cast<unsigned long long*>(
                                            L.series + 2 * ((s + 1u) / (u32)L.every - 1u)));
}

struct BatchItem {
    int lat;
    int pad;
    long long begin, end;  // words
};

constexpr int kBatchWarps = 8;

__global__ void __launch_bounds__(kBatchWarps * 32) batch_msc_kernel(
    const BatchLattice* __restrict__ lats, const BatchItem* __restrict__ items, int n_items,
    long long epoch_rel, const long long* epoch_base)
{
    __shared__ QueueSlots q_all[kBatchWarps];
    __shared__ uint4 lvmask[16];
    // (launched without programmatic serialization: its early-launched blocks would hold their
    // 17 KB work stacks while waiting, and the batch measured slower with it)
    // the epoch, relative to the device counter in replayed graph chunks
    const long long epoch = epoch_rel + (epoch_base ? *epoch_base : 0);
    const u32 color = (u32)(epoch & 1);
    const int warp = threadIdx.x >> 5;
    long long m_acc = 0, e_acc = 0;  // flushed per lattice, as in batch_int8_kernel
    for (int it = blockIdx.x; it < n_items; it += gridDim.x) {
        const BatchItem item = items[it];
        const BatchLattice& L = lats[item.lat];
        const u32 s = (u32)((epoch - L.join_epoch) >> 1);  // sweeps done (< 2^31)
        const bool meas = color == 1 && L.every > 0 && ((s + 1u) % (u32)L.every) == 0;
        MscHalf p;
        p.own = static_cast<u64*>(L.c[color]);
        p.other = static_cast<const u64*>(L.c[color ^ 1]);
        p.rows = L.rows;
        p.nw = L.nw;
        p.t = L.t0 + s;
        p.color = color;
        p.k0 = L.k0;
        p.k1 = L.k1;
        p.thr4 = L.table[3];
        p.thr8 = L.table[4];
        p.nw_magic = L.nw_magic;
        p.stats = nullptr;
        p.ctl = nullptr;
        p.meas = meas ? reinterpret_cast<unsigned long long*>(
                            L.series + 2 * ((s + 1u) / (u32)L.every - 1u))
                      : nullptr;
        if (threadIdx.x < 16) lvmask[threadIdx.x] = level_masks(p.thr4, p.thr8, threadIdx.x);
        __syncthreads();
        const long long len = item.end - item.begin;
        long long per = (len + kBatchWarps - 1) / kBatchWarps;
        per = (per + 31) / 32 * 32;
        const long long b = item.begin + warp * per;
        const long long e = min(b + per, item.end);
        msc_queue_range(p, b, e, L.nw_shift, q_all[warp], lvmask);
        if (meas) {
            // the warp's words are final: measure them (the other colour is unchanged)
            __syncwarp();
            msc_measure_range(p, b, e, L.nw_shift, m_acc, e_acc);
            if (it + (int)gridDim.x >= n_items || items[it + gridDim.x].lat != item.lat) {
                block_accumulate2(m_acc, e_acc, p.meas);
                m_acc = e_acc = 0;
            }
        }
        __syncthreads();
    }
}

__global__ void batch_epoch_set(long long* counter, long long epoch) { *counter = epoch; }

// ----------------------------------------------------------------------------- host engine ---

using Clock = std::chrono::steady_clock;

struct Job {
    int64_t id = 0;
    int state = ISING_JOB_PENDING;
    ising_job spec;
    std::vector<int8_t> init;  // host copy of an initial lattice (ISING_INIT_LATTICE)
    int rows = 0, lh = 0, ly = 0, lz = 1, nw = 0;
    int pitch = 0;  // int8: bytes between rows on the device (lh rounded up to 16)
    size_t colour_bytes = 0, series_pairs = 0, device_bytes = 0;
    void* c[2] = {nullptr, nullptr};
    long long* d_series = nullptr;
    long long* h_series = nullptr;  // pinned
    int8_t* h_lattice = nullptr;    // pinned, keep_lattice only
    long long join_epoch = -1;
    cudaEvent_t done_event = nullptr;
    Clock::time_point t_submit, t_start, t_done;
    std::string error;
};

struct KernelClass {
    int variant, v, ndim, rule, mixed;  // mixed: rows padded (lh % 16 != 0)
    bool operator<(const KernelClass& o) const
    {
        return std::tie(variant, v, ndim, rule, mixed) <
               std::tie(o.variant, o.v, o.ndim, o.rule, o.mixed);
    }
};

// The launches of one int8 class.
struct Int8Class {
    KernelClass kc;
    bool one;  // one chunk per thread
    std::vector<Int8Launch> launches;
};

// memcpy of a finished lattice into the caller's memory, by up to four threads for large ones: the
// caller's pages are usually new, and one thread faulting and filling them copies about 5 GB/s.
static void copy_lattice(int8_t* dst, const int8_t* src, size_t n)
{
    constexpr size_t kPart = (size_t)2 << 20;
    size_t parts = std::min<size_t>(4, n / kPart);
    parts = std::min<size_t>(parts, std::thread::hardware_concurrency());
    if (parts < 2) {
        memcpy(dst, src, n);
        return;
    }
    std::thread helpers[3];
    const size_t step = n / parts & ~(size_t)4095;
    size_t begin = 0;
    for (size_t i = 0; i + 1 < parts; ++i) {
        try {
            helpers[i] = std::thread([=] { memcpy(dst + begin, src + begin, step); });
        } catch (...) {  // no thread to be had: the rest is copied here
            break;
        }
        begin += step;
    }
    memcpy(dst + begin, src + begin, n - begin);
    for (std::thread& t : helpers)
        if (t.joinable()) t.join();
}

class Engine {
public:
    Engine(int device, int64_t budget) : device_(device), budget_(budget) {}

    int init()
    {
        cudaError_t e = cudaSetDevice(device_);
        if (e != cudaSuccess) return cuda_fail(e, "cudaSetDevice");
        e = cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking);
        if (e != cudaSuccess) return cuda_fail(e, "cudaStreamCreate");
        sms_ = device_sm_count(device_);
        // The engine's own stream-ordered pool keeps freed lattice memory (up to the budget)
        // mapped across synchronisations, so admitting a job after another finished reuses it
        // instead of mapping fresh pages; the device's default pool is left untouched.
        cudaMemPoolProps props;
        memset(&props, 0, sizeof props);
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device_;
        e = cudaMemPoolCreate(&pool_, &props);
        if (e != cudaSuccess) return cuda_fail(e, "cudaMemPoolCreate");
        uint64_t keep = (uint64_t)budget_;
        e = cudaMemPoolSetAttribute(pool_, cudaMemPoolAttrReleaseThreshold, &keep);
        if (e != cudaSuccess) return cuda_fail(e, "cudaMemPoolSetAttribute");
        e = cudaMalloc((void**)&d_epoch_, sizeof(long long));
        if (e != cudaSuccess) return cuda_fail(e, "cudaMalloc (epoch counter)");
        return ISING_OK;
    }

    ~Engine()
    {
        cudaSetDevice(device_);
        for (Aux& a : aux_) cudaStreamSynchronize(a.stream);
        if (stream_) cudaStreamSynchronize(stream_);
        for (auto& kv : jobs_) free_job(*kv.second);
        if (d_lats_) cudaFreeAsync(d_lats_, stream_);
        if (d_items_) cudaFreeAsync(d_items_, stream_);
        if (stream_) cudaStreamSynchronize(stream_);
        if (chunk_exec_) cudaGraphExecDestroy(chunk_exec_);
        for (auto& x : old_execs_) {
            cudaGraphExecDestroy(x.first);
            cudaEventDestroy(x.second);
        }
        if (d_epoch_) cudaFree(d_epoch_);
        for (auto& kv : pinned_free_) cudaFreeHost(kv.second);
        for (cudaEvent_t ev : epoch_events_) cudaEventDestroy(ev);
        for (Aux& a : aux_) {
            cudaEventDestroy(a.event);
            cudaStreamDestroy(a.stream);
        }
        if (fork_event_) cudaEventDestroy(fork_event_);
        if (stream_) cudaStreamDestroy(stream_);
        if (pool_) cudaMemPoolDestroy(pool_);
        cudaGetLastError();
    }

    // Validates the job and queues it; returns its id.
    int submit(const ising_job& spec, int64_t* id)
    {
        auto j = std::make_unique<Job>();
        int rc = validate(spec, *j);
        if (rc != ISING_OK) return rc;
        j->spec = spec;
        if (spec.init == ISING_INIT_LATTICE) {
            const size_t n = (size_t)j->rows * 2 * j->lh;
            j->init.assign(spec.lattice, spec.lattice + n);
        }
        j->spec.lattice = nullptr;
        if ((int64_t)j->device_bytes > budget_)
            return fail(ISING_ERR_NOMEM, "job needs %zu device bytes, over the %lld-byte budget",
                        j->device_bytes, (long long)budget_);
        // the pinned host buffers of the results are taken now, on the submitting thread:
        // page-locking memory while the job finishes would stall the sweeps in flight
        cudaError_t e = cudaSuccess;
        if (j->series_pairs)
            e = pinned_get((void**)&j->h_series, j->series_pairs * 2 * sizeof(long long));
        if (e == cudaSuccess && spec.keep_lattice)
            e = pinned_get((void**)&j->h_lattice, (size_t)j->rows * 2 * j->lh);
        if (e != cudaSuccess) {
            cudaGetLastError();
            free_job(*j);
            return fail(ISING_ERR_NOMEM, "pinned result buffers of a job");
        }
        j->id = ++last_id_;
        j->t_submit = Clock::now();
        *id = j->id;
        pending_.push_back(j->id);
        jobs_[j->id] = std::move(j);
        return ISING_OK;
    }

    bool busy() const { return !active_.empty() || !pending_.empty() || !finishing_.empty(); }
    bool has_work() const { return !active_.empty() || !pending_.empty(); }
    size_t active_count() const { return active_.size(); }
    size_t pending_count() const { return pending_.size(); }
    long long epoch() const { return epoch_; }
    int64_t used_bytes() const { return used_; }

    // One half-sweep of every active lattice (admitting pending jobs at even epochs).
    // Issues the next epoch, or the next replayed chunk of 2 * chunk_sweeps_ epochs when the
    // batch is stable and `budget` (epochs the caller still allows; <= 0: no limit) holds it.
    int step(long long budget = 0)
    {
        cudaError_t e = cudaSetDevice(device_);
        if (e != cudaSuccess) return cuda_fail(e, "cudaSetDevice");
        if ((epoch_ & 1) == 0) {
            int rc = admit();
            if (rc != ISING_OK) return rc;
        }
        if (active_.empty()) return ISING_OK;
        if (dirty_) {
            drop_chunk();
            int rc = rebuild();
            if (rc != ISING_OK) return rc;
        }
        reap_chunks();
        if (chunk_ready() && (budget <= 0 || 2 * chunk_sweeps_ <= budget)) {
            int rc = run_chunk();
            if (rc == ISING_OK) rc = retire();
            if (rc == ISING_OK) rc = throttle();
            return rc;
        }
        e = launch_epoch(epoch_, nullptr);
        if (e != cudaSuccess) return cuda_fail(e, "batch launch");
        ++epoch_;
        if ((epoch_ & 1) == 0) {
            int rc = join();
            if (rc == ISING_OK) rc = retire();
            if (rc != ISING_OK) return rc;
            rc = throttle();
            if (rc != ISING_OK) return rc;
        }
        return ISING_OK;
    }

    // Marks finished result copies as done; returns how many completed.
    int poll()
    {
        int n = 0;
        for (auto it = finishing_.begin(); it != finishing_.end();) {
            Job& j = *jobs_[*it];
            const cudaError_t e = cudaEventQuery(j.done_event);
            if (e == cudaSuccess) {
                j.state = ISING_JOB_DONE;
                j.t_done = Clock::now();
                cudaEventDestroy(j.done_event);
                j.done_event = nullptr;
                it = finishing_.erase(it);
                ++n;
            } else if (e == cudaErrorNotReady) {
                ++it;
            } else {
                return cuda_fail(e, "result event");
            }
        }
        return n;
    }

    int wait_finishing()
    {
        const int rc = join();
        if (rc != ISING_OK) return rc;
        cudaError_t e = cudaStreamSynchronize(stream_);
        if (e != cudaSuccess) return cuda_fail(e, "cudaStreamSynchronize");
        poll();
        return ISING_OK;
    }

    Job* find(int64_t id)
    {
        auto it = jobs_.find(id);
        return it == jobs_.end() ? nullptr : it->second.get();
    }

    int result(int64_t id, int64_t* series_out, int8_t* lattice_out, double* latency)
    {
        Job* j = find(id);
        if (!j) return fail(ISING_ERR_INVALID, "unknown job %lld", (long long)id);
        if (j->state != ISING_JOB_DONE)
            return fail(ISING_ERR_STATE, "job %lld is not done", (long long)id);
        if (series_out && j->series_pairs)
            memcpy(series_out, j->h_series, j->series_pairs * 2 * sizeof(long long));
        if (lattice_out) {
            if (!j->h_lattice)
                return fail(ISING_ERR_STATE, "job %lld was not submitted with keep_lattice",
                            (long long)id);
            copy_lattice(lattice_out, j->h_lattice, (size_t)j->rows * 2 * j->lh);
        }
        if (latency)
            *latency = std::chrono::duration<double>(j->t_done - j->t_submit).count();
        return ISING_OK;
    }

    int release(int64_t id)
    {
        auto it = jobs_.find(id);
        if (it == jobs_.end()) return fail(ISING_ERR_INVALID, "unknown job %lld", (long long)id);
        Job& j = *it->second;
        if (j.state == ISING_JOB_ACTIVE || j.state == ISING_JOB_FINISHING)
            return fail(ISING_ERR_STATE, "job %lld is still running", (long long)id);
        if (j.state == ISING_JOB_PENDING)
            pending_.erase(std::remove(pending_.begin(), pending_.end(), id), pending_.end());
        free_job(j);
        jobs_.erase(it);
        return ISING_OK;
    }

    int64_t budget() const { return budget_; }
    cudaStream_t stream() const { return stream_; }

    // Launch knobs of the batch (identical results for every value); applied at the next
    // rebuild of the work list.
    int set_knob(int knob, int value)
    {
        if (knob == ISING_KNOB_BAND) {
            if (value < 1 || value > 64) return fail(ISING_ERR_INVALID, "band cap must be 1..64");
            band_cap_ = value;
        } else if (knob == ISING_KNOB_ITEMS_PER_SLOT) {
            if (value < 1 || value > 64)
                return fail(ISING_ERR_INVALID, "items per slot must be 1..64");
            items_per_slot_ = value;
        } else if (knob == ISING_KNOB_GRAPH_CHUNK) {
            if (value < 0 || value > 64)
                return fail(ISING_ERR_INVALID, "batch graph chunk must be 0..64 sweeps");
            chunk_sweeps_ = value;
            drop_chunk();
        } else {
            return fail(ISING_ERR_INVALID, "knob %d does not apply to a batch", knob);
        }
        dirty_ = true;
        return ISING_OK;
    }

    int get_knob(int knob, int* value) const
    {
        if (knob == ISING_KNOB_BAND) *value = band_cap_;
        else if (knob == ISING_KNOB_ITEMS_PER_SLOT) *value = (int)items_per_slot_;
        else if (knob == ISING_KNOB_GRAPH_CHUNK) *value = (int)chunk_sweeps_;
        else return fail(ISING_ERR_INVALID, "knob %d does not apply to a batch", knob);
        return ISING_OK;
    }

private:
    int validate(const ising_job& s, Job& j)
    {
        if (s.ndim != 2 && s.ndim != 3)
            return fail(ISING_ERR_INVALID, "only 2D and 3D lattices are supported");
        for (int i = 0; i < s.ndim; ++i)
            if (s.shape[i] < 2 || s.shape[i] % 2)
                return fail(ISING_ERR_INVALID, "all extents must be even and >= 2");
        if (s.variant != ISING_VARIANT_INT8 && s.variant != ISING_VARIANT_MSC)
            return fail(ISING_ERR_INVALID, "unknown variant %d", s.variant);
        if (s.algorithm != ISING_METROPOLIS && s.algorithm != ISING_HEATBATH)
            return fail(ISING_ERR_INVALID, "unknown algorithm %d", s.algorithm);
        if (s.variant == ISING_VARIANT_MSC && (s.ndim != 2 || s.algorithm != ISING_METROPOLIS))
            return fail(ISING_ERR_INVALID, "msc supports 2D Metropolis only");
        const int64_t lx = s.shape[s.ndim - 1];
        if (lx % (s.variant == ISING_VARIANT_MSC ? 128 : 8))
            return fail(ISING_ERR_INVALID, "last extent must be a multiple of %d",
                        s.variant == ISING_VARIANT_MSC ? 128 : 8);
        if (s.table_n != 2 * s.ndim + 1)
            return fail(ISING_ERR_INVALID, "table must have %d entries", 2 * s.ndim + 1);
        if (s.n_sweeps < 0 || s.measure_every < 0)
            return fail(ISING_ERR_INVALID, "negative sweep count or interval");
        if (s.init != ISING_INIT_COLD && s.init != ISING_INIT_PHILOX && s.init != ISING_INIT_LATTICE)
            return fail(ISING_ERR_INVALID, "unknown init %d", s.init);
        if (s.init == ISING_INIT_LATTICE && !s.lattice)
            return fail(ISING_ERR_INVALID, "ISING_INIT_LATTICE needs a lattice");
        const int64_t ly = s.shape[s.ndim - 2], lz = s.ndim == 3 ? s.shape[0] : 1;
        if (ly * lz > 0x7FFFFFFF || lx / 2 > 0x7FFFFFFF)
            return fail(ISING_ERR_INVALID, "lattice too large");
        if (s.variant == ISING_VARIANT_INT8 && ly * lz * ((lx / 2 + 15) / 16) > 0x7FFFFFFF)
            return fail(ISING_ERR_INVALID, "lattice too large for the batch (2^31 chunks)");
        j.rows = (int)(ly * lz);
        j.lh = (int)(lx / 2);
        j.ly = (int)ly;
        j.lz = (int)lz;
        j.nw = (int)(lx / 128);
        j.pitch = (j.lh + 15) / 16 * 16;
        j.colour_bytes = s.variant == ISING_VARIANT_MSC ? (size_t)j.rows * j.nw * 8
                                                       : (size_t)j.rows * j.pitch;
        j.series_pairs = s.measure_every > 0 ? (size_t)(s.n_sweeps / s.measure_every) : 0;
        j.device_bytes = 2 * j.colour_bytes + j.series_pairs * 2 * sizeof(long long);
        return ISING_OK;
    }

    int admit()
    {
        for (auto it = pending_.begin(); it != pending_.end();) {
            Job& j = *jobs_[*it];
            if (used_ + (int64_t)j.device_bytes > budget_) {
                ++it;  // later, smaller jobs may still fit
                continue;
            }
            int rc = start_job(j);
            if (rc != ISING_OK) return rc;
            it = pending_.erase(it);
        }
        return ISING_OK;
    }

    int start_job(Job& j)
    {
        cudaError_t e;
        for (int c = 0; c < 2; ++c) {
            e = dev_alloc(&j.c[c], j.colour_bytes);
            if (e != cudaSuccess) return cuda_fail(e, "cudaMallocAsync (job lattice)");
        }
        if (j.series_pairs) {
            const size_t sb = j.series_pairs * 2 * sizeof(long long);
            e = dev_alloc((void**)&j.d_series, sb);
            if (e == cudaSuccess) e = cudaMemsetAsync(j.d_series, 0, sb, stream_);
            if (e != cudaSuccess) return cuda_fail(e, "job series");
        }
        const ising_job& s = j.spec;
        const int max_blocks = sms_ * 8;
        if (s.init == ISING_INIT_COLD) {
            const int v = s.variant == ISING_VARIANT_MSC ? 0xFF : 0x01;
            for (int c = 0; c < 2 && e == cudaSuccess; ++c)
                e = cudaMemsetAsync(j.c[c], v, j.colour_bytes, stream_);
        } else if (s.init == ISING_INIT_PHILOX) {
            e = launch_philox_start(j.c[0], j.c[1], j.rows, j.lh, j.pitch,
                                    s.variant == ISING_VARIANT_MSC, (u32)s.seed,
                                    (u32)(s.seed >> 32), max_blocks, stream_);
        } else {
            const size_t full = (size_t)j.rows * 2 * j.lh;
            int8_t* stage = nullptr;
            e = dev_alloc((void**)&stage, full);
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(stage, j.init.data(), full, cudaMemcpyHostToDevice, stream_);
            if (e == cudaSuccess) {
                if (s.variant == ISING_VARIANT_MSC)
                    e = launch_msc_pack(stage, (u64*)j.c[0], (u64*)j.c[1], j.rows, 0, j.nw,
                                        max_blocks, stream_);
                else
                    e = launch_int8_split(stage, (int8_t*)j.c[0], (int8_t*)j.c[1], j.rows, 0,
                                          j.lh, j.pitch, j.ly, max_blocks, stream_);
            }
            if (stage) cudaFreeAsync(stage, stream_);
            std::vector<int8_t>().swap(j.init);
        }
        if (e != cudaSuccess) return cuda_fail(e, "job start");
        used_ += (int64_t)j.device_bytes;
        j.join_epoch = epoch_;
        j.state = ISING_JOB_ACTIVE;
        j.t_start = Clock::now();
        if (s.n_sweeps == 0) {
            j.state = ISING_JOB_ACTIVE;
            return finish_job(j);
        }
        active_.push_back(j.id);
        dirty_ = true;
        return ISING_OK;
    }

    // Builds the launch lists, grouped by kernel class: for int8 classes the lattice
    // descriptors of each launch (chunks of kInt8PerLaunch), for msc the lattice table and the
    // work items in device memory.
    int rebuild()
    {
        int jrc = join();
        if (jrc != ISING_OK) return jrc;
        std::vector<BatchLattice> lats;              // msc lattices
        std::map<KernelClass, std::vector<Int8Desc>> int8_descs;
        std::map<KernelClass, long long> class_units;  // chunk-rows (int8) or words (msc)
        std::vector<std::pair<KernelClass, int>> msc_of;  // (class, index in lats)
        for (int64_t id : active_) {
            Job& j = *jobs_[id];
            const ising_job& s = j.spec;
            u32 table[7];
            for (int i = 0; i < 7; ++i) table[i] = i < s.table_n ? s.table[i] : 0xFFFFFFFFu;
            KernelClass kc{s.variant, 0, s.ndim, 0, 0};
            if (s.variant == ISING_VARIANT_MSC) {
                BatchLattice L;
                memset(&L, 0, sizeof L);
                L.c[0] = j.c[0];
                L.c[1] = j.c[1];
                L.series = j.d_series;
                L.join_epoch = j.join_epoch;
                L.rows = j.rows;
                L.nw = j.nw;
                L.nw_shift = (j.nw & (j.nw - 1)) == 0 ? __builtin_ctz((unsigned)j.nw) : -1;
                L.nw_magic = magic_for(j.nw);
                L.every = (int)s.measure_every;
                L.t0 = (u32)s.t0;
                L.k0 = (u32)s.seed;
                L.k1 = (u32)(s.seed >> 32);
                memcpy(L.table, table, sizeof table);
                class_units[kc] += (long long)j.rows * j.nw;
                msc_of.emplace_back(kc, (int)lats.size());
                lats.push_back(L);
            } else {
                Int8Desc D;
                memset(&D, 0, sizeof D);
                D.c[0] = j.c[0];
                D.c[1] = j.c[1];
                D.series = j.d_series;
                D.join_epoch = j.join_epoch;
                D.every = (int)s.measure_every;
                D.t0 = (u32)s.t0;
                D.k0 = (u32)s.seed;
                D.k1 = (u32)(s.seed >> 32);
                memcpy(D.table, table, sizeof table);
                D.rows = j.rows;
                D.lh = j.lh;
                D.ly = j.ly;
                D.lz = j.lz;
                D.pitch = j.pitch;  // rows padded to 16 bytes: chunk width 16
                D.cpr = (j.lh + 15) / 16;
                kc.v = 16;
                kc.mixed = (j.lh % 16) != 0;
                kc.rule = select_rule(s.variant, s.algorithm, s.ndim, table);
                class_units[kc] += (long long)j.rows * D.cpr;
                int8_descs[kc].push_back(D);
            }
        }
        // int8: the class's band height is the longest power of two up to the band cap that
        // still leaves kBandBlocks (or items_per_slot, if fewer) blocks of one slot per thread per
        // resident block; blocks of a lattice hold per_block slots, items_per_slot blocks per
        // resident block
        int8_launches_.clear();
        for (auto& kv : int8_descs) {
            const KernelClass& kc = kv.first;
            const long long units = class_units[kc];
            int band = 1;
            while (band * 2 <= band_cap_) band *= 2;
            const long long want = std::min(items_per_slot_, kBandBlocks) * 256 * slots(kc);
            while (band > 1 && units / band < want) band >>= 1;
            long long per = item_size(units / band, slots(kc), items_per_slot_, kInt8ItemMin,
                                      kInt8ItemMax);
            per = (per + 255) / 256 * 256;
            const bool one = units < (kc.ndim == 3 ? kOneUnits3 : kOneUnits2) * sms_;
            if (one) {
                band = 1;
                per = kOneThreads;
            }
            std::vector<Int8Launch> launches;
            for (size_t i = 0; i < kv.second.size(); ++i) {
                if (i % kInt8PerLaunch == 0) {
                    launches.emplace_back();
                    memset(&launches.back(), 0, sizeof(Int8Launch));
                }
                Int8Launch& P = launches.back();
                Int8Desc D = kv.second[i];
                D.band = std::min(std::min(band, int8_band_limit(kc.ndim, D.cpr)), D.ly);
                D.bpp = (D.ly + D.band - 1) / D.band;
                const long long nslots = (long long)D.lz * D.bpp * D.cpr;
                D.nslots = (int)nslots;
                D.cpr_magic = fast_div_magic((u32)D.cpr, (unsigned long long)nslots);
                D.bpp_magic = fast_div_magic((u32)D.bpp, (unsigned long long)D.lz * D.bpp);
                D.per_block = (int)per;
                const int prev = P.n ? P.lat[P.n - 1].block_begin +
                                           (P.lat[P.n - 1].nslots + P.lat[P.n - 1].per_block - 1) /
                                               P.lat[P.n - 1].per_block
                                     : 0;
                D.block_begin = prev;
                P.lat[P.n++] = D;
            }
            int8_launches_.push_back(Int8Class{kc, one, std::move(launches)});
        }
        // msc: one word per thread for small totals, else work items of whole 256-word runs over
        // the class's lattices
        msc_one_.clear();
        std::map<KernelClass, std::vector<BatchItem>> by_class;
        if (!msc_of.empty() && class_units[msc_of[0].first] < kOneWords * sms_) {
            for (const auto& m : msc_of) {
                if (msc_one_.empty() || msc_one_.back().n == kInt8PerLaunch) {
                    msc_one_.emplace_back();
                    memset(&msc_one_.back(), 0, sizeof(MscLaunch));
                }
                MscLaunch& P = msc_one_.back();
                const BatchLattice& L = lats[m.second];
                MscDesc D;
                memset(&D, 0, sizeof D);
                D.c[0] = static_cast<u64*>(L.c[0]);
                D.c[1] = static_cast<u64*>(L.c[1]);
                D.series = L.series;
                D.join_epoch = L.join_epoch;
                D.nw_magic = L.nw_magic;
                D.every = L.every;
                D.rows = L.rows;
                D.nw = L.nw;
                D.nw_shift = L.nw_shift;
                D.t0 = L.t0;
                D.k0 = L.k0;
                D.k1 = L.k1;
                D.thr4 = L.table[3];
                D.thr8 = L.table[4];
                D.block_begin = P.n ? (int)msc_grid(P) : 0;
                P.lat[P.n++] = D;
            }
            msc_of.clear();
        }
        for (const auto& m : msc_of) {
            const KernelClass& kc = m.first;
            const BatchLattice& L = lats[m.second];
            const long long words = (long long)L.rows * L.nw;
            long long per = item_size(class_units[kc], slots(kc), items_per_slot_, kMscItemMin,
                                      kMscItemMax);
            per = (per + 255) / 256 * 256;
            for (long long b = 0; b < words; b += per)
                by_class[kc].push_back(BatchItem{m.second, 0, b, std::min(words, b + per)});
        }
        std::vector<BatchItem> items;
        classes_.clear();
        for (auto& kv : by_class) {
            classes_.emplace_back(kv.first, std::make_pair((int)items.size(), (int)kv.second.size()));
            items.insert(items.end(), kv.second.begin(), kv.second.end());
        }
        int rc = upload(lats.data(), lats.size() * sizeof(BatchLattice), (void**)&d_lats_, &lats_cap_);
        if (rc == ISING_OK)
            rc = upload(items.data(), items.size() * sizeof(BatchItem), (void**)&d_items_, &items_cap_);
        if (rc != ISING_OK) return rc;
        plan_streams();
        dirty_ = false;
        return ISING_OK;
    }

    // Every class advances on a stream of its own when there are several: their lattices are
    // independent, and a class alone often leaves most of the GPU waiting.  The engine's stream
    // waits for all of them at every sweep (join), they wait for it only after it did something
    // (fork): admissions, results, work lists, graph chunks.
    // Without streams or events to be had, all classes stay on the engine's stream.
    void plan_streams()
    {
        const size_t n = int8_launches_.size() + (msc_one_.empty() ? 0 : 1) + classes_.size();
        forked_ = false;
        n_aux_ = n > 1 && class_streams(n) ? n : 0;
    }

    // Makes n class streams and the fork event; whether all of them exist.
    bool class_streams(size_t n)
    {
        if (!fork_event_ &&
            cudaEventCreateWithFlags(&fork_event_, cudaEventDisableTiming) != cudaSuccess) {
            fork_event_ = nullptr;
            cudaGetLastError();
            return false;
        }
        while (aux_.size() < n) {
            Aux a;
            cudaError_t e = cudaStreamCreateWithFlags(&a.stream, cudaStreamNonBlocking);
            if (e == cudaSuccess) e = cudaEventCreateWithFlags(&a.event, cudaEventDisableTiming);
            if (e != cudaSuccess) {
                if (a.stream) cudaStreamDestroy(a.stream);
                cudaGetLastError();
                return false;
            }
            aux_.push_back(a);
        }
        return true;
    }

    // The class streams wait for the engine's.
    cudaError_t fork()
    {
        if (!n_aux_ || forked_) return cudaSuccess;
        cudaError_t e = cudaEventRecord(fork_event_, stream_);
        for (size_t i = 0; i < n_aux_ && e == cudaSuccess; ++i)
            e = cudaStreamWaitEvent(aux_[i].stream, fork_event_, 0);
        forked_ = e == cudaSuccess;
        return e;
    }

    // The engine's stream waits for the class streams.
    int join()
    {
        if (!joinable_) return ISING_OK;
        for (size_t i = 0; i < n_aux_; ++i) {
            cudaError_t e = cudaEventRecord(aux_[i].event, aux_[i].stream);
            if (e == cudaSuccess) e = cudaStreamWaitEvent(stream_, aux_[i].event, 0);
            if (e != cudaSuccess) return cuda_fail(e, "batch class join");
        }
        joinable_ = false;
        return ISING_OK;
    }

    // Blocks of an int8 launch: the last lattice's block_begin plus its blocks.
    static unsigned int8_grid(const Int8Launch& P)
    {
        const Int8Desc& L = P.lat[P.n - 1];
        return (unsigned)(L.block_begin + (L.nslots + L.per_block - 1) / L.per_block);
    }

    static unsigned msc_grid(const MscLaunch& P)
    {
        const MscDesc& L = P.lat[P.n - 1];
        const long long words = (long long)L.rows * L.nw;
        return (unsigned)(L.block_begin + (words + kOneThreads - 1) / kOneThreads);
    }

    // Resident blocks of a class's kernel on the whole device.
    long long slots(const KernelClass& kc)
    {
        const void* fn = kc.variant == ISING_VARIANT_MSC
                             ? (const void*)batch_msc_kernel
                             : (const void*)batch_int8_kernel<16, 2, kMetroFast, false, 16>;
        // (one occupancy for all int8 classes: they share the launch bounds)
        return (long long)sms_ * blocks_per_sm(fn, kc.variant == ISING_VARIANT_MSC
                                                       ? kBatchWarps * 32 : 256);
    }

    int upload(const void* src, size_t bytes, void** dst, size_t* cap)
    {
        if (bytes == 0) return ISING_OK;
        if (bytes > *cap) {
            if (*dst) cudaFreeAsync(*dst, stream_);
            size_t nc = std::max(bytes, *cap * 2);
            cudaError_t e = dev_alloc(dst, nc);
            if (e != cudaSuccess) return cuda_fail(e, "cudaMallocAsync (work list)");
            *cap = nc;
        }
        // pageable source: staged by the driver before the call returns
        cudaError_t e = cudaMemcpyAsync(*dst, src, bytes, cudaMemcpyHostToDevice, stream_);
        if (e != cudaSuccess) return cuda_fail(e, "work list upload");
        return ISING_OK;
    }

    int blocks_per_sm(const void* fn, int threads)
    {
        int& per_sm = occupancy_[fn];
        if (per_sm < 1 &&
            (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, 0) != cudaSuccess ||
             per_sm < 1)) {
            cudaGetLastError();
            per_sm = 2;
        }
        return per_sm;
    }

    int grid_for(const void* fn, int n_items, int threads = 256)
    {
        const int g = sms_ * blocks_per_sm(fn, threads);
        return n_items < g ? n_items : g;
    }

    template <int NDIM, int RULE, bool MIXED, int N>
    cudaError_t launch_int8_kernel(bool one, const Int8LaunchN<N>& P, unsigned grid, cudaStream_t st)
    {
        if (one)
            return launch_pdl(batch_int8_one_kernel<NDIM, RULE, MIXED, N>, dim3(grid),
                              dim3(kOneThreads), st, P);
        return launch_pdl(batch_int8_kernel<16, NDIM, RULE, MIXED, N>, dim3(grid), dim3(256), st, P);
    }

    template <int NDIM, bool MIXED, int N>
    cudaError_t launch_int8_cap(const Int8Class& c, const Int8Launch& full, cudaStream_t st)
    {
        Int8LaunchN<N> P;
        P.epoch = full.epoch;
        P.epoch_base = full.epoch_base;
        P.n = full.n;
        P.pad = 0;
        memcpy(P.lat, full.lat, (size_t)full.n * sizeof(Int8Desc));
        const unsigned grid = int8_grid(full);
        switch (c.kc.rule) {
        case kMetroFast: return launch_int8_kernel<NDIM, kMetroFast, MIXED, N>(c.one, P, grid, st);
        case kHeat: return launch_int8_kernel<NDIM, kHeat, MIXED, N>(c.one, P, grid, st);
        case kMetroGeneric:
            return launch_int8_kernel<NDIM, kMetroGeneric, MIXED, N>(c.one, P, grid, st);
        default: return cudaErrorInvalidValue;
        }
    }

    template <int NDIM, bool MIXED>
    cudaError_t launch_int8_n(const Int8Class& c, const Int8Launch& P, cudaStream_t st)
    {
        if (P.n <= 16) return launch_int8_cap<NDIM, MIXED, 16>(c, P, st);
        if (P.n <= 64) return launch_int8_cap<NDIM, MIXED, 64>(c, P, st);
        return launch_int8_cap<NDIM, MIXED, kInt8PerLaunch>(c, P, st);
    }

    // int8 rows are padded to 16 bytes, so the chunk width is always 16; lattices whose rows are
    // a multiple of 16 get the kernel without the partial-chunk code.
    cudaError_t launch_int8(const Int8Class& c, const Int8Launch& P, cudaStream_t st)
    {
        if (c.kc.ndim == 3)
            return c.kc.mixed ? launch_int8_n<3, true>(c, P, st) : launch_int8_n<3, false>(c, P, st);
        return c.kc.mixed ? launch_int8_n<2, true>(c, P, st) : launch_int8_n<2, false>(c, P, st);
    }

    template <int N>
    cudaError_t launch_msc_one_cap(const MscLaunch& full, cudaStream_t st)
    {
        MscLaunchN<N> P;
        P.epoch = full.epoch;
        P.epoch_base = full.epoch_base;
        P.n = full.n;
        P.pad = 0;
        memcpy(P.lat, full.lat, (size_t)full.n * sizeof(MscDesc));
        return launch_pdl(batch_msc_one_kernel<N>, dim3(msc_grid(full)), dim3(kOneThreads), st, P);
    }

    cudaError_t launch_msc_one(const MscLaunch& P, cudaStream_t st)
    {
        if (P.n <= 16) return launch_msc_one_cap<16>(P, st);
        if (P.n <= 64) return launch_msc_one_cap<64>(P, st);
        return launch_msc_one_cap<kInt8PerLaunch>(P, st);
    }

    cudaError_t launch_msc(int off, int n, long long epoch, const long long* epoch_base,
                           cudaStream_t st)
    {
        auto fn = batch_msc_kernel;
        const dim3 grid(grid_for((const void*)fn, n, kBatchWarps * 32)), block(kBatchWarps * 32);
        fn<<<grid, block, 0, st>>>(d_lats_, d_items_ + off, n, epoch, epoch_base);
        return cudaGetLastError();
    }

    // Every class's launches of one epoch (absolute, or relative to *epoch_base).
    cudaError_t launch_epoch(long long epoch, const long long* epoch_base)
    {
        cudaError_t e = fork();
        size_t i = 0;
        auto next_stream = [&] { return n_aux_ ? aux_[i++].stream : stream_; };
        for (auto& cl : int8_launches_) {
            const cudaStream_t st = next_stream();
            for (Int8Launch& P : cl.launches) {
                P.epoch = epoch;
                P.epoch_base = epoch_base;
                if (e == cudaSuccess) e = launch_int8(cl, P, st);
            }
        }
        if (!msc_one_.empty()) {
            const cudaStream_t st = next_stream();
            for (MscLaunch& P : msc_one_) {
                P.epoch = epoch;
                P.epoch_base = epoch_base;
                if (e == cudaSuccess) e = launch_msc_one(P, st);
            }
        }
        for (const auto& cl : classes_) {
            const cudaStream_t st = next_stream();
            if (e == cudaSuccess)
                e = launch_msc(cl.second.first, cl.second.second, epoch, epoch_base, st);
        }
        joinable_ = n_aux_ > 0;
        return e;
    }

    // ---- graph chunks: kChunkSweeps sweeps of a stable batch replayed from one graph ----
    // While no job can join (admission happens at even epochs, and pending jobs that did not
    // fit can only fit after a job retires) and every active job has kChunkSweeps sweeps left,
    // the batch's launches repeat with only the epoch changing: they are captured once per
    // membership, reading the epoch from a device counter set before each replay.
    static constexpr long long kChunkSweeps = 32;  // default of the ISING_KNOB_GRAPH_CHUNK knob
    static constexpr long long kChunkReplays = 4;  // chunks of sweeps left needed for a capture

    long long min_sweeps_left() const
    {
        long long m = LLONG_MAX;
        for (int64_t id : active_) {
            const Job& j = *jobs_.at(id);
            m = std::min(m, (long long)j.spec.n_sweeps - (epoch_ - j.join_epoch) / 2);
        }
        return m;
    }

    bool chunk_ready() const
    {
        if ((epoch_ & 1) || active_.empty() || chunk_sweeps_ == 0) return false;
        return min_sweeps_left() >= chunk_sweeps_ * (chunk_exec_ ? 1 : kChunkReplays);
    }

    int run_chunk()
    {
        cudaError_t e;
        if (!chunk_exec_) {
            e = cudaStreamBeginCapture(stream_, cudaStreamCaptureModeThreadLocal);
            if (e != cudaSuccess) return cuda_fail(e, "cudaStreamBeginCapture (batch)");
            cudaError_t le = cudaSuccess;
            forked_ = false;  // the class streams join the capture, each a branch of the graph
            for (long long k = 0; k < 2 * chunk_sweeps_ && le == cudaSuccess; ++k)
                le = launch_epoch(k, d_epoch_);
            const int jrc = le == cudaSuccess ? join() : ISING_OK;
            joinable_ = false;
            cudaGraph_t graph = nullptr;
            e = cudaStreamEndCapture(stream_, &graph);
            if (jrc != ISING_OK) {
                if (graph) cudaGraphDestroy(graph);
                return jrc;
            }
            if (le != cudaSuccess || e != cudaSuccess) {
                if (graph) cudaGraphDestroy(graph);
                return cuda_fail(le != cudaSuccess ? le : e, "batch graph capture");
            }
            e = cudaGraphInstantiate(&chunk_exec_, graph, 0);
            cudaGraphDestroy(graph);
            if (e != cudaSuccess) {
                chunk_exec_ = nullptr;
                return cuda_fail(e, "cudaGraphInstantiate (batch)");
            }
        }
        batch_epoch_set<<<1, 1, 0, stream_>>>(d_epoch_, epoch_);
        e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaGraphLaunch(chunk_exec_, stream_);
        if (e != cudaSuccess) return cuda_fail(e, "batch graph launch");
        forked_ = false;  // the class streams have yet to wait for the chunk
        epoch_ += 2 * chunk_sweeps_;
        return ISING_OK;
    }

    // Drops the chunk graph (membership changed); it is destroyed once its launches are done.
    void drop_chunk()
    {
        if (!chunk_exec_) return;
        cudaEvent_t ev = nullptr;
        if (cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) == cudaSuccess &&
            cudaEventRecord(ev, stream_) == cudaSuccess) {
            old_execs_.emplace_back(chunk_exec_, ev);
        } else {
            cudaStreamSynchronize(stream_);
            cudaGraphExecDestroy(chunk_exec_);
            if (ev) cudaEventDestroy(ev);
        }
        chunk_exec_ = nullptr;
    }

    void reap_chunks()
    {
        for (auto it = old_execs_.begin(); it != old_execs_.end();) {
            if (cudaEventQuery(it->second) == cudaSuccess) {
                cudaGraphExecDestroy(it->first);
                cudaEventDestroy(it->second);
                it = old_execs_.erase(it);
            } else {
                ++it;
            }
        }
        cudaGetLastError();  // cudaErrorNotReady from the queries
    }

    int retire()
    {
        for (auto it = active_.begin(); it != active_.end();) {
            Job& j = *jobs_[*it];
            if ((epoch_ - j.join_epoch) / 2 >= j.spec.n_sweeps) {
                int rc = finish_job(j);
                if (rc != ISING_OK) return rc;
                it = active_.erase(it);
                dirty_ = true;
            } else {
                ++it;
            }
        }
        return ISING_OK;
    }

    // Enqueues the result copies after the job's last half-sweep and frees its lattice.
    int finish_job(Job& j)
    {
        cudaError_t e = cudaSuccess;
        if (j.series_pairs) {
            const size_t sb = j.series_pairs * 2 * sizeof(long long);
            if (!j.h_series) e = pinned_get((void**)&j.h_series, sb);
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(j.h_series, j.d_series, sb, cudaMemcpyDeviceToHost, stream_);
        }
        if (e == cudaSuccess && j.spec.keep_lattice) {
            const size_t full = (size_t)j.rows * 2 * j.lh;
            int8_t* stage = nullptr;
            if (!j.h_lattice) e = pinned_get((void**)&j.h_lattice, full);
            if (e == cudaSuccess) e = dev_alloc((void**)&stage, full);
            if (e == cudaSuccess) {
                if (j.spec.variant == ISING_VARIANT_MSC)
                    e = launch_msc_unpack((const u64*)j.c[0], (const u64*)j.c[1], stage, j.rows, 0,
                                          j.nw, sms_ * 8, stream_);
                else
                    e = launch_int8_merge((const int8_t*)j.c[0], (const int8_t*)j.c[1], stage,
                                          j.rows, 0, j.lh, j.pitch, j.ly, sms_ * 8, stream_);
            }
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(j.h_lattice, stage, full, cudaMemcpyDeviceToHost, stream_);
            if (stage) cudaFreeAsync(stage, stream_);
        }
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&j.done_event, cudaEventDisableTiming);
        if (e == cudaSuccess) e = cudaEventRecord(j.done_event, stream_);
        if (e != cudaSuccess) return cuda_fail(e, "job results");
        for (int c = 0; c < 2; ++c) {
            cudaFreeAsync(j.c[c], stream_);
            j.c[c] = nullptr;
        }
        if (j.d_series) {
            cudaFreeAsync(j.d_series, stream_);
            j.d_series = nullptr;
        }
        used_ -= (int64_t)j.device_bytes;
        j.state = ISING_JOB_FINISHING;
        finishing_.push_back(j.id);
        return ISING_OK;
    }

    // Records the end of the sweep (or graph chunk) just issued; the host stays at most about
    // kMaxAhead sweeps ahead of the device (see throttle_event), so a newly admitted job starts
    // soon after it joins.
    static constexpr long long kMaxAhead = 8;

    int throttle()
    {
        cudaEvent_t ev = nullptr;
        if (!free_events_.empty()) {
            ev = free_events_.back();
            free_events_.pop_back();
        } else {
            cudaError_t e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
            if (e != cudaSuccess) return cuda_fail(e, "cudaEventCreate");
            epoch_events_.push_back(ev);
        }
        cudaEventRecord(ev, stream_);
        inflight_.emplace_back(ev, epoch_);
        return ISING_OK;
    }

public:
    // The event to wait for before issuing more work (nullptr: not too far ahead).  Callers
    // wait without holding any lock the submitters need, then call throttle_done().
    cudaEvent_t throttle_event() const
    {
        return !inflight_.empty() && epoch_ - inflight_.front().second > 2 * kMaxAhead
                   ? inflight_.front().first
                   : nullptr;
    }

    void throttle_done()
    {
        free_events_.push_back(inflight_.front().first);
        inflight_.pop_front();
    }

    int wait_throttle()
    {
        while (cudaEvent_t ev = throttle_event()) {
            const cudaError_t e = cudaEventSynchronize(ev);
            if (e != cudaSuccess) return cuda_fail(e, "throttle");
            throttle_done();
        }
        return ISING_OK;
    }

private:

    void free_job(Job& j)
    {
        if (j.done_event) cudaEventDestroy(j.done_event);
        j.done_event = nullptr;
        for (int c = 0; c < 2; ++c)
            if (j.c[c]) cudaFreeAsync(j.c[c], stream_);
        if (j.d_series) cudaFreeAsync(j.d_series, stream_);
        if (j.h_series) pinned_put(j.h_series, j.series_pairs * 2 * sizeof(long long));
        if (j.h_lattice) pinned_put(j.h_lattice, (size_t)j.rows * 2 * j.lh);
        j.c[0] = j.c[1] = nullptr;
        j.d_series = nullptr;
        j.h_series = nullptr;
        j.h_lattice = nullptr;
    }

    cudaError_t dev_alloc(void** p, size_t bytes)
    {
        return cudaMallocFromPoolAsync(p, bytes, pool_, stream_);
    }

    // Pinned host buffers for results are reused across jobs (size classes of powers of two
    // from 4 KiB): page-locking memory for every finished job would stall the serving loop.
    static size_t pinned_class(size_t bytes)
    {
        size_t c = 4096;
        while (c < bytes) c <<= 1;
        return c;
    }

    cudaError_t pinned_get(void** p, size_t bytes)
    {
        const size_t c = pinned_class(bytes);
        auto it = pinned_free_.find(c);
        if (it != pinned_free_.end()) {
            *p = it->second;
            pinned_free_.erase(it);
            return cudaSuccess;
        }
        return cudaMallocHost(p, c);
    }

    void pinned_put(void* p, size_t bytes) { pinned_free_.emplace(pinned_class(bytes), p); }

    int device_;
    int64_t budget_;
    int64_t used_ = 0;
    int sms_ = 148;
    cudaStream_t stream_ = nullptr;
    cudaMemPool_t pool_ = nullptr;
    std::multimap<size_t, void*> pinned_free_;  // reusable pinned result buffers by size class
    long long epoch_ = 0;
    int64_t last_id_ = 0;
    int band_cap_ = kBandCap;
    long long items_per_slot_ = kItemsPerSlot;
    long long* d_epoch_ = nullptr;       // device epoch counter of replayed graph chunks
    cudaGraphExec_t chunk_exec_ = nullptr;
    std::vector<std::pair<cudaGraphExec_t, cudaEvent_t>> old_execs_;
    long long chunk_sweeps_ = kChunkSweeps;  // 0: no graph chunks
    std::map<int64_t, std::unique_ptr<Job>> jobs_;
    std::deque<int64_t> pending_;
    std::vector<int64_t> active_;
    std::vector<int64_t> finishing_;
    bool dirty_ = false;
    BatchLattice* d_lats_ = nullptr;
    BatchItem* d_items_ = nullptr;
    size_t lats_cap_ = 0, items_cap_ = 0;
    std::vector<std::pair<KernelClass, std::pair<int, int>>> classes_;  // msc work items
    std::vector<Int8Class> int8_launches_;
    std::vector<MscLaunch> msc_one_;  // the msc class, one word per thread
    struct Aux {
        cudaStream_t stream = nullptr;
        cudaEvent_t event = nullptr;
    };
    std::vector<Aux> aux_;           // class streams
    size_t n_aux_ = 0;               // class streams in use (0: all on stream_)
    cudaEvent_t fork_event_ = nullptr;
    bool forked_ = false;            // the class streams have waited for stream_
    bool joinable_ = false;          // stream_ has yet to wait for the class streams
    std::vector<cudaEvent_t> epoch_events_, free_events_;
    std::map<const void*, int> occupancy_;
    std::deque<std::pair<cudaEvent_t, long long>> inflight_;  // (event, epoch recorded at)
};

}  // namespace ising

using namespace ising;

// ------------------------------------------------------------------------------- batch API ---
struct ising_batch {
    std::unique_ptr<Engine> eng;
};

extern "C" {

int ising_batch_create(int device, int64_t memory_budget, ising_batch** out)
{
    if (!out) return fail(ISING_ERR_INVALID, "null output pointer");
    *out = nullptr;
    if (memory_budget <= 0) return fail(ISING_ERR_INVALID, "memory budget must be positive");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) {
        cudaGetLastError();
        return fail(ISING_ERR_INVALID, "device %d not available", device);
    }
    auto b = new ising_batch();
    b->eng.reset(new Engine(device, memory_budget));
    int rc = b->eng->init();
    if (rc != ISING_OK) {
        delete b;
        return rc;
    }
    *out = b;
    return ISING_OK;
}

int ising_batch_add(ising_batch* b, const ising_job* job, int64_t* id)
{
    if (!b || !job || !id) return fail(ISING_ERR_INVALID, "null argument");
    return b->eng->submit(*job, id);
}

int ising_batch_run(ising_batch* b, int64_t max_epochs, int64_t* epochs_run)
{
    if (!b) return fail(ISING_ERR_INVALID, "null batch");
    int64_t n = 0;  // half-sweep epochs issued (a replayed chunk issues many)
    while (b->eng->has_work() && (max_epochs <= 0 || n < max_epochs)) {
        const size_t before = b->eng->active_count() + b->eng->pending_count();
        const long long e0 = b->eng->epoch();
        int rc = b->eng->step(max_epochs > 0 ? max_epochs - n : 0);
        if (rc == ISING_OK) rc = b->eng->wait_throttle();
        if (rc != ISING_OK) return rc;
        n += b->eng->epoch() - e0;
        if (b->eng->active_count() == 0 && b->eng->pending_count() > 0 &&
            b->eng->pending_count() == before)
            return fail(ISING_ERR_NOMEM, "pending jobs do not fit the memory budget");
    }
    if (epochs_run) *epochs_run = n;
    return b->eng->wait_finishing();
}

int ising_batch_status(ising_batch* b, int64_t id, int* state, int64_t* sweeps_done)
{
    if (!b || !state) return fail(ISING_ERR_INVALID, "null argument");
    b->eng->poll();
    Job* j = b->eng->find(id);
    if (!j) return fail(ISING_ERR_INVALID, "unknown job %lld", (long long)id);
    *state = j->state;
    if (sweeps_done) {
        long long s = 0;
        if (j->state == ISING_JOB_DONE || j->state == ISING_JOB_FINISHING) s = j->spec.n_sweeps;
        else if (j->state == ISING_JOB_ACTIVE) s = (b->eng->epoch() - j->join_epoch) / 2;
        *sweeps_done = s;
    }
    return ISING_OK;
}

int ising_batch_result(ising_batch* b, int64_t id, int64_t* series_out, int8_t* lattice_out)
{
    if (!b) return fail(ISING_ERR_INVALID, "null batch");
    b->eng->poll();
    return b->eng->result(id, series_out, lattice_out, nullptr);
}

int ising_batch_release(ising_batch* b, int64_t id)
{
    if (!b) return fail(ISING_ERR_INVALID, "null batch");
    return b->eng->release(id);
}

int ising_batch_set_knob(ising_batch* b, int knob, int value)
{
    if (!b) return fail(ISING_ERR_INVALID, "null batch");
    return b->eng->set_knob(knob, value);
}

int ising_batch_get_knob(ising_batch* b, int knob, int* value)
{
    if (!b || !value) return fail(ISING_ERR_INVALID, "null argument");
    return b->eng->get_knob(knob, value);
}

int ising_batch_destroy(ising_batch* b)
{
    delete b;
    return ISING_OK;
}

}  // extern "C"

// ----------------------------------------------------------------------------- serving API ---
struct ising_server {
    std::unique_ptr<Engine> eng;
    std::mutex mu;
    std::condition_variable cv_work, cv_done;
    std::thread worker;
    bool stop = false;
    int error = ISING_OK;
    std::string error_msg;
};

static void server_loop(ising_server* s)
{
    std::unique_lock<std::mutex> lk(s->mu);
    while (true) {
        s->cv_work.wait(lk, [s] { return s->stop || s->eng->busy(); });
        if (s->stop && !s->eng->busy()) break;
        if (s->eng->has_work()) {
            // one sweep (two half-sweeps) per turn, then let submitters in
            for (int k = 0; k < 2 && s->error == ISING_OK; ++k) {
                const int rc = s->eng->step();
                if (rc != ISING_OK) {
                    s->error = rc;
                    s->error_msg = g_last_error;
                }
            }
            // bound the run-ahead without holding the lock submitters and waiters need
            while (cudaEvent_t ev = s->eng->throttle_event()) {
                lk.unlock();
                const cudaError_t e = cudaEventSynchronize(ev);
                lk.lock();
                if (e != cudaSuccess) {
                    s->error = cuda_fail(e, "throttle");
                    s->error_msg = g_last_error;
                    break;
                }
                s->eng->throttle_done();
            }
        } else {
            lk.unlock();
            cudaStreamSynchronize(s->eng->stream());
            lk.lock();
        }
        if (s->eng->poll() > 0) s->cv_done.notify_all();
        if (s->error != ISING_OK) {
            s->cv_done.notify_all();
            break;
        }
        // brief release so submitters and waiters can take the lock
        lk.unlock();
        std::this_thread::yield();
        lk.lock();
    }
}

extern "C" {

int ising_server_create(int device, int64_t memory_budget, ising_server** out)
{
    if (!out) return fail(ISING_ERR_INVALID, "null output pointer");
    *out = nullptr;
    if (memory_budget <= 0) return fail(ISING_ERR_INVALID, "memory budget must be positive");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) {
        cudaGetLastError();
        return fail(ISING_ERR_INVALID, "device %d not available", device);
    }
    auto s = new ising_server();
    s->eng.reset(new Engine(device, memory_budget));
    int rc = s->eng->init();
    if (rc != ISING_OK) {
        delete s;
        return rc;
    }
    s->worker = std::thread([s, device] {
        cudaSetDevice(device);
        server_loop(s);
    });
    *out = s;
    return ISING_OK;
}

int ising_server_submit(ising_server* s, const ising_job* job, int64_t* id)
{
    if (!s || !job || !id) return fail(ISING_ERR_INVALID, "null argument");
    std::lock_guard<std::mutex> lk(s->mu);
    if (s->error != ISING_OK) return fail(s->error, "server stopped: %s", s->error_msg.c_str());
    int rc = s->eng->submit(*job, id);
    if (rc == ISING_OK) s->cv_work.notify_one();
    return rc;
}

int ising_server_wait(ising_server* s, int64_t id, double timeout_s, int* state)
{
    if (!s || !state) return fail(ISING_ERR_INVALID, "null argument");
    std::unique_lock<std::mutex> lk(s->mu);
    Job* j = s->eng->find(id);
    if (!j) return fail(ISING_ERR_INVALID, "unknown job %lld", (long long)id);
    auto done = [&] { return s->error != ISING_OK || s->eng->find(id)->state == ISING_JOB_DONE; };
    if (timeout_s < 0) s->cv_done.wait(lk, done);
    else s->cv_done.wait_for(lk, std::chrono::duration<double>(timeout_s), done);
    *state = s->eng->find(id)->state;
    if (s->error != ISING_OK) return fail(s->error, "server stopped: %s", s->error_msg.c_str());
    return ISING_OK;
}

int ising_server_result(ising_server* s, int64_t id, int64_t* series_out, int8_t* lattice_out,
                        double* latency_s)
{
    if (!s) return fail(ISING_ERR_INVALID, "null server");
    std::lock_guard<std::mutex> lk(s->mu);
    return s->eng->result(id, series_out, lattice_out, latency_s);
}

int ising_server_release(ising_server* s, int64_t id)
{
    if (!s) return fail(ISING_ERR_INVALID, "null server");
    std::lock_guard<std::mutex> lk(s->mu);
    return s->eng->release(id);
}

int ising_server_status(ising_server* s, int64_t* pending, int64_t* active, int64_t* used_bytes,
                        int64_t* epoch)
{
    if (!s) return fail(ISING_ERR_INVALID, "null server");
    std::lock_guard<std::mutex> lk(s->mu);
    if (pending) *pending = (int64_t)s->eng->pending_count();
    if (active) *active = (int64_t)s->eng->active_count();
    if (used_bytes) *used_bytes = s->eng->used_bytes();
    if (epoch) *epoch = s->eng->epoch();
    return ISING_OK;
}

int ising_server_set_knob(ising_server* s, int knob, int value)
{
    if (!s) return fail(ISING_ERR_INVALID, "null server");
    std::lock_guard<std::mutex> lk(s->mu);
    return s->eng->set_knob(knob, value);
}

int ising_server_destroy(ising_server* s)
{
    if (!s) return ISING_OK;
    {
        std::lock_guard<std::mutex> lk(s->mu);
        s->stop = true;
    }
    s->cv_work.notify_all();
    if (s->worker.joinable()) s->worker.join();
    delete s;
    return ISING_OK;
}

}  // extern "C"
