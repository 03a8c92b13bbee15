// int8 compressed-checkerboard half-sweep (2D/3D, Metropolis/heat bath) with the fused
// integer (M, E) reduction.
//
// Same results as pyising's NumpyCheckerboard._half_sweep (src/pyising/backends/
// numpy_backend.py:26-44) and the CUDA C int8_half kernel (src/pyising/backends/cuda/
// ising.cu:25-87): site n = row*Lh + j of colour c draws word n%4 of
// Philox((n/4, t, c, 0), seed) (src/pyising/philox.py:54-64).
//
// Work split: a thread owns V consecutive colour sites of one row (V = 16: one 128-bit load
// per array, four Philox blocks).  Spins stay packed in 32-bit words and the neighbour
// counting is byte-parallel (SWAR): with +1 = 0x01 and -1 = 0xFF, bits 1 to 7 of a byte are the
// "down" flag.  A loaded word of the opposite colour is masked once with 0x04040404, so the sum
// of a site's neighbour words holds four times its down neighbours D: the byte offset of an
// entry in a table of 32-bit thresholds.
//
// Decision: one shared-memory lookup, one comparison and one predicated operation per site.
//   Heat bath: +1 iff u < table[U], U = up neighbours = 2d - D.
//   Metropolis flips iff X <= 0 or u < table[(X + 2d)/2], X = s*h = 2d - 2A, A = anti-aligned
//   neighbours = D for an up spin, 2d - D for a down spin.  The lookup index is 4 D + 32 (spin
//   down), the entry the largest uniform that flips: table[2d - A] - 1 for A < d, 2^32 - 1 (every
//   uniform) for A >= d.  A table with a zero among its A < d entries (no uniform flips) has no
//   such entry and takes the general rule.
#pragma once

#include "common.cuh"

namespace ising {

template <int W>
struct Words {
    u32 v[W];
};

template <int W>
__device__ __forceinline__ Words<W> load_words(const int8_t* p)
{
    Words<W> r;
    if constexpr (W == 4) {
        const uint4 q = *reinterpret_cast<const uint4*>(p);
        r.v[0] = q.x; r.v[1] = q.y; r.v[2] = q.z; r.v[3] = q.w;
    } else if constexpr (W == 2) {
        const uint2 q = *reinterpret_cast<const uint2*>(p);
        r.v[0] = q.x; r.v[1] = q.y;
    } else {
        r.v[0] = *reinterpret_cast<const u32*>(p);
    }
    return r;
}

template <int W>
__device__ __forceinline__ Words<W> load_words_ro(const int8_t* p)
{
    Words<W> r;
    if constexpr (W == 4) {
        const uint4 q = __ldg(reinterpret_cast<const uint4*>(p));
        r.v[0] = q.x; r.v[1] = q.y; r.v[2] = q.z; r.v[3] = q.w;
    } else if constexpr (W == 2) {
        const uint2 q = __ldg(reinterpret_cast<const uint2*>(p));
        r.v[0] = q.x; r.v[1] = q.y;
    } else {
        r.v[0] = __ldg(reinterpret_cast<const unsigned int*>(p));
    }
    return r;
}

// The opposite colour read from L2, bypassing L1: needed inside one launch that runs several
// half-sweeps, where other SMs rewrite rows this SM may have cached.
template <int W>
__device__ __forceinline__ Words<W> load_words_cg(const int8_t* p)
{
    Words<W> r;
    if constexpr (W == 4) {
        const uint4 q = __ldcg(reinterpret_cast<const uint4*>(p));
        r.v[0] = q.x; r.v[1] = q.y; r.v[2] = q.z; r.v[3] = q.w;
    } else if constexpr (W == 2) {
        const uint2 q = __ldcg(reinterpret_cast<const uint2*>(p));
        r.v[0] = q.x; r.v[1] = q.y;
    } else {
        r.v[0] = __ldcg(reinterpret_cast<const unsigned int*>(p));
    }
    return r;
}

template <int W, bool CG>
__device__ __forceinline__ Words<W> load_other(const int8_t* p)
{
    if constexpr (CG) return load_words_cg<W>(p);
    else return load_words_ro<W>(p);
}

template <int W>
__device__ __forceinline__ void store_words(int8_t* p, const Words<W>& r)
{
    if constexpr (W == 4) {
        *reinterpret_cast<uint4*>(p) = make_uint4(r.v[0], r.v[1], r.v[2], r.v[3]);
    } else if constexpr (W == 2) {
        *reinterpret_cast<uint2*>(p) = make_uint2(r.v[0], r.v[1]);
    } else {
        *reinterpret_cast<u32*>(p) = r.v[0];
    }
}

// Words of the opposite colour as the neighbour sums take them: 4 for a down spin, 0 for up.
template <int W>
__device__ __forceinline__ Words<W> downs(Words<W> w)
{
#pragma unroll
    for (int k = 0; k < W; ++k) w.v[k] &= kBit2;
    return w;
}

// The lookup table of a block (kLookupWords words of shared memory), indexed by the byte offset
// 4 D (heat bath; also the general Metropolis rule's thresholds) or 4 D + 32 (own spin down).
// Padding bytes hold any value, so every offset that their masked sums can form is in range:
// 4 * 6 + 32 bytes at most.  One thread fills it.
constexpr int kLookupWords = 16;

template <int NDIM, int RULE>
__device__ __forceinline__ void fill_lookup(u32* rt, const u32* table)
{
    constexpr int d = NDIM;
#pragma unroll
    for (int i = 0; i < kLookupWords; ++i) {
        const int D = i & 7, a = i < 8 ? D : 2 * d - D;  // a: anti-aligned neighbours
        if (D > 2 * d) {
            rt[i] = 0u;
        } else if constexpr (RULE == kHeat) {
            rt[i] = table[2 * d - D];
        } else if constexpr (RULE == kMetroFast) {
            rt[i] = a < d ? table[2 * d - a] - 1u : 0xFFFFFFFFu;
        } else {
            rt[i] = a < d ? table[2 * d - a] : 0u;
        }
    }
}

__device__ __forceinline__ u32 lookup(const u32* rt, u32 idx, int i)
{
    // byte i of idx, as a dot product: that runs on the multiplier pipe, a permute or shift on
    // the logic pipe, which bounds the kernel
    const u32 off = __dp4a(idx, 1u << (8 * i), 0u);
    return *reinterpret_cast<const u32*>(reinterpret_cast<const char*>(rt) + off);
}

// Predicated operations on one byte of a word of four spins: a comparison and the operation
// itself.  (The compiler's own form of such selects was a comparison, a conditional move and a
// select or add per site; its moves ran on the multiplier pipe that the Philox products need.)
__device__ __forceinline__ void add_if_less(u32& w, u32 u, u32 thr, u32 x)
{
    asm("{\n\t.reg .pred p;\n\tsetp.lt.u32 p, %1, %2;\n\t@p add.u32 %0, %0, %3;\n\t}"
        : "+r"(w)
        : "r"(u), "r"(thr), "r"(x));
}

__device__ __forceinline__ void add_if_not_greater(u32& w, u32 u, u32 thr, u32 x)
{
    asm("{\n\t.reg .pred p;\n\tsetp.le.u32 p, %1, %2;\n\t@p add.u32 %0, %0, %3;\n\t}"
        : "+r"(w)
        : "r"(u), "r"(thr), "r"(x));
}

// Bit 7 of each byte, over the whole byte (prmt's sign mode, which __byte_perm does not have).
__device__ __forceinline__ u32 byte_signs(u32 v)
{
    u32 r;
    asm("prmt.b32 %0, %1, 0, 0xBA98;" : "=r"(r) : "r"(v));
    return r;
}

// New spins of the four sites in word `s` given four times their down neighbours `d4` (one byte
// per site) and their four uniforms; `rt` is the block's lookup table (fill_lookup).
template <int NDIM, int RULE>
__device__ __forceinline__ u32 decide4(u32 s, u32 d4, const u32x4& r, const u32* rt)
{
    constexpr int d = NDIM;
    const u32 u[4] = {r.x, r.y, r.z, r.w};
    if constexpr (RULE == kObserve) {
        return s;
    } else if constexpr (RULE == kHeat) {
        u32 ns = 0xFFFFFFFFu;
#pragma unroll
        for (int i = 0; i < 4; ++i) add_if_less(ns, u[i], lookup(rt, d4, i), 0u - (0xFEu << (8 * i)));
        return ns;
    } else if constexpr (RULE == kMetroFast) {
        const u32 idx = d4 + (s & kBit5);
        u32 flips = 0u;
#pragma unroll
        for (int i = 0; i < 4; ++i) add_if_not_greater(flips, u[i], lookup(rt, idx, i), 1u << (8 * i));
        return s ^ (flips * 0xFEu);
    } else {
        // any table: A >= d flips whatever the uniform (the lookup holds 0 there)
        const u32 idx = d4 + (s & kBit5);
        const u32 up = d4 + (u32)(0x80 - 4 * d) * 0x01010101u;  // bit 7: D >= d
        const u32 dn = (u32)(0x80 + 4 * d) * 0x01010101u - d4;  // bit 7: D <= d
        u32 flips = (((up & ~s) | (dn & s)) >> 7) & 0x01010101u;
#pragma unroll
        for (int i = 0; i < 4; ++i) add_if_less(flips, u[i], lookup(rt, idx, i), 1u << (8 * i));
        return s ^ (flips * 0xFEu);
    }
}

// New spins of V consecutive colour sites of a row (parity `par` = (y + z + colour) & 1) from their
// own words `s` and the masked words (downs) of the opposite colour: the same row
// `c`, the rows above/below `nu`/`nd`, the planes above/below `zu`/`zd` (3D) and the horizontal
// neighbour byte outside the chunk `edge` (masked too); with MEAS adds the chunk's (M, E)
// contribution to m_acc / e_acc.  With RULE == kObserve nothing is updated (measurement only).
// `draw(k)` returns the four uniforms of the chunk's word k.
//
// MIXED = false: every chunk is full (lh % V == 0).  MIXED = true: rows are padded to a multiple
// of V bytes and a row's last chunk holds wv < W valid words; such a chunk runs the same
// instructions as a full one (no divergence inside a warp), with the padding words selected
// away: their random numbers are drawn and discarded, their bytes stored back unchanged, and
// the right-hand neighbour of the last valid word is the row's wrapped edge byte.
template <int V, int NDIM, int RULE, bool MIXED, bool MEAS, class Draw>
__device__ __forceinline__ Words<V / 4> int8_update(const Draw& draw, int par, int wv,
                                                    const Words<V / 4>& s,
                                                    const Words<V / 4>& c,
                                                    const Words<V / 4>& nu,
                                                    const Words<V / 4>& nd,
                                                    const Words<V / 4>& zu,
                                                    const Words<V / 4>& zd, u32 edge,
                                                    const u32* rt, long long& m_acc,
                                                    long long& e_acc)
{
    constexpr int W = V / 4;
    // Neighbour sums first, so the neighbour words are dead before the Philox blocks.
    u32 d4[W];
    int other_down = 0;  // down spins of the opposite colour at the same indices (for M)
#pragma unroll
    for (int k = 0; k < W; ++k) {
        u32 hz;  // the horizontal neighbours that are not at the sites' own indices
        if (par) {
            u32 nx = edge;
            if (k + 1 < W) nx = (!MIXED || k + 1 < wv) ? c.v[k + 1] : edge;
            hz = __byte_perm(c.v[k], nx, 0x4321);
        } else {
            hz = k > 0 ? __byte_perm(c.v[k], c.v[k - 1], 0x2107) : __byte_perm(c.v[k], edge, 0x2104);
        }
        d4[k] = c.v[k] + nu.v[k] + nd.v[k] + hz;
        if constexpr (NDIM == 3) d4[k] += zu.v[k] + zd.v[k];
        if constexpr (MEAS) {
            const int od = __popc(c.v[k]);
            other_down += (!MIXED || k < wv) ? od : 0;
        }
    }

    Words<W> ns;
#pragma unroll
    for (int k = 0; k < W; ++k) {
        if constexpr (RULE == kObserve) {
            ns.v[k] = s.v[k];
        } else {
            const u32 d = decide4<NDIM, RULE>(s.v[k], d4[k], draw(k), rt);
            ns.v[k] = (!MIXED || k < wv) ? d : s.v[k];
        }
    }

    if constexpr (MEAS) {
        // Bonds of this colour's sites: s*h = 2d - 2A' per site, A' = anti-aligned neighbours of
        // the new spin: D if it is up, 2d - D if it is down; E = -sum s*h.
        constexpr u32 k8d = 0x01010101u * (u32)(8 * NDIM);
        int anti4 = 0, down = 0;
#pragma unroll
        for (int k = 0; k < W; ++k) {
            const u32 sel = byte_signs(ns.v[k]);
            const u32 a4 = (d4[k] & ~sel) | ((k8d - d4[k]) & sel);
            const bool valid = !MIXED || k < wv;
            anti4 += valid ? byte_sum(a4) : 0;
            down += valid ? __popc(ns.v[k] & kBit2) : 0;
        }
        const int nv = 4 * wv;                      // valid sites of this chunk
        m_acc += 2 * nv - 2 * (down + other_down);  // this colour's sites + the other's
        e_acc += anti4 / 2 - 2 * NDIM * nv;         // -(2d n - 2 anti)
    }
    return ns;
}

// The four uniforms of word k of the chunk whose first four sites have Philox counter q0.
template <int NDIM>
struct DrawSites {
    const Int8Half& p;
    u32 q0;
    __device__ __forceinline__ u32x4 operator()(int k) const
    {
        return philox4x32_10<NDIM == 2>(q0 + (u32)k, p.t, p.color, 0u, p.k0, p.k1);
    }
};

template <bool MIXED, int W>
__device__ __forceinline__ int valid_words(const Int8Half& p, int j0)
{
    if constexpr (!MIXED) return W;
    const int left = (p.lh - j0) >> 2;
    return left < W ? left : W;
}

// Horizontal neighbour byte outside a chunk's wv valid words (periodic in x).
__device__ __forceinline__ int edge_index(const Int8Half& p, int par, int j0, int wv)
{
    return par ? (j0 + 4 * wv == p.lh ? 0 : j0 + 4 * wv) : (j0 == 0 ? p.lh - 1 : j0 - 1);
}

// Philox counter of the four sites from j0 of row `row`: the logical site index row*lh + j over
// 4, independent of the pitch.
__device__ __forceinline__ u32 site_counter(const Int8Half& p, long long row, int j0)
{
    return (u32)((unsigned long long)(row * p.lh + j0) >> 2);
}

// One chunk (V sites from j0) of row `row` = (z, y): loads its neighbourhood, then int8_update.
// CG reads the opposite colour from L2 (needed when one launch runs several half-sweeps).
template <int V, int NDIM, int RULE, bool CG, bool MIXED, bool MEAS, class Draw>
__device__ __forceinline__ void int8_chunk(const Int8Half& p, const Draw& draw, long long row,
                                           int y, int z, int j0, const u32* rt, long long& m_acc,
                                           long long& e_acc)
{
    constexpr int W = V / 4;
    const int par = (y + z + (int)p.color) & 1;
    const int wv = valid_words<MIXED, W>(p, j0);
    const long long rb = row * p.pitch;
    const int8_t* orow = p.other + rb;
    const Words<W> s = load_words<W>(p.own + rb + j0);
    const Words<W> c = downs(load_other<W, CG>(orow + j0));
    const int yu = z * p.ly + (y + 1 == p.ly ? 0 : y + 1);
    const int yd = z * p.ly + (y == 0 ? p.ly - 1 : y - 1);
    const Words<W> nu = downs(load_other<W, CG>(p.other + (long long)yu * p.pitch + j0));
    const Words<W> nd = downs(load_other<W, CG>(p.other + (long long)yd * p.pitch + j0));
    Words<W> zu = nu, zd = nd;
    if constexpr (NDIM == 3) {
        const int pu = (z + 1 == p.lz ? 0 : z + 1) * p.ly + y;
        const int pd = (z == 0 ? p.lz - 1 : z - 1) * p.ly + y;
        zu = downs(load_other<W, CG>(p.other + (long long)pu * p.pitch + j0));
        zd = downs(load_other<W, CG>(p.other + (long long)pd * p.pitch + j0));
    }
    const int je = edge_index(p, par, j0, wv);
    const u32 edge =
        (CG ? (u32)(uint8_t)__ldcg(orow + je) : (u32)(uint8_t)__ldg(orow + je)) & kBit2;
    const Words<W> ns = int8_update<V, NDIM, RULE, MIXED, MEAS>(
        draw, par, wv, s, c, nu, nd, zu, zd, edge, rt, m_acc, e_acc);
    if constexpr (RULE != kObserve) store_words<W>(p.own + rb + j0, ns);
}

// Where a band walk is: the row's own words, the row itself and its neighbour planes in the
// opposite colour.
struct BandRow {
    int8_t* own;
    const int8_t* c;
    const int8_t* zu;
    const int8_t* zd;
    u32 q;  // Philox counter of the chunk's first four sites in this row
};

// One row of a band, of parity `par`: the masked rows nd, c and nu are at hand.
template <int V, int NDIM, int RULE, bool MIXED, bool MEAS>
__device__ __forceinline__ void int8_band_row(const Int8Half& p, const BandRow& b, int par, int wv,
                                              int step_l, int step_r, const Words<V / 4>& c,
                                              const Words<V / 4>& nu, const Words<V / 4>& nd,
                                              const u32* rt, long long& m_acc, long long& e_acc)
{
    constexpr int W = V / 4;
    Words<W> zu = nu, zd = nd;
    if constexpr (NDIM == 3) {
        zu = downs(load_words_ro<W>(b.zu));
        zd = downs(load_words_ro<W>(b.zd));
    }
    const u32 edge = (u32)(uint8_t)__ldg(b.c + (par ? step_r : step_l)) & kBit2;
    const Words<W> s = load_words<W>(b.own);
    const Words<W> ns = int8_update<V, NDIM, RULE, MIXED, MEAS>(
        DrawSites<NDIM>{p, b.q}, par, wv, s, c, nu, nd, zu, zd, edge, rt, m_acc, e_acc);
    if constexpr (RULE != kObserve) store_words<W>(b.own, ns);
}

// Band schedule: chunk column j0 of rows y0 .. y1-1 of plane z, top to bottom.  The three
// opposite-colour rows a row needs (y-1, y, y+1) slide down the band, so each row loads and masks
// one new opposite-colour row (plus the planes z +- 1 in 3D) instead of three.  A band of an even
// number of rows takes two rows per step: the row parity, which side the horizontal neighbours
// are on, is then fixed in the code, and the sliding rows are renamed every second row only.  Not
// so padded rows that are updated and measured: two such rows in flight need more than the 64
// registers of four blocks per SM (spilled, a measured sweep of 3D 300x300x304 took 58.4 us, row by
// row 44.7).  (PAIRS: batches have measured and unmeasured rows in one kernel.)
template <int RULE, bool MIXED, bool MEAS>
constexpr bool kRowPairs = !(MIXED && MEAS && RULE != kObserve);

template <int V, int NDIM, int RULE, bool MIXED, bool MEAS,
          bool PAIRS = kRowPairs<RULE, MIXED, MEAS>>
__device__ __forceinline__ void int8_band(const Int8Half& p, int z, int y0, int y1, int j0,
                                          const u32* rt, long long& m_acc, long long& e_acc)
{
    constexpr int W = V / 4;
    const int wv = valid_words<MIXED, W>(p, j0);
    const int ly = p.ly, pitch = p.pitch;
    const u32 qstep = (u32)p.lh >> 2;
    const long long row0 = (long long)z * ly + y0;
    const int8_t* plane = p.other + (long long)z * ly * pitch + j0;  // row 0 of the plane
    const int step_r = j0 + 4 * wv == p.lh ? -j0 : 4 * wv, step_l = j0 == 0 ? p.lh - 1 : -1;
    BandRow b;
    b.own = p.own + row0 * pitch + j0;
    b.c = plane + (long long)y0 * pitch;
    b.q = site_counter(p, row0, j0);
    b.zu = b.zd = b.c;
    if constexpr (NDIM == 3) {
        b.zu = p.other + ((long long)(z + 1 == p.lz ? 0 : z + 1) * ly + y0) * pitch + j0;
        b.zd = p.other + ((long long)(z == 0 ? p.lz - 1 : z - 1) * ly + y0) * pitch + j0;
    }
    auto advance = [&] {
        b.own += pitch;
        b.c += pitch;
        b.q += qstep;
        if constexpr (NDIM == 3) {
            b.zu += pitch;
            b.zd += pitch;
        }
    };
    Words<W> nd = downs(load_words_ro<W>(y0 == 0 ? plane + (long long)(ly - 1) * pitch : b.c - pitch));
    Words<W> c = downs(load_words_ro<W>(b.c));
    const int par0 = (y0 + z + (int)p.color) & 1;
    auto pairs = [&](auto par) {
        constexpr int P = decltype(par)::value;
#pragma unroll 1
        for (int y = y0; y < y1; y += 2) {
            const Words<W> d1 = downs(load_words_ro<W>(b.c + pitch));  // y is even: y + 1 < ly
            int8_band_row<V, NDIM, RULE, MIXED, MEAS>(p, b, P, wv, step_l, step_r, c, d1, nd, rt,
                                                      m_acc, e_acc);
            advance();
            const Words<W> d2 = downs(load_words_ro<W>(y + 2 == ly ? plane : b.c + pitch));
            int8_band_row<V, NDIM, RULE, MIXED, MEAS>(p, b, 1 - P, wv, step_l, step_r, d1, d2, c,
                                                      rt, m_acc, e_acc);
            advance();
            nd = d1;
            c = d2;
        }
    };
    if constexpr (PAIRS) {
        if (((y0 | y1) & 1) == 0) {
            if (par0) pairs(std::integral_constant<int, 1>{});
            else pairs(std::integral_constant<int, 0>{});
            return;
        }
    }
#pragma unroll 1
    for (int y = y0; y < y1; ++y) {
        const Words<W> nu = downs(load_words_ro<W>(y + 1 == ly ? plane : b.c + pitch));
        int8_band_row<V, NDIM, RULE, MIXED, MEAS>(p, b, (par0 + y - y0) & 1, wv, step_l, step_r, c,
                                                  nu, nd, rt, m_acc, e_acc);
        advance();
        nd = c;
        c = nu;
    }
}

}  // namespace ising
