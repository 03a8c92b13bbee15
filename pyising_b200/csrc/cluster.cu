// Swendsen-Wang cluster updates of an int8 lattice (2D/3D), in its checkerboard layout.
//
// Local updates slow down critically near T_c (autocorrelation ~ L^2.17 sweeps in 2D); pyising
// equilibrates its starts and measures its Binder cumulants with a CPU Wolff sampler
// (src/pyising/cluster.py:32-104, src/pyising/validate.py:45-50,127-150).  Here the cluster
// update runs on the device: Swendsen-Wang (Phys. Rev. Lett. 58, 86 (1987)) with the
// connected components found by a lock-free union-find.
//
// One update at step t:
//   1. every bond joins a colour-0 site to a colour-1 site (the lattice is bipartite), so each
//      colour-0 site owns its 2d bonds and each bond is seen once.  A bond between aligned
//      spins is active with probability p = 1 - exp(-2 beta) (threshold p_bond on a uniform
//      u32 from Philox((n, t, kBondTag, k), key)).  The union-find runs on two levels, so that
//      the near-spanning clusters of the critical region do not funnel every union through a
//      few global roots: a CTA owns a tile of R rows x W positions of one plane, both colours
//      (16 x 32 by default), unites the active bonds inside the tile in shared memory, then
//      writes each site's tile-local root as its global label (sw_local_kernel); a second
//      kernel unites the active bonds that leave their tile in global memory (sw_cross_kernel).
//      (The single-level variant, every bond united in global memory by sw_bond_kernel, is kept
//      behind the cluster_tile knob.)
//      On both levels roots are linked larger-under-smaller with atomicCAS and finds halve
//      paths with plain stores (parents only ever move up the tree, so a stale read is still
//      an ancestor); the tile order of sites is their global order, so the final root of a
//      cluster is its smallest site whatever the tile size;
//   2. every label is replaced by its root (a read-only walk: only thread i writes label[i]);
//      in 2D the flips walk to the roots themselves instead;
//   3. every cluster flips with probability 1/2: bit (root & 127) of
//      Philox((root >> 7, t, kFlipTag, 0), key), the same for all its sites.
// Site g = c * S + row * lh + j (S = rows * lh sites per colour, the logical compressed index).
// Labels are int32 (lattices of fewer than 2^31 sites).  Every retry loop is bounded: a thread
// that exceeds the bound sets the error word and stops, and the host reports ISING_ERR_TIMEOUT.
#include "capi_internal.h"
#include "tile_forest.h"

namespace ising {

constexpr u32 kBondTag = 0x53570001u;  // Philox counter word 2 of the bond uniforms
constexpr u32 kFlipTag = 0x53570002u;  // ... of the cluster flip bits
// Bounded loops: one union (its finds and retries) or one root walk may take at most kStepLimit
// steps in global memory (about 0.3 s of dependent L2 reads; legitimate walks are far shorter) or
// kTileSteps in a tile's shared memory (tile_forest.h; a few milliseconds).  A thread that runs out
// sets the error word, and every loop in global memory gives up as soon as any thread has set it,
// which it reads every kErrPoll steps.  So one cycle in the labels (which a correct union-find never
// makes) ends the launch within milliseconds and the host reports ISING_ERR_TIMEOUT with the
// context intact.
constexpr int kStepLimit = 1 << 20;
constexpr int kErrPoll = 64;

struct StepBudget {
    int left = kStepLimit;
    bool dead = false;
};

// One more step of a bounded loop; false (and the error word set) when the budget is spent or
// another thread has set the error word.
__device__ __forceinline__ bool step(StepBudget& b, int* err)
{
    if (b.dead) return false;
    if (--b.left < 0) {
        atomicExch(err, 1);
        b.dead = true;
        return false;
    }
    if ((b.left & (kErrPoll - 1)) == 0 && *(volatile int*)err) {
        b.dead = true;
        return false;
    }
    return true;
}

struct ClusterArgs {
    int8_t* c[2];
    int* label;
    unsigned char* bonds;  // per colour-0 site, bit k = bond k active
    int* err;
    long long S;           // sites per colour
    long long rows;
    int lh, ly, lz, pitch, ndim;
    u32 t, k0, k1, p_bond;
};

__device__ __forceinline__ int uf_find(int* label, int x, int* err, StepBudget& b)
{
    while (step(b, err)) {
        const int p = __ldcg(label + x);
        if (p == x) return x;
        const int gp = __ldcg(label + p);
        if (gp != p) label[x] = gp;  // path halving
        x = gp;
    }
    return x;
}

// The root of x without writing anything: flattening must not halve paths, or a halving store
// (label[x] = grandparent) could overwrite the root another thread has just written to label[x].
__device__ __forceinline__ int uf_root(const int* label, int x, int* err)
{
    StepBudget b;
    while (step(b, err)) {
        const int p = __ldcg(label + x);
        if (p == x) return x;
        x = p;
    }
    return x;
}

__device__ __forceinline__ void uf_union(int* label, int a, int b, int* err)
{
    StepBudget budget;  // shared by the finds and the retries of this union
    while (step(budget, err)) {
        a = uf_find(label, a, err, budget);
        b = uf_find(label, b, err, budget);
        if (budget.dead || a == b) return;
        if (a > b) {
            const int t = a;
            a = b;
            b = t;
        }
        // link root b under root a, unless b stopped being a root meanwhile
        const int old = atomicCAS(label + b, b, a);
        if (old == b) return;
        b = old;
    }
}

// Test hook (ISING_KNOB_TEST_LABEL_CYCLE): a two-site cycle in the labels, which the root walks
// after it can only leave through their step budgets.
__global__ void sw_cycle_kernel(int* label, long long S)
{
    label[0] = (int)S;
    label[S] = 0;
}

// Colour-1 positions of the 2d bonds of colour-0 site n (the order of the bond bits): the same
// index, the other horizontal neighbour, y + 1, y - 1, z + 1, z - 1 (periodic).
__device__ __forceinline__ void bond_ends(const ClusterArgs& a, long long n, long long nb[6])
{
    const long long row = n / a.lh;
    const int j = (int)(n - row * a.lh);
    const int y = (int)(row % a.ly), z = (int)(row / a.ly);
    const int par = (y + z) & 1;  // colour 0
    const long long plane = (long long)z * a.ly;
    nb[0] = row * a.lh + j;
    nb[1] = row * a.lh + (par ? (j + 1 == a.lh ? 0 : j + 1) : (j == 0 ? a.lh - 1 : j - 1));
    nb[2] = (plane + (y + 1 == a.ly ? 0 : y + 1)) * a.lh + j;
    nb[3] = (plane + (y == 0 ? a.ly - 1 : y - 1)) * a.lh + j;
    nb[4] = ((long long)(z + 1 == a.lz ? 0 : z + 1) * a.ly + y) * a.lh + j;
    nb[5] = ((long long)(z == 0 ? a.lz - 1 : z - 1) * a.ly + y) * a.lh + j;
}

__device__ __forceinline__ int8_t colour1_spin(const ClusterArgs& a, long long m)
{
    const long long mrow = m / a.lh;
    return a.c[1][mrow * a.pitch + (m - mrow * a.lh)];
}

// Shared-memory union of one tile (same rules as the global one).
__device__ __forceinline__ void tile_union(int* lab, int a, int b, int* err)
{
    int left = kTileSteps;  // shared by the finds and the retries of this union
    while (true) {
        a = tile_find(lab, a, left);
        b = tile_find(lab, b, left);
        if (left < 0) {
            atomicExch(err, 1);
            return;
        }
        if (a == b) return;
        if (a > b) {
            const int t = a;
            a = b;
            b = t;
        }
        const int old = atomicCAS(lab + b, b, a);
        if (old == b) return;
        b = old;
    }
}

// Rectangular tiles: a tile is R rows x W positions of one plane (y in [y0, y0 + R), j in
// [j0, j0 + W), clipped at the plane's edges), of both colours; its local index of position
// (r, c) is r * W + c for colour 0 and R * W + r * W + c for colour 1, which orders a tile's
// sites as their global indices do.
struct TileGeo {
    int R, W;        // rows and positions per tile
    int tx, ty;      // tiles per row of positions, per plane
    u32 w_magic;     // fast_div magic of W (quotients of positions of a tile)
};

__device__ __forceinline__ void tile_origin(const ClusterArgs& a, const TileGeo& g, long long b,
                                           int& z, int& y0, int& j0)
{
    const long long per_plane = (long long)g.tx * g.ty;
    z = (int)(b / per_plane);
    const int rem = (int)(b - (long long)z * per_plane);
    const int by = rem / g.tx;
    y0 = by * g.R;
    j0 = (rem - by * g.tx) * g.W;
}

// Tile b: draws the bonds of the tile's colour-0 sites, stores their masks, unites the active
// bonds that stay in the tile (shared memory) and writes every tile site's label: the global index
// of its tile-local root.
//
// A warp takes a row of the tile (tiles narrower than a warp: as many rows as fit), a lane the sites
// of one position of both colours.  The row's horizontal bonds form runs of a chain; ballots of the two bonds of each colour-0 site give every
// site its run's smallest site as parent at once, without a union.  The vertical bonds then unite
// runs, once per pair of runs and row (a match over the warp picks one lane of each pair), and so do
// the bonds around the lattice where a tile holds its whole width or height.  Near
// T_c, where most sites of a tile are in one cluster, one union per bond had long walks and many
// failed compare-and-swaps.  Measured on one B200, equilibrated at T_c, this kernel 91 -> 30 us at
// 1024^2, the unions between tiles 37 -> 15 us, whole updates 141 -> 58 us at 1024^2 and 1588 ->
// 440 us at 4096^2; joining the rows' seams in the order of blocks of 1, 2, 4, ... rows was slower
// (80 against 71 us).
constexpr int kLocalThreads = 256;

__global__ void __launch_bounds__(kLocalThreads) sw_local_kernel(const ClusterArgs a, const TileGeo g)
{
    extern __shared__ int lab[];  // [2 R W] labels, then [R W] bytes of bond masks
    int z, y0, j0;
    tile_origin(a, g, blockIdx.x, z, y0, j0);
    const int R = g.R, W = g.W, RW = R * W;  // W <= 32
    const int rn = a.ly - y0 < R ? a.ly - y0 : R;  // rows of this tile
    const int wn = a.lh - j0 < W ? a.lh - j0 : W;  // positions per row of this tile
    unsigned char* masks = reinterpret_cast<unsigned char*>(lab + 2 * RW);
    // lanes per row: the least power of two from wn on; 1 << up rows per warp, this lane's the sub-th
    const int up = wn > 16 ? 0 : wn > 8 ? 1 : wn > 4 ? 2 : 3;
    const int lane = (int)(threadIdx.x & 31u), c = lane & ((32 >> up) - 1);
    const int base = lane - c, sub = lane >> (5 - up);
    const u32 below = (1u << base) - 1u;                       // the lanes of the warp's rows before
    const u32 inside = ((1u << (wn - 1)) - 1u) << base;        // of this row's sites but the last
    const int first = ((int)(threadIdx.x >> 5) << up), step_r = (int)(blockDim.x >> 5) << up;
    const bool wrap_x = g.tx == 1, wrap_y = g.ty == 1;         // the tile reaches around the lattice
    const long long plane = (long long)z * a.ly;
    for (int rw = first; rw < rn; rw += step_r) {  // (the same for all lanes of a warp)
        const int r = rw + sub;
        const bool in = c < wn && r < rn;
        const int y = y0 + r, j = j0 + c;
        const int par = (y + z) & 1;  // 1: the row's other horizontal neighbour is at j + 1
        // the spins the row's bonds join: its own, the opposite colour's of the rows y, y + 1, y - 1
        // (and planes z + 1, z - 1), and the horizontal neighbour from the next lane or, at the
        // tile's edge, from memory
        const long long row = plane + y;
        const int8_t* c1 = a.c[1] + row * a.pitch;
        const int s1 = in ? c1[j] : 0;
        int side = __shfl_sync(0xFFFFFFFFu, s1, par ? lane + 1 : lane - 1);
        unsigned mask = 0;
        if (in) {
            if (par ? c + 1 == wn : c == 0)
                side = c1[par ? (j + 1 == a.lh ? 0 : j + 1) : (j == 0 ? a.lh - 1 : j - 1)];
            const u32 q = (u32)row * (u32)a.lh + (u32)j;  // < 2^30
            const int s = a.c[0][row * a.pitch + j];
            const long long step = a.pitch, wrap = (long long)(a.ly - 1) * a.pitch;
            const int above = c1[(y + 1 == a.ly ? -wrap : step) + j];
            const int dn = c1[(y == 0 ? wrap : -step) + j];
            const u32x4 r0 = philox4x32_10(q, a.t, kBondTag, 0u, a.k0, a.k1);
            mask = (r0.x < a.p_bond && s1 == s ? 1u : 0u) | (r0.y < a.p_bond && side == s ? 2u : 0u) |
                   (r0.z < a.p_bond && above == s ? 4u : 0u) | (r0.w < a.p_bond && dn == s ? 8u : 0u);
            if (a.ndim == 3) {
                const u32x4 r1 = philox4x32_10(q, a.t, kBondTag, 1u, a.k0, a.k1);
                const long long pl = (long long)a.ly * a.pitch, zwrap = (a.lz - 1) * pl;
                const int zu = c1[(z + 1 == a.lz ? -zwrap : pl) + j];
                const int zd = c1[(z == 0 ? zwrap : -pl) + j];
                mask |= (r1.x < a.p_bond && zu == s ? 16u : 0u) |
                        (r1.y < a.p_bond && zd == s ? 32u : 0u);
            }
            a.bonds[q] = (unsigned char)mask;
            masks[r * W + c] = (unsigned char)mask;
        }
        // bonds inside the row and tile (not around the lattice): to the own index, to j +- 1
        const bool inner = par ? c + 1 < wn : c > 0;
        const u32 m0 = __ballot_sync(0xFFFFFFFFu, mask & 1u);
        const u32 m1 = __ballot_sync(0xFFFFFFFFu, inner && (mask & 2u) != 0);
        // bit of lane l: its colour-0 site is in one run with that of lane l + 1 (in the same row)
        const u32 link = (par ? m1 & (m0 >> 1) : m0 & (m1 >> 1)) & inside;
        auto run_start = [&](int at) {  // position of the first colour-0 site of the run of lane `at`
            const u32 breaks = ~link & ((1u << at) - 1u) & ~below;
            return max(32 - __clz((int)breaks), base) - base;  // 0 without a break
        };
        if (in) {
            const int i0 = r * W, i1 = RW + r * W + c;
            lab[i0 + c] = i0 + run_start(lane);
            int parent = i1;
            if ((m0 >> lane) & 1u) parent = i0 + run_start(lane);
            else if (par && c > 0 && ((m1 >> (lane - 1)) & 1u)) parent = i0 + run_start(lane - 1);
            else if (!par && c + 1 < wn && ((m1 >> (lane + 1)) & 1u))
                parent = i0 + run_start(lane + 1);
            lab[i1] = parent;
        }
    }
    __syncthreads();
    volatile int* vlab = lab;
    for (int rw = first; rw < rn; rw += step_r) {
        const int r = rw + sub;
        const bool in = c < wn && r < rn;
        const unsigned mask = in ? masks[r * W + c] : 0u;
        // y + 1, y - 1, and around the row
        for (int k = 2; k < (wrap_x ? 5 : 4); ++k) {
            int nr = r, nc = c;
            bool active = ((mask >> (k == 4 ? 1 : k)) & 1u) != 0;
            if (k == 2) {
                nr = r + 1 < rn ? r + 1 : 0;
                active = active && (r + 1 < rn || wrap_y);
            } else if (k == 3) {
                nr = r > 0 ? r - 1 : rn - 1;
                active = active && (r > 0 || wrap_y);
            } else {
                const int par = (y0 + r + z) & 1;
                nc = par ? 0 : wn - 1;
                active = active && c == wn - 1 - nc;
            }
            const u32 act = __ballot_sync(0xFFFFFFFFu, active);
            if (active) {
                const int u = vlab[r * W + c], v = vlab[RW + nr * W + nc];
                const u32 peers = __match_any_sync(act, (u32)u << 16 | (u32)v);
                if (lane == __ffs((int)peers) - 1) tile_union(lab, u, v, a.err);
            }
            __syncwarp();
        }
    }
    __syncthreads();
    for (int rw = first; rw < rn; rw += step_r) {
        const int r = rw + sub;
        if (c >= wn || r >= rn) continue;
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) {
            int left = kTileSteps;
            const int root = tile_root(lab, cc * RW + r * W + c, left);
            if (left < 0) atomicExch(a.err, 1);
            const int rc = root >= RW;
            const u32 rl = (u32)(root - rc * RW), rr = fast_div(rl, (u32)W, g.w_magic);
            const int gi = (int)(cc * a.S) + (int)(plane + y0 + r) * a.lh + j0 + c;
            const int gr = (int)(rc * a.S) + (int)(plane + y0 + (int)rr) * a.lh + j0 +
                           (int)(rl - rr * (u32)W);
            a.label[gi] = gr;
        }
    }
}

// Single-level variant (cluster_tile knob 1): every site its own tree, then every colour-0 site
// draws its bonds and unites the active ones in global memory directly.
__global__ void sw_init_kernel(int* label, long long n)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        label[i] = (int)i;
}

__global__ void sw_bond_kernel(const ClusterArgs a)
{
    const int nbonds = 2 * a.ndim;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < a.S;
         q += (long long)gridDim.x * blockDim.x) {
        const long long row = q / a.lh;
        const int8_t s = a.c[0][row * a.pitch + (q - row * a.lh)];
        long long nb[6];
        bond_ends(a, q, nb);
        const u32x4 r0 = philox4x32_10((u32)q, a.t, kBondTag, 0u, a.k0, a.k1);
        u32x4 r1 = {0u, 0u, 0u, 0u};
        if (a.ndim == 3) r1 = philox4x32_10((u32)q, a.t, kBondTag, 1u, a.k0, a.k1);
        const u32 u[6] = {r0.x, r0.y, r0.z, r0.w, r1.x, r1.y};
        unsigned mask = 0;
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            if (k >= nbonds) break;
            if (u[k] < a.p_bond && colour1_spin(a, nb[k]) == s) {
                mask |= 1u << k;
                uf_union(a.label, (int)q, (int)(a.S + nb[k]), a.err);
            }
        }
        a.bonds[q] = (unsigned char)mask;
    }
}

// The active bonds between tiles, united in global memory: the two bonds across every seam between
// tile rows (the last one around the lattice) at each position, the one bond across every seam
// between tile columns at each row, and in 3D the two z bonds of every colour-0 site.  Lanes run
// along a seam, where neighbouring bonds mostly join the same two tile clusters: one lane per pair
// of labels in a warp does the union.  A thread takes `parts` z bonds one after another: the rows of
// two tiles in neighbouring planes mostly join the same two clusters, too, and in an ordered lattice
// those unions get in each other's way when all of them start at once (cluster_z_parts).
__global__ void __launch_bounds__(256) sw_cross_kernel(const ClusterArgs a, const TileGeo g, int parts)
{
    const long long lh = a.lh, ly = a.ly, lz = a.lz;
    // (a single tile row or column has no seam: its tiles unite the bonds around the lattice too)
    const long long per_rows = g.ty > 1 ? (long long)g.ty * lz * lh : 0;  // per direction
    const long long per_cols = g.tx > 1 ? (long long)g.tx * a.rows : 0;
    const long long end_rows = 2 * per_rows, end_cols = end_rows + per_cols;
    const long long begin_z = (end_cols + 31) / 32 * 32, z_part = 2 * a.S / parts;  // S % 4 == 0
    const long long n = a.ndim == 3 ? begin_z + z_part : end_cols;
    const long long stride = (long long)gridDim.x * blockDim.x;
    const int lane = (int)(threadIdx.x & 31u);
    int part = 0;  // of the z bonds; the same for all lanes of a warp
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i - lane < n;) {
        long long q = -1, m = 0;  // colour-0 and colour-1 positions of the bond
        int k = 0;
        if (i < end_rows) {
            const int up = i >= per_rows;
            const u32 e = (u32)(i - up * per_rows);  // < S < 2^31
            const u32 seam = e / (u32)lh;
            const long long j = e - seam * (u32)lh;
            const long long z = seam / (u32)g.ty, ty = seam - (u32)z * (u32)g.ty;
            const long long last = (ty + 1) * g.R < ly ? (ty + 1) * g.R - 1 : ly - 1;
            const long long next = last + 1 == ly ? 0 : last + 1;
            k = up ? 3 : 2;
            q = (z * ly + (up ? next : last)) * lh + j;
            m = (z * ly + (up ? last : next)) * lh + j;
        } else if (i < end_cols) {
            const u32 e = (u32)(i - end_rows);  // < S
            const long long seam = e / (u32)a.rows;
            const long long row = e - (u32)seam * (u32)a.rows;
            const long long z = (u32)row / (u32)ly, y = row - z * ly;
            const long long last = (seam + 1) * g.W < lh ? (seam + 1) * g.W - 1 : lh - 1;
            const long long next = last + 1 == lh ? 0 : last + 1;
            const int par = (int)(y + z) & 1;
            k = 1;
            q = row * lh + (par ? last : next);
            m = row * lh + (par ? next : last);
        } else if (i >= begin_z && i < n) {
            const long long bond = i - begin_z + part * z_part;
            const int up = bond >= a.S;
            q = bond - up * a.S;
            k = up ? 5 : 4;
            const long long pl = ly * lh;
            const long long z = (u32)q / (u32)pl;
            m = q + (up ? (z == 0 ? (lz - 1) * pl : -pl) : (z + 1 == lz ? -(lz - 1) * pl : pl));
        }
        const bool active = q >= 0 && ((a.bonds[q] >> k) & 1u) != 0;
        const u32 act = __ballot_sync(0xFFFFFFFFu, active);
        if (active) {
            const int u = __ldcg(a.label + q), v = __ldcg(a.label + a.S + m);
            const u32 peers = __match_any_sync(act, (unsigned long long)(u32)u << 32 | (u32)v);
            if (lane == __ffs((int)peers) - 1) uf_union(a.label, u, v, a.err);
        }
        __syncwarp();
        if (i - lane >= begin_z && ++part < parts) continue;
        part = 0;
        i += stride;
    }
}

// Every label becomes its root; only thread i writes label[i], and every value it can hold
// meanwhile (its old parent or the root) is an ancestor, so other threads' walks stay valid.
__global__ void sw_flatten_kernel(int* label, long long n, int* err)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        label[i] = uf_root(label, (int)i, err);
}

// Step 3.  A thread takes four consecutive sites, one word of spins (rows are a multiple of four
// sites).  WALK: it walks up to their roots itself (read-only, the four walks side by side), with
// no flattening pass before; otherwise the labels are flat already.
template <bool WALK>
__global__ void __launch_bounds__(256) sw_flip_kernel(const ClusterArgs a)
{
    const long long n = a.S / 2;  // words of both colours
    const int lw = a.lh >> 2;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        // (nothing writes labels meanwhile: the walks may hit L1, where the upper tree soon is)
        const int4 first = __ldg(reinterpret_cast<const int4*>(a.label) + i);
        int x[4] = {first.x, first.y, first.z, first.w};
        if constexpr (WALK) {
            StepBudget budget;
            bool more = true;
            while (more && step(budget, a.err)) {
                more = false;
                int p[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) p[k] = __ldg(a.label + x[k]);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    more = more || p[k] != x[k];
                    x[k] = p[k];
                }
            }
        }
        u32 flips = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const u32 root = (u32)x[k];
            const u32x4 r = philox4x32_10(root >> 7, a.t, kFlipTag, 0u, a.k0, a.k1);
            const u32 w = (root & 64) ? ((root & 32) ? r.w : r.z) : ((root & 32) ? r.y : r.x);
            flips |= ((w >> (root & 31)) & 1u) << (8 * k);
        }
        const int c = 2 * i >= n ? 1 : 0;
        const u32 m = (u32)(i - (c ? n / 2 : 0));  // word of the colour, < 2^30
        const u32 row = m / (u32)lw;
        u32* p = reinterpret_cast<u32*>((c ? a.c[1] : a.c[0]) + (long long)row * a.pitch) +
                 (m - row * (u32)lw);
        *p ^= flips * 0xFEu;  // +1 <-> -1
    }
}

static int cluster_setup(ising_sim* h)
{
    if (h->variant != ISING_VARIANT_INT8)
        return fail(ISING_ERR_INVALID, "cluster updates: int8 lattices only");
    const long long n = 2 * h->rows * (long long)h->lh;
    if (n >= 0x7FFFFFFFll)
        return fail(ISING_ERR_INVALID, "cluster updates: lattices of fewer than 2^31 sites");
    if (!h->d_label) {  // labels, the error word, then one bond mask per colour-0 site
        // from the handles' pool (cudaMalloc took 2 ms of the first call of every handle), on a
        // stream that is then waited for: usable from any stream
        cudaError_t e = pool_alloc(h->device, (void**)&h->d_label,
                                   (size_t)n * sizeof(int) + 256 + (size_t)(n / 2),
                                   h->own_stream_handle);
        if (e == cudaSuccess) e = cudaStreamSynchronize(h->own_stream_handle);
        if (e != cudaSuccess) {
            cudaGetLastError();
            h->d_label = nullptr;
            return fail(ISING_ERR_NOMEM, "allocation of the cluster labels (%lld sites)", n);
        }
    }
    return ISING_OK;
}

// Tile shape of the shared-memory union-find: about T positions (the handle's cluster_tile
// knob, else kTileAuto) as R rows x W positions, W = 32 (16 for small T) or the row length;
// T = 0: the single-level union-find in global memory (knob value 1).  Small tiles give many
// CTAs and short trees, square-ish ones keep most bonds inside their tile.
constexpr int kTileAuto = 512;
constexpr int kTileMaxPositions = 6144;             // the knob's largest value
constexpr int kTileSiteBytes = 2 * sizeof(int) + 1;  // shared memory per position

static int cluster_tiles(const ising_sim* h, TileGeo* g)
{
    if (h->cluster_tile == 1) return 0;
    const int T = h->cluster_tile > 0 ? h->cluster_tile : kTileAuto;
    g->W = T >= 256 ? 32 : 16;
    if (g->W > h->lh) g->W = h->lh;
    g->R = T / g->W;
    if (g->R < 1) g->R = 1;
    if (g->R > h->ly) g->R = h->ly;
    g->tx = (h->lh + g->W - 1) / g->W;
    g->ty = (h->ly + g->R - 1) / g->R;
    g->w_magic = fast_div_magic((u32)g->W, (unsigned long long)g->R * g->W);
    return g->tx * g->ty * h->lz;
}

// z bonds per thread of the unions between tiles.  Four in lattices whose z bonds would all start at
// once, that are well ordered (3D bonds are critical at p = 0.358) and not too small to profit: one
// B200, us per update, one / four: at beta 0.28 8x8x4096 165 / 75, 64^3 125 / 80, 16x16x1024 157 / 82,
// 48^3 88 / 65; but 128x16x16 43 / 48, 128^3 363 / 701, and at the critical beta 8x8x4096 38 / 48, 64^3
// 42 / 51.
static int cluster_z_parts(const ClusterArgs& a, int threads)
{
    const bool fits = 2 * a.S <= threads && 6 * a.S >= threads;
    return a.ndim == 3 && a.p_bond >= 0x66666666u && fits ? 4 : 1;
}

static unsigned char* cluster_masks(ising_sim* h, long long S)
{
    return reinterpret_cast<unsigned char*>(h->d_label) + 2 * S * sizeof(int) + 256;
}

// One labeling (step 1-2) and, when `flip`, the cluster flips (step 3).
static int cluster_step(ising_sim* h, u32 t, u64 seed, u32 p_bond, bool flip)
{
    ClusterArgs a;
    a.c[0] = (int8_t*)h->c[0];
    a.c[1] = (int8_t*)h->c[1];
    a.S = h->rows * (long long)h->lh;
    a.label = h->d_label;
    a.err = reinterpret_cast<int*>(reinterpret_cast<char*>(h->d_label) + 2 * a.S * sizeof(int));
    a.bonds = cluster_masks(h, a.S);
    a.rows = h->rows;
    a.lh = h->lh;
    a.ly = h->ly;
    a.lz = h->lz;
    a.pitch = h->pitch;
    a.ndim = h->ndim;
    a.t = t;
    a.k0 = (u32)seed;
    a.k1 = (u32)(seed >> 32);
    a.p_bond = p_bond;
    const int grid = h->sm_count * 8;
    TileGeo g;
    const int tiles = cluster_tiles(h, &g);
    if (tiles > 0) {
        const size_t smem = (size_t)g.R * g.W * kTileSiteBytes;
        if (smem > 48 * 1024) {  // one value for every thread and handle that shares the function
            const cudaError_t e = cudaFuncSetAttribute(
                sw_local_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                kTileMaxPositions * kTileSiteBytes);
            if (e != cudaSuccess) return cuda_fail(e, "cluster tile size");
        }
        // (many tiles: four warps each and more tiles per SM, 1024^2 61.6 / 65.5 us per update; few:
        // eight, 256^2 43 / 35 us)
        const int threads = tiles >= 4 * h->sm_count ? kLocalThreads / 2 : kLocalThreads;
        sw_local_kernel<<<(unsigned)tiles, threads, smem, h->stream>>>(a, g);
        if (g.tx > 1 || g.ty > 1 || h->ndim == 3)  // else one tile holds the lattice
            sw_cross_kernel<<<grid, 256, 0, h->stream>>>(a, g, cluster_z_parts(a, grid * 256));
    } else {
        sw_init_kernel<<<grid, 256, 0, h->stream>>>(a.label, 2 * a.S);
        sw_bond_kernel<<<grid, 256, 0, h->stream>>>(a);
    }
    if (h->test_label_cycle) sw_cycle_kernel<<<1, 1, 0, h->stream>>>(a.label, a.S);
    // 2D: the flips walk to the roots themselves (no flattening pass); 3D, where the trees of
    // the tiles' roots are deeper (every z bond leaves its tile), measured faster flattened first
    // (256^3: 1046 vs 1131 us per update; 1024^2: 79 vs 85 us the other way round)
    const bool walk = flip && h->ndim == 2;
    if (!walk) sw_flatten_kernel<<<grid, 256, 0, h->stream>>>(a.label, 2 * a.S, a.err);
    if (walk) sw_flip_kernel<true><<<grid, 256, 0, h->stream>>>(a);
    else if (flip) sw_flip_kernel<false><<<grid, 256, 0, h->stream>>>(a);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "cluster update launch");
    return ISING_OK;
}

static int cluster_error(ising_sim* h)
{
    const long long S = h->rows * (long long)h->lh;
    int err = 0;
    cudaError_t e = cudaMemcpyAsync(&err, reinterpret_cast<char*>(h->d_label) + 2 * S * sizeof(int),
                                    sizeof(int), cudaMemcpyDeviceToHost, h->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
    if (e != cudaSuccess) return cuda_fail(e, "cluster update");
    if (err) return fail(ISING_ERR_TIMEOUT, "a bounded union-find loop of the cluster update gave up");
    return ISING_OK;
}

}  // namespace ising

using namespace ising;

extern "C" int ising_cluster_sweep(ising_sim* h, uint64_t step0, int64_t n_steps, uint64_t seed,
                                   uint32_t p_bond, int64_t* series_out)
{
    if (!h) return fail(ISING_ERR_INVALID, "null handle");
    if (n_steps < 0) return fail(ISING_ERR_INVALID, "negative step count");
    cudaError_t e = cudaSetDevice(h->device);
    if (e != cudaSuccess) return cuda_fail(e, "cudaSetDevice");
    int rc = cluster_setup(h);
    if (rc != ISING_OK) return rc;
    if (series_out && n_steps > 0) {
        rc = ensure_series(h, n_steps);
        if (rc != ISING_OK) return rc;
        e = cudaMemsetAsync(h->d_series, 0, (size_t)n_steps * 2 * sizeof(long long), h->stream);
        if (e != cudaSuccess) return cuda_fail(e, "cudaMemsetAsync (series)");
    }
    const long long S = h->rows * (long long)h->lh;
    e = cudaMemsetAsync(reinterpret_cast<char*>(h->d_label) + 2 * S * sizeof(int), 0, sizeof(int),
                        h->stream);
    if (e != cudaSuccess) return cuda_fail(e, "cudaMemsetAsync");
    for (int64_t k = 0; k < n_steps; ++k) {
        rc = cluster_step(h, (u32)(step0 + (uint64_t)k), seed, p_bond, true);
        if (rc == ISING_OK && series_out)
            rc = observe(h, reinterpret_cast<unsigned long long*>(h->d_series + 2 * k));
        if (rc != ISING_OK) return rc;
    }
    rc = cluster_error(h);
    if (rc == ISING_OK && series_out && n_steps > 0) {
        e = cudaMemcpyAsync(series_out, h->d_series, (size_t)n_steps * 2 * sizeof(long long),
                            cudaMemcpyDeviceToHost, h->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
        if (e != cudaSuccess) return cuda_fail(e, "cluster series copy");
    }
    return rc;
}

extern "C" int ising_cluster_labels(ising_sim* h, uint64_t step, uint64_t seed, uint32_t p_bond,
                                    int32_t* labels_out, uint8_t* bonds_out)
{
    if (!h || !labels_out || !bonds_out) return fail(ISING_ERR_INVALID, "null argument");
    cudaError_t e = cudaSetDevice(h->device);
    if (e != cudaSuccess) return cuda_fail(e, "cudaSetDevice");
    int rc = cluster_setup(h);
    if (rc != ISING_OK) return rc;
    const long long S = h->rows * (long long)h->lh;
    e = cudaMemsetAsync(reinterpret_cast<char*>(h->d_label) + 2 * S * sizeof(int), 0, sizeof(int),
                        h->stream);
    if (e != cudaSuccess) return cuda_fail(e, "cudaMemsetAsync");
    rc = cluster_step(h, (u32)step, seed, p_bond, false);
    if (rc == ISING_OK) rc = cluster_error(h);
    if (rc == ISING_OK) {
        e = cudaMemcpyAsync(labels_out, h->d_label, (size_t)(2 * S) * sizeof(int),
                            cudaMemcpyDeviceToHost, h->stream);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(bonds_out, cluster_masks(h, S), (size_t)S, cudaMemcpyDeviceToHost,
                                h->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
        if (e != cudaSuccess) rc = cuda_fail(e, "cluster labels copy");
    }
    return rc;
}
