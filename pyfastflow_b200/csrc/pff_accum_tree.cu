// libpff drainage accumulation by hierarchical tile contraction: the upstream sums
// that pyfastflow's accumulate_constant_Q forms by rake and compress
// (pyfastflow/flow/downstream_propag.py:21-179 driven by flow/flowfields.py:254-292),
// computed with a different decomposition.
//
// Q[i] = sum of the seeds of every cell whose receiver path passes through i
// (i included); counts[i] = the number of such cells.  The sums are formed
// exactly: counts as uint32, seeds as 64-bit fixed point (seed * 2^s rounded to
// an integer, with s chosen from max|seed| so that no sum can overflow), and Q is
// the fixed-point total rounded once to f32.  Integer sums do not depend on the
// order of additions, so the result is deterministic although every level uses
// atomics.  The reference's f32 rake-and-compress sums differ from the exact sum
// by their own rounding: counts are identical, Q agrees to f32 rounding.
//
// Decomposition (each level is one kernel launch up and one down):
//   level 0   32 x 32 cell tiles, one CTA each.  In shared memory every cell's
//             in-tile upstream sum is formed by pointer doubling (below): about
//             log2 of the longest in-tile path rounds, every cell busy in every
//             round, no serial chain.  Cells whose receiver lies in another tile
//             ("exits") become the nodes of level 1, carrying their in-tile totals.
//   level L   blocks of S_L x S_L tiles (S_1 = 8, S_{L+1} = 2 S_L).  A node's
//             parent at level L is the terminal (within the lower-level block) of
//             the cell or node its flow enters; pointer-doubling rounds run over
//             a block's nodes in shared memory.  Nodes whose parent lies in another block are
//             the next level's nodes.  The top level is one block over the grid.
//   down      from the top: each level's nodes receive the totals of the nodes of
//             the level above that drain into them (integer atomics), and the rounds
//             run again with those inflows added to the seeds, giving every node
//             its full total; at level 0 the inflows of a tile's entries are added
//             along their in-tile paths to the totals kept from the way up.
// A constant seed needs only the counts: its totals are count x seed.
// A receiver cycle shows as a successor pointer that outlives the rounds; it is
// reported in the status word (the result is then unspecified).
#include <algorithm>
#include <cmath>
#include "pff_coop.cuh"
#include "pff_internal.h"

namespace pff {

constexpr int TR_T = 32;                 // tile side in cells
constexpr int TR_TC = TR_T * TR_T;       // cells per tile
constexpr int TR_T0_THREADS = 256;
constexpr int TR_LB_THREADS = 1024;
constexpr int TR_S1 = 8;                 // level-1 block side in tiles
constexpr int TR_MAXLEV = 20;
constexpr int TR_SMEM_NODES = 8192;      // nodes of a block kept in shared memory
constexpr int TR_NODE_BYTES = 24;        // lo, hi, cnt, lpar, jmp, tn
constexpr int TR_ALL_TILES = 4;          // one launch for the whole accumulation up to so many tiles per SM

// status bits
constexpr int TR_ERR_RCV = 1;       // a receiver index out of range
constexpr int TR_ERR_CYCLE = 2;     // a receiver cycle
constexpr int TR_ERR_CAP = 4;       // more exits in a tile than the capacity (local = 0 only)
constexpr int TR_ERR_NONLOCAL = 8;  // local = 1 but a receiver leads into another tile's interior
constexpr int TR_ERR_SEED = 16;     // a non-finite seed

struct TreeLevel {
    long long *W;        // in-block total carried up (fixed point)
    unsigned *C;         // in-block count carried up
    int *rawpar;         // parent before resolution (level 1: a cell; else a position one level down)
    int *par;            // resolved parent position at this level, or -1
    int *up;             // position at the next level of this node's block terminal, or -1
    long long *In;       // inflow from the level above (fixed point)
    unsigned *Inc;       // inflow count
    int *src;            // position of this node one level down (levels >= 2)
    int *cnt;            // nodes per block (appended by the level below)
    int side;            // block side in tiles
    int nbx, nby;        // blocks per row / column
};

struct TreeArgs {
    int nx, ny, ntx, nty, N;
    int slots;           // node slots per level (tiles x cap0)
    int cap0;            // node slots per tile
    int nlev;            // block levels 1..nlev (nlev = top)
    int local;           // receivers lead only to tile-perimeter cells of other tiles
    unsigned char *marker;  // cell receives inflow from another tile this call
    long long *In0;
    unsigned *Inc0;
    int *up0;            // per cell: level-1 position of its tile terminal, or -1
    long long *T0;       // per cell: in-tile total (weighted seeds)
    unsigned *C0;        // per cell: in-tile count
    int *status;         // [0] error bits, [1] max |seed| bits, [8] grid barrier
    BarWait wait;
    int *out;            // the caller's copy of status[0] (mapped host memory), or null
    int nzero;           // ints from status on that start at zero (status, then the levels' counts)
    long long *scr_acc;  // fallback storage for blocks larger than TR_SMEM_NODES
    unsigned *scr_cnt;
    int *scr_lpar, *scr_pend, *scr_tn;
    long long *scr_acc2;  // start-of-round copies for those blocks
    unsigned *scr_cnt2;
    TreeLevel lv[TR_MAXLEV + 1];
};

// ---- block geometry (row-major blocks, closed-form tile offsets) ------------------
struct BlockGeo {
    int tile_off;   // first tile index of the block in the level's slot order
    int tiles;      // tiles in the block
};
__host__ __device__ __forceinline__ BlockGeo block_geo(int bx, int by, int side, int ntx, int nty)
{
    const int h = min(side, nty - by * side), w = min(side, ntx - bx * side);
    BlockGeo g;
    g.tile_off = by * side * ntx + bx * side * h;
    g.tiles = w * h;
    return g;
}

// ---- fixed point --------------------------------------------------------------------
// s such that N * max|seed| * 2^s < 2^62: no partial sum can overflow int64.
__device__ __forceinline__ int fixed_shift(unsigned maxbits, int N)
{
    const float m = __uint_as_float(maxbits);
    if (!(m > 0.f)) return 0;
    int e;
    const unsigned E = (maxbits >> 23) & 0xffu;
    if (E) e = (int)E - 126;    // m = f * 2^e with f in [0.5, 1): m < 2^e
    else frexpf(m, &e);
    const int nb = 32 - __clz(N);  // N < 2^nb
    return 62 - (e + nb);
}
// round(w * 2^s) to the nearest integer, ties to even, from the IEEE-754 fields:
// w = +-m * 2^(E-150) (m with its implicit bit; E = 0: m * 2^-149).  Exact in
// 64 bits for every |w| <= max|seed| (fixed_shift keeps m * 2^(e+s) < 2^62).
__device__ __forceinline__ long long to_fixed(float w, int s)
{
    const unsigned b = __float_as_uint(w);
    const unsigned E = (b >> 23) & 0xffu;
    unsigned long long m = b & 0x7fffffu;
    int e;
    if (E) { m |= 0x800000u; e = (int)E - 150; }
    else e = -149;
    const int sh = e + s;
    unsigned long long v;
    if (sh >= 0) v = sh < 40 ? m << sh : 0;  // (larger shifts only for non-finite seeds, flagged elsewhere)
    else {
        const int k = -sh;
        if (k > 40) v = 0;
        else {
            const unsigned long long q = m >> k, rem = m & ((1ull << k) - 1), half = 1ull << (k - 1);
            v = q + ((rem > half || (rem == half && (q & 1))) ? 1 : 0);
        }
    }
    return (b >> 31) ? -(long long)v : (long long)v;
}
__device__ __forceinline__ float from_fixed(long long v, int s)
{
    // one correct rounding to f32, then an exact power-of-two scaling
    float f = __ll2float_rn(v);
    while (s > 126) { f = __fmul_rn(f, 0x1p-126f); s -= 126; }
    while (s < -126) { f = __fmul_rn(f, 0x1p126f); s += 126; }
    return __fmul_rn(f, __int_as_float((127 - s) << 23));
}

// max |seed| over the grid (as f32 bits: non-negative floats order as integers)
__device__ __forceinline__ void tree_seedmax(const float *__restrict__ w, int N, int *status)
{
    unsigned m = 0;
    bool bad = false;
    auto take = [&](float x) {
        const float a = fabsf(x);
        if (!(a <= 3.4028235e38f)) bad = true;
        else m = max(m, __float_as_uint(a));
    };
    const int stride = gridDim.x * blockDim.x, t0 = blockIdx.x * blockDim.x + threadIdx.x;
    if (((uintptr_t)w & 15) == 0) {  // 16-byte loads, then the tail
        const float4 *w4 = reinterpret_cast<const float4 *>(w);
        for (int q = t0; q < N / 4; q += stride) {
            const float4 v = __ldg(w4 + q);
            take(v.x); take(v.y); take(v.z); take(v.w);
        }
        for (int i = (N / 4) * 4 + t0; i < N; i += stride) take(w[i]);
    } else {
        for (int i = t0; i < N; i += stride) take(w[i]);
    }
    for (int o = 16; o; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0 && m) atomicMax((unsigned *)&status[1], m);
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(&status[0], TR_ERR_SEED);
}

__global__ void k_tree_seedmax(const float *__restrict__ w, int N, int *status) { tree_seedmax(w, N, status); }

// ---- accumulation by pointer doubling -------------------------------------------------------
// Within a block, with A the donor -> receiver adjacency restricted to the block,
// the upstream sums are Q = sum_j A^j w = prod_i (I + A^(2^i)) w (A is nilpotent
// on a forest).  Round i applies (I + A^(2^i)): every node adds its current sum
// to the node 2^i steps downstream (integer atomics), and the successor pointers
// double; a pointer dies when its path leaves the block or ends at a root.  All
// nodes work in every round, so there is no serial chain; the rounds stop when
// every pointer is dead (after ceil(log2 of the longest in-block path) rounds).
// A pointer still alive after log2(n) + 1 rounds lies on a receiver cycle.
//
// jmp[k]: successor 2^i steps down, or -1.  Register copies of each thread's
// nodes (RPT per thread) hold the start-of-round values.
template <int RPT, int NT, bool VAL>
__device__ __forceinline__ bool doubling_rounds(int n, int *jmp, unsigned *lo, unsigned *hi, unsigned *cnt,
                                                int max_rounds)
{
    // totals as 32-bit halves: the low half's atomic returns the old value, and the
    // adder that wraps it carries into the high half (each wrap counted once)
    for (int r = 0; r < max_rounds; ++r) {
        int sj[RPT], nj[RPT];
        unsigned sl[RPT], sh[RPT], sc[RPT];
        bool live = false;
#pragma unroll
        for (int j = 0; j < RPT; ++j) {
            const int k = threadIdx.x + j * NT;
            sj[j] = -1;
            if (k < n) {
                sj[j] = jmp[k];
                if (sj[j] >= 0) {
                    if (VAL) {
                        sl[j] = lo[k];
                        sh[j] = hi[k];
                    }
                    sc[j] = cnt[k];
                    nj[j] = jmp[sj[j]];
                    live = true;
                }
            }
        }
        if (!__syncthreads_or(live)) return true;
#pragma unroll
        for (int j = 0; j < RPT; ++j) {
            if (sj[j] >= 0) {
                const int k = threadIdx.x + j * NT;
                if (VAL) {
                    const unsigned old = atomicAdd(&lo[sj[j]], sl[j]);
                    atomicAdd(&hi[sj[j]], sh[j] + (old + sl[j] < old ? 1u : 0u));
                }
                atomicAdd(&cnt[sj[j]], sc[j]);
                jmp[k] = nj[j];
            }
        }
        __syncthreads();
    }
    // a pointer that is still alive: a path longer than the block (a cycle)
    bool live = false;
    for (int k = threadIdx.x; k < n; k += NT) live |= jmp[k] >= 0;
    return !__syncthreads_or(live);
}

// ---- level 0: a group of 256 threads per tile ---------------------------------------------
// The cells of a tw x th tile that another tile's exit can enter: its perimeter when the
// receivers are local, else every cell.  Entry e as a local index (row * 32 + column).
__device__ __forceinline__ int tree_entries(const TreeArgs &a, int tw, int th)
{
    if (!a.local) return tw * th;
    return tw + (th > 1 ? tw : 0) + max(th - 2, 0) * (tw > 1 ? 2 : 1);
}
__device__ __forceinline__ int tree_entry(const TreeArgs &a, int e, int tw, int th)
{
    int lx, ly;
    if (!a.local) { ly = e / tw; lx = e - ly * tw; }
    else if (e < tw) { lx = e; ly = 0; }
    else if (e < 2 * tw && th > 1) { lx = e - tw; ly = th - 1; }
    else if (tw > 1) { const int f = e - 2 * tw; lx = (f & 1) ? tw - 1 : 0; ly = 1 + (f >> 1); }
    else { lx = 0; ly = 1 + e - 2; }
    return ly * TR_T + lx;
}

// Pass 0, level 0, one tile by a group of 256 threads (t: thread of the group; sync: the
// group's barrier).  The same doubling rounds as doubling_rounds(), with each 64-bit total
// held as two 32-bit halves in shared memory: 32-bit shared atomics are single
// operations, 64-bit ones are not.  The low half's atomic returns the old value, so the
// adder whose addition wraps it adds the carry to the high half; every wrap is counted
// exactly once, and the 64-bit sum is exact.
//
// VAL = false (a constant seed): only the counts are formed; a total is count x seed, the
// same integer.
//
// Writes the in-tile totals of every cell (T0, C0), the level-1 nodes of the exits, and
// up0 for the cells other tiles can drain into.
//
// Bound by the rounds' shared-memory atomics (about 7 rounds; 72 % issue active).
template <bool VAL, class Sync>
__device__ __forceinline__ void tree_tile_up(const TreeArgs &a, const int32_t *__restrict__ rcv,
                                             const float *__restrict__ w, int s, int tile, unsigned char *smem, int t,
                                             Sync sync)
{
    constexpr int RPT = TR_TC / TR_T0_THREADS;
    unsigned *cnt = reinterpret_cast<unsigned *>(smem), *lo = cnt + TR_TC, *hi = lo + (VAL ? TR_TC : 0);
    uint16_t *jmp = reinterpret_cast<uint16_t *>(hi + (VAL ? TR_TC : 0));
    int16_t *lpar = reinterpret_cast<int16_t *>(jmp + TR_TC);  // -2 no cell, -1 root, -3 exit, else in-tile receiver
    int *sv = reinterpret_cast<int *>(lpar + TR_TC);           // [0] exits, [1] base, [2] error, [3] live rounds flag
    constexpr uint16_t DEAD = 0xffff;
    const int tx = tile % a.ntx, ty = tile / a.ntx;
    const int x0 = tx * TR_T, y0 = ty * TR_T;
    const int tw = min(TR_T, a.nx - x0), th = min(TR_T, a.ny - y0);
    const int lx = t & (TR_T - 1), ly0 = t >> 5;  // a thread's cells: rows ly0 + 8 j
    if (t < 4) sv[t] = 0;
    sync();
    int rr[RPT];
    float wv[RPT];
#pragma unroll
    for (int j = 0; j < RPT; ++j) {
        const bool in = lx < tw && ly0 + 8 * j < th;
        const int gi = (y0 + ly0 + 8 * j) * a.nx + x0 + lx;
        rr[j] = in ? rcv[gi] : -1;
        wv[j] = VAL && in ? w[gi] : 0.f;
    }
    unsigned alive = 0;  // this thread's cells whose pointer is still alive
    bool exit_[RPT];
#pragma unroll
    for (int j = 0; j < RPT; ++j) {
        const int k = t + j * TR_T0_THREADS, ly = ly0 + 8 * j;
        int lp = -2;
        unsigned long long v = 0;
        if (lx < tw && ly < th) {
            const int gi = (y0 + ly) * a.nx + x0 + lx;
            int r = rr[j];
            if (r < 0 || r >= a.N) { atomicOr(&sv[2], TR_ERR_RCV); r = gi; }
            const int d = r - gi;
            if (d == 0) lp = -1;
            else if (d == 1 && lx + 1 < tw) lp = k + 1;  // D4 neighbours without a division
            else if (d == -1 && lx > 0) lp = k - 1;
            else if (d == a.nx && ly + 1 < th) lp = k + TR_T;
            else if (d == -a.nx && ly > 0) lp = k - TR_T;
            else {
                const int ry = r / a.nx, rx = r - ry * a.nx;
                lp = (rx >= x0 && rx < x0 + tw && ry >= y0 && ry < y0 + th) ? (ry - y0) * TR_T + rx - x0 : -3;
            }
            if (VAL) v = (unsigned long long)to_fixed(wv[j], s);
        }
        lpar[k] = (int16_t)lp;
        exit_[j] = lp == -3;
        jmp[k] = lp >= 0 ? (uint16_t)lp : DEAD;
        alive |= (lp >= 0 ? 1u : 0u) << j;
        cnt[k] = lp != -2 ? 1u : 0u;
        if (VAL) {
            lo[k] = (unsigned)v;
            hi[k] = (unsigned)(v >> 32);
        }
    }
    sync();
    // doubling rounds: the longest in-tile path is < 1024 = 2^10 cells
    bool cyc = false;
    for (int r = 0;; ++r) {
        int sj[RPT], nj[RPT];
        unsigned sl[RPT], sh[RPT], sc[RPT];
        if (alive) sv[3] = r + 1;
#pragma unroll
        for (int j = 0; j < RPT; ++j) {
            const int k = t + j * TR_T0_THREADS;
            sj[j] = -1;
            if (alive >> j & 1u) {
                sj[j] = jmp[k];
                if (VAL) {
                    sl[j] = lo[k];
                    sh[j] = hi[k];
                }
                sc[j] = cnt[k];
                nj[j] = jmp[sj[j]];
                if (nj[j] == DEAD) alive &= ~(1u << j);
            }
        }
        sync();
        if (sv[3] != r + 1) break;
        if (r == 10) { cyc = true; break; }  // a path longer than the tile: a cycle
#pragma unroll
        for (int j = 0; j < RPT; ++j) {
            if (sj[j] >= 0) {
                const int k = t + j * TR_T0_THREADS;
                if (VAL) {
                    const unsigned old = atomicAdd(&lo[sj[j]], sl[j]);
                    atomicAdd(&hi[sj[j]], sh[j] + (old + sl[j] < old ? 1u : 0u));
                }
                atomicAdd(&cnt[sj[j]], sc[j]);
                jmp[k] = (uint16_t)nj[j];
            }
        }
        sync();
    }
    if (cyc && t == 0) atomicOr(&sv[2], TR_ERR_CYCLE);

    // totals, and exits -> level-1 nodes of this tile's level-1 block
    const TreeLevel &L1 = a.lv[1];
    const int bx = tx / L1.side, by = ty / L1.side;
    const int b1 = by * L1.nbx + bx;
    const BlockGeo g1 = block_geo(bx, by, L1.side, a.ntx, a.nty);
    int rank[RPT];
#pragma unroll
    for (int j = 0; j < RPT; ++j) {
        const unsigned m = __ballot_sync(0xffffffffu, exit_[j]);
        int base = 0;
        if (m && (t & 31) == 0) base = atomicAdd(&sv[0], __popc(m));
        rank[j] = __shfl_sync(0xffffffffu, base, 0) + __popc(m & ((1u << (t & 31)) - 1u));
    }
    sync();
    if (t == 0) {
        const int n = sv[0];
        int base = n ? atomicAdd(&L1.cnt[b1], n) : 0;
        if (base + n > g1.tiles * a.cap0) {
            atomicOr(&sv[2], TR_ERR_CAP);
            base = -1;
        }
        sv[1] = base;
    }
    sync();
    const int base = sv[1], slot0 = g1.tile_off * a.cap0 + base;
    int *q = reinterpret_cast<int *>(cnt);  // level-1 position of each exit, once its count is written
#pragma unroll
    for (int j = 0; j < RPT; ++j) {
        const int k = t + j * TR_T0_THREADS, ly = ly0 + 8 * j;
        int qk = -1;
        if (lx < tw && ly < th) {
            const int gi = (y0 + ly) * a.nx + x0 + lx;
            const long long tot = VAL ? (long long)(((unsigned long long)hi[k] << 32) | lo[k]) : 0;
            const unsigned c = cnt[k];
            a.C0[gi] = c;
            if (VAL) a.T0[gi] = tot;
            if (exit_[j] && base >= 0) {
                const int r = rr[j];
                qk = slot0 + rank[j];
                if (VAL) L1.W[qk] = tot;
                L1.C[qk] = c;
                L1.rawpar[qk] = r;
                L1.src[qk] = gi;
                if (VAL) a.In0[r] = 0;
                a.Inc0[r] = 0;
                a.marker[r] = 1;
                if (a.local) {  // the entry must be on the perimeter of its own tile
                    const int ry = r / a.nx, rx = r - ry * a.nx;
                    const int ex = rx % TR_T, ey = ry % TR_T;
                    if (!(ex == 0 || ey == 0 || ex == TR_T - 1 || ey == TR_T - 1 || rx == a.nx - 1 || ry == a.ny - 1))
                        atomicOr(&sv[2], TR_ERR_NONLOCAL);
                }
            }
        }
        q[k] = qk;
    }
    sync();
    // up0 = level-1 position of the cell's tile terminal (if that is an exit), for
    // the cells another tile's exit can enter: the perimeter when local, every cell
    // otherwise; each walks down to its terminal
    const int per = tree_entries(a, tw, th);
    for (int e = t; e < per; e += TR_T0_THREADS) {
        int u = tree_entry(a, e, tw, th);
        const int gi = (y0 + (u >> 5)) * a.nx + x0 + (u & (TR_T - 1));
        for (int st = 0; st < TR_TC && lpar[u] >= 0; ++st) u = lpar[u];
        a.up0[gi] = lpar[u] == -3 ? q[u] : -1;
    }
    if (t == 0 && sv[2]) atomicOr(&a.status[0], sv[2]);
}

// The last pass, level 0: each cell's full total = its in-tile total plus the inflows of the
// tile's entries upstream of it.  The entries (at most 124 when local, most tiles have
// 30-60) each walk their in-tile path and add; every other cell only reads its total back.
// The pass was a second run of the doubling rounds with the inflows in the seeds (318 us
// at 4096^2 against 382 for the first); reading the totals back costs 12 B per cell.
template <bool VAL, class Sync>
__device__ __forceinline__ void tree_tile_finish(const TreeArgs &a, const int32_t *__restrict__ rcv, int s, long long cval,
                                                 float *Q, unsigned *counts, int tile, unsigned char *smem, int t,
                                                 Sync sync)
{
    constexpr int RPT = TR_TC / TR_T0_THREADS;
    unsigned *cnt = reinterpret_cast<unsigned *>(smem), *lo = cnt + TR_TC, *hi = lo + (VAL ? TR_TC : 0);
    int16_t *lpar = reinterpret_cast<int16_t *>(hi + (VAL ? TR_TC : 0));  // in-tile receiver or -1
    const int tx = tile % a.ntx, ty = tile / a.ntx;
    const int x0 = tx * TR_T, y0 = ty * TR_T;
    const int tw = min(TR_T, a.nx - x0), th = min(TR_T, a.ny - y0);
    const int lx = t & (TR_T - 1), ly0 = t >> 5;
    int rr[RPT];
    unsigned cv[RPT];
    long long tv[RPT];
#pragma unroll
    for (int j = 0; j < RPT; ++j) {
        const bool in = lx < tw && ly0 + 8 * j < th;
        const int gi = (y0 + ly0 + 8 * j) * a.nx + x0 + lx;
        rr[j] = in ? rcv[gi] : -1;
        cv[j] = in ? a.C0[gi] : 0u;
        tv[j] = VAL && in ? a.T0[gi] : 0;
    }
#pragma unroll
    for (int j = 0; j < RPT; ++j) {
        const int k = t + j * TR_T0_THREADS, ly = ly0 + 8 * j;
        int lp = -1;
        if (lx < tw && ly < th) {
            const int gi = (y0 + ly) * a.nx + x0 + lx, r = rr[j], d = r - gi;
            if (d == 1 && lx + 1 < tw) lp = k + 1;
            else if (d == -1 && lx > 0) lp = k - 1;
            else if (d == a.nx && ly + 1 < th) lp = k + TR_T;
            else if (d == -a.nx && ly > 0) lp = k - TR_T;
            else if (d != 0 && r >= 0 && r < a.N) {
                const int ry = r / a.nx, rx = r - ry * a.nx;
                if (rx >= x0 && rx < x0 + tw && ry >= y0 && ry < y0 + th) lp = (ry - y0) * TR_T + rx - x0;
            }
        }
        lpar[k] = (int16_t)lp;
        cnt[k] = cv[j];
        if (VAL) {
            lo[k] = (unsigned)(unsigned long long)tv[j];
            hi[k] = (unsigned)((unsigned long long)tv[j] >> 32);
        }
    }
    sync();
    const int per = tree_entries(a, tw, th);
    for (int e = t; e < per; e += TR_T0_THREADS) {
        int u = tree_entry(a, e, tw, th);
        const int gi = (y0 + (u >> 5)) * a.nx + x0 + (u & (TR_T - 1));
        if (!a.marker[gi]) continue;
        const unsigned ic = a.Inc0[gi];
        const unsigned long long iv = VAL ? (unsigned long long)a.In0[gi] : 0;
        for (int st = 0; st < TR_TC && u >= 0; ++st) {
            atomicAdd(&cnt[u], ic);
            if (VAL) {
                const unsigned old = atomicAdd(&lo[u], (unsigned)iv);
                atomicAdd(&hi[u], (unsigned)(iv >> 32) + (old + (unsigned)iv < old ? 1u : 0u));
            }
            u = lpar[u];
        }
    }
    sync();
#pragma unroll
    for (int j = 0; j < RPT; ++j) {
        const int k = t + j * TR_T0_THREADS, ly = ly0 + 8 * j;
        if (lx < tw && ly < th) {
            const int gi = (y0 + ly) * a.nx + x0 + lx;
            const unsigned c = cnt[k];
            if (Q) {
                const long long v = VAL ? (long long)(((unsigned long long)hi[k] << 32) | lo[k]) : cval * (long long)c;
                Q[gi] = from_fixed(v, s);
            }
            if (counts) counts[gi] = c;
        }
    }
}

template <bool VAL>
struct TreeTile {
    static constexpr int BYTES = TR_TC * 4 * (VAL ? 3 : 1) + TR_TC * 4 + 16;  // shared memory of a tile pass
};

// the shift of the fixed-point seeds
__device__ __forceinline__ int tree_shift(const TreeArgs &a, const float *w, float value)
{
    return fixed_shift(w ? (unsigned)vload(a.status + 1) : __float_as_uint(fabsf(value)), a.N);
}

template <bool VAL>
__global__ void __launch_bounds__(TR_T0_THREADS) k_tree_up(const int32_t *__restrict__ rcv, const float *__restrict__ w,
                                                           float value, TreeArgs a)
{
    __shared__ __align__(16) unsigned char sm[TreeTile<VAL>::BYTES];
    tree_tile_up<VAL>(a, rcv, w, tree_shift(a, w, value), blockIdx.x, sm, threadIdx.x, []() { __syncthreads(); });
}

template <bool VAL>
__global__ void __launch_bounds__(TR_T0_THREADS) k_tree_finish(const int32_t *__restrict__ rcv, const float *__restrict__ w,
                                                               float value, float *Q, unsigned *counts, TreeArgs a)
{
    __shared__ __align__(16) unsigned char sm[TreeTile<VAL>::BYTES];
    const int s = tree_shift(a, w, value);
    // the status is final since the passes before; after a problem Q keeps its seeds for the
    // caller's other path
    if (vload(a.status) == 0)
        tree_tile_finish<VAL>(a, rcv, s, w ? 0 : to_fixed(value, s), Q, counts, blockIdx.x, sm, threadIdx.x,
                              []() { __syncthreads(); });
    if (a.out && blockIdx.x == 0 && threadIdx.x == 0) {
        *(volatile int *)a.out = a.status[0];
        __threadfence_system();
    }
}

// ---- levels >= 1: one CTA per block -----------------------------------------------------------
// MODE 0 up (local totals, next-level nodes, up pointers), 1 down (totals with the
// inflows, scattered one level down), 2 top (up with no exits, then scattered).
template <int MODE, bool VAL>
__device__ __forceinline__ void tree_level(int L, const TreeArgs &a, int b, unsigned char *tsm)
{
    __shared__ int s_n, s_base, s_err;
    const TreeLevel &V = a.lv[L];
    const int bx = b % V.nbx, by = b / V.nbx;
    const BlockGeo g = block_geo(bx, by, V.side, a.ntx, a.nty);
    const int base = g.tile_off * a.cap0;
    const int n = min(V.cnt[b], g.tiles * a.cap0);  // appends past the capacity were refused and flagged
    if (n <= 0) return;
    unsigned *lo, *hi;  // totals as 32-bit halves
    unsigned *cnt;
    int *lpar, *jmp, *tn;
    const bool in_smem = n <= TR_SMEM_NODES;
    if (in_smem) {
        lo = (unsigned *)tsm;
        hi = lo + TR_SMEM_NODES;
        cnt = hi + TR_SMEM_NODES;
        lpar = (int *)(cnt + TR_SMEM_NODES);
        jmp = lpar + TR_SMEM_NODES;
        tn = jmp + TR_SMEM_NODES;
    } else {  // a block too large for shared memory works in its slice of the scratch
        lo = (unsigned *)a.scr_acc + base;  // scr_acc: 2 S unsigned
        hi = (unsigned *)a.scr_acc + a.slots + base;
        cnt = a.scr_cnt + base;
        lpar = a.scr_lpar + base;
        jmp = a.scr_pend + base;
        tn = a.scr_tn + base;
    }
    if (threadIdx.x == 0) { s_n = 0; s_err = 0; }
    for (int k = threadIdx.x; k < n; k += TR_LB_THREADS) {
        const int pos = base + k;
        int p;
        if (MODE == 1) {
            p = V.par[pos];
        } else {
            const int rp = V.rawpar[pos];
            if (rp < 0 || rp >= (L == 1 ? a.N : a.slots)) {
                atomicOr(&s_err, TR_ERR_RCV);
                p = -1;
            } else {
                p = L == 1 ? a.up0[rp] : a.lv[L - 1].up[rp];
            }
            if (p < -1 || p >= a.slots) {  // an entry that was never given a terminal (local = 1 violated)
                atomicOr(&s_err, TR_ERR_NONLOCAL);
                p = -1;
            }
            V.par[pos] = p;
        }
        const int lp = p < 0 ? -1 : (p >= base && p < base + n ? p - base : -3);
        lpar[k] = lp;
        jmp[k] = lp >= 0 ? lp : -1;
        unsigned long long sv = VAL ? (unsigned long long)V.W[pos] : 0;
        unsigned sc = V.C[pos];
        if (MODE == 1) {
            if (VAL) sv += (unsigned long long)V.In[pos];
            sc += V.Inc[pos];
        } else {
            if (VAL) V.In[pos] = 0;
            V.Inc[pos] = 0;
        }
        if (VAL) {
            lo[k] = (unsigned)sv;
            hi[k] = (unsigned)(sv >> 32);
        }
        cnt[k] = sc;
    }
    __syncthreads();
    int rounds = 1;
    while ((1 << rounds) < n) ++rounds;
    bool ok;
    if (in_smem) {
        ok = doubling_rounds<TR_SMEM_NODES / TR_LB_THREADS, TR_LB_THREADS, VAL>(n, jmp, lo, hi, cnt, rounds + 1);
    } else {
        // the same rounds with the start-of-round values in a second scratch (tn holds the next pointers)
        ok = true;
        for (int r = 0;; ++r) {
            bool live = false;
            for (int k = threadIdx.x; k < n; k += TR_LB_THREADS) {
                const int j = jmp[k];
                tn[k] = j >= 0 ? jmp[j] : -1;
                live |= j >= 0;
            }
            if (!__syncthreads_or(live)) break;
            if (r > rounds) { ok = false; break; }
            for (int k = threadIdx.x; k < n; k += TR_LB_THREADS) {  // start-of-round snapshot
                const int j = jmp[k];
                if (j >= 0) {
                    if (VAL) a.scr_acc2[base + k] = (long long)(((unsigned long long)hi[k] << 32) | lo[k]);
                    a.scr_cnt2[base + k] = cnt[k];
                }
            }
            __syncthreads();
            for (int k = threadIdx.x; k < n; k += TR_LB_THREADS) {
                const int j = jmp[k];
                if (j >= 0) {
                    if (VAL) {
                        const unsigned long long x = (unsigned long long)a.scr_acc2[base + k];
                        const unsigned old = atomicAdd(&lo[j], (unsigned)x);
                        atomicAdd(&hi[j], (unsigned)(x >> 32) + (old + (unsigned)x < old ? 1u : 0u));
                    }
                    atomicAdd(&cnt[j], a.scr_cnt2[base + k]);
                }
            }
            __syncthreads();
            for (int k = threadIdx.x; k < n; k += TR_LB_THREADS) jmp[k] = tn[k];
            __syncthreads();
        }
    }
    if (!ok && threadIdx.x == 0) s_err |= TR_ERR_CYCLE;
    __syncthreads();

    if (MODE != 0) {
        // every node of this level drains into a node one level down (in another
        // block of that level): add its total to that node's inflow
        for (int k = threadIdx.x; k < n; k += TR_LB_THREADS) {
            const int pos = base + k;
            if (L == 1) {
                const int cell = V.rawpar[pos];
                if (cell < 0 || cell >= a.N) continue;  // flagged in the up pass
                if (VAL) atomicAdd((unsigned long long *)&a.In0[cell], ((unsigned long long)hi[k] << 32) | lo[k]);
                atomicAdd(&a.Inc0[cell], cnt[k]);
            } else {
                const TreeLevel &D = a.lv[L - 1];
                const int sp = V.src[pos];
                const int t = (sp >= 0 && sp < a.slots) ? D.par[sp] : -1;
                if (t < 0 || t >= a.slots) continue;
                if (VAL) atomicAdd((unsigned long long *)&D.In[t], ((unsigned long long)hi[k] << 32) | lo[k]);
                atomicAdd(&D.Inc[t], cnt[k]);
            }
        }
        __syncthreads();
        if (threadIdx.x == 0 && s_err) atomicOr(&a.status[0], s_err);
        return;
    }

    // up: block terminals, then the exits become nodes of the next level
    for (int k = threadIdx.x; k < n; k += TR_LB_THREADS) tn[k] = lpar[k] >= 0 ? lpar[k] : k;
    __syncthreads();
    for (int r = 0; r <= rounds; ++r) {
        bool ch = false;
        for (int k = threadIdx.x; k < n; k += TR_LB_THREADS) {
            const int t = tn[k], tt = tn[t];
            if (tt != t) { tn[k] = tt; ch = true; }
        }
        if (!__syncthreads_or(ch)) break;
    }
    const TreeLevel &U = a.lv[L + 1];
    const int ubx = bx / 2, uby = by / 2;
    const int ub = uby * U.nbx + ubx;
    const BlockGeo ug = block_geo(ubx, uby, U.side, a.ntx, a.nty);
    int mine = 0;
    for (int k = threadIdx.x; k < n; k += TR_LB_THREADS) mine += lpar[k] == -3;
    for (int o = 16; o; o >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, o);
    if ((threadIdx.x & 31) == 0 && mine) atomicAdd(&s_n, mine);
    __syncthreads();
    if (threadIdx.x == 0) {
        s_base = s_n ? atomicAdd(&U.cnt[ub], s_n) : 0;
        if (s_base + s_n > ug.tiles * a.cap0) { s_err |= TR_ERR_CAP; s_n = -1; }
        s_n = s_n < 0 ? -1 : 0;
    }
    __syncthreads();
    const int slot0 = ug.tile_off * a.cap0 + s_base;
    for (int k = threadIdx.x; k < n; k += TR_LB_THREADS) {
        int q = -1;
        if (lpar[k] == -3 && s_n >= 0) {
            const int pos = base + k;
            q = slot0 + atomicAdd(&s_n, 1);
            if (VAL) U.W[q] = (long long)(((unsigned long long)hi[k] << 32) | lo[k]);
            U.C[q] = cnt[k];
            U.rawpar[q] = V.par[pos];
            U.src[q] = pos;
        }
        jmp[k] = q;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < n; k += TR_LB_THREADS) {
        const int t = tn[k];
        V.up[base + k] = lpar[t] == -3 ? jmp[t] : -1;
    }
    if (threadIdx.x == 0 && s_err) atomicOr(&a.status[0], s_err);
}

template <int MODE, bool VAL>
__global__ void __launch_bounds__(TR_LB_THREADS) k_tree_level(int L, TreeArgs a)
{
    extern __shared__ __align__(16) unsigned char tsm[];
    tree_level<MODE, VAL>(L, a, blockIdx.x, tsm);
}

// The whole accumulation in one cooperative launch, a grid barrier between the passes, for
// grids whose passes are shorter than their launches: at 512 x 512 the seven launches,
// four memsets and the status read took 64 us of device time and 111 us in all.  Larger
// grids take the separate launches, whose tile passes hold twice the threads per SM.
template <bool VAL>
__global__ void __launch_bounds__(TR_LB_THREADS, 1) k_tree_all(const int32_t *__restrict__ rcv, const float *__restrict__ w,
                                                               float value, float *Q, unsigned *counts, TreeArgs a)
{
    extern __shared__ __align__(16) unsigned char tsm[];
    __shared__ int dead;
    const int gtid = blockIdx.x * TR_LB_THREADS + threadIdx.x, gthreads = gridDim.x * TR_LB_THREADS;
    const int grp = threadIdx.x / TR_T0_THREADS, gt = threadIdx.x & (TR_T0_THREADS - 1);
    constexpr int ngrp = TR_LB_THREADS / TR_T0_THREADS;
    if (threadIdx.x == 0) dead = 0;
    if (gridDim.x == 1)  // one block clears its counters itself
        for (int k = threadIdx.x; k < a.nzero; k += TR_LB_THREADS) a.status[k] = 0;
    GridBar bar{a.status + 8, a.wait};
    __syncthreads();
    if (((uintptr_t)a.marker & 15) == 0) {
        for (int k = gtid; k < (a.N + 15) / 16; k += gthreads)  // the array is padded to 256 bytes
            reinterpret_cast<uint4 *>(a.marker)[k] = make_uint4(0, 0, 0, 0);
    } else {
        for (int k = gtid; k < a.N; k += gthreads) a.marker[k] = 0;
    }
    if (VAL) tree_seedmax(w, a.N, a.status);
    if (!bar.sync(&dead)) return;
    const int s = tree_shift(a, w, value), ntiles = a.ntx * a.nty;
    auto gsync = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(grp + 1), "n"(TR_T0_THREADS) : "memory"); };
    unsigned char *gsm = tsm + grp * ((TreeTile<VAL>::BYTES + 15) / 16 * 16);
    for (int k = grp * gridDim.x + blockIdx.x; k < ntiles; k += ngrp * gridDim.x) {
        tree_tile_up<VAL>(a, rcv, w, s, k, gsm, gt, gsync);
        gsync();
    }
    if (!bar.sync(&dead)) return;
    for (int L = 1; L < a.nlev; ++L) {
        for (int b = blockIdx.x; b < a.lv[L].nbx * a.lv[L].nby; b += gridDim.x) {
            tree_level<0, VAL>(L, a, b, tsm);
            __syncthreads();
        }
        if (!bar.sync(&dead)) return;
    }
    if (blockIdx.x == 0) tree_level<2, VAL>(a.nlev, a, 0, tsm);
    if (!bar.sync(&dead)) return;
    for (int L = a.nlev - 1; L >= 1; --L) {
        for (int b = blockIdx.x; b < a.lv[L].nbx * a.lv[L].nby; b += gridDim.x) {
            tree_level<1, VAL>(L, a, b, tsm);
            __syncthreads();
        }
        if (!bar.sync(&dead)) return;
    }
    const long long cval = w ? 0 : to_fixed(value, s);
    const int n = vload(a.status) == 0 ? ntiles : 0;  // after a problem Q keeps its seeds
    for (int k = grp * gridDim.x + blockIdx.x; k < n; k += ngrp * gridDim.x) {
        tree_tile_finish<VAL>(a, rcv, s, cval, Q, counts, k, gsm, gt, gsync);
        gsync();
    }
    if (a.out && gtid == 0) {
        *(volatile int *)a.out = vload(a.status);
        __threadfence_system();
    }
}

// ---- host --------------------------------------------------------------------------------------
struct TreePlan {
    int ntx, nty, ntiles, nlev, cap0;
    long long slots;
    int nb[TR_MAXLEV + 1], nbx[TR_MAXLEV + 1], nby[TR_MAXLEV + 1], side[TR_MAXLEV + 1];
};

static TreePlan tree_plan(int nx, int ny, int local)
{
    TreePlan p{};
    p.ntx = (nx + TR_T - 1) / TR_T;
    p.nty = (ny + TR_T - 1) / TR_T;
    p.ntiles = p.ntx * p.nty;
    p.cap0 = local ? 128 : 256;
    p.slots = (long long)p.ntiles * p.cap0;
    int side = TR_S1, L = 1;
    for (;;) {
        p.side[L] = side;
        p.nbx[L] = (p.ntx + side - 1) / side;
        p.nby[L] = (p.nty + side - 1) / side;
        p.nb[L] = p.nbx[L] * p.nby[L];
        if (p.nb[L] == 1 || L == TR_MAXLEV - 1) break;
        side *= 2;
        ++L;
    }
    p.nlev = L;
    return p;
}

// The workspace's layout; a.status and the levels' counts are contiguous.
static TreeArgs tree_carve(const TreePlan &p, int nx, int ny, int local, void *workspace, size_t bytes, size_t *used)
{
    Carver cv(workspace, bytes);
    const int N = nx * ny;
    TreeArgs a{};
    a.nx = nx; a.ny = ny; a.ntx = p.ntx; a.nty = p.nty; a.N = N;
    a.cap0 = p.cap0; a.nlev = p.nlev; a.local = local ? 1 : 0;
    a.slots = (int)p.slots;
    a.marker = cv.take<unsigned char>(N);
    a.In0 = cv.take<long long>(N);
    a.T0 = cv.take<long long>(N);
    a.Inc0 = cv.take<unsigned>(N);
    a.C0 = cv.take<unsigned>(N);
    a.up0 = cv.take<int>(N);
    a.nzero = 64;
    for (int L = 1; L <= p.nlev; ++L) a.nzero += p.nb[L];
    a.status = cv.take<int>(a.nzero);
    const size_t S = (size_t)p.slots;
    a.scr_acc = cv.take<long long>(S);
    a.scr_cnt = cv.take<unsigned>(S);
    a.scr_lpar = cv.take<int>(S);
    a.scr_pend = cv.take<int>(S);
    a.scr_tn = cv.take<int>(S);
    a.scr_acc2 = cv.take<long long>(S);
    a.scr_cnt2 = cv.take<unsigned>(S);
    int *cnt = a.status ? a.status + 64 : nullptr;
    for (int L = 1; L <= p.nlev; ++L) {
        TreeLevel &V = a.lv[L];
        V.W = cv.take<long long>(S);
        V.In = cv.take<long long>(S);
        V.C = cv.take<unsigned>(S);
        V.Inc = cv.take<unsigned>(S);
        V.rawpar = cv.take<int>(S);
        V.par = cv.take<int>(S);
        V.up = cv.take<int>(S);
        V.src = cv.take<int>(S);
        V.cnt = cnt;
        if (cnt) cnt += p.nb[L];
        V.side = p.side[L];
        V.nbx = p.nbx[L];
        V.nby = p.nby[L];
    }
    // the top level's exits would go to level nlev+1: there are none (one block)
    a.lv[p.nlev + 1] = a.lv[p.nlev];
    if (used) *used = cv.off;
    return a;
}

static size_t tree_bytes(const TreePlan &p, int nx, int ny)
{
    size_t used = 0;
    tree_carve(p, nx, ny, 1, nullptr, 0, &used);
    return used + 4096;
}

template <bool VAL>
static int launch_tree(const TreePlan &p, const TreeArgs &a_, const int32_t *receivers, const float *weights, float value,
                       float *Q, uint32_t *counts, cudaStream_t st)
{
    TreeArgs a = a_;
    a.wait = bar_wait(BAR_TREE);
    int dev = 0, nsm = 148, coop = 0;
    PFF_CUDA(cudaGetDevice(&dev));
    PFF_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    PFF_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
    const size_t smem = (size_t)TR_SMEM_NODES * TR_NODE_BYTES;  // per-device attribute: set on every call
    if (coop && p.ntiles <= TR_ALL_TILES * nsm) {
        // a block has room for 4 tiles at a time, but tiles on SMs of their own are faster
        const int blocks = p.ntiles <= TR_LB_THREADS / TR_T0_THREADS ? 1 : std::min(nsm, p.ntiles);
        if (blocks > 1) PFF_CUDA(cudaMemsetAsync(a.status, 0, sizeof(int) * (size_t)a.nzero, st));
        PFF_CUDA(cudaFuncSetAttribute(k_tree_all<VAL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        void *args[] = {(void *)&receivers, (void *)&weights, &value, &Q, &counts, &a};
        PFF_CUDA(cudaLaunchCooperativeKernel((void *)k_tree_all<VAL>, blocks, TR_LB_THREADS, args, smem, st));
        count_launch();
        return check_cuda("pff_accumulate_tree");
    }
    PFF_CUDA(cudaMemsetAsync(a.marker, 0, (size_t)a.N, st));
    PFF_CUDA(cudaMemsetAsync(a.status, 0, sizeof(int) * (size_t)a.nzero, st));
    if (VAL) {
        const int grid = std::min(div_up(a.N, 256), nsm * 8);
        { k_tree_seedmax<<<grid, 256, 0, st>>>(weights, a.N, a.status); count_launch(); }
    }
    PFF_CUDA(cudaFuncSetAttribute(k_tree_level<0, VAL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    PFF_CUDA(cudaFuncSetAttribute(k_tree_level<1, VAL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    PFF_CUDA(cudaFuncSetAttribute(k_tree_level<2, VAL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    PFF_PROBED("k_tree_tile<up>", st, k_tree_up<VAL><<<p.ntiles, TR_T0_THREADS, 0, st>>>(receivers, weights, value, a));
    count_launch();
    for (int L = 1; L < p.nlev; ++L) {
        k_tree_level<0, VAL><<<p.nb[L], TR_LB_THREADS, smem, st>>>(L, a);
        count_launch();
    }
    { k_tree_level<2, VAL><<<1, TR_LB_THREADS, smem, st>>>(p.nlev, a); count_launch(); }
    for (int L = p.nlev - 1; L >= 1; --L) {
        k_tree_level<1, VAL><<<p.nb[L], TR_LB_THREADS, smem, st>>>(L, a);
        count_launch();
    }
    PFF_PROBED("k_tree_tile<down>", st,
               k_tree_finish<VAL><<<p.ntiles, TR_T0_THREADS, 0, st>>>(receivers, weights, value, Q, counts, a));
    count_launch();
    return check_cuda("pff_accumulate_tree");
}

static int accumulate_tree(const int32_t *receivers, const float *weights, float value, float *Q, uint32_t *counts, int nx,
                           int ny, int local, void *workspace, size_t workspace_bytes, int *out, cudaStream_t st)
{
    if (nx < 1 || ny < 1 || (long long)nx * ny > (1LL << 30) || !receivers || (!Q && !counts)) {
        set_error("pff_accumulate_tree: bad arguments");
        return PFF_ERR_ARG;
    }
    const TreePlan p = tree_plan(nx, ny, local);
    if (!workspace || workspace_bytes < tree_bytes(p, nx, ny)) {
        set_error("pff_accumulate_tree: workspace too small");
        return PFF_ERR_WORKSPACE;
    }
    if (!weights && !(fabsf(value) <= 3.4028235e38f)) {
        set_error("pff_accumulate_tree: non-finite seed value");
        return PFF_ERR_ARG;
    }
    TreeArgs a = tree_carve(p, nx, ny, local, workspace, workspace_bytes, nullptr);
    a.out = out;
    return weights ? launch_tree<true>(p, a, receivers, weights, value, Q, counts, st)
                   : launch_tree<false>(p, a, receivers, weights, value, Q, counts, st);
}

}  // namespace pff

using namespace pff;

extern "C" size_t pff_accumulate_tree_workspace_bytes(int nx, int ny, int local)
{
    if (nx < 1 || ny < 1 || (long long)nx * ny > (1LL << 30)) return 0;
    return tree_bytes(tree_plan(nx, ny, local), nx, ny);
}

extern "C" int pff_accumulate_tree(const int32_t *receivers, const float *weights, float value, float *Q,
                                   uint32_t *counts, int nx, int ny, int local, void *workspace,
                                   size_t workspace_bytes, void *stream)
{
    clear_error();
    return accumulate_tree(receivers, weights, value, Q, counts, nx, ny, local, workspace, workspace_bytes, nullptr,
                           S(stream));
}

extern "C" int pff_accumulate_tree_run(const int32_t *receivers, const float *weights, float value, float *Q,
                                       uint32_t *counts, int nx, int ny, int local, void *workspace,
                                       size_t workspace_bytes, int *status, void *stream)
{
    clear_error();
    if (!status) {
        set_error("pff_accumulate_tree_run: null pointer");
        return PFF_ERR_ARG;
    }
    int *host = nullptr, *dptr = nullptr;
    PFF_TRY(pinned_ints(&host, &dptr));
    host[0] = -1;
    PFF_TRY(accumulate_tree(receivers, weights, value, Q, counts, nx, ny, local, workspace, workspace_bytes, dptr,
                            S(stream)));
    PFF_CUDA(cudaStreamSynchronize(S(stream)));
    PFF_TRY(check_cuda("pff_accumulate_tree_run"));
    *status = *(volatile int *)host;
    if (*status < 0) {
        set_error("pff_accumulate_tree_run: the passes did not end");
        return PFF_ERR_NOCONV;
    }
    return PFF_OK;
}

extern "C" int pff_accumulate_tree_status(int nx, int ny, int local, void *workspace, size_t workspace_bytes,
                                          int *status, void *stream)
{
    clear_error();
    if (!status || nx < 1 || ny < 1) {
        set_error("pff_accumulate_tree_status: bad arguments");
        return PFF_ERR_ARG;
    }
    const TreePlan p = tree_plan(nx, ny, local);
    if (!workspace || workspace_bytes < tree_bytes(p, nx, ny)) {
        set_error("pff_accumulate_tree_status: workspace too small");
        return PFF_ERR_WORKSPACE;
    }
    const TreeArgs a = tree_carve(p, nx, ny, local, workspace, workspace_bytes, nullptr);
    int words[2] = {0, 0};
    PFF_TRY(read_ints(IntReads().add(a.status, 1).add(a.status + 8, 1), words, S(stream)));
    if (words[1] & BAR_HALT) {
        set_error("pff_accumulate_tree_status: the passes did not end");
        return PFF_ERR_NOCONV;
    }
    *status = words[0];
    return PFF_OK;
}
