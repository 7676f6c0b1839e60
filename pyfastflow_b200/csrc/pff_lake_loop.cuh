// The carve reroute's outer loop (lakeflow.py:498-538) as one persistent cooperative
// kernel, and the same loop for the tiles of a ragged batch (pff_batch.cu).
//
// What bounds it: latency.  One outer iteration is about ten dependent steps over
// lists (border cells, pits, path segments, touched tiles) that shrink by 2-3x per
// iteration.  As separate kernels in a device-driven graph an iteration cost about 27
// launches of 2 us and their gaps (135-140 us per iteration at 1001 x 777, of which
// the work was a third).  Here a step ends with a grid barrier (about 1 us over 148
// blocks; __syncthreads alone when one block is enough) and every block takes the loop's
// decisions itself from counters it reads after the barrier.
//
// Nothing is N-wide after the first saddle pass:
//   - labels are not rewritten between iterations: the current label of a cell is
//     fin[bid[i]], with fin brought up to date once per iteration over the first pit list;
//   - the receivers' second copy rec_, the carve tags and the tile terminals J are
//     brought up to date over the tiles the carve touched.
// One block of 1024 threads per SM: the barrier's cost grows with the number of
// blocks, and 32 warps hide the gathers of the list steps.
#pragma once
#include "pff_common.cuh"
#include "pff_coop.cuh"
#include "pff_tiles.cuh"

namespace pff {

__device__ __forceinline__ long long invalid_key() { return pack_key(1e8f, 42); }  // lakeflow.py:127


// Exact quotient and remainder of n / d for 0 <= n < 2^31 and d >= 2 without the
// integer divide sequence: with m = floor(2^32 / d) or m = floor((2^32 - 1) / d) (one
// less only when d divides 2^32), q = umulhi(n, m) is floor(n / d) or one less
// (n m / 2^32 > n / d - 2 n / 2^32 > n / d - 1), and one correction of the remainder
// fixes it.
__device__ __forceinline__ void divmod_nx(int n, int d, unsigned m, int &q, int &r)
{
    q = (int)__umulhi((unsigned)n, m);
    r = n - q * d;
    if (r >= d) { ++q; r -= d; }
}

// Tile-local indices q of a thread's receivers r (its cells: rows ly0 + 4 k of column lx of
// the w x h tile at (row0, col0), local index t + 256 k, grid index i0 + 4 k nx; r < 0: no
// cell): the receiver's, or the cell's own where it is a root or its receiver lies outside.
// True if some receiver outside is not a tile-border cell (a receiver one column or row away
// always is one).
__device__ __forceinline__ bool tile_locals(const int (&r)[TILE_PER_THREAD], int (&q)[TILE_PER_THREAD], int i0, int t,
                                            int lx, int ly0, int row0, int col0, int w, int h, int nx, int ny,
                                            unsigned mnx)
{
    static_assert(TILE_THREADS == 4 * TILE_W, "a thread's cells are 4 rows apart");
    int far = 0;  // receivers that are not the grid neighbour (wrapped edges, or no D4 link)
#pragma unroll
    for (int k = 0; k < TILE_PER_THREAD; ++k) {
        const int c = t + k * TILE_THREADS, d = r[k] - (i0 + 4 * k * nx);
        const int sx = (d == 1) - (d == -1), sy = (d == nx) - (d == -nx);
        const bool in = r[k] >= 0 && (unsigned)(lx + sx) < (unsigned)w && (unsigned)(ly0 + 4 * k + sy) < (unsigned)h;
        q[k] = in ? c + sx + TILE_W * sy : c;
        if (r[k] >= 0 && d != 0 && (sx | sy) == 0) far |= 1 << k;
    }
    bool nonlocal = false;
    if (!far) return nonlocal;
#pragma unroll
    for (int k = 0; k < TILE_PER_THREAD; ++k) {
        if (!(far >> k & 1)) continue;
        int rr, rc;
        divmod_nx(r[k], nx, mnx, rr, rc);
        if (rr >= row0 && rr < row0 + h && rc >= col0 && rc < col0 + w) q[k] = (rr - row0) * TILE_W + rc - col0;
        else if (!is_tile_border(nx, ny, rr, rc)) nonlocal = true;
    }
    return nonlocal;
}

// A thread's 8 pointers q to their tile terminals.  Four rounds of pointer doubling in p
// (16-bit local pointers; a pointer then spans 16 cells or ends), then every pointer is
// followed on its own over the settled array, without barriers: most paths in a tile
// are shorter than 64 cells.  At most 2048 / 16 steps; true if a pointer is then still
// moving (a cycle).
// Bound by the shared-memory gathers' latency and bank conflicts.
template <class Sync>
__device__ __forceinline__ bool tile_jump(uint16_t *p, int (&q)[TILE_PER_THREAD], int t, Sync sync)
{
    int qq[TILE_PER_THREAD];
    unsigned act = (1u << TILE_PER_THREAD) - 1;  // pointers not known to be terminals
#pragma unroll 1
    for (int round = 0; round < 4; ++round) {
#pragma unroll
        for (int k = 0; k < TILE_PER_THREAD; ++k)
            if (act >> k & 1) qq[k] = p[q[k]];
#pragma unroll
        for (int k = 0; k < TILE_PER_THREAD; ++k)
            if (act >> k & 1) {
                if (qq[k] != q[k]) {
                    p[t + k * TILE_THREADS] = (uint16_t)qq[k];
                    q[k] = qq[k];
                } else {
                    act &= ~(1u << k);
                }
            }
        sync();
    }
#pragma unroll 1
    for (int step = 0; act && step < TILE_CELLS / 16 + 1; ++step) {
#pragma unroll
        for (int k = 0; k < TILE_PER_THREAD; ++k)
            if (act >> k & 1) qq[k] = p[q[k]];
#pragma unroll
        for (int k = 0; k < TILE_PER_THREAD; ++k)
            if (act >> k & 1) {
                if (qq[k] == q[k]) act &= ~(1u << k);
                q[k] = qq[k];
            }
    }
    return act != 0;
}

// Tile terminals of one tile by a group of 256 threads (t: thread of the group): J[i] = the receiver of the last in-tile cell of
// i's path (the root itself, or the first cell past the tile).  info[0] pits (pits ==
// nullptr: no pit list), info[2] set if some exit target is not a tile-border cell
// (receivers that are not D4 neighbours).  copy: also rec_copy = rec.
//
template <int MODE, class Sync>
__device__ __forceinline__ void tile_terminal_one(const int32_t *rec, int32_t *J, int32_t *R, int *pits, int *info,
                                                  const Grid &g, int tx, int ty, uint16_t *p, int *rv,
                                                  int32_t *rec_copy, int t, Sync sync)
{
    const int nx = g.nx, ny = g.ny;
    const unsigned mnx = 0xffffffffu / (unsigned)nx;
    const int col0 = tx * TILE_W, row0 = ty * TILE_H;
    const int w = min(TILE_W, nx - col0), h = min(TILE_H, ny - row0);
    const int lx = t & (TILE_W - 1), ly0 = t / TILE_W;
    const int i0 = (row0 + ly0) * nx + col0 + lx;
    int r[TILE_PER_THREAD], q[TILE_PER_THREAD];
#pragma unroll
    for (int k = 0; k < TILE_PER_THREAD; ++k) r[k] = (lx < w && ly0 + 4 * k < h) ? rec[i0 + 4 * k * nx] : -1;
    bool nonlocal = tile_locals(r, q, i0, t, lx, ly0, row0, col0, w, h, nx, ny, mnx);
    int term = 0;  // cells that are terminals
#pragma unroll
    for (int k = 0; k < TILE_PER_THREAD; ++k) {
        const int c = t + k * TILE_THREADS;
        p[c] = (uint16_t)q[k];
        rv[c] = r[k];
        if (q[k] == c) term |= 1 << k;
        if (rec_copy && r[k] >= 0) rec_copy[i0 + 4 * k * nx] = r[k];
    }
    sync();
    nonlocal |= tile_jump(p, q, t, sync);
    // a tile off the grid's rim has no cell that can leave (modes 0-2)
    const bool rim = MODE == 3 || row0 == 0 || col0 == 0 || row0 + h == ny || col0 + w == nx;
#pragma unroll
    for (int k = 0; k < TILE_PER_THREAD; ++k) {
        const int c = t + k * TILE_THREADS, ly = ly0 + 4 * k, i = i0 + 4 * k * nx;
        bool pit = false;
        if (r[k] >= 0) {
            const int j = rv[q[k]];
            J[i] = j;
            if (lx == 0 || ly == 0 || lx == w - 1 || ly == h - 1 || r[k] == i) R[i] = j;
            if (q[k] == c && !(term >> k & 1)) nonlocal = true;  // a cycle in the tile
            pit = pits && r[k] == i;
            if (rim && pit) pit = !can_leave<MODE>(g, i, row0 + ly, col0 + lx);
        }
        const unsigned m = __ballot_sync(0xffffffffu, pit);
        if (m) {
            const int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
            int base = 0;
            if (lane == leader) base = atomicAdd(info, __popc(m));
            base = __shfl_sync(0xffffffffu, base, leader);
            if (pit) pits[base + __popc(m & ((1u << lane) - 1u))] = i;
        }
    }
    if (nonlocal) info[2] = 1;
}

// The saddle candidate of a border cell goes to atomicMin(saddle + bi, key) (pass 2).
// In the border-list pass, where most lanes hold a candidate and neighbouring list
// entries share basins, saddle_min_warp makes that one atomic per basin per warp
// (in the N-wide strip pass it cost more than it saved): the lanes holding a
// candidate group by basin (match.any), take the group's minimum key as two 32-bit
// reductions (the key's signed order is the unsigned order of key ^ 2^63: high
// words first, then the low words of the lanes that hold the minimal high word),
// and the group's first lane applies it.  The minimum over the same keys: the
// saddle is the one the per-cell atomics produce.
__device__ __forceinline__ void saddle_min_warp(long long *saddle, int bi, long long key, bool has)
{
    const unsigned act = __ballot_sync(0xffffffffu, has);
    if (!has) return;
    const unsigned peers = __match_any_sync(act, bi);
    const unsigned long long u = (unsigned long long)key ^ 0x8000000000000000ull;
    const unsigned hi = (unsigned)(u >> 32), lo = (unsigned)u;
    const unsigned mh = __reduce_min_sync(peers, hi);
    const unsigned ml = __reduce_min_sync(peers, hi == mh ? lo : 0xffffffffu);
    if ((int)(threadIdx.x & 31) == __ffs(peers) - 1)
        atomicMin(saddle + bi, (long long)((((unsigned long long)mh << 32) | ml) ^ 0x8000000000000000ull));
}

// Passes 1-2 for one cell; key: the lowest (z', neighbour basin) of a border cell (a
// saddle candidate if below the invalid key).  Returns 0 for a cell off every
// border, 1 for a border cell of the outlet basin 0, 2 for a border cell of a pit basin.
template <bool WRITE = true>
__device__ __forceinline__ int saddle_cell(int i, int bi, float zi, const int (&jn)[4], const int (&bn)[4],
                                           const float (&zn)[4], uint8_t *is_border, float *zp, long long &key)
{
    bool border = false;
    float zmin = 1e9f;
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if (jn[k] != -1 && bn[k] != bi) { border = true; zmin = fminf(zmin, zn[k]); }
    if (WRITE) is_border[i] = border;
    const float zpi = border ? fmaxf(zi, zmin) : 1e9f;
    if (WRITE) zp[i] = zpi;
    if (!border) return 0;
    long long res = 0x7fffffffffffffffll;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (jn[k] == -1 || bn[k] == bi) continue;
        const long long c = pack_key(zpi, bn[k]);
        res = c < res ? c : res;
    }
    key = res;
    return bi != 0 ? 2 : 1;
}

// how the loop ended (final state words: [0] iteration, [1] outer, [2] n_outer, [3] state)
enum { RR_RUN = 0, RR_NOPITS = 1, RR_DONE = 2, RR_GENERAL = 3, RR_RESUME = 4, RR_WALKERR = 5, RR_BOUND = 6 };

__device__ __forceinline__ int d_ceil_log2(long long n)
{
    int r = 0;
    long long p = 1;
    while (p < n) { p <<= 1; ++r; }
    return r;
}

constexpr int LOOP_THREADS = 1024;              // threads of a block (the batch also runs it with 256 and 512)
constexpr int LOOP_CAP = 128;                   // list entries buffered per warp
constexpr int LOOP_ITS = 33, LOOP_CTR = 40;     // per-iteration counter slots (outer <= 32)
constexpr int LOOP_JUMPS = 16;                  // label jump rounds (8 links each: chains up to 9^16)
enum { LC_NP = 0, LC_NA = 1, LC_NSEG = 2, LC_NDIRTY = 3, LC_ODD = 4, LC_FLAG = 8 };  // in an iteration's slots
constexpr int LOOP_GROUP_BYTES = LOOP_CAP * 16 * 8;  // per 256 threads: 8 warps' border-list entries of 16 B
constexpr int LOOP_SMEM = LOOP_THREADS / TILE_THREADS * LOOP_GROUP_BYTES;
static_assert(LOOP_GROUP_BYTES >= TILE_CELLS * 6, "a tile pass uses its group's memory");

// The blocks that work on one grid.  All blocks of a cooperative launch:
struct GridTeam {
    GridBar bar;
    int *dead;
    __device__ __forceinline__ int rank() const { return blockIdx.x; }
    __device__ __forceinline__ int size() const { return gridDim.x; }
    __device__ __forceinline__ bool sync() { return bar.sync(dead); }
};
// The blocks of a cluster (resident together by construction):
struct ClusterTeam {
    int r, n;
    __device__ __forceinline__ int rank() const { return r; }
    __device__ __forceinline__ int size() const { return n; }
    __device__ __forceinline__ bool sync()
    {
        if (n == 1) {
            __syncthreads();
        } else {
            asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        }
        return true;
    }
};

struct LoopArgs {
    int32_t *bid, *rec, *rec_, *J;
    const float *z;
    float *zp;
    uint8_t *isb;
    long long *sad, *out;
    int32_t *snode;
    uint8_t *tag, *tag_;
    uint8_t *inv;
    int32_t *fin, *nf;
    int *pit0, *pits[2];   // the first pit list; those of later iterations: [(it - it0) & 1]
    int *alist[2];         // border cells (the first list marks pit-basin cells by the sign bit)
    int *abid;             // later lists: a border cell's label,
    long long *akey;       // and its lowest (z', neighbour basin) key
    int *segs, *dirty, *dtiles;
    int *it_ctr;           // LOOP_ITS x LOOP_CTR counters, zeroed before the prologue
    int *info;             // prologue: [0] pits, [2] non-D4 receivers, [4] unresolved labels, [5] no labels
    int *ctl, *ctl_out;    // final state words (RR_*), and the caller's copy
    int *bar;              // barrier arrivals
    BarWait wait, labels_wait;
    Grid g;
};

__device__ __forceinline__ void group_sync(int id) { asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(TILE_THREADS) : "memory"); }
__device__ __forceinline__ bool group_or(int id, bool p)
{
    int r;
    asm volatile("{\n .reg .pred p, q;\n setp.ne.s32 p, %1, 0;\n bar.red.or.pred q, %2, %3, p;\n selp.s32 %0, 1, 0, q;\n}\n"
                 : "=r"(r)
                 : "r"((int)p), "r"(id), "n"(TILE_THREADS)
                 : "memory");
    return r != 0;
}

__device__ __forceinline__ void loop_mark(const LoopArgs &A, int *nd, int tile)
{
    if (vload(A.dirty + tile) == 0 && atomicExch(A.dirty + tile, 1) == 0) A.dtiles[atomicAdd(nd, 1)] = tile;
}

struct TileXY {
    int ntx;
    unsigned mnx;
    int nx;
    __device__ __forceinline__ int of(int i) const
    {
        int row, col;
        divmod_nx(i, nx, mnx, row, col);
        return row / TILE_H * ntx + col / TILE_W;
    }
};

// Bring a touched tile up to date: rec_ = rec (and, going on, the tags cleared: the
// tagged cells are those whose receiver the carve changed), and its tile terminals.
__device__ __forceinline__ void loop_tile(const LoopArgs &A, int tile, int ntx, unsigned mnx, int t, int bar_id,
                                          unsigned char *smem, bool go_on)
{
    uint16_t *p = reinterpret_cast<uint16_t *>(smem);
    int *rv = reinterpret_cast<int *>(smem + 2 * TILE_CELLS);
    const int nx = A.g.nx, ny = A.g.ny;
    const int ty = tile / ntx, tx = tile - ty * ntx;
    const int row0 = ty * TILE_H, col0 = tx * TILE_W;
    const int w = min(TILE_W, nx - col0), h = min(TILE_H, ny - row0);
    const int lx = t & (TILE_W - 1), ly0 = t / TILE_W;
    const int i0 = (row0 + ly0) * nx + col0 + lx;
    int r[TILE_PER_THREAD], o[TILE_PER_THREAD];
#pragma unroll
    for (int k = 0; k < TILE_PER_THREAD; ++k) {
        const bool in = lx < w && ly0 + 4 * k < h;
        r[k] = in ? A.rec[i0 + 4 * k * nx] : -1;
        o[k] = in ? A.rec_[i0 + 4 * k * nx] : -1;
    }
#pragma unroll
    for (int k = 0; k < TILE_PER_THREAD; ++k)
        if (r[k] != o[k]) {
            const int i = i0 + 4 * k * nx;
            A.rec_[i] = r[k];
            if (go_on) A.tag[i] = A.tag_[i] = 0;
        }
    if (!go_on) return;
    int q[TILE_PER_THREAD];
    tile_locals(r, q, i0, t, lx, ly0, row0, col0, w, h, nx, ny, mnx);
#pragma unroll
    for (int k = 0; k < TILE_PER_THREAD; ++k) {
        p[t + k * TILE_THREADS] = (uint16_t)q[k];
        rv[t + k * TILE_THREADS] = r[k];
    }
    group_sync(bar_id);
    tile_jump(p, q, t, [&]() { group_sync(bar_id); });
#pragma unroll
    for (int k = 0; k < TILE_PER_THREAD; ++k)
        if (r[k] >= 0) A.J[i0 + 4 * k * nx] = rv[q[k]];
    group_sync(bar_id);  // the buffers are reused by the group's next tile
}

// One path segment: tag the cells of start's path inside its tile by pointer doubling
// (after round r every cell within 2^(r+1) - 1 steps is on), until the start's own
// doubled pointer has left the tile, then reverse the links (rec[receiver] = cell).
__device__ __forceinline__ void loop_walk(const LoopArgs &A, int s0, int ntx, unsigned mnx, int t, int bar_id,
                                          unsigned char *smem, int *nd, const TileXY &txy)
{
    constexpr uint16_t NONE = 0xffff;
    uint16_t *jmp = reinterpret_cast<uint16_t *>(smem);  // two buffers
    uint8_t *on = smem + 4 * TILE_CELLS;
    const int nx = A.g.nx, ny = A.g.ny;
    int srow, scol;
    divmod_nx(s0, nx, mnx, srow, scol);
    const int ty = srow / TILE_H, tx = scol / TILE_W;
    const int row0 = ty * TILE_H, col0 = tx * TILE_W;
    const int w = min(TILE_W, nx - col0), h = min(TILE_H, ny - row0);
    const int start = (srow - row0) * TILE_W + scol - col0;
    const int lx = t & (TILE_W - 1), ly0 = t / TILE_W;
    const int i0 = (row0 + ly0) * nx + col0 + lx;
    int r[TILE_PER_THREAD], j[TILE_PER_THREAD];
#pragma unroll
    for (int k = 0; k < TILE_PER_THREAD; ++k)
        r[k] = (lx < w && ly0 + 4 * k < h) ? A.rec_[i0 + 4 * k * nx] : -1;
    tile_locals(r, j, i0, t, lx, ly0, row0, col0, w, h, nx, ny, mnx);
#pragma unroll
    for (int k = 0; k < TILE_PER_THREAD; ++k) {
        const int c = t + k * TILE_THREADS;
        if (j[k] == c) j[k] = NONE;
        jmp[c] = (uint16_t)j[k];
        on[c] = c == start;
    }
    group_sync(bar_id);
    for (int rd = 0; rd < 11; ++rd) {  // 2^11 = TILE_CELLS
        const uint16_t *jc = jmp + (rd & 1) * TILE_CELLS;
        uint16_t *jn = jmp + ((rd & 1) ^ 1) * TILE_CELLS;
        if (jc[start] == NONE) break;  // the same value for the whole group
#pragma unroll
        for (int k = 0; k < TILE_PER_THREAD; ++k) {
            const int c = t + k * TILE_THREADS;
            if (j[k] != NONE) {
                if (on[c]) on[j[k]] = 1;
                j[k] = jc[j[k]];
            }
            jn[c] = (uint16_t)j[k];
        }
        group_sync(bar_id);
    }
    bool local = false;
#pragma unroll
    for (int k = 0; k < TILE_PER_THREAD; ++k) {
        if (!on[t + k * TILE_THREADS]) continue;
        const int i = i0 + 4 * k * nx;
        A.tag[i] = 1;
        A.tag_[i] = 1;
        if (r[k] == i) continue;  // the root
        A.rec[r[k]] = i;
        const int tl = txy.of(r[k]);
        if (tl == ty * ntx + tx) local = true;
        else loop_mark(A, nd, tl);
    }
    if (group_or(bar_id, local) && t == 0) loop_mark(A, nd, ty * ntx + tx);
}

// a barrier that gave up ends the work
#define LOOP_SYNC()                        \
    do {                                   \
        if (!T.sync()) return RR_BOUND;    \
    } while (0)

// The outer iterations of one grid.  BATCH: a batch tile, whose basin, border and z'
// arrays are scratch: they are initialised for the pits only, and nothing is written that
// only a caller would read.  KEYED: the first border list carries labels and keys (from
// reroute_first_border, not from the strip pass).  it and outer on entry: the iteration to
// begin with, and (if that is not the first) the loop's bound.  Returns the final
// state (the same in every thread), the iteration it stopped in, its bound and count.
template <int MODE, bool BATCH, bool KEYED, class Team>
__device__ __forceinline__ int reroute_loop(const LoopArgs &A, Team &T, unsigned char *loop_smem, int &it, int &outer,
                                            int &n_outer)
{
    const Grid g = A.g;
    const int nx = g.nx, N = g.N();
    const unsigned mnx = 0xffffffffu / (unsigned)nx;
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, wib = tid >> 5;
    const int nblk = T.size(), gtid = T.rank() * nt + tid, gthreads = nblk * nt;
    const int grp = tid / TILE_THREADS, gt = tid & (TILE_THREADS - 1), ngrp = nt / TILE_THREADS;
    unsigned char *gsm = loop_smem + grp * LOOP_GROUP_BYTES;
    const TileXY txy{(nx + TILE_W - 1) / TILE_W, mnx, nx};
    const long long iv = invalid_key();
    const int np0 = vload(A.info);
    const int it0 = it;
    int state = RR_RUN;
    n_outer = 0;
    if (it0 == 0) outer = np0 > 0 ? d_ceil_log2(np0) + 1 : 0;  // :500
    if (vload(A.info + 5)) state = RR_BOUND;                   // the labels' launch gave up
    else if (np0 == 0) state = it0 == 0 ? RR_NOPITS : RR_DONE;      // :496-497, :512-514
    else if (vload(A.info + 2) || vload(A.info + 4)) state = RR_GENERAL;  // not D4, or a receiver cycle in the input
    if (state == RR_RUN) {
        // clear the carve tags of an earlier call
        if ((((uintptr_t)A.tag | (uintptr_t)A.tag_) & 15) == 0) {
            const uint4 zero = make_uint4(0, 0, 0, 0);
            for (int k = gtid; k < N / 16; k += gthreads) {
                reinterpret_cast<uint4 *>(A.tag)[k] = zero;
                reinterpret_cast<uint4 *>(A.tag_)[k] = zero;
            }
            for (int k = (N & ~15) + gtid; k < N; k += gthreads) A.tag[k] = A.tag_[k] = 0;
        } else {
            for (int k = gtid; k < N; k += gthreads) A.tag[k] = A.tag_[k] = 0;
        }
        if (gtid == 0) {
            A.fin[0] = 0;
            A.nf[0] = ~0;
        }
    }
    while (state == RR_RUN) {
        const int rel = it - it0;  // the lists and counters begin with this call
        const bool first = rel == 0;
        int *C = A.it_ctr + rel * LOOP_CTR, *Cn = C + LOOP_CTR;
        const int np = first ? np0 : vload(C + LC_NP);
        const int *pits = first ? A.pit0 : A.pits[rel & 1];
        int *pnext = A.pits[(rel + 1) & 1];
        const int *alist = A.alist[rel & 1];
        auto label = [&](int i) -> int {
            const int b = A.bid[i];
            return first ? b : A.fin[b];
        };
        // ---- passes 1-2 over the previous border cells (the first list comes from the strip pass)
        if (!first) {
            const int *aprev = A.alist[(rel & 1) ^ 1];
            int *anext = A.alist[rel & 1];
            const int n = vload(C - LOOP_CTR + LC_NA);
            // each warp on its own: the entries that stay on a border collect in its buffer,
            // and the next trip's cells are loaded ahead
            int *bufi = reinterpret_cast<int *>(loop_smem) + wib * LOOP_CAP * 4, *bufb = bufi + LOOP_CAP;
            long long *bufk = reinterpret_cast<long long *>(bufb + LOOP_CAP);
            int nb = 0;
            auto flush = [&]() {
                __syncwarp();
                int base = 0;
                if (lane == 0 && nb) base = atomicAdd(C + LC_NA, nb);
                base = __shfl_sync(0xffffffffu, base, 0);
                for (int q = lane; q < nb; q += 32) {
                    anext[base + q] = bufi[q];
                    A.abid[base + q] = bufb[q];
                    A.akey[base + q] = bufk[q];
                }
                __syncwarp();
                nb = 0;
            };
            int k0 = (T.rank() * (nt / 32) + wib) * 32;
            int inext = k0 + lane < n ? aprev[k0 + lane] : -1;
            for (; k0 < n; k0 += gthreads) {
                const bool has = k0 + lane < n;
                const int i = inext & 0x7FFFFFFF;
                const int kn = k0 + gthreads + lane;
                inext = kn < n ? aprev[kn] : -1;
                int code = 0, bi = 0;
                long long key = 0;
                if (has) {
                    int row, col;
                    divmod_nx(i, nx, mnx, row, col);
                    int jn[4], bn[4];
                    float zn[4];
                    neighbours4<MODE>(g, i, row, col, jn);
                    bi = A.bid[i];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        bn[q] = jn[q] != -1 ? A.bid[jn[q]] : 0;
                        zn[q] = jn[q] != -1 ? A.z[jn[q]] : 0.f;
                    }
                    const float zi = A.z[i];
                    bi = A.fin[bi];
#pragma unroll
                    for (int q = 0; q < 4; ++q) bn[q] = A.fin[bn[q]];
                    code = saddle_cell<!BATCH>(i, bi, zi, jn, bn, zn, A.isb, A.zp, key);
                }
                saddle_min_warp(A.sad, bi, key, code != 0 && key < iv);
                const unsigned m = __ballot_sync(0xffffffffu, code != 0);
                if (code != 0) {
                    const int at = nb + __popc(m & ((1u << lane) - 1u));
                    bufi[at] = i;
                    bufb[at] = bi;
                    bufk[at] = key;
                }
                nb += __popc(m);
                if (nb > LOOP_CAP - 32) flush();
            }
            flush();
            LOOP_SYNC();
        }
        // ---- pass 3: the saddle node is the largest qualifying cell index
        const int na = vload(C + LC_NA);
        // cell i of basin bi with z' equal to the saddle's: is a neighbour in its basin?
        auto claim = [&](int i, int bi, int tb) {
            int row, col, jn[4];
            divmod_nx(i, nx, mnx, row, col);
            neighbours4<MODE>(g, i, row, col, jn);
            bool here = false;
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (jn[q] != -1 && label(jn[q]) == tb) here = true;
            if (here) atomicMax(A.snode + bi, i);
        };
        if (first && !KEYED) {
            for (int k = gtid; 4 * k < na; k += gthreads) {  // the list's memory is padded to 16 bytes
                const int4 v = reinterpret_cast<const int4 *>(alist)[k];
                int i[4] = {v.x, v.y, v.z, v.w}, bi[4];
                float zpi[4];
                long long s[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const bool on = 4 * k + q < na && i[q] < 0;  // a border cell of a pit basin
                    i[q] &= 0x7FFFFFFF;
                    bi[q] = on ? A.bid[i[q]] : 0;
                    zpi[q] = on ? A.zp[i[q]] : 0.f;
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) s[q] = bi[q] ? A.sad[bi[q]] : iv;
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (bi[q] && zpi[q] == key_value(s[q])) claim(i[q], bi[q], key_index(s[q]));
            }
        } else {
            for (int k = gtid; k < na; k += gthreads) {
                const int bi = A.abid[k];
                const long long key = A.akey[k];
                if (bi == 0) continue;
                const long long s = A.sad[bi];
                // the cell's lowest key is the basin's, or only the sign of a zero differs
                if (key == s) atomicMax(A.snode + bi, alist[k]);
                else if (key_value(s) == 0.f && key_value(key) == 0.f) claim(alist[k], bi, key_index(s));
            }
        }
        LOOP_SYNC();
        // ---- pass 4: the outlet is the lowest foreign neighbour of the saddle node
        for (int k = gtid; k < np; k += gthreads) {
            const int b = pits[k] + 1;
            if (b >= N || A.sad[b] == iv) continue;
            const int node = A.snode[b];
            if (node < 0) continue;
            float tz = 1e9f;
            int r = -1, row, col, jn[4];
            divmod_nx(node, nx, mnx, row, col);
            neighbours4<MODE>(g, node, row, col, jn);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if (jn[q] == -1) continue;
                const float zj = A.z[jn[q]];
                if (label(jn[q]) != b && tz > zj) { tz = zj; r = jn[q]; }
            }
            if (r > -1) {
                const long long c = pack_key(tz, r);
                if (c < A.out[b]) A.out[b] = c;
            }
        }
        LOOP_SYNC();
        // ---- per basin: pass 5 (the larger basin of each 2-cycle, decided on this snapshot of
        //      the outlets; the invalid entries are written in the next step), link the saddle
        //      node, the label it merges into, the pits left, and its path's segment starts,
        //      one tile at a time through J
        {
            auto two_cycle = [&](int b, long long o) -> bool {
                const int bd1 = label(key_index(o));
                if (bd1 == 0 || bd1 >= b) return false;
                const int ro2 = key_index(A.out[bd1]);
                return ro2 >= 0 && ro2 < N && label(ro2) == b;
            };
            const int D = N > 42 ? label(42) : 0;  // see k_saddle_p5_serial_fix
            int *buf = reinterpret_cast<int *>(loop_smem) + wib * LOOP_CAP;
            int nb = 0;  // warp-uniform
            auto flush = [&]() {
                __syncwarp();
                int base = 0;
                if (lane == 0 && nb) base = atomicAdd(C + LC_NSEG, nb);
                base = __shfl_sync(0xffffffffu, base, 0);
                for (int q = lane; q < nb; q += 32)
                    if (base + q < N) A.segs[base + q] = buf[q];
                __syncwarp();
                nb = 0;
            };
            for (int kb = (T.rank() * (nt / 32) + wib) * 32; kb < np; kb += gthreads) {
                const int k = kb + lane;
                bool keep = false;
                int x = -1, p = -1;
                if (k < np) {
                    p = pits[k];
                    const int b = p + 1;
                    if (b < N) {
                        long long o = A.out[b];
                        bool dead_b = o != iv && two_cycle(b, o);
                        if (b == D && !dead_b && o != iv) {
                            const int bd1 = label(key_index(o));
                            if (bd1 != 0 && bd1 < D) {
                                const long long o1 = A.out[bd1];
                                dead_b = o1 != iv && two_cycle(bd1, o1);
                            }
                        }
                        if (dead_b) {
                            o = iv;
                            A.inv[b] = 1;
                        }
                        x = dead_b ? -1 : A.snode[b];
                        if (o != iv) {
                            const int node = key_index(o);
                            A.rec[x] = node;
                            loop_mark(A, C + LC_NDIRTY, txy.of(x));
                            A.nf[b] = label(node);
                        } else {
                            keep = true;
                            if (x != -1) C[LC_ODD] = 1;  // a path reversed without an outlet link
                        }
                    } else {
                        keep = true;
                    }
                    if (keep) A.nf[b] = ~b;
                }
                const unsigned m = __ballot_sync(0xffffffffu, keep);
                if (m) {
                    int base = 0;
                    if (lane == 0) base = atomicAdd(Cn + LC_NP, __popc(m));
                    base = __shfl_sync(0xffffffffu, base, 0);
                    if (keep) pnext[base + __popc(m & ((1u << lane) - 1u))] = p;
                }
                int tl = x >= 0 ? txy.of(x) : -1;
                for (int step = 0; step <= N && __any_sync(0xffffffffu, x >= 0); ++step) {
                    const unsigned e = __ballot_sync(0xffffffffu, x >= 0);
                    if (x >= 0) buf[nb + __popc(e & ((1u << lane) - 1u))] = x;
                    nb += __popc(e);
                    if (nb > LOOP_CAP - 32) flush();
                    if (x >= 0) {  // J[x] in x's own tile is the pit: the walk ends there
                        x = A.J[x];
                        const int t2 = txy.of(x);
                        if (t2 == tl) x = -1;
                        tl = t2;
                    }
                }
            }
            flush();
        }
        LOOP_SYNC();
        // ---- walk the segments; the labels' first jump round shares the step
        const int nseg_all = vload(C + LC_NSEG), nseg = min(nseg_all, N);
        const bool last = it + 1 >= outer, odd = vload(C + LC_ODD) != 0, over = nseg_all > N;
        for (int k = gtid; k < np; k += gthreads) {
            const int b = pits[k] + 1;
            if (b < N && A.inv[b]) {
                A.out[b] = iv;
                A.sad[b] = iv;
                A.snode[b] = -1;
            }
        }
        // a group of 256 threads takes about 5 us per segment whatever its length, a thread
        // about 0.6 us per cell; segments are many while the paths are short
        if (nseg > 2 * ngrp * nblk) {
            for (int k = gtid; k < nseg; k += gthreads) {
                const int start = A.segs[k], tl = txy.of(start);
                int x = start;
                bool local = false;
                for (int step = 0; step < TILE_CELLS + 1; ++step) {
                    A.tag[x] = 1;
                    A.tag_[x] = 1;
                    const int nxt = A.rec_[x];
                    if (nxt == x) break;
                    A.rec[nxt] = x;
                    const int t2 = txy.of(nxt);
                    if (t2 != tl) { loop_mark(A, C + LC_NDIRTY, t2); break; }
                    local = true;
                    x = nxt;
                }
                if (local) loop_mark(A, C + LC_NDIRTY, tl);
            }
        } else {
            for (int k = grp * nblk + T.rank(); k < nseg; k += nblk * ngrp) {
                loop_walk(A, A.segs[k], txy.ntx, mnx, gt, grp + 1, gsm, C + LC_NDIRTY, txy);
            }
        }
        // nf[b]: the label basin b merges into, or ~label once known to be final.  A chain
        // that never ends is a cycle of basins the carve closed.
        bool settled = false;
        for (int r = 0; r < LOOP_JUMPS; ++r) {
            bool ch = false;
            if (!last && !odd) {
                for (int k = gtid; k < np; k += gthreads) {
                    const int b = pits[k] + 1;
                    int x = vload(A.nf + b);
                    if (x < 0) continue;
                    for (int s = 0; s < 8 && x >= 0; ++s) x = vload(A.nf + x);
                    A.nf[b] = x;
                    ch |= x >= 0;
                }
                if (__any_sync(0xffffffffu, ch) && lane == 0) C[LC_FLAG + r] = 1;
            }
            LOOP_SYNC();
            if (last || odd || vload(C + LC_FLAG + r) == 0) { settled = true; break; }
        }
        // ---- the loop's decisions, in the reference's order (:500, :512-514)
        ++n_outer;
        if (over) state = RR_WALKERR;
        else if (odd) state = RR_RESUME;            // the reference's N-wide steps from here on
        else if (last) state = RR_DONE;
        else if (!settled) state = RR_RESUME;       // the carve closed a receiver cycle
        else if (vload(Cn + LC_NP) == 0) { ++n_outer; state = RR_DONE; }
        else if (rel + 2 >= LOOP_ITS) state = RR_BOUND;
        const bool go_on = state == RR_RUN;
        const int ndirty = vload(C + LC_NDIRTY);
        for (int k = grp * nblk + T.rank(); k < ndirty; k += nblk * ngrp) {
            const int tile = A.dtiles[k];
            loop_tile(A, tile, txy.ntx, mnx, gt, grp + 1, gsm, go_on);
            if (gt == 0) A.dirty[tile] = 0;
        }
        if (!go_on) break;
        for (int k = gtid; k < np0; k += gthreads) {  // labels: fin[b] = final(fin[b])
            const int b = A.pit0[k] + 1, x = first ? b : A.fin[b];
            if (x) A.fin[b] = ~A.nf[x];
        }
        for (int k = gtid; k <= np; k += gthreads) {  // the basins' entries of this iteration
            const int b = k < np ? pits[k] + 1 : 0;
            A.sad[b] = iv;
            A.out[b] = iv;
            A.snode[b] = -1;
            A.inv[b] = 0;
        }
        LOOP_SYNC();
        ++it;
    }
    if (!BATCH && (state == RR_DONE || state == RR_WALKERR)) {  // basin_id_init (:537)
        if (MODE != 3 && (nx & 3) == 0 && ((uintptr_t)A.bid & 15) == 0) {
            for (int q = gtid; 4 * q < N; q += gthreads) {
                int row, col, lab[4];
                divmod_nx(4 * q, nx, mnx, row, col);
#pragma unroll
                for (int k = 0; k < 4; ++k) lab[k] = can_leave<MODE>(g, 4 * q + k, row, col + k) ? 0 : 4 * q + k + 1;
                reinterpret_cast<int4 *>(A.bid)[q] = make_int4(lab[0], lab[1], lab[2], lab[3]);
            }
        } else {
            for (int i = gtid; i < N; i += gthreads) {
                int row, col;
                divmod_nx(i, nx, mnx, row, col);
                A.bid[i] = can_leave<MODE>(g, i, row, col) ? 0 : i + 1;
            }
        }
    }
    return state;
}

// Labels of the first iteration: pointer jumping of R over the tile-border cells (8 links
// per round and thread; chains of tiles up to 9^16 long), then one gather per cell and
// the basins' initial entries (20 B per cell: the stores overlap the gathers).
template <int MODE, bool BATCH, class Team>
__device__ __forceinline__ int reroute_labels(const LoopArgs &A, int32_t *R, Team &T)
{
    if (vload(A.info) == 0 || vload(A.info + 2)) return RR_RUN;  // the same for every block
    const Grid g = A.g;
    const int nx = g.nx, N = g.N();
    const unsigned mnx = 0xffffffffu / (unsigned)nx;
    const int ntx = (nx + TILE_W - 1) / TILE_W;
    const long long nslots = (long long)ntx * ((g.ny + TILE_H - 1) / TILE_H) * BORDER_SLOTS;
    const int gtid = T.rank() * blockDim.x + threadIdx.x, gthreads = T.size() * blockDim.x;
    int *flags = A.bar + 16;
    for (int r = 0; r < LOOP_JUMPS; ++r) {
        bool ch = false;
        for (long long k = gtid; k < nslots; k += gthreads) {
            const int e = border_cell(nx, g.ny, ntx, k);
            if (e < 0) continue;
            int x = vload(R + e), y = vload(R + x);
            if (y == x) continue;
            for (int s = 0; s < 8 && y != x; ++s) {
                x = y;
                y = vload(R + x);
            }
            R[e] = x;
            ch |= y != x;
        }
        if (__any_sync(0xffffffffu, ch) && (threadIdx.x & 31) == 0) flags[r] = 1;
        LOOP_SYNC();
        if (vload(flags + r) == 0) break;
    }
    const long long iv = invalid_key();
    bool cyc = false;
    if (!BATCH && MODE != 3 && (nx & 3) == 0 &&
        (((uintptr_t)A.J | (uintptr_t)A.bid | (uintptr_t)A.sad | (uintptr_t)A.out | (uintptr_t)A.snode) & 15) == 0 &&
        ((uintptr_t)A.inv & 3) == 0) {
        for (int q = gtid; 4 * q < N; q += gthreads) {
            const int4 j = reinterpret_cast<const int4 *>(A.J)[q];
            const int rt[4] = {R[j.x], R[j.y], R[j.z], R[j.w]};
            reinterpret_cast<longlong2 *>(A.sad)[2 * q] = reinterpret_cast<longlong2 *>(A.sad)[2 * q + 1] =
                make_longlong2(iv, iv);
            reinterpret_cast<longlong2 *>(A.out)[2 * q] = reinterpret_cast<longlong2 *>(A.out)[2 * q + 1] =
                make_longlong2(iv, iv);
            reinterpret_cast<int4 *>(A.snode)[q] = make_int4(-1, -1, -1, -1);
            reinterpret_cast<uchar4 *>(A.inv)[q] = make_uchar4(0, 0, 0, 0);
            int lab[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                cyc |= A.rec_[rt[k]] != rt[k];  // a receiver cycle: labels need the general path
                int row, col;
                divmod_nx(rt[k], nx, mnx, row, col);
                lab[k] = can_leave<MODE>(g, rt[k], row, col) ? 0 : rt[k] + 1;
            }
            reinterpret_cast<int4 *>(A.bid)[q] = make_int4(lab[0], lab[1], lab[2], lab[3]);
        }
    } else {
        constexpr int U = 4;  // cells per trip, their gathers in flight together
        for (int i0 = gtid; i0 < N; i0 += U * gthreads) {
            int rt[U], rr[U];
#pragma unroll
            for (int u = 0; u < U; ++u) rt[u] = i0 + u * gthreads < N ? A.J[i0 + u * gthreads] : 0;
#pragma unroll
            for (int u = 0; u < U; ++u) rt[u] = i0 + u * gthreads < N ? R[rt[u]] : 0;
#pragma unroll
            for (int u = 0; u < U; ++u) rr[u] = A.rec_[rt[u]];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int i = i0 + u * gthreads;
                if (i >= N) break;
                if (!BATCH) {
                    A.sad[i] = iv;
                    A.out[i] = iv;
                    A.snode[i] = -1;
                    A.inv[i] = 0;
                }
                cyc |= rr[u] != rt[u];
                int row, col;
                divmod_nx(rt[u], nx, mnx, row, col);
                A.bid[i] = can_leave<MODE>(g, rt[u], row, col) ? 0 : rt[u] + 1;
            }
        }
    }
    if (BATCH) {
        const int np = vload(A.info);
        for (int k = gtid; k <= np; k += gthreads) {
            const int b = k < np ? A.pit0[k] + 1 : 0;
            A.sad[b] = iv;
            A.out[b] = iv;
            A.snode[b] = -1;
            A.inv[b] = 0;
        }
    } else if (gtid == 0) {
        A.sad[N] = iv;
        A.out[N] = iv;
        A.snode[N] = -1;
        A.inv[N] = 0;
    }
    if (cyc) A.info[4] = 1;
    return RR_RUN;
}

// The tile pass over the whole grid: rec_ = rec, tile terminals and the pit list.
template <int MODE, class Team>
__device__ __forceinline__ void reroute_tiles(const LoopArgs &A, int32_t *R, Team &T, unsigned char *smem)
{
    const int grp = threadIdx.x / TILE_THREADS, gt = threadIdx.x & (TILE_THREADS - 1), ngrp = blockDim.x / TILE_THREADS;
    const Grid g = A.g;
    const int ntx = (g.nx + TILE_W - 1) / TILE_W, ntiles = ntx * ((g.ny + TILE_H - 1) / TILE_H);
    unsigned char *gsm = smem + grp * LOOP_GROUP_BYTES;
    for (int k = grp * T.size() + T.rank(); k < ntiles; k += ngrp * T.size()) {
        tile_terminal_one<MODE>(A.rec, A.J, R, A.pit0, A.info, g, k % ntx, k / ntx,
                                reinterpret_cast<uint16_t *>(gsm), reinterpret_cast<int *>(gsm + 2 * TILE_CELLS), A.rec_,
                                gt, [&]() { group_sync(grp + 1); });
        group_sync(grp + 1);  // the buffers are reused by the group's next tile
    }
}

// Passes 1-2 of the first iteration over every cell; the border cells with their labels
// and keys.  A warp takes 32 consecutive cells: neighbours and their labels come from L1.
template <int MODE, bool WRITE, class Team>
__device__ __forceinline__ void reroute_first_border(const LoopArgs &A, Team &T, unsigned char *smem)
{
    if (vload(A.info) == 0 || vload(A.info + 2) || vload(A.info + 4)) return;
    const Grid g = A.g;
    const int nx = g.nx, N = g.N(), lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const unsigned mnx = 0xffffffffu / (unsigned)nx;
    const int gthreads = T.size() * blockDim.x;
    int *bufi = reinterpret_cast<int *>(smem) + wib * LOOP_CAP * 4, *bufb = bufi + LOOP_CAP;
    long long *bufk = reinterpret_cast<long long *>(bufb + LOOP_CAP);
    int *na = A.it_ctr + LC_NA;
    int nb = 0;
    auto flush = [&]() {
        __syncwarp();
        int base = 0;
        if (lane == 0 && nb) base = atomicAdd(na, nb);
        base = __shfl_sync(0xffffffffu, base, 0);
        for (int q = lane; q < nb; q += 32) {
            A.alist[0][base + q] = bufi[q];
            A.abid[base + q] = bufb[q];
            A.akey[base + q] = bufk[q];
        }
        __syncwarp();
        nb = 0;
    };
    for (int k0 = (T.rank() * (blockDim.x >> 5) + wib) * 64; k0 < N; k0 += 2 * gthreads) {
        int jn[2][4], bn[2][4], bi[2];
        float zn[2][4], zi[2];
        bool on[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {  // two cells per thread, their loads in flight together
            const int i = k0 + 32 * u + lane;
            on[u] = false;
            if (i < N) {
                int row, col;
                divmod_nx(i, nx, mnx, row, col);
                if (can_leave<MODE>(g, i, row, col)) {
                    if (WRITE) A.zp[i] = A.z[i];
                } else {
                    on[u] = true;
                    neighbours4<MODE>(g, i, row, col, jn[u]);
                    bi[u] = A.bid[i];
                    zi[u] = A.z[i];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        bn[u][q] = jn[u][q] != -1 ? A.bid[jn[u][q]] : 0;
                        zn[u][q] = jn[u][q] != -1 ? A.z[jn[u][q]] : 0.f;
                    }
                }
            }
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int i = k0 + 32 * u + lane;
            int code = 0;
            long long key = 0;
            if (on[u]) code = saddle_cell<WRITE>(i, bi[u], zi[u], jn[u], bn[u], zn[u], A.isb, A.zp, key);
            if (code != 0 && key < invalid_key()) atomicMin(A.sad + bi[u], key);
            const unsigned m = __ballot_sync(0xffffffffu, code != 0);
            if (code != 0) {
                const int at = nb + __popc(m & ((1u << lane) - 1u));
                bufi[at] = i;
                bufb[at] = bi[u];
                bufk[at] = key;
            }
            nb += __popc(m);
            if (nb > LOOP_CAP - 32) flush();
        }
    }
    flush();
}

}  // namespace pff
