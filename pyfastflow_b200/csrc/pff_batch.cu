// libpff ragged batch: hundreds of independent DEM tiles of uneven sizes routed
// (receivers -> carve reroute -> accumulate) in ONE persistent launch over a packed
// layout.  Each CTA takes whole tiles from a queue (largest first) and runs the
// entire chain for its tile with block-wide barriers between passes: tiles are
// independent, so nothing synchronises across CTAs and the launch needs no host
// round trip (it can be captured in a CUDA graph).
//
// Within a tile the steps are the reference's own (pyfastflow/flow/receivers.py:31-58,
// lakeflow.py:466-538, downstream_propag.py:59-179, flowfields.py:254-292) with the
// pinned semantics of the single-grid path: serial last writer for the saddle node
// and for path reversal (largest index), the serial 2-cycle pass, serial labelling of
// receiver cycles (emulated), snapshot rake-and-compress rounds with donors in
// ascending index.  Results are bit-identical to routing each tile on its own.
#include <algorithm>
#include <vector>
#include "pff_internal.h"
#include "pff_lake_loop.cuh"
#include "pff_pow.cuh"

namespace pff {

// Packed per-cell and per-basin arrays of the batch (device pointers).
struct BatchArrays {
    const float *z;
    const uint8_t *codes;  // packed boundary codes of the custom-mode tiles (may be null without such tiles)
    int32_t *rcv;      // out: rerouted receivers (tile-local indices)
    float *grad;       // out: steepest gradient of the original receivers
    float *Q;          // in: per-cell seed, out: upstream sum
    uint32_t *counts;  // out: upstream cell counts
    int32_t *rec_, *rec__, *bid, *mark;
    float *zp;
    uint8_t *isb, *tag, *tag_;
    long long *saddle, *outlet;  // N+1 per tile
    int32_t *snode;              // N+1 per tile
    uint8_t *inv;                // N+1 per tile
    int32_t *dnr, *dnr_;         // 4 per cell
    int32_t *ndnr, *ndnr_, *src;
    float *p_;
    uint32_t *c_;
    const BatchTile *tiles;  // in largest-first order
    int *queue;              // [0] next tile
    const int *small;        // whether the batch is k_batch_small's; null: it is not
    int *status;             // [0] error bits (see pff_batch_status)
};


constexpr int LB_SIDE = 32, LB_CELLS = LB_SIDE * LB_SIDE;  // label sub-blocks

// Cells up to which GraphFlood's reroutes are the reference's steps by one block: 5 iterations on 40 tiles of
// 24 x 24 take 483 us, 563 by the list loop; of 32 x 32 753 and 644.
constexpr int GF_SMALL = 900;

struct BatchShm {
    LoopArgs la;  // the current tile's reroute
    int loop[64 + LOOP_ITS * LOOP_CTR];  // its state words, barrier flags and counters (the first block's are used)
    int any[3];   // team_any's flags (the first block's are used)
    int any_r;
    int it_outer[2];
    int red;
    int cur;
    int ws[32];
    int lp[LB_CELLS];   // sub-block pointers (local indices)
    int tgt[LB_CELLS];  // sub-block cells' receivers (tile indices)
};

__host__ __device__ __forceinline__ int bceil_log2(long long n)
{
    int r = 0;
    long long p = 1;
    while (p < n) { p <<= 1; ++r; }
    return r;
}

__device__ __forceinline__ long long inv_key() { return pack_key(1e8f, 42); }

// Block-wide sum (every thread gets it).
__device__ __forceinline__ int bsum(int v, BatchShm &sh)
{
    __syncthreads();
    if (threadIdx.x == 0) sh.red = 0;
    __syncthreads();
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(&sh.red, v);
    __syncthreads();
    const int r = sh.red;
    __syncthreads();
    return r;
}

// Block-wide exclusive prefix sum of v (blockDim a multiple of 32); *total = sum.
__device__ __forceinline__ int bscan(int v, BatchShm &sh, int *total)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int x = v;
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    __syncthreads();
    if (lane == 31) sh.ws[wid] = x;
    __syncthreads();
    if (wid == 0) {
        int s = lane < nw ? sh.ws[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        if (lane < nw) sh.ws[lane] = s;
    }
    __syncthreads();
    const int before = (wid ? sh.ws[wid - 1] : 0) + x - v;
    *total = sh.ws[nw - 1];
    __syncthreads();
    return before;
}

#define FOR_CELLS(i, N) for (int i = threadIdx.x; i < (N); i += blockDim.x)

template <int MODE>
__device__ __forceinline__ bool leave(const Grid &g, int i)
{
    return can_leave_i<MODE>(g, i);
}

// ---- labels: basin_id_init + propagate_basin on a copy of rec_ (lakeflow.py:47-80, 507-511)
//
// Acyclic receivers: the fixed point of pointer jumping, reached in parallel.  On a
// receiver cycle the reference's serial in-place rounds give a result that depends
// only on the cycle's cells visited in ascending index; it is emulated here and every
// cell draining into the cycle takes the cycle's label.
template <int MODE>
__device__ void tile_labels(const Grid &g, int N, const int32_t *rec_, int32_t *work, int32_t *bid, int32_t *mark,
                            int32_t *scr, int rounds, BatchShm &sh, int *status)
{
    FOR_CELLS(i, N) {
        bid[i] = leave<MODE>(g, i) ? 0 : i + 1;
        work[i] = rec_[i];
        mark[i] = 0;
    }
    __syncthreads();
    for (int r = 0; r < rounds; ++r) {
        int ch = 0;
        FOR_CELLS(i, N) {
            const int p = work[i];
            const int b = bid[p], pp = work[p];
            if (bid[i] != b) { bid[i] = b; ch = 1; }
            if (pp != p) { work[i] = pp; ch = 1; }
        }
        if (!__syncthreads_or(ch)) break;
    }
    // After the rounds every pointer sits on a true root or on a cycle cell.
    int unresolved = 0;
    FOR_CELLS(i, N) {
        const int x = work[i];
        unresolved |= (rec_[x] != x);
    }
    if (!__syncthreads_or(unresolved)) return;
    // Mark every cycle cell: walkers claim cells and stop at the first cell another
    // walker claimed, which covers each cycle exactly once.
    FOR_CELLS(i, N) {
        int x = work[i];
        if (rec_[x] == x) continue;
        for (int s = 0; s <= N; ++s) {
            if (atomicExch(mark + x, 1)) break;
            x = rec_[x];
        }
    }
    __syncthreads();
    // cycle cells in ascending index order: cells[a], pos[cell] = a
    int32_t *cells = scr, *pos = scr + N, *lrec = scr + 2LL * N, *lb = scr + 3LL * N;
    int L = 0;
    for (int base = 0; base < N; base += blockDim.x) {
        const int i = base + threadIdx.x;
        const int f = (i < N && mark[i]) ? 1 : 0;
        int tot;
        const int p = bscan(f, sh, &tot);
        if (f) { cells[L + p] = i; pos[i] = L + p; }
        L += tot;
    }
    __syncthreads();
    FOR_CELLS(a, L) {
        const int c = cells[a];
        lrec[a] = pos[rec_[c]];
        lb[a] = leave<MODE>(g, c) ? 0 : c + 1;
    }
    __syncthreads();
    if (threadIdx.x == 0)
        for (int r = 0; r < rounds; ++r)
            for (int a = 0; a < L; ++a) {
                lb[a] = lb[lrec[a]];
                lrec[a] = lrec[lrec[a]];
            }
    __syncthreads();
    int bad = 0;
    FOR_CELLS(a, L) bad |= (lb[a] != lb[pos[rec_[cells[a]]]]);  // one label per cycle
    if (__syncthreads_or(bad) && threadIdx.x == 0) atomicOr(status, BST_CYCLE_LABELS);
    FOR_CELLS(i, N) {
        const int x = work[i];
        if (rec_[x] != x) bid[i] = lb[pos[x]];
    }
    __syncthreads();
}

// ---- labels, fast form for acyclic receivers -----------------------------------------
//
// The fixed point of the labelling is bid[i] = root(i)+1, or 0 when the root can leave.
// Roots are found in three steps: (A) each 32 x 32 sub-block is pointer-jumped in shared
// memory to its cells' terminals (an in-block root, or the last in-block cell of the
// path); J[i] = the terminal's receiver, i.e. the root itself or the entry cell of the
// next sub-block, which lies on that sub-block's perimeter; (B) pointer jumping on J over
// the perimeter cells only; (C) one gather.  A receiver cycle shows up as a pointer that
// does not settle or a final target that is not a root; the caller then runs the
// general labelling, which reproduces the serial result on cycles.
template <int MODE>
__device__ bool tile_labels_blocks(const Grid &g, int N, const int32_t *rec_, int32_t *J, int32_t *bid, BatchShm &sh)
{
    const int nx = g.nx, ny = g.ny;
    const int nbx = (nx + LB_SIDE - 1) / LB_SIDE, nby = (ny + LB_SIDE - 1) / LB_SIDE;
    int bad = 0;
    // (A) sub-block terminals
    for (int blk = 0; blk < nbx * nby; ++blk) {
        const int x0 = (blk % nbx) * LB_SIDE, y0 = (blk / nbx) * LB_SIDE;
        for (int l = threadIdx.x; l < LB_CELLS; l += blockDim.x) {
            const int x = x0 + (l & (LB_SIDE - 1)), y = y0 + l / LB_SIDE;
            int p = l, t = -1;
            if (x < nx && y < ny) {
                const int i = y * nx + x;
                t = rec_[i];
                const int ry = t / nx, rx = t - ry * nx;
                if (t != i && rx >= x0 && rx < x0 + LB_SIDE && ry >= y0 && ry < y0 + LB_SIDE)
                    p = (ry - y0) * LB_SIDE + (rx - x0);
            }
            sh.lp[l] = p;
            sh.tgt[l] = t;
        }
        __syncthreads();
        for (int r = 0; r < 10; ++r) {  // chains inside a block are shorter than 2^10 cells
            int q[LB_CELLS / 256];      // blockDim >= 256: at most 4 cells per thread
#pragma unroll
            for (int c = 0; c < LB_CELLS / 256; ++c) {
                const int l = threadIdx.x + c * blockDim.x;
                if (l < LB_CELLS) q[c] = sh.lp[sh.lp[l]];
            }
            __syncthreads();
#pragma unroll
            for (int c = 0; c < LB_CELLS / 256; ++c) {
                const int l = threadIdx.x + c * blockDim.x;
                if (l < LB_CELLS) sh.lp[l] = q[c];
            }
            __syncthreads();
        }
        for (int l = threadIdx.x; l < LB_CELLS; l += blockDim.x) {
            const int x = x0 + (l & (LB_SIDE - 1)), y = y0 + l / LB_SIDE;
            if (x >= nx || y >= ny) continue;
            const int t = sh.lp[l];
            if (sh.lp[t] != t) bad = 1;  // a cycle inside the block
            J[y * nx + x] = sh.tgt[t];
        }
        __syncthreads();
    }
    if (__syncthreads_or(bad)) return false;
    // (B) pointer jumping over the perimeter cells (every J value is a root or one of them)
    const int PER = 4 * LB_SIDE - 4;
    const int nper = nbx * nby * PER;
    bool settled = false;
    for (int r = 0; r < 64; ++r) {
        int ch = 0;
        for (int k = threadIdx.x; k < nper; k += blockDim.x) {
            const int blk = k / PER, e = k - blk * PER;
            const int x0 = (blk % nbx) * LB_SIDE, y0 = (blk / nbx) * LB_SIDE;
            const int bw = min(LB_SIDE, nx - x0), bh = min(LB_SIDE, ny - y0);  // the block's extent in the tile
            int lx, ly;  // position e on the perimeter of the bw x bh block
            if (e < LB_SIDE) { lx = e; ly = 0; }
            else if (e < 2 * LB_SIDE) { lx = e - LB_SIDE; ly = bh - 1; }
            else if (e < 3 * LB_SIDE - 2) { lx = 0; ly = e - 2 * LB_SIDE + 1; }
            else { lx = bw - 1; ly = e - (3 * LB_SIDE - 2) + 1; }
            if (lx >= bw || ly >= bh || (e >= 2 * LB_SIDE && ly >= bh - 1)) continue;
            const int x = x0 + lx, y = y0 + ly;
            const int i = y * nx + x;
            const int a = J[i], b2 = J[a];
            if (b2 != a) { J[i] = b2; ch = 1; }
        }
        if (!__syncthreads_or(ch)) { settled = true; break; }
    }
    if (!settled) return false;
    // (C) gather, and check that every target is a true root
    FOR_CELLS(i, N) {
        int t = J[i];
        if (rec_[t] != t) t = J[t];
        if (rec_[t] != t) { bad = 1; continue; }
        bid[i] = leave<MODE>(g, t) ? 0 : t + 1;
    }
    return !__syncthreads_or(bad);
}

// ---- saddlesort passes 1-5 (lakeflow.py:106-281) ------------------------------------
template <int MODE>
__device__ void tile_saddlesort(const Grid &g, int N, const int32_t *bid, uint8_t *isb, float *zp, long long *sad,
                                int32_t *snode, long long *out, uint8_t *inv, const float *z, const int32_t *pl,
                                int np)
{
    // With labels of acyclic receivers (pl given) the only basin ids are 0 and pit + 1 for
    // the current pits (pl, np entries): those entries are reset and the per-basin passes
    // run over the pit list.  Otherwise (labels of a receiver cycle, pl == nullptr) every
    // basin id 0..N is reset and scanned, as in the reference.  Basin N is skipped by the
    // per-basin passes, as the reference's loops over b < N skip it.
    const long long iv = inv_key();
    const int ninit = pl ? np + 1 : N + 1, nscan = pl ? np : N;
    for (int k = threadIdx.x; k < ninit; k += blockDim.x) {
        const int b = pl ? (k < np ? pl[k] + 1 : 0) : k;
        sad[b] = iv;
        out[b] = iv;
        snode[b] = -1;
        inv[b] = 0;
    }
    __syncthreads();
    // passes 1 and 2: z' and the per-basin lowest packed (z', neighbour basin)
    FOR_CELLS(i, N) {
        const float zi = z[i];
        if (leave<MODE>(g, i)) {
            zp[i] = zi;
            isb[i] = 0;  // never written by the reference: its zero initial value
            continue;
        }
        const int row = i / g.nx, col = i - row * g.nx;
        const int bi = bid[i];
        int js[4];
        neighbours4<MODE>(g, i, row, col, js);
        bool border = false;
        float zn = 1e9f;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (js[k] != -1 && bid[js[k]] != bi) {
                border = true;
                zn = fminf(zn, z[js[k]]);
            }
        isb[i] = border;
        const float zpi = border ? fmaxf(zi, zn) : 1e9f;
        zp[i] = zpi;
        if (!border) continue;
        long long res = iv;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (js[k] == -1) continue;
            const int bj = bid[js[k]];
            if (bj != bi) {
                const long long c = pack_key(zpi, bj);
                res = c < res ? c : res;
            }
        }
        if (res != iv) atomicMin(sad + bi, res);
    }
    __syncthreads();
    // pass 3: saddle node = largest qualifying index (serial last writer)
    FOR_CELLS(i, N) {
        if (!isb[i]) continue;
        const int bi = bid[i];
        if (bi == 0) continue;
        const long long s = sad[bi];
        const float tz = key_value(s);
        const int tb = key_index(s);
        const float zpi = zp[i];
        const int row = i / g.nx, col = i - row * g.nx;
        int js[4];
        neighbours4<MODE>(g, i, row, col, js);
        bool here = false;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (js[k] != -1 && bid[js[k]] == tb && zpi == tz) here = true;
        if (here) atomicMax(snode + bi, i);
    }
    __syncthreads();
    // pass 4: outlet = lowest foreign neighbour of the saddle node (first k wins)
    for (int k0 = threadIdx.x; k0 < nscan; k0 += blockDim.x) {
        const int b = pl ? pl[k0] + 1 : k0;
        if (b == 0 || b >= N || sad[b] == iv) continue;
        const int node = snode[b];
        if (node < 0) continue;
        float tz = 1e9f;
        int r = -1;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int j = neighbour_i<MODE>(g, node, k);
            if (j == -1) continue;
            const float zj = z[j];
            if (bid[j] != b && tz > zj) {
                tz = zj;
                r = j;
            }
        }
        if (r > -1) out[b] = pack_key(tz, r);
    }
    __syncthreads();
    // pass 5: 2-cycles b -> b' -> b with b' < b, snapshot reads, plus the one basin
    // (bid[42]) whose serial outcome can differ from the snapshot
    for (int k0 = threadIdx.x; k0 < nscan; k0 += blockDim.x) {
        const int b = pl ? pl[k0] + 1 : k0;
        if (b == 0 || b >= N) continue;
        const long long ob = out[b];
        if (ob == iv) continue;
        const int bd1 = bid[key_index(ob)];
        if (bd1 == 0) continue;
        const int ro2 = key_index(out[bd1]);
        const int bd2 = (ro2 >= 0 && ro2 < N) ? bid[ro2] : -1;
        if (bd2 == b && bd1 < b) inv[b] = 1;
    }
    __syncthreads();
    if (threadIdx.x == 0 && N > 42) {
        const int D = bid[42];
        if (D > 0 && D < N && out[D] != iv) {
            const int bd1 = bid[key_index(out[D])];
            if (bd1 != 0 && bd1 < D && inv[bd1]) inv[D] = 1;
        }
    }
    __syncthreads();
    for (int k0 = threadIdx.x; k0 < nscan; k0 += blockDim.x) {
        const int b = pl ? pl[k0] + 1 : k0;
        if (b < N && inv[b]) {
            out[b] = iv;
            sad[b] = iv;
            snode[b] = -1;
        }
    }
    __syncthreads();
}

// ---- reroute_carve (lakeflow.py:308-438); leaves the result in rec and rec_ ----------
//
// The reference tags the saddle nodes and propagates the tags by pointer jumping until
// no tag changes; a round adds the next 2^r cells of every tagged path, so the fixed
// point is the union of the saddle nodes' forward orbits under rec_ (down to each
// pit, or around a receiver cycle).  The jumped pointers are discarded by the
// finalisation, so only that tag set matters: here each saddle node walks its own
// orbit, stopping at a cell already tagged (the rest of that orbit is another
// walker's) or at a root.
__device__ void tile_carve(int N, int32_t *rec, int32_t *rec_, int32_t *claim, uint8_t *tag, const int32_t *snode,
                           const long long *out, const int32_t *pl, int np, int *status)
{
    const long long iv = inv_key();
    FOR_CELLS(i, N) {
        tag[i] = 0;
        claim[i] = -1;
    }
    __syncthreads();
    int overrun = 0;
    const int nscan = pl ? np : N;  // the pits' basins, or every basin id (see tile_saddlesort)
    for (int k0 = threadIdx.x; k0 < nscan; k0 += blockDim.x) {
        const int b = pl ? pl[k0] + 1 : k0;
        if (b >= N) continue;
        int x = snode[b];
        if (x == -1) continue;
        int s = 0;
        for (; s <= N; ++s) {
            if (tag[x]) break;
            tag[x] = 1;
            const int nx_ = rec_[x];
            if (nx_ == x) break;
            x = nx_;
        }
        if (s > N) overrun = 1;
    }
    if (__syncthreads_or(overrun) && threadIdx.x == 0) atomicOr(status, BST_CARVE);
    // finalise: pre-carve receivers, path reversal (largest index wins), saddle links
    FOR_CELLS(i, N) {
        const int r0 = rec_[i];
        rec[i] = r0;
        if (tag[r0] && tag[i] && i != r0) atomicMax(claim + r0, i);
    }
    __syncthreads();
    FOR_CELLS(x, N) {
        const int c = claim[x];
        if (c >= 0) rec[x] = c;
    }
    __syncthreads();
    for (int k0 = threadIdx.x; k0 < nscan; k0 += blockDim.x) {
        const int b = pl ? pl[k0] + 1 : k0;
        if (b >= N) continue;
        const long long ob = out[b];
        if (ob != iv) rec[snode[b]] = key_index(ob);
    }
    __syncthreads();
    FOR_CELLS(i, N) rec_[i] = rec[i];
    __syncthreads();
}

// ---- rake-and-compress (downstream_propag.py:21-179), f32 and u32 payloads ---------------
__device__ __forceinline__ bool bget_src(const int32_t *src, int t, int it)
{
    const int e = src[t];
    bool flip = e < 0;
    if (abs(e) == it + 1) flip = !flip;
    return flip;
}

// Only nodes that still have donors are visited: a node with none left does nothing
// in any later round, so the rounds run over a compacted active list (la -> lb).
__device__ void tile_accumulate(int N, const int32_t *rcv, float *p, uint32_t *c, int32_t *dnr, int32_t *dnr_,
                                int32_t *ndnr, int32_t *ndnr_, int32_t *src, float *p_, uint32_t *c_, int32_t *la,
                                int32_t *lb, BatchShm &sh)
{
    FOR_CELLS(t, N) {
        ndnr[t] = 0;
        src[t] = 0;
        c[t] = 1u;
    }
    __syncthreads();
    FOR_CELLS(t, N) {  // rcv2donor (:78-96); D4 receivers give at most 4 donors
        const int r = rcv[t];
        if (r == t) continue;
        const int slot = atomicAdd(ndnr + r, 1);
        if (slot < 4) dnr[4LL * r + slot] = t;
    }
    __syncthreads();
    int nact = 0;
    for (int b0 = 0; b0 < N; b0 += blockDim.x) {  // sort donors (ascending: the serial slot order), list actives
        const int r = b0 + threadIdx.x;
        int f = 0;
        if (r < N) {
            const int n = min(ndnr[r], 4);
            int *d = dnr + 4LL * r;
            for (int a = 1; a < n; ++a) {
                const int x = d[a];
                int b = a - 1;
                while (b >= 0 && d[b] > x) {
                    d[b + 1] = d[b];
                    --b;
                }
                d[b + 1] = x;
            }
            f = n > 0;
        }
        int tot;
        const int q = bscan(f, sh, &tot);
        if (f) la[nact + q] = r;
        nact += tot;
    }
    __syncthreads();
    const int logn = bceil_log2(N) + 1;
    for (int it = 0; it <= logn && nact > 0; ++it) {
        int worked_any = 0, nnext = 0;
        for (int b0 = 0; b0 < nact; b0 += blockDim.x) {
            const int k = b0 + threadIdx.x;
            int keep = 0, tid = -1;
            if (k < nact) {
                tid = la[k];
                const bool flip = bget_src(src, tid, it);
                int todo = flip ? ndnr_[tid] : ndnr[tid];
                const long long base = 4LL * tid;
                int donors[4] = {-1, -1, -1, -1};
                bool worked = false;
                float padd = 0.f;
                uint32_t cadd = 0;
                int i = 0;
                while (i < todo && i < 4) {
                    if (donors[i] == -1) donors[i] = flip ? dnr_[base + i] : dnr[base + i];
                    const int did = donors[i];
                    const bool fd = bget_src(src, did, it);
                    const int nd = fd ? ndnr_[did] : ndnr[did];
                    if (nd <= 1) {
                        if (!worked) {
                            padd = flip ? p_[tid] : p[tid];
                            cadd = flip ? c_[tid] : c[tid];
                        }
                        worked = true;
                        padd = __fadd_rn(padd, fd ? p_[did] : p[did]);
                        cadd += fd ? c_[did] : c[did];
                        if (nd == 0) {
                            --todo;
                            if (todo > i) donors[i] = flip ? dnr_[base + todo] : dnr[base + todo];
                            --i;
                        } else {
                            donors[i] = fd ? dnr_[4LL * did] : dnr[4LL * did];
                        }
                    }
                    ++i;
                }
                if (worked) {
                    worked_any = 1;
                    const int m = todo < 4 ? todo : 4;
                    if (flip) {
                        ndnr[tid] = todo;
                        p[tid] = padd;
                        c[tid] = cadd;
                        for (int j = 0; j < m; ++j) dnr[base + j] = donors[j];
                    } else {
                        ndnr_[tid] = todo;
                        p_[tid] = padd;
                        c_[tid] = cadd;
                        for (int j = 0; j < m; ++j) dnr_[base + j] = donors[j];
                    }
                    src[tid] = (flip ? 1 : -1) * (it + 1);
                }
                keep = todo > 0;
            }
            int tot;
            const int q = bscan(keep, sh, &tot);
            if (keep) lb[nnext + q] = tid;
            nnext += tot;
        }
        // a round in which nothing worked leaves the state, and every later round, unchanged
        if (!__syncthreads_or(worked_any)) break;
        int32_t *t = la;
        la = lb;
        lb = t;
        nact = nnext;
    }
    FOR_CELLS(t, N) {  // fuse(Q, src, Q_, logn)
        if (bget_src(src, t, logn)) {
            p[t] = p_[t];
            c[t] = c_[t];
        }
    }
    __syncthreads();
}

// ---- teams ---------------------------------------------------------------------------
// The blocks of a cluster work on one tile together; team_at gives the address of a
// shared variable of the team's first block.
template <class T>
__device__ __forceinline__ T *team_at(T *p, const ClusterTeam &Tm)
{
    if (Tm.n == 1) return p;
    T *q;
    asm("mapa.u64 %0, %1, 0;" : "=l"(q) : "l"(p));
    return q;
}
#define FOR_TEAM(i, N) for (int i = Tm.r * blockDim.x + threadIdx.x; i < (N); i += Tm.n * blockDim.x)
// U cells per thread and trip (cells i0, i0 + stride, ...), so that their loads are in
// flight together: the passes are bound by load latency at 32 warps per SM
#define FOR_TEAM_U(i0, stride, U, N)                                                    \
    for (int stride = Tm.n * blockDim.x, i0 = Tm.r * blockDim.x + threadIdx.x; i0 < (N); \
         i0 += (U) * stride)

// whether any thread of the team has p (a barrier)
__device__ __forceinline__ bool team_any(bool p, BatchShm &sh, ClusterTeam &Tm)
{
    if (Tm.n == 1) return __syncthreads_or(p);
    const int r = sh.any_r;
    int *any = team_at(sh.any, Tm);
    if (__any_sync(0xffffffffu, p) && (threadIdx.x & 31) == 0) any[r] = 1;
    if (Tm.r == 0 && threadIdx.x == 0) sh.any[(r + 1) % 3] = 0;  // last read two calls ago
    Tm.sync();
    const bool res = *(volatile int *)(any + r) != 0;
    if (threadIdx.x == 0) sh.any_r = (r + 1) % 3;
    __syncthreads();
    return res;
}

// receivers (receivers.py:31-58): strict >, first k wins ties (and the gradient and a copy of the
// receivers if grad and rec_ are not null).
template <int MODE, int U>
__device__ __forceinline__ void receivers_cells(const Grid &g, float dx, const float *z, int32_t *rec, int32_t *rec_,
                                                float *grad, ClusterTeam Tm)
{
    const int N = g.nx * g.ny;
    const unsigned mnx = 0xffffffffu / (unsigned)g.nx;
    FOR_TEAM_U(i0, stride, U, N) {
        int js[U][4];
        float zi[U], zn[U][4];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = i0 + u * stride;
            if (i >= N) break;
            int row, col;
            divmod_nx(i, g.nx, mnx, row, col);
            neighbours4<MODE>(g, i, row, col, js[u]);
            zi[u] = z[i];
#pragma unroll
            for (int k = 0; k < 4; ++k) zn[u][k] = js[u][k] != -1 ? z[js[u][k]] : zi[u];
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = i0 + u * stride;
            if (i >= N) break;
            // one quotient per cell, as in k_receivers_lean: division by dx is monotone, and the
            // first direction whose rounded quotient is the largest has a drop within 2^-21 of
            // the largest drop; when that direction's drop is the largest itself, it is the
            // answer.  Anything else (a near tie, a quotient that under- or overflows) takes
            // the ordered scan.
            float d[4], dmax = 0.f;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                d[k] = js[u][k] != -1 ? __fsub_rn(zi[u], zn[u][k]) : 0.f;
                dmax = fmaxf(dmax, d[k]);
            }
            int r = i;
            float sr = 0.f;
            if (dmax > 0.f) {
                const float near = __fmul_rn(dmax, 1.0f - 0x1p-21f);
                int kf = 3;
                float df = d[3];
#pragma unroll
                for (int k = 2; k >= 0; --k)
                    if (d[k] >= near) { kf = k; df = d[k]; }
                sr = __fdiv_rn(dmax, dx);
                r = kf == 0 ? js[u][0] : (kf == 1 ? js[u][1] : (kf == 2 ? js[u][2] : js[u][3]));
                if (df != dmax || !(sr >= 0x1p-100f && sr <= 0x1p100f)) {
                    r = i;
                    sr = 0.f;
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const float q = d[k] > 0.f ? __fdiv_rn(d[k], dx) : 0.f;
                        if (q > sr) {
                            sr = q;
                            r = js[u][k];
                        }
                    }
                }
            }
            rec[i] = r;
            if (rec_) rec_[i] = r;
            if (grad) grad[i] = sr;
        }
    }
    Tm.sync();
}

template <int MODE>
__device__ __noinline__ void tile_receivers(const Grid &g, float dx, const float *z, int32_t *rec, float *grad,
                                            ClusterTeam Tm)
{
    receivers_cells<MODE, 2>(g, dx, z, rec, nullptr, grad, Tm);
}

// reroute_flow(carve=True) (lakeflow.py:466-538), the reference's own steps by one block,
// from outer iteration it (with rec_ == rec; outer as the first iteration set it, or -1 to set
// it here).
template <int MODE>
__device__ __forceinline__ void reroute_steps(const Grid &g, const BatchTile &T, const BatchArrays &A, const float *z,
                                              BatchShm &sh, int it, int outer)
{
    const int N = g.nx * g.ny;
    const long long o = T.off, ob = T.boff;
    int32_t *rec = A.rcv + o, *rec_ = A.rec_ + o, *rec__ = A.rec__ + o, *bid = A.bid + o;
    const int lrounds = bceil_log2(N) + 1;
    int32_t *pl = A.ndnr + o;  // pit list (scratch of the accumulation / diffusion, free here)
    auto list_pits = [&]() {   // depression_counter (lakeflow.py:25-44), as an ascending list
        int n = 0;
        for (int b0 = 0; b0 < N; b0 += blockDim.x) {
            const int i = b0 + threadIdx.x;
            const int f = (i < N && rec_[i] == i && !leave<MODE>(g, i)) ? 1 : 0;
            int tot;
            const int q = bscan(f, sh, &tot);
            if (f) pl[n + q] = i;
            n += tot;
        }
        __syncthreads();
        return n;
    };
    for (; outer < 0 || it < outer; ++it) {
        const int nd = list_pits();
        if (nd == 0) break;  // (the labels the reference computes first are overwritten)
        if (outer < 0) outer = bceil_log2(nd) + 1;  // :500
        const bool acyclic = tile_labels_blocks<MODE>(g, N, rec_, rec__, bid, sh);
        if (!acyclic) tile_labels<MODE>(g, N, rec_, rec__, bid, A.mark + o, A.dnr + 4 * o, lrounds, sh, A.status);
        const int32_t *bl = acyclic ? pl : nullptr;  // basin ids: the pits', or any (labels of a cycle)
        tile_saddlesort<MODE>(g, N, bid, A.isb + o, A.zp + o, A.saddle + ob, A.snode + ob, A.outlet + ob,
                              A.inv + ob, z, bl, nd);
        tile_carve(N, rec, rec_, A.mark + o, A.tag + o, A.snode + ob, A.outlet + ob, bl, nd, A.status);
    }
}

template <int MODE>
__device__ __noinline__ void tile_reroute_steps(const Grid &g, const BatchTile &T, const BatchArrays &A, const float *z,
                                                BatchShm &sh, int it, int outer)
{
    reroute_steps<MODE>(g, T, A, z, sh, it, outer);
}

// A small tile, start to end, by one block: the reference's steps need fewer barriers than the list
// loop and its front.
template <int MODE>
__device__ __forceinline__ void small_tile(const BatchTile *tile, const BatchArrays &A, BatchShm &sh)
{
    const BatchTile T = *tile;
    const Grid g{T.nx, T.ny, MODE, MODE == 3 ? A.codes + T.off : nullptr};
    const long long o = T.off;
    const float *z = A.z + o;
    receivers_cells<MODE, 1>(g, T.dx, z, A.rcv + o, A.rec_ + o, A.grad + o, ClusterTeam{0, 1});
    reroute_steps<MODE>(g, T, A, z, sh, 0, -1);
    tile_accumulate(T.nx * T.ny, A.rcv + o, A.Q + o, A.counts + o, A.dnr + 4 * o, A.dnr_ + 4 * o, A.ndnr + o,
                    A.ndnr_ + o, A.src + o, A.p_ + o, A.c_ + o, A.mark + o, A.rec__ + o, sh);
}

// The same reroute by the single grid's device loop, the team's blocks together; a tile
// where the carve closes a receiver cycle goes on with the reference's steps.
//
// The steps are functions of their own: inlined into one kernel they spilled 2-3 KB of
// registers at 1024 threads.
template <int MODE>
__device__ __noinline__ void batch_front_steps(const LoopArgs &L, int32_t *R, ClusterTeam Tm, unsigned char *smem)
{
    reroute_tiles<MODE>(L, R, Tm, smem);
    Tm.sync();
    reroute_labels<MODE, true>(L, R, Tm);
    Tm.sync();
    reroute_first_border<MODE, false>(L, Tm, smem);
    Tm.sync();
}
template <int MODE>
__device__ __noinline__ int batch_loop(const LoopArgs &L, ClusterTeam Tm, unsigned char *smem, int *it_outer)
{
    int it = it_outer[0], outer = it_outer[1], n_outer = 0;
    const int state = reroute_loop<MODE, true, true>(L, Tm, smem, it, outer, n_outer);
    __syncthreads();
    if (threadIdx.x == 0) {
        it_outer[0] = it;
        it_outer[1] = outer;
    }
    Tm.sync();
    return state;
}

template <int MODE>
__device__ __noinline__ void tile_reroute(const BatchTile &T, const BatchArrays &A, const float *z, BatchShm &sh,
                                          ClusterTeam Tm, unsigned char *smem)
{
    const Grid g{T.nx, T.ny, MODE, MODE == 3 ? A.codes + T.off : nullptr};
    const int N = g.nx * g.ny;
    const long long o = T.off, ob = T.boff;
    int32_t *R = reinterpret_cast<int32_t *>(A.p_) + o;  // later the segment list
    if (Tm.r == 0)
        for (int k = threadIdx.x; k < 64 + LOOP_ITS * LOOP_CTR; k += blockDim.x) sh.loop[k] = 0;
    if (threadIdx.x == 0) {
        LoopArgs &L = sh.la;
        int *ctr = team_at(sh.loop, Tm);
        int32_t *d = A.dnr + 4 * o, *e = A.dnr_ + 4 * o;  // 4 N entries each
        const int ntiles = (g.nx + TILE_W - 1) / TILE_W * ((g.ny + TILE_H - 1) / TILE_H);  // at most N / 4
        L.bid = A.bid + o; L.rec = A.rcv + o; L.rec_ = A.rec_ + o; L.J = A.rec__ + o;
        L.z = z; L.zp = nullptr; L.isb = nullptr;
        L.sad = A.saddle + ob; L.out = A.outlet + ob; L.snode = A.snode + ob;
        L.tag = A.tag + o; L.tag_ = A.tag_ + o; L.inv = A.inv + ob;
        L.fin = d; L.nf = d + N + 1;
        L.alist[0] = d + 2 * N + 2;
        L.dirty = d + 3 * N + 2; L.dtiles = L.dirty + ntiles;
        L.akey = reinterpret_cast<long long *>(e); L.abid = e + 2 * N; L.pit0 = e + 3 * N;
        L.pits[0] = A.ndnr + o; L.pits[1] = A.ndnr_ + o;
        L.alist[1] = A.mark + o;
        L.segs = R;
        L.ctl = ctr; L.ctl_out = nullptr;
        L.info = ctr + 16; L.bar = ctr + 24; L.it_ctr = ctr + 64;
        L.g = g;
    }
    __syncthreads();
    const int ntiles = (g.nx + TILE_W - 1) / TILE_W * ((g.ny + TILE_H - 1) / TILE_H);
    if (threadIdx.x == 0) sh.it_outer[0] = sh.it_outer[1] = 0;
    for (;;) {
        FOR_TEAM(k, ntiles) sh.la.dirty[k] = 0;
        Tm.sync();
        batch_front_steps<MODE>(sh.la, R, Tm, smem);
        const int state = batch_loop<MODE>(sh.la, Tm, smem, sh.it_outer);
        if (state == RR_WALKERR && Tm.r == 0 && threadIdx.x == 0) atomicOr(A.status, BST_CARVE);
        if (state != RR_GENERAL && state != RR_RESUME) break;
        // the carve closed a receiver cycle, or left one: one iteration of the reference's
        // steps by the first block (their N-wide passes take 5-30 ms on a tile of 10^6
        // cells), then the fast loop again from the receivers it leaves
        const int gi = state == RR_RESUME ? sh.it_outer[0] + 1 : sh.it_outer[0], outer = sh.it_outer[1];
        if (gi >= outer) break;
        if (Tm.r == 0) {
            tile_reroute_steps<MODE>(g, T, A, z, sh, gi, gi + 1);
            __syncthreads();
            for (int k = threadIdx.x; k < 64 + LOOP_ITS * LOOP_CTR; k += blockDim.x) sh.loop[k] = 0;
        }
        Tm.sync();
        if (threadIdx.x == 0) sh.it_outer[0] = gi + 1;
        __syncthreads();
        if (gi + 1 >= outer) break;
    }
    Tm.sync();
}

template <int MODE>
__device__ __forceinline__ void route_tile(const BatchTile &T, const BatchArrays &A, BatchShm &sh, ClusterTeam &Tm,
                                           unsigned char *smem)
{
    const Grid g{T.nx, T.ny, MODE, MODE == 3 ? A.codes + T.off : nullptr};
    const int N = T.nx * T.ny;
    const long long o = T.off;
    const float *z = A.z + o;
    tile_receivers<MODE>(g, T.dx, z, A.rcv + o, A.grad + o, Tm);
    tile_reroute<MODE>(T, A, z, sh, Tm, smem);
    // accumulate: Q holds the seed (flowfields.py:272-292).  Tiles the front takes (modes 0-2,
    // 3 x 3 and more) are accumulated after this launch, all together
    if (T.item0 >= 0 || Tm.r != 0) return;
    tile_accumulate(N, A.rcv + o, A.Q + o, A.counts + o, A.dnr + 4 * o, A.dnr_ + 4 * o, A.ndnr + o, A.ndnr_ + o,
                    A.src + o, A.p_ + o, A.c_ + o, A.mark + o, A.rec__ + o, sh);
}

// ---- GraphFlood on a tile (gf_fields.py:126-141) --------------------------------------
//
// One iteration: receivers, carve reroute, fill with delta (fill_topo.py:17-45,
// snapshot rounds), 5 diffusion sweeps (gf_hydrodynamics.py:24-75, sums in the
// serial order), Manning update (gf_hydrodynamics.py:79-129).  Per-tile constants
// are the f32 values the single-grid Flooder passes: dx2, prec*dx^2, manning.
struct GfParams {
    const float *cst;  // per tile (caller order): dx2, prec_dx2, manning, stop threshold on max|dh|
    float edgesw, dt, eps;
    int niter;
    int crit;          // 0: stop when max|dh| < threshold; 1: when mean|dh| < threshold; -1: never
    float *h;          // packed, in/out
    int32_t *iters;    // per tile (caller order): iterations run
    float *res;        // per tile: last max|dh| and mean|dh| (2 floats)
    float *trace;      // optional, per tile: niter x (max|dh|, mean|dh|)
};

// max and sum of v over the team (max as unsigned bits: |x| >= 0, NaN above all)
__device__ __forceinline__ void bmaxsum(float m, float sum, BatchShm &sh, ClusterTeam &Tm, float *om, float *os)
{
    unsigned mu = __float_as_uint(m);
    for (int o = 16; o; o >>= 1) {
        mu = max(mu, __shfl_xor_sync(0xffffffffu, mu, o));
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
    }
    int *ws = team_at(sh.ws, Tm);
    Tm.sync();
    if (Tm.r == 0 && threadIdx.x == 0) { sh.ws[0] = 0; sh.ws[1] = 0; }
    Tm.sync();
    if ((threadIdx.x & 31) == 0) {
        atomicMax((unsigned *)&ws[0], mu);
        atomicAdd((float *)&ws[1], sum);
    }
    Tm.sync();
    *om = __uint_as_float((unsigned)vload(ws));
    *os = __int_as_float(vload(ws + 1));
    Tm.sync();
}

// The steps of an iteration are functions of their own: inlined into one kernel they
// spilled registers at 1024 threads.

// fill_z_add_delta (fill_topo.py:99-125): rounds on snapshots of the records {pointer,
// surface}; the buffer that holds the final ones is returned.
__device__ __noinline__ const int2 *gf_fill(int N, int2 *fa, int2 *fb, const int32_t *rec, float *zh, float *h, float *href,
                                    int nr, float eps, BatchShm &sh, ClusterTeam Tm)
{
    FOR_TEAM(i, N) {
        const int r = rec[i];
        fa[i] = make_int2(r == i ? (i | (int)0x80000000) : r, __float_as_int(zh[i]));
    }
    Tm.sync();
    int2 *a = fa, *b = fb;
    for (int r = 0; r < nr; ++r) {
        const float inc = (float)(ldexp(1.0, r - 1) * (double)eps);
        bool ch = false;
        FOR_TEAM_U(i0, stride, 4, N) {
            int2 sv[4], tv[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int i = i0 + u * stride;
                sv[u] = i < N ? a[i] : make_int2(0, 0);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) tv[u] = a[sv[u].x & 0x7FFFFFFF];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int i = i0 + u * stride, q = sv[u].x & 0x7FFFFFFF;
                if (i >= N) break;
                int2 n = sv[u];
                if (q != i) {
                    const int qq = tv[u].x & 0x7FFFFFFF;
                    const float zi = __int_as_float(n.y), zq = __int_as_float(tv[u].y);
                    n.x = qq;
                    if (!(qq == q && zi > (tv[u].x < 0 ? zq : zh[q]))) n.y = __float_as_int(fmaxf(zi, __fadd_rn(zq, inc)));
                    ch |= n.x != sv[u].x || n.y != sv[u].y;
                }
                b[i] = n;
            }
        }
        const bool any = team_any(ch, sh, Tm);
        int2 *t = a; a = b; b = t;
        // a round that changed nothing is a fixed point of every later round
        if (!any) break;
    }
    FOR_TEAM(i, N) {
        const float zf = __int_as_float(a[i].y), hi = h[i], zi = zh[i];
        href[i] = hi;
        h[i] = __fadd_rn(hi, __fsub_rn(zf, zi));
        zh[i] = zf;
    }
    Tm.sync();
    return a;
}

// diffuse_Q_constant_prec (gf_hydrodynamics.py:24-75): a cell's outgoing weights once (-1:
// not a source), then 5 gather sweeps; the last one's result is in the returned array.
template <int MODE>
__device__ __noinline__ void gf_weights(const Grid &g, float dx, const float *zh, float *w, ClusterTeam Tm)
{
    const int N = g.nx * g.ny, nx = g.nx;
    const unsigned mnx = 0xffffffffu / (unsigned)nx;
    FOR_TEAM_U(i0, stride, 2, N) {
        int js[2][4];
        float zi[2], zn[2][4];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int i = i0 + u * stride;
            int row, col;
            divmod_nx(i, nx, mnx, row, col);
            if (i < N && !can_leave<MODE>(g, i, row, col)) neighbours4<MODE>(g, i, row, col, js[u]);
            else js[u][0] = js[u][1] = js[u][2] = js[u][3] = -1;  // leaving cells have no slopes
            zi[u] = i < N ? zh[i] : 0.f;
#pragma unroll
            for (int k = 0; k < 4; ++k) zn[u][k] = js[u][k] != -1 ? zh[js[u][k]] : zi[u];
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int i = i0 + u * stride;
            if (i >= N) break;
            float sk[4];
            float sums = 0.f;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                sk[k] = (js[u][k] != -1) ? fmaxf(0.f, __fdiv_rn(__fsub_rn(zi[u], zn[u][k]), dx)) : 0.f;
                sums = __fadd_rn(sums, sk[k]);
            }
            const bool src = !(sums == 0.f);
#pragma unroll
            for (int k = 0; k < 4; ++k) w[(size_t)k * N + i] = src ? __fdiv_rn(sk[k], sums) : -1.f;
        }
    }
    Tm.sync();
}
template <int MODE>
__device__ __noinline__ const float *gf_sweeps(const Grid &g, const float *w, float *Q, float *temp, float prec_dx2,
                                       ClusterTeam Tm)
{
    const int N = g.nx * g.ny, nx = g.nx;
    const unsigned mnx = 0xffffffffu / (unsigned)nx;
    const bool sym = MODE != 3 && nx >= 3 && g.ny >= 3;
    float *qa = Q, *qb = temp;
    for (int sw = 0; sw < 5; ++sw) {
        FOR_TEAM_U(j0, stride, 2, N) {
            float wv[2][4], qv[2][4];
            int js[2][4];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int j = j0 + u * stride;
                int row, col;
                divmod_nx(j, nx, mnx, row, col);
                // modes 0-2 on grids of at least 3 x 3: j's sources are its own neighbours,
                // and neighbour k sends to j through its opposite link 3 - k
                if (sym && j < N) neighbours4<MODE>(g, j, row, col, js[u]);
                else js[u][0] = js[u][1] = js[u][2] = js[u][3] = -1;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int i = js[u][k];
                    wv[u][k] = i != -1 ? w[(size_t)(3 - k) * N + i] : -1.f;
                    qv[u][k] = i != -1 ? qa[i] : 0.f;
                }
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int j = j0 + u * stride;
                if (j >= N) break;
                float acc = prec_dx2;
                if (sym) {
                    // ascending source: top, left, right, bottom, except beside a wrap
                    int (&x)[4] = js[u];
                    if (MODE != 0 && !(x[0] < x[1] && x[1] < x[2] && x[2] < x[3])) {
                        auto cs = [&](int p, int q) {
                            if (x[p] > x[q]) {
                                const int ti = x[p]; x[p] = x[q]; x[q] = ti;
                                float tf = wv[u][p]; wv[u][p] = wv[u][q]; wv[u][q] = tf;
                                tf = qv[u][p]; qv[u][p] = qv[u][q]; qv[u][q] = tf;
                            }
                        };
                        cs(0, 1); cs(2, 3); cs(0, 2); cs(1, 3); cs(1, 2);
                    }
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (!(wv[u][k] < 0.f)) acc = __fadd_rn(acc, __fmul_rn(wv[u][k], qv[u][k]));
                } else {
                    int row, col, c[8];
                    divmod_nx(j, nx, mnx, row, col);
                    const int n = donor_candidates(g, j, row, col, c);
                    for (int q = 0; q < n; ++q) {
                        const int i = c[q];
                        if (w[i] < 0.f) continue;
                        const float qi = qa[i];
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            if (neighbour_i<MODE>(g, i, k) == j)
                                acc = __fadd_rn(acc, __fmul_rn(w[(size_t)k * N + i], qi));
                    }
                }
                qb[j] = acc;
            }
        }
        Tm.sync();
        float *t = qa; qa = qb; qb = t;
    }
    return qa;
}

// Manning update (gf_hydrodynamics.py:79-129; h receives tdh twice, :127-129); slopes from
// the fill's records a, which hold the filled surface; the diffused qa goes into Q.
// Returns this thread's largest |dh| and the sum.
__device__ __noinline__ float2 gf_update(int N, const int2 *a, const int32_t *rec, const float *qa, float *Q, float *h,
                                 float *zh, const float *href, float dx, float dx2, float manning,
                                 float edgesw, float dt, ClusterTeam Tm)
{
    float m = 0.f, sum = 0.f;
    FOR_TEAM(i, N) {
        const int r = rec[i];
        const float zi = __int_as_float(a[i].y), qi = qa[i], hi = h[i];
        float tS = edgesw;
        if (r != i) tS = fmaxf(__fdiv_rn(__fsub_rn(zi, __int_as_float(a[r].y)), dx), 1e-4f);
        Q[i] = qi;
        float Qo = __fmul_rn(dx, pow53(hi));
        Qo = __fdiv_rn(Qo, manning);
        Qo = __fmul_rn(Qo, __fsqrt_rn(tS));
        float tdh = __fdiv_rn(__fsub_rn(qi, Qo), dx2);
        tdh = __fmul_rn(tdh, dt);
        const float h1 = __fadd_rn(hi, tdh);
        if (h1 < 0.f) tdh = __fadd_rn(tdh, h1);
        const float hn = __fadd_rn(h1, tdh);
        h[i] = hn;
        zh[i] = __fadd_rn(zi, tdh);
        const float e = fabsf(__fsub_rn(hn, href[i]));
        m = __uint_as_float(max(__float_as_uint(m), __float_as_uint(e)));
        sum += e;
    }
    return make_float2(m, sum);
}

template <int MODE>
__device__ __forceinline__ void gf_tile(const BatchTile &T, const BatchArrays &A, const GfParams &P, BatchShm &sh,
                                        ClusterTeam &Tm, unsigned char *smem)
{
    const Grid g{T.nx, T.ny, MODE, MODE == 3 ? A.codes + T.off : nullptr};
    const int N = T.nx * T.ny;
    const long long o = T.off;
    float *zh = const_cast<float *>(A.z) + o, *h = P.h + o, *Q = A.Q + o;
    int32_t *rec = A.rcv + o;
    // scratch of the routing arrays, free once the reroute is done
    int2 *fa = reinterpret_cast<int2 *>(A.dnr + 4 * o), *fb = fa + N;  // fill records {pointer, surface}
    float *w = reinterpret_cast<float *>(A.dnr_) + 4 * o;
    float *temp = reinterpret_cast<float *>(A.ndnr) + o;
    float *href = reinterpret_cast<float *>(A.c_) + o;
    const float dx = T.dx, dx2 = P.cst[4 * T.id], prec_dx2 = P.cst[4 * T.id + 1], manning = P.cst[4 * T.id + 2];
    const float thr = P.cst[4 * T.id + 3];
    const int nr = bceil_log2(N);
    int it = 0;
    float rmax = 0.f, rmean = 0.f;
    for (; it < P.niter; ++it) {
        tile_receivers<MODE>(g, dx, zh, rec, nullptr, Tm);
        if (N <= GF_SMALL) {
            if (Tm.r == 0) {
                FOR_CELLS(i, N) A.rec_[o + i] = rec[i];
                __syncthreads();
                tile_reroute_steps<MODE>(g, T, A, zh, sh, 0, -1);
            }
            Tm.sync();
        } else {
            tile_reroute<MODE>(T, A, zh, sh, Tm, smem);
        }
        const int2 *a = gf_fill(N, fa, fb, rec, zh, h, href, nr, P.eps, sh, Tm);
        gf_weights<MODE>(g, dx, zh, w, Tm);
        const float *qa = gf_sweeps<MODE>(g, w, Q, temp, prec_dx2, Tm);
        const float2 e = gf_update(N, a, rec, qa, Q, h, zh, href, dx, dx2, manning, P.edgesw, P.dt, Tm);
        bmaxsum(e.x, e.y, sh, Tm, &rmax, &rmean);
        rmean /= (float)N;
        if (P.trace && Tm.r == 0 && threadIdx.x == 0) {
            P.trace[((size_t)T.id * P.niter + it) * 2] = rmax;
            P.trace[((size_t)T.id * P.niter + it) * 2 + 1] = rmean;
        }
        if ((P.crit == 0 && rmax < thr) || (P.crit == 1 && rmean < thr)) { ++it; break; }
    }
    if (Tm.r == 0 && threadIdx.x == 0) {
        P.iters[T.id] = it;
        P.res[2 * T.id] = rmax;
        P.res[2 * T.id + 1] = rmean;
    }
}

// The next tile of the queue for the whole team (largest first), or -1.
__device__ __forceinline__ int next_tile(int ntiles, int *queue, BatchShm &sh, ClusterTeam &Tm)
{
    Tm.sync();  // the previous tile is done, and its number read
    if (Tm.r == 0 && threadIdx.x == 0) sh.cur = atomicAdd(queue, 1);
    Tm.sync();
    const int k = *(volatile int *)team_at(&sh.cur, Tm);
    Tm.sync();
    return k < ntiles ? k : -1;
}

__device__ __forceinline__ ClusterTeam cluster_team()
{
    ClusterTeam Tm;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(Tm.r));
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(Tm.n));
    return Tm;
}

// Persistent: each team takes the next tile until the queue is empty.
__global__ void __launch_bounds__(1024) k_batch_route(int ntiles, BatchArrays A)
{
    extern __shared__ __align__(16) unsigned char batch_smem[];
    __shared__ BatchShm sh;
    if (A.small && *A.small) return;  // k_batch_small's batch
    ClusterTeam Tm = cluster_team();
    if (threadIdx.x == 0) sh.any[0] = sh.any[1] = sh.any[2] = sh.any_r = 0;
    for (;;) {
        const int k = next_tile(ntiles, A.queue, sh, Tm);
        if (k < 0) return;
        const BatchTile T = A.tiles[k];
        switch (T.mode) {
        case 0: route_tile<0>(T, A, sh, Tm, batch_smem); break;
        case 1: route_tile<1>(T, A, sh, Tm, batch_smem); break;
        case 2: route_tile<2>(T, A, sh, Tm, batch_smem); break;
        case 3:
            if (A.codes) route_tile<3>(T, A, sh, Tm, batch_smem);
            else if (threadIdx.x == 0) atomicOr(A.status, BST_MODE);
            break;
        default:
            if (threadIdx.x == 0) atomicOr(A.status, BST_MODE);
            break;
        }
    }
}

// A batch of small tiles, one block per tile.  A kernel of its own: without the list loop's shared
// memory the steps' scratch stays in L1 (2000 tiles of 32 x 32 cells 1476 us, 1791 inside
// k_batch_route), and with nothing else inlined they spill nothing.
__global__ void __launch_bounds__(1024) k_batch_small(int ntiles, BatchArrays A)
{
    __shared__ BatchShm sh;
    if (!*A.small) return;
    for (;;) {
        if (threadIdx.x == 0) sh.cur = atomicAdd(A.queue, 1);
        __syncthreads();
        const int k = sh.cur;
        __syncthreads();
        if (k >= ntiles) return;
        switch (A.tiles[k].mode) {
        case 0: small_tile<0>(A.tiles + k, A, sh); break;
        case 1: small_tile<1>(A.tiles + k, A, sh); break;
        case 2: small_tile<2>(A.tiles + k, A, sh); break;
        case 3:
            if (A.codes) small_tile<3>(A.tiles + k, A, sh);
            else if (threadIdx.x == 0) atomicOr(A.status, BST_MODE);
            break;
        default:
            if (threadIdx.x == 0) atomicOr(A.status, BST_MODE);
            break;
        }
        __syncthreads();
    }
}

// Persistent GraphFlood: each team runs whole tiles to their stop, largest first.
__global__ void __launch_bounds__(1024) k_batch_graphflood(int ntiles, BatchArrays A, GfParams P)
{
    extern __shared__ __align__(16) unsigned char batch_smem[];
    __shared__ BatchShm sh;
    ClusterTeam Tm = cluster_team();
    if (threadIdx.x == 0) sh.any[0] = sh.any[1] = sh.any[2] = sh.any_r = 0;
    for (;;) {
        const int k = next_tile(ntiles, A.queue, sh, Tm);
        if (k < 0) return;
        const BatchTile T = A.tiles[k];
        switch (T.mode) {
        case 0: gf_tile<0>(T, A, P, sh, Tm, batch_smem); break;
        case 1: gf_tile<1>(T, A, P, sh, Tm, batch_smem); break;
        case 2: gf_tile<2>(T, A, P, sh, Tm, batch_smem); break;
        case 3:
            if (A.codes) gf_tile<3>(T, A, P, sh, Tm, batch_smem);
            else if (threadIdx.x == 0) atomicOr(A.status, BST_MODE);
            break;
        default:
            if (threadIdx.x == 0) atomicOr(A.status, BST_MODE);
            break;
        }
    }
}

__global__ void k_batch_reset(int *ctr, int *acc_ctr)
{
    if (threadIdx.x < 2) ctr[threadIdx.x] = 0;
    if (acc_ctr) acc_ctr[threadIdx.x] = 0;
}

// Workspace layout, identical for the plan and the launches.
struct BatchWs {
    BatchArrays A;
    BatchTile *tiles, *by_offset;  // largest first; in packed order
    int *ctr;
    int *limits, *items, *acc_ctr;
    int32_t *priv;  // 4 per cell: the memory of rec_, rec__, bid and mark
    bool ok;
};

// Work items of the accumulation front: a tile nx x ny has ceil(nx/64) ceil(ny/24) <=
// nx ny / 37 + 1 of them (tiles of at least 3 x 3; 3 x (24 k + 1) comes closest).
static size_t batch_item_cap(long long total, int ntiles) { return (size_t)(total / 37 + ntiles); }

static BatchWs carve_batch(void *ws, size_t wsb, long long total, int ntiles, size_t *used = nullptr)
{
    Carver cv(ws, wsb);
    const size_t n = (size_t)total, nb = n + (size_t)ntiles;
    BatchWs w{};
    BatchArrays &A = w.A;
    w.ctr = cv.take<int>(64);
    w.tiles = cv.take<BatchTile>((size_t)ntiles);
    w.by_offset = cv.take<BatchTile>((size_t)ntiles);
    w.limits = cv.take<int>(64);
    w.items = cv.take<int>(batch_item_cap(total, ntiles));
    w.acc_ctr = cv.take<int>(BATCH_ACC_CTR);
    w.priv = cv.take<int32_t>(4 * n);
    A.rec_ = w.priv;
    A.rec__ = A.rec_ + n;
    A.bid = A.rec__ + n;
    A.mark = A.bid + n;
    A.zp = cv.take<float>(n);
    A.isb = cv.take<uint8_t>(n);
    A.tag = cv.take<uint8_t>(n);
    A.tag_ = cv.take<uint8_t>(n);
    A.saddle = cv.take<long long>(nb);
    A.outlet = cv.take<long long>(nb);
    A.snode = cv.take<int32_t>(nb);
    A.inv = cv.take<uint8_t>(nb);
    A.dnr = cv.take<int32_t>(4 * n);
    A.dnr_ = cv.take<int32_t>(4 * n);
    A.ndnr = cv.take<int32_t>(n);
    A.ndnr_ = cv.take<int32_t>(n);
    A.src = cv.take<int32_t>(n);
    A.p_ = cv.take<float>(n);
    A.c_ = cv.take<uint32_t>(n);
    A.tiles = w.tiles;
    A.queue = w.ctr;
    A.status = w.ctr + 1;
    w.ok = A.c_ != nullptr;
    if (used) *used = cv.off;
    return w;
}

}  // namespace pff

using namespace pff;

extern "C" size_t pff_batch_workspace_bytes(long long total_cells, int ntiles)
{
    if (total_cells <= 0 || ntiles <= 0) return 0;
    size_t used = 0;
    carve_batch(nullptr, 0, total_cells, ntiles, &used);
    return used + 256;
}

namespace pff {
// Blocks per tile (a cluster).  More blocks shorten the largest tile's chain, which bounds a
// batch whose tiles differ much, and fill the GPU when tiles are few; each costs a share of
// cluster barriers.
static int batch_team(long long total, int ntiles, int slots)
{
    const long long avg = total / ntiles;
    int t = 1;
    while (t < 8 && (long long)ntiles * t * 2 <= slots && avg >= 2048LL * t) t *= 2;
    if (avg >= 65536) t = std::max(t, 4);
    return t;
}

// A batch whose largest tile has at most so many cells is k_batch_small's, by the threads of a block
// (1024, 512, 256).  The steps beat the list loop while barriers cost more than passes over
// every cell.  Tiles of 24 x 24 cells: 40 of them take 118 us with 1024 threads and 183 by the loop, 2000
// take 900 and 1150; 48 x 48: 205 and 250, but 2000 of them 2198 and 2126, and 40 of 56 x 56
// with 512 threads 264 and 259; with 256 threads 40 of 40 x 40 237 and 239.  Mixed batches go by their
// largest tile, the last to end: 40 of 24 to 60 cells a side 219 and 234, of 24 to 75 289 and
// 275.  Where tiles outnumber the SMs the smaller ones make up for it: 200 of 24 to 75 384 and
// 476 (but of 64 x 64 567 and 503), with 512 threads 280 of 37 to 60 328 and
// 367 (220 of 40 to 66 368 and 344).
constexpr int SMALL_CLASSES = 3;
static int small_class(int threads) { return threads == 1024 ? 0 : (threads == 512 ? 1 : 2); }
static int small_cells(int cls, int ntiles, long long total)
{
    if (cls == 2) return 1900;
    if (ntiles > 300) return 2600;
    const bool many = ntiles > 148 && total <= (cls == 0 ? 2800LL : 2400LL) * ntiles;
    return cls == 0 ? (many ? 5600 : 3600) : (many ? 4400 : 3100);
}

struct BatchShape {
    int threads, ctas_per_sm, team, blocks;
};

// The launch of `kernel` for the shape asked for: ctas_per_sm clamped to [1, occupancy].
template <class K>
static int batch_shape(K kernel, int threads, int ctas_per_sm, long long total, int ntiles, BatchShape *s)
{
    int dev = 0, nsm = 148, occ = 1;
    PFF_CUDA(cudaGetDevice(&dev));
    PFF_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    const size_t smem = (size_t)(threads / TILE_THREADS) * LOOP_GROUP_BYTES;
    PFF_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, LOOP_SMEM));
    PFF_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, threads, smem));
    if (ctas_per_sm < 1) ctas_per_sm = 1;
    if (ctas_per_sm > occ) ctas_per_sm = occ > 0 ? occ : 1;
    const int team = batch_team(total, ntiles, nsm * ctas_per_sm);
    *s = BatchShape{threads, ctas_per_sm, team, std::min(std::max(nsm * ctas_per_sm / team, 1), ntiles) * team};
    return PFF_OK;
}

// GraphFlood with the shape left to the library (ctas_per_sm < 1).  More tiles than SMs: two
// half-size blocks per SM hold twice the tiles at once, and the steps are bound by latency,
// not by threads (256 tiles of 128 x 128 on 148 SMs took two rounds of one block each).
static int gf_choose(int ntiles, int *threads, int *ctas_per_sm)
{
    if (*ctas_per_sm >= 1) return PFF_OK;
    int dev = 0, nsm = 148;
    PFF_CUDA(cudaGetDevice(&dev));
    PFF_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    *ctas_per_sm = 1;
    if (*threads == 1024 && ntiles > nsm) {
        *threads = 512;
        *ctas_per_sm = 2;
    }
    return PFF_OK;
}

template <class K, class... Args>
static int launch_batch(K kernel, int threads, int ctas_per_sm, long long total, int ntiles, cudaStream_t st, Args... args)
{
    BatchShape s{};
    PFF_TRY(batch_shape(kernel, threads, ctas_per_sm, total, ntiles, &s));
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)s.blocks);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = (size_t)(threads / TILE_THREADS) * LOOP_GROUP_BYTES;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)s.team;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    PFF_CUDA(cudaLaunchKernelEx(&cfg, kernel, args...));
    count_launch();
    return PFF_OK;
}

static int batch_check(long long total, int ntiles, void *ws, size_t wsb, const char *who)
{
    if (ntiles <= 0 || total <= 0) {
        set_error("%s: empty batch", who);
        return PFF_ERR_ARG;
    }
    if (!ws || wsb < pff_batch_workspace_bytes(total, ntiles)) {
        set_error("%s: workspace too small", who);
        return PFF_ERR_WORKSPACE;
    }
    return PFF_OK;
}
}  // namespace pff

extern "C" long long pff_batch_plan(const int32_t *tile_nx, const int32_t *tile_ny, const int32_t *tile_mode,
                                    const float *tile_dx, int ntiles, long long *tile_offset, int32_t *order,
                                    void *workspace, size_t workspace_bytes, void *stream)
{
    clear_error();
    if (ntiles <= 0 || !tile_nx || !tile_ny || !tile_mode || !tile_dx || !tile_offset) {
        set_error("pff_batch_plan: bad arguments");
        return -PFF_ERR_ARG;
    }
    long long off = 0;
    for (int t = 0; t < ntiles; ++t) {
        const int nx = tile_nx[t], ny = tile_ny[t], md = tile_mode[t];
        if (nx < 2 || ny < 2 || md < 0 || md > 3 || (long long)nx * ny * 4 >= (1LL << 31) ||
            !(tile_dx[t] > 0.f)) {
            set_error("pff_batch_plan: tile %d: bad size %dx%d, mode %d or dx (modes 0-3)", t, nx, ny,
                      md);
            return -PFF_ERR_ARG;
        }
        tile_offset[t] = off;
        off += (long long)nx * ny;
    }
    const long long total = off;
    if (!workspace) return total;  // size query
    const int rc = batch_check(total, ntiles, workspace, workspace_bytes, "pff_batch_plan");
    if (rc) return -rc;
    // largest tiles first (longest-processing-time order); equal sizes by tile index
    int *ord = new int[ntiles];
    for (int t = 0; t < ntiles; ++t) ord[t] = t;
    auto cells = [&](int t) { return (long long)tile_nx[t] * tile_ny[t]; };
    std::stable_sort(ord, ord + ntiles, [&](int a, int b) { return cells(a) > cells(b); });
    std::vector<BatchTile> hp(ntiles), ht(ntiles);  // packed order, largest first
    std::vector<int> items;
    int limits[3 + SMALL_CLASSES] = {64, 0, 0};  // from [3] on, per class, whether the batch is k_batch_small's
    bool small = true;  // with every launch shape
    for (int c = 0; c < SMALL_CLASSES; ++c) {
        limits[3 + c] = cells(ord[0]) <= small_cells(c, ntiles, total);
        small = small && limits[3 + c];
    }
    for (int t = 0; t < ntiles; ++t) {
        const int nx = tile_nx[t], ny = tile_ny[t], logn = bceil_log2(cells(t)) + 1;
        // packed cell ids of the accumulation are 32-bit
        const bool front = !small && batch_front_takes(nx, ny, tile_mode[t]) && total < 2000000000LL;
        hp[t] = BatchTile{tile_offset[t], tile_offset[t] + t, nx, ny, tile_mode[t], t, tile_dx[t],
                          front ? (int)items.size() : -1, logn, 0};
        if (!front) continue;
        items.insert(items.end(), (size_t)batch_front_items(nx, ny), t);
        limits[0] = std::min(limits[0], logn);
        limits[1] = std::max(limits[1], logn);
    }
    limits[2] = (int)items.size();
    for (int k = 0; k < ntiles; ++k) {
        ht[k] = hp[ord[k]];
        if (order) order[k] = ord[k];
    }
    BatchWs w = carve_batch(workspace, workspace_bytes, total, ntiles);
    cudaStream_t st = S(stream);
    cudaError_t e1 = cudaMemcpyAsync(w.tiles, ht.data(), sizeof(BatchTile) * ntiles, cudaMemcpyHostToDevice, st);
    if (e1 == cudaSuccess)
        e1 = cudaMemcpyAsync(w.by_offset, hp.data(), sizeof(BatchTile) * ntiles, cudaMemcpyHostToDevice, st);
    if (e1 == cudaSuccess) e1 = cudaMemcpyAsync(w.limits, limits, sizeof(limits), cudaMemcpyHostToDevice, st);
    if (e1 == cudaSuccess && !items.empty())
        e1 = cudaMemcpyAsync(w.items, items.data(), sizeof(int) * items.size(), cudaMemcpyHostToDevice, st);
    const cudaError_t e2 = cudaStreamSynchronize(st);  // the host arrays must outlive the copies
    delete[] ord;
    if (e1 != cudaSuccess || e2 != cudaSuccess) {
        set_error("pff_batch_plan: descriptor upload: %s", cudaGetErrorString(e1 != cudaSuccess ? e1 : e2));
        return -PFF_ERR_CUDA;
    }
    return total;
}

extern "C" int pff_batch_route(const float *z, const uint8_t *codes, int32_t *receivers, float *gradient, float *Q,
                               uint32_t *counts, long long total_cells, int ntiles, int threads, int ctas_per_sm,
                               void *workspace, size_t workspace_bytes, void *stream)
{
    clear_error();
    PFF_TRY(batch_check(total_cells, ntiles, workspace, workspace_bytes, "pff_batch_route"));
    if (!z || !receivers || !gradient || !Q || !counts) {
        set_error("pff_batch_route: null pointer");
        return PFF_ERR_ARG;
    }
    if (threads != 256 && threads != 512 && threads != 1024) {
        set_error("pff_batch_route: threads must be 256, 512 or 1024 (got %d)", threads);
        return PFF_ERR_ARG;
    }
    BatchWs w = carve_batch(workspace, workspace_bytes, total_cells, ntiles);
    BatchArrays A = w.A;
    A.z = z;
    A.codes = codes;
    A.rcv = receivers;
    A.grad = gradient;
    A.Q = Q;
    A.counts = counts;
    cudaStream_t st = S(stream);
    { k_batch_reset<<<1, BATCH_ACC_CTR, 0, st>>>(w.ctr, w.acc_ctr); count_launch(); }
    const int cls = small_class(threads);
    if (total_cells <= (long long)small_cells(cls, ntiles, total_cells) * ntiles) {  // else the largest tile is larger
        A.small = w.limits + 3 + cls;
        int dev = 0, nsm = 148, occ = 1;
        PFF_CUDA(cudaGetDevice(&dev));
        PFF_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
        PFF_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_batch_small, threads, 0));
        const int grid = std::min(nsm * std::max(std::min(ctas_per_sm, occ), 1), ntiles);
        { k_batch_small<<<grid, threads, 0, st>>>(ntiles, A); count_launch(); }
    }
    PFF_TRY(launch_batch(k_batch_route, threads, ctas_per_sm, total_cells, ntiles, st, ntiles, A));
    if (total_cells < 2000000000LL) {
        BatchAcc b{};
        b.rcv = receivers; b.Q = Q; b.counts = counts;
        b.bufA = A.dnr; b.bufB = A.dnr_; b.priv = w.priv;
        b.la[0] = A.ndnr; b.la[1] = A.ndnr_;
        b.lf[0] = A.src; b.lf[1] = reinterpret_cast<int *>(A.p_);
        b.ctr = w.acc_ctr; b.status = A.status; b.small = A.small;
        b.by_offset = w.by_offset; b.items = w.items; b.limits = w.limits;
        b.total = total_cells; b.ntiles = ntiles;
        PFF_TRY(launch_batch_accumulate(b, st));
    }
    return check_cuda("pff_batch_route");
}

extern "C" int pff_batch_status(long long total_cells, int ntiles, void *workspace, size_t workspace_bytes,
                                int *status, void *stream)
{
    clear_error();
    PFF_TRY(batch_check(total_cells, ntiles, workspace, workspace_bytes, "pff_batch_status"));
    if (!status) {
        set_error("pff_batch_status: null pointer");
        return PFF_ERR_ARG;
    }
    BatchWs w = carve_batch(workspace, workspace_bytes, total_cells, ntiles);
    cudaStream_t st = S(stream);
    PFF_CUDA(cudaMemcpyAsync(status, w.A.status, sizeof(int), cudaMemcpyDeviceToHost, st));
    PFF_CUDA(cudaStreamSynchronize(st));
    return PFF_OK;
}

extern "C" int pff_batch_graphflood(float *zh, const uint8_t *codes, float *h, float *Q, const float *tile_consts,
                                    float edgesw, float dt,
                                    int niter, int crit, int32_t *iters, float *residuals, float *trace,
                                    long long total_cells, int ntiles, int threads, int ctas_per_sm, void *workspace,
                                    size_t workspace_bytes, void *stream)
{
    clear_error();
    PFF_TRY(batch_check(total_cells, ntiles, workspace, workspace_bytes, "pff_batch_graphflood"));
    if (!zh || !h || !Q || !tile_consts || !iters || !residuals || niter < 0 || crit < -1 || crit > 1) {
        set_error("pff_batch_graphflood: bad arguments");
        return PFF_ERR_ARG;
    }
    if (threads != 256 && threads != 512 && threads != 1024) {
        set_error("pff_batch_graphflood: threads must be 256, 512 or 1024 (got %d)", threads);
        return PFF_ERR_ARG;
    }
    BatchWs w = carve_batch(workspace, workspace_bytes, total_cells, ntiles);
    BatchArrays A = w.A;
    A.z = zh;
    A.codes = codes;
    A.Q = Q;
    A.rcv = A.src;  // the rerouted receivers of each iteration (the accumulation arrays are unused)
    A.grad = nullptr;
    A.counts = nullptr;
    GfParams P{tile_consts, edgesw, dt, 1e-3f, niter, crit, h, iters, residuals, trace};
    cudaStream_t st = S(stream);
    { k_batch_reset<<<1, BATCH_ACC_CTR, 0, st>>>(w.ctr, nullptr); count_launch(); }
    PFF_TRY(gf_choose(ntiles, &threads, &ctas_per_sm));
    PFF_TRY(launch_batch(k_batch_graphflood, threads, ctas_per_sm, total_cells, ntiles, st, ntiles, A, P));
    return check_cuda("pff_batch_graphflood");
}

extern "C" int pff_batch_shape(int graphflood, long long total_cells, int ntiles, int *threads, int *ctas_per_sm,
                               int *team)
{
    clear_error();
    if (!threads || !ctas_per_sm || !team || total_cells <= 0 || ntiles <= 0 ||
        (*threads != 256 && *threads != 512 && *threads != 1024)) {
        set_error("pff_batch_shape: bad arguments");
        return PFF_ERR_ARG;
    }
    BatchShape s{};
    if (graphflood) {
        PFF_TRY(gf_choose(ntiles, threads, ctas_per_sm));
        PFF_TRY(batch_shape(k_batch_graphflood, *threads, *ctas_per_sm, total_cells, ntiles, &s));
    } else {
        PFF_TRY(batch_shape(k_batch_route, *threads, *ctas_per_sm, total_cells, ntiles, &s));
    }
    *threads = s.threads;
    *ctas_per_sm = s.ctas_per_sm;
    *team = s.team;
    return PFF_OK;
}
