// libpff accumulation: donor inversion and rake-and-compress tree contraction.
//
// Semantics follow pyfastflow/flow/downstream_propag.py exactly:
//   - donor slots hold donors in ascending cell index (the reference's serial
//     atomic order, :88-96);
//   - each round reads a consistent start-of-round snapshot through the
//     ping-pong buffers and per-node epoch tags src = +-(round+1) (:21-56), so
//     the result is independent of thread scheduling and bit-identical to the
//     serial execution, f32 sums included.
// The structure of the contraction (which donor is raked or compressed in which
// round) does not depend on the payload, so one pass carries both the f32
// payload p and an exact uint32 count payload c.
#include <cub/block/block_scan.cuh>
#include <algorithm>
#include <type_traits>
#include "pff_coop.cuh"
#include "pff_internal.h"

namespace pff {

__global__ void k_rcv2donor_scatter(const int32_t *__restrict__ rcv, int32_t *dnr, int32_t *ndnr, int N)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= N) return;
    const int r = rcv[t];
    if (r == t) return;
    const int slot = atomicAdd(ndnr + r, 1);
    if (slot < 4) dnr[4 * (long long)r + slot] = t;
}

// Order each node's (at most 4) donor slots by ascending donor index.
__global__ void k_sort_donors(int32_t *dnr, const int32_t *__restrict__ ndnr, int N)
{
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= N) return;
    const int n = min(ndnr[r], 4);
    if (n < 2) return;
    int4 *p4 = reinterpret_cast<int4 *>(dnr) + r;
    int4 v = *p4;
    int d[4] = {v.x, v.y, v.z, v.w};
    for (int a = 1; a < n; ++a) {
        int x = d[a], b = a - 1;
        while (b >= 0 && d[b] > x) { d[b + 1] = d[b]; --b; }
        d[b + 1] = x;
    }
    *p4 = make_int4(d[0], d[1], d[2], d[3]);
}

__device__ __forceinline__ bool get_src(const int32_t *src, int t, int it)
{
    const int e = src[t];
    bool flip = e < 0;
    if (abs(e) == it + 1) flip = !flip;
    return flip;
}

// One rake-and-compress round (downstream_propag.py:157-179).
// If CNT, a second payload c/c_ (uint32) follows the same contraction.
// round_flags (optional): round_flags[it] != 0 if any node worked this round;
// a round whose predecessor did no work returns at once (nothing can change).
template <bool CNT>
__global__ void __launch_bounds__(256) k_rake(int32_t *dnr, int32_t *ndnr, float *p, int32_t *src,
                                              int32_t *dnr_, int32_t *ndnr_, float *p_, uint32_t *c,
                                              uint32_t *c_, int it, int N, int *round_flags)
{
    if (round_flags && it > 0 && *(volatile int *)(round_flags + it - 1) == 0) return;
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    if (tid >= N) return;
    const bool flip = get_src(src, tid, it);
    int todo = flip ? ndnr_[tid] : ndnr[tid];
    if (todo <= 0) return;
    const long long base = 4LL * tid;
    const long long lim = 4LL * N;
    int donors[4] = {-1, -1, -1, -1};
    bool worked = false;
    float padd = 0.f;
    uint32_t cadd = 0;
    int i = 0;
    while (i < todo && i < 4) {
        if (donors[i] == -1) donors[i] = flip ? dnr_[base + i] : dnr[base + i];
        const int did = donors[i];
        const bool fd = get_src(src, did, it);
        const int nd = fd ? ndnr_[did] : ndnr[did];
        if (nd <= 1) {
            if (!worked) {
                padd = flip ? p_[tid] : p[tid];
                if (CNT) cadd = flip ? c_[tid] : c[tid];
            }
            worked = true;
            padd = __fadd_rn(padd, fd ? p_[did] : p[did]);
            if (CNT) cadd += fd ? c_[did] : c[did];
            if (nd == 0) {
                --todo;
                if (todo > i && base + todo < lim) donors[i] = flip ? dnr_[base + todo] : dnr[base + todo];
                --i;
            } else {
                donors[i] = fd ? dnr_[4LL * did] : dnr[4LL * did];
            }
        }
        ++i;
    }
    if (!worked) return;
    const int m = todo < 4 ? todo : 4;
    if (flip) {
        ndnr[tid] = todo;
        p[tid] = padd;
        if (CNT) c[tid] = cadd;
        for (int j = 0; j < m; ++j) dnr[base + j] = donors[j];
    } else {
        ndnr_[tid] = todo;
        p_[tid] = padd;
        if (CNT) c_[tid] = cadd;
        for (int j = 0; j < m; ++j) dnr_[base + j] = donors[j];
    }
    src[tid] = (flip ? 1 : -1) * (it + 1);
    if (round_flags) round_flags[it] = 1;
}

template <class T>
__global__ void k_fuse(T *A, const int32_t *__restrict__ src, const T *__restrict__ B, int it, int N)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= N) return;
    if (get_src(src, t, it)) A[t] = B[t];
}

__global__ void k_fill_u32(uint32_t *a, uint32_t v, int N)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < N) a[t] = v;
}

static int ceil_log2(long long n)
{
    int r = 0;
    long long p = 1;
    while (p < n) { p <<= 1; ++r; }
    return r;
}

// ---------------------------------------------------------------------------
// Whole accumulation with compacted active lists.
//
// The schedule is the reference's rake-and-compress (same rounds, same snapshot
// reads, same per-node donor order), so every f32 sum is formed exactly as in
// the reference; only nodes that still have donors are visited.  Node state:
//   public  {ndnr, p, c, d0}   16 B, read by the node's receiver -> double buffered
//   private {d1, d2, d3, -}    16 B, read and written only by the node itself
// Active nodes rewrite their public record into the next buffer every round;
// a node that finishes in round r has its final record copied into the other
// buffer during round r+1 (that buffer is write-only in round r+1).
struct __align__(16) Pub {
    int ndnr;
    float p;
    uint32_t c;
    int d0;
};

// Fallback path (receivers that are not D4 neighbours, or no grid given): scatter + sort.
__device__ __forceinline__ void acc_init(Pub *A, Pub *B, int4 *priv, const float *Q, uint32_t *counts, int N)
{
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < N; t += gridDim.x * blockDim.x) {
        const Pub s{0, Q[t], 1u, -1};
        A[t] = s;
        B[t] = s;
        priv[t] = make_int4(-1, -1, -1, -1);
        if (counts) counts[t] = 1u;
    }
}

__device__ __forceinline__ void acc_scatter(const int32_t *rcv, Pub *A, int4 *priv, int N, int *overflow)
{
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < N; t += gridDim.x * blockDim.x) {
        const int r = rcv[t];
        if (r == t) continue;
        const int slot = atomicAdd(&A[r].ndnr, 1);
        if (slot == 0) A[r].d0 = t;
        else if (slot < 4) reinterpret_cast<int *>(priv + r)[slot - 1] = t;
        else *overflow = 1;  // more than 4 donors: the reference's slots overflow into the next node's
    }
}

// Block-aggregated append of up to two predicates (order kept within a block).
template <int BS>
__device__ __forceinline__ void block_append2(bool pa, bool pf, int t, int *la, int *na, int *lf, int *nf)
{
    using Scan = cub::BlockScan<int, BS>;
    __shared__ typename Scan::TempStorage tmp;
    __shared__ int base_a, base_f;
    const int v = (pa ? 1 : 0) | (pf ? 0x10000 : 0);
    int ex, tot;
    Scan(tmp).ExclusiveSum(v, ex, tot);
    if (threadIdx.x == 0) {
        base_a = (tot & 0xFFFF) ? atomicAdd(na, tot & 0xFFFF) : 0;
        base_f = (nf && (tot >> 16)) ? atomicAdd(nf, tot >> 16) : 0;
    }
    __syncthreads();
    if (pa) la[base_a + (ex & 0xFFFF)] = t;
    if (pf) lf[base_f + (ex >> 16)] = t;
    __syncthreads();
}

// Sort each node's donor slots ascending, copy its public record to the second
// buffer, and list the nodes that have donors (round-0 active list).
template <int BS>
__device__ __forceinline__ void acc_list0(Pub *A, Pub *B, int4 *priv, int *list, int *nlist, int N)
{
    const int stride = gridDim.x * BS, trips = (N + stride - 1) / stride;
    for (int k = 0; k < trips; ++k) {
        const int t = k * stride + blockIdx.x * BS + threadIdx.x;
        int n = 0;
        if (t < N) {
            Pub s = A[t];
            n = s.ndnr;
            if (n >= 2) {
                int4 q = priv[t];
                int d[4] = {s.d0, q.x, q.y, q.z};
                const int m = n < 4 ? n : 4;
                for (int a = 1; a < m; ++a) {
                    int x = d[a], b = a - 1;
                    while (b >= 0 && d[b] > x) { d[b + 1] = d[b]; --b; }
                    d[b + 1] = x;
                }
                s.d0 = d[0];
                A[t].d0 = d[0];
                priv[t] = make_int4(d[1], d[2], d[3], -1);
            }
            if (n > 0) B[t] = s;
        }
        block_append2<BS>(n > 0, false, t, list, nlist, nullptr, nullptr);
    }
}

__global__ void __launch_bounds__(256) k_acc_init(Pub *A, Pub *B, int4 *priv, const float *Q, uint32_t *counts, int N)
{
    acc_init(A, B, priv, Q, counts, N);
}
__global__ void __launch_bounds__(256) k_acc_scatter(const int32_t *rcv, Pub *A, int4 *priv, int N, int *overflow)
{
    acc_scatter(rcv, A, priv, N, overflow);
}
__global__ void __launch_bounds__(256) k_acc_list0(Pub *A, Pub *B, int4 *priv, int *list, int *nlist, int N)
{
    acc_list0<256>(A, B, priv, list, nlist, N);
}

// Gather-form initialisation for D4 receivers: the donors of t are the cells
// among its grid neighbours and wrap partners whose receiver is t; visiting
// them in ascending index gives the reference's serial slot order without
// atomics or a sort.  Builds both public buffers, the private slots, the
// counts and the round-0 active list in one pass.  Sets *nonlocal if some
// receiver is not one of these candidates (then the scatter path redoes it).
template <int MODE, int BS>
__global__ void __launch_bounds__(BS) k_acc_gather(const int32_t *__restrict__ rcv, Pub *A, Pub *B, int4 *priv,
                                                   const float *__restrict__ Q, uint32_t *counts, int *list,
                                                   int *nlist, int *nonlocal, int *overflow, Grid g)
{
    const int col = blockIdx.x * 32 + (threadIdx.x & 31);
    const int row = blockIdx.y * (BS / 32) + (threadIdx.x >> 5);
    const bool in = col < g.nx && row < g.ny;
    const int t = row * g.nx + col;
    int nd = 0;
    if (in) {
        const int rt = rcv[t];
        bool ok = rt == t;
        int d[4] = {-1, -1, -1, -1};
        if (MODE != 3) {
            // the neighbour relation of modes 0-2 is symmetric: the donors of t are
            // among its own neighbours; sort them ascending (5 compare-swaps)
            int cn[4];
            neighbours4<MODE>(g, t, row, col, cn);
            int c0 = cn[0], c1 = cn[1], c2 = cn[2], c3 = cn[3];
            // -1 (no neighbour) sorts last
            auto key = [](int v) { return (unsigned)v; };
            auto cs = [&](int &a, int &b) { if (key(a) > key(b)) { int x = a; a = b; b = x; } };
            cs(c0, c1); cs(c2, c3); cs(c0, c2); cs(c1, c3); cs(c1, c2);
            const int cc[4] = {c0, c1, c2, c3};
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                const int j = cc[a];
                if (j < 0 || (a > 0 && j == cc[a - 1])) continue;
                if (j == rt) ok = true;
                if (rcv[j] == t) {
                    if (nd < 4) d[nd] = j;
                    ++nd;
                }
            }
        } else {
            int c[8];
            const int n = donor_candidates(g, t, row, col, c);
            for (int a = 0; a < n; ++a) {
                const int j = c[a];
                if (j == rt) ok = true;
                if (rcv[j] == t) {
                    if (nd < 4) d[nd] = j;
                    ++nd;
                }
            }
        }
        if (!ok) *nonlocal = 1;
        if (nd > 4) *overflow = 1;
        const Pub s{nd, Q[t], 1u, d[0]};
        A[t] = s;
        if (nd == 0) {
            // leaves: final from the start, in both buffers; active nodes rewrite B
            // in round 0 and write their counts when they finish
            B[t] = s;
            if (counts) counts[t] = 1u;
        }
        if (nd >= 2) priv[t] = make_int4(d[1], d[2], d[3], -1);
    }
    block_append2<BS>(nd > 0, false, t, list, nlist, nullptr, nullptr);
}

__device__ __forceinline__ int sel4(int k, int a, int b, int c, int d)
{
    return k == 0 ? a : (k == 1 ? b : (k == 2 ? c : d));
}
__device__ __forceinline__ void set4(int k, int v, int &a, int &b, int &c, int &d)
{
    a = k == 0 ? v : a;
    b = k == 1 ? v : b;
    c = k == 2 ? v : c;
    d = k == 3 ? v : d;
}
__device__ __forceinline__ Pub pick4(int q, const Pub &a, const Pub &b, const Pub &c, const Pub &d)
{
    return q == 0 ? a : (q == 1 ? b : (q == 2 ? c : d));
}

// The scan for a node with two donors of n0 and n1 donors (their first ones f0 and f1): which
// are absorbed, and the slots left.  A removed first donor leaves its slot to the second.
struct Two {
    int todo, w0, w1;
    bool a0, a1;
};
__device__ __forceinline__ Two two_donors(int n0, int n1, int own0, int own1, int f0, int f1)
{
    const int x0 = n0 == 1 ? f0 : own0, x1 = n1 == 1 ? f1 : own1;
    return Two{(n0 != 0) + (n1 != 0), n0 != 0 ? x0 : x1, x1, n0 <= 1, n1 <= 1};
}

// The result of an active node's round into the next buffers: 0 keeps donors, 1 finished
// (Q and count written).
__device__ __forceinline__ int acc_store(int t, const Pub &s, bool worked, int todo, float p, uint32_t c, int w0, int w1,
                                         int w2, int w3, Pub *nxt, int4 *priv, float *Q, uint32_t *counts)
{
    if (!worked) {
        nxt[t] = s;
        return 0;
    }
    nxt[t] = Pub{todo, p, c, todo > 0 ? w0 : s.d0};
    if (todo > 1) priv[t] = make_int4(w1, w2, w3, -1);
    if (todo > 0) return 0;
    Q[t] = p;
    if (counts) counts[t] = c;
    return 1;
}

// The reference's swap-remove scan (downstream_propag.py:131-162) of a node t with record s over
// the start-of-round states P0 .. P3 of its donors `own`, loaded up front (every one it
// can need is a start-of-round slot); slot k holds donor w_k whose preloaded state is q_k.
__device__ __forceinline__ int acc_scan(int t, const Pub &s, const int (&own)[4], const Pub &P0, const Pub &P1,
                                        const Pub &P2, const Pub &P3, Pub *nxt, int4 *priv, float *Q, uint32_t *counts)
{
    int todo = s.ndnr;
    int w0 = own[0], w1 = own[1], w2 = own[2], w3 = own[3];
    int q0 = 0, q1 = 1, q2 = 2, q3 = 3;
    bool worked = false;
    float padd = s.p;
    uint32_t cadd = s.c;
    int i = 0;
#pragma unroll
    for (int step = 0; step < 8; ++step) {  // each step advances i or removes a donor
        if (i >= todo || i >= 4) break;
        const int q = sel4(i, q0, q1, q2, q3);
        const Pub ds = pick4(q, P0, P1, P2, P3);
        if (ds.ndnr <= 1) {
            worked = true;
            padd = __fadd_rn(padd, ds.p);
            cadd += ds.c;
            if (ds.ndnr == 0) {
                --todo;
                if (todo > i && todo < 4) {
                    set4(i, sel4(todo, own[0], own[1], own[2], own[3]), w0, w1, w2, w3);
                    set4(i, todo, q0, q1, q2, q3);
                }
            } else {
                set4(i, ds.d0, w0, w1, w2, w3);
                ++i;
            }
        } else {
            ++i;
        }
    }
    return acc_store(t, s, worked, todo, padd, cadd, w0, w1, w2, w3, nxt, priv, Q, counts);
}

// A node with three or more donors (2-3 % of them).
__device__ __noinline__ int acc_node_many(int t, const Pub *cur, Pub *nxt, int4 *priv, float *Q, uint32_t *counts)
{
    const Pub s = cur[t];
    const int4 pq = priv[t];
    const int own[4] = {s.d0, pq.x, pq.y, pq.z};
    const Pub P0 = cur[own[0]], P1 = cur[own[1]], P2 = cur[own[2]];
    const Pub P3 = s.ndnr > 3 ? cur[own[3]] : s;
    return acc_scan(t, s, own, P0, P1, P2, P3, nxt, priv, Q, counts);
}

// An active node's round: its record s, its first donor's P0, its second donor d1 and that one's P1
// (where it has two).
__device__ __forceinline__ int acc_node(int t, const Pub &s, int d1, const Pub &P0, const Pub &P1, const Pub *cur, Pub *nxt,
                                        int4 *priv, float *Q, uint32_t *counts)
{
    if (s.ndnr > 2) return acc_node_many(t, cur, nxt, priv, Q, counts);
    const Two r = s.ndnr == 2 ? two_donors(P0.ndnr, P1.ndnr, s.d0, d1, P0.d0, P1.d0)
                              : Two{P0.ndnr != 0, P0.ndnr == 1 ? P0.d0 : s.d0, -1, P0.ndnr <= 1, false};
    float p = s.p;
    uint32_t c = s.c;
    if (r.a0) { p = __fadd_rn(p, P0.p); c += P0.c; }
    if (r.a1) { p = __fadd_rn(p, P1.p); c += P1.c; }
    return acc_store(t, s, r.a0 || r.a1, r.todo, p, c, r.w0, r.w1, -1, -1, nxt, priv, Q, counts);
}

// Every remaining round in one cooperative launch, a grid barrier between rounds.  Round
// it reads cnt[2 it] active nodes (list la[it & 1]) and cnt[2 it + 1] nodes that
// finished in round it - 1 (list lf[it & 1]; copied into the buffer written this
// round; with fin_q, round first0 also writes their Q and count: the nodes that
// finished inside the tile front), and ends when both are zero.
//
// What bounds it: the late rounds, whose lists are nearly empty.  One launch per round
// cost 2-4 us each for about 20 of them (285 us for the 24 rounds at 2048 x 2048); a
// barrier costs 1.3 us, and the empty ones at the end are skipped.  The early rounds wait on
// dependent loads (entry, record, slots, donors; DRAM 23 % busy at 32 warps per SM), so a
// warp takes 64 entries, two per thread, and issues each level's loads for both.  It
// collects what it keeps in shared memory, so the lists stay in runs of ascending cells
// whose donors share cache lines.
constexpr int ACC_THREADS = 1024, ACC_CAP = 128;
struct AccRounds {
    const int32_t *rcv;
    Pub *buf[2];
    int4 *priv;
    float *Q;
    uint32_t *counts;
    int *la[2], *lf[2];
    int *cnt;        // 2 per round
    int *nonlocal, *overflow;
    int N, first, logn;
    int *bar, *over_out;
    BarWait wait;
    // ragged batch: rounds end tile by tile (N is then the packed total, nonlocal unused)
    const BatchTile *tiles;
    int ntiles;
    const int *limits;  // [0] smallest, [1] largest logn of the tiles
    int *status;        // BST_* bits
};

// One round over a long list as a launch of its own, where no tile front takes the first rounds
// (custom boundaries, or no grid): 40 warps per SM, and one atomic per list and 256 entries
// where the cooperative rounds have 32 and one per 64 to 128; the lists keep their order.
// Nodes with three or four donors, for which that kernel calls a function, stay with their
// warp.  Every round by
// k_acc_rounds and with these: custom boundaries 2522 and 2339 us at 4096 x 4096, 698 and 682
// at 2048 x 2048, no grid 336 and 296 at 1200 x 1200.  Not the last round, nor after the
// gather has found other receivers.
constexpr int ACC_WIDE = 1 << 20;     // nodes from which they are used
constexpr int ACC_WIDE_ROUNDS = 7;    // 4 rounds: 2452 us at 4096 x 4096
template <int BS>
__global__ void __launch_bounds__(BS, 5) k_acc_round_wide(AccRounds a, int it)
{
    if (*a.nonlocal) return;
    const Pub *cur = a.buf[it & 1];
    Pub *nxt = a.buf[(it & 1) ^ 1];
    const int *la = a.la[it & 1], *lf = a.lf[it & 1];
    int *c2 = a.cnt + 2 * (it + 1);
    const int nA = a.cnt[2 * it], total = nA + a.cnt[2 * it + 1];
    const int stride = gridDim.x * BS, trips = (total + stride - 1) / stride;
    for (int k = 0; k < trips; ++k) {
        const int idx = k * stride + blockIdx.x * BS + threadIdx.x;
        int t = -1, res = 2;
        if (idx < nA) {
            t = la[idx];
            const Pub s = cur[t];
            int own[4] = {s.d0, -1, -1, -1};
            if (s.ndnr > 1) {
                const int4 pq = a.priv[t];
                own[1] = pq.x; own[2] = pq.y; own[3] = pq.z;
            }
            Pub P0 = s, P1 = s, P2 = s, P3 = s;
            P0 = cur[own[0]];
            if (s.ndnr > 1) P1 = cur[own[1]];
            if (s.ndnr > 2) P2 = cur[own[2]];
            if (s.ndnr > 3) P3 = cur[own[3]];
            res = acc_scan(t, s, own, P0, P1, P2, P3, nxt, a.priv, a.Q, a.counts);
        } else if (idx < total) {
            t = lf[idx - nA];
            nxt[t] = cur[t];
        }
        block_append2<BS>(res == 0, res == 1, t, a.la[(it & 1) ^ 1], c2, a.lf[(it & 1) ^ 1], c2 + 1);
    }
}

__global__ void __launch_bounds__(ACC_THREADS, 1) k_acc_rounds(AccRounds a)
{
    __shared__ int sa[ACC_THREADS / 32][ACC_CAP], sf[ACC_THREADS / 32][ACC_CAP];
    __shared__ int dead;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int gthreads = gridDim.x * ACC_THREADS;
    if (threadIdx.x == 0) dead = 0;
    GridBar bar{a.bar, a.wait};
    __syncthreads();
    int it = a.first, logn = a.logn, logmin = a.logn;
    if (a.tiles) {
        logmin = a.limits[0];
        logn = a.limits[1];
    } else if (*a.nonlocal) {  // the same for every block
        if (blockIdx.x == 0 && threadIdx.x == 0) a.cnt[0] = a.cnt[2 * it] = a.cnt[2 * it + 1] = 0;
        acc_init(a.buf[0], a.buf[1], a.priv, a.Q, a.counts, a.N);
        if (!bar.sync(&dead)) return;
        acc_scatter(a.rcv, a.buf[0], a.priv, a.N, a.overflow);
        if (!bar.sync(&dead)) return;
        acc_list0<ACC_THREADS>(a.buf[0], a.buf[1], a.priv, a.la[0], a.cnt, a.N);
        if (!bar.sync(&dead)) return;
        it = 0;
    }
    const int it0 = it;
    for (; it <= logn; ++it) {
        const int p = it & 1;
        const Pub *cur = a.buf[p];
        Pub *nxt = a.buf[p ^ 1];
        const int nA = vload(a.cnt + 2 * it), nF = vload(a.cnt + 2 * it + 1), total = nA + nF;
        if (total == 0) break;
        const int *la = a.la[p], *lf = a.lf[p];
        int *la2 = a.la[p ^ 1], *lf2 = a.lf[p ^ 1], *c2 = a.cnt + 2 * (it + 1);
        const bool fin_q = it == it0 && it > 0;
        int na = 0, nf = 0;  // buffered, warp-uniform
        auto flush = [&](int *buf, int &n, int *list, int *count) {
            __syncwarp();
            int base = 0;
            if (lane == 0 && n) base = atomicAdd(count, n);
            base = __shfl_sync(0xffffffffu, base, 0);
            for (int q = lane; q < n; q += 32) list[base + q] = buf[q];
            __syncwarp();
            n = 0;
        };
        for (int k0 = (blockIdx.x * (ACC_THREADS / 32) + wib) * 64; k0 < total; k0 += 2 * gthreads) {
            int t[2], d1[2], res[2];
            Pub sc[2], P0[2], P1[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int idx = k0 + 32 * u + lane;
                t[u] = idx < nA ? la[idx] : (idx < total ? lf[idx - nA] : -1);
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) sc[u] = t[u] >= 0 ? cur[t[u]] : Pub{0, 0.f, 0u, -1};
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const bool act = k0 + 32 * u + lane < nA;
                d1[u] = act && sc[u].ndnr == 2 ? a.priv[t[u]].x : -1;
                P0[u] = act ? cur[sc[u].d0] : sc[u];
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) P1[u] = d1[u] >= 0 ? cur[d1[u]] : P0[u];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int idx = k0 + 32 * u + lane;
                res[u] = 2;
                if (idx < nA) {
                    bool last = it == logn;
                    if (a.tiles && it >= logmin) {  // the tile's own last round
                        int lo = 0, hi = a.ntiles - 1;  // tiles sorted by offset: see k_batch_front
                        while (lo < hi) {
                            const int mid = (lo + hi + 1) >> 1;
                            if (a.tiles[mid].off <= t[u]) lo = mid;
                            else hi = mid - 1;
                        }
                        last = it == a.tiles[lo].logn;
                    }
                    const Pub &s = sc[u];
                    if (last) {  // the start-of-round value is the result (fuse(.., logn), :59-74)
                        a.Q[t[u]] = s.p;
                        if (a.counts) a.counts[t[u]] = s.c;
                    } else {
                        res[u] = acc_node(t[u], s, d1[u], P0[u], P1[u], cur, nxt, a.priv, a.Q, a.counts);
                    }
                } else if (idx < total) {
                    nxt[t[u]] = sc[u];
                    if (fin_q) {
                        a.Q[t[u]] = sc[u].p;
                        if (a.counts) a.counts[t[u]] = sc[u].c;
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const unsigned ma = __ballot_sync(0xffffffffu, res[u] == 0), mf = __ballot_sync(0xffffffffu, res[u] == 1);
                if (res[u] == 0) sa[wib][na + __popc(ma & ((1u << lane) - 1u))] = t[u];
                if (res[u] == 1) sf[wib][nf + __popc(mf & ((1u << lane) - 1u))] = t[u];
                na += __popc(ma);
                nf += __popc(mf);
            }
            if (na > ACC_CAP - 64) flush(sa[wib], na, la2, c2);
            if (nf > ACC_CAP - 64) flush(sf[wib], nf, lf2, c2 + 1);
        }
        if (na) flush(sa[wib], na, la2, c2);
        if (nf) flush(sf[wib], nf, lf2, c2 + 1);
        if (!bar.sync(&dead)) {  // a single grid's caller misses over_out
            if (a.status && blockIdx.x == 0 && threadIdx.x == 0) atomicOr(a.status, BST_ROUNDS);
            return;
        }
    }
    if (a.over_out && blockIdx.x == 0 && threadIdx.x == 0) {
        ((volatile int *)a.over_out)[0] = *a.overflow;
        __threadfence_system();
    }
}

// ---------------------------------------------------------------------------
// The first FR rounds over spatial tiles (D4 receivers, modes 0-2).
//
// Every donor link joins grid neighbours, and a compress replaces a donor by the
// donor's own donor, so at the start of round r a node's slots point at most 2^r
// hops upstream and its state depends only on the initial states within 2^r - 1
// hops.  The initial state of a cell needs the receivers of its neighbours, one
// more cell.  So one CTA loads a tile plus a halo of 2^FR cells (receivers and
// seeds), builds the initial states in shared memory, and runs the rounds with
// the rule of acc_node and acc_node_many: round r only over the cells within
// 2^FR - 2^(r+1) of the tile (what the later rounds of the tile's cells read),
// the last round in registers for the tile's cells alone.
//
// Outputs, for the tile's cells: the round-FR record in `cur_out` (the buffer
// round FR reads); leaves (no donors ever) also in `nxt_out` with their count 1;
// nodes still active go to the round-FR active list; nodes that finished inside
// the front go to the round-FR finished list, whose copy also writes their Q and
// count (Q is read here as the seeds of neighbouring tiles' halos, so it is
// written only after this launch).  Sets *nonlocal if some receiver is neither
// the cell nor a grid neighbour (then the scatter path redoes everything).
template <int FR>
struct Front {
    static constexpr int H = 1 << FR;
    static constexpr int TW = 64, TH = FR == 1 ? 16 : 24;
    static constexpr int RW = TW + 2 * H, RH = TH + 2 * H, NR = RW * RH;
    static constexpr int BS = 512;
    static constexpr size_t SMEM = (size_t)NR * (6 * 4 + 3 * 2 + 1);
    static_assert(NR < 0xFFFF, "local ids are 16-bit");
    static_assert((TW * TH) % BS == 0, "uniform output trips");
};

// One node's round on shared-memory snapshots (the rule of acc_node and acc_node_many; local ids).
struct FrontNode {
    int todo;
    float p;
    uint32_t c;
    int w0, w1, w2, w3;
    bool worked;
};

__device__ __forceinline__ FrontNode front_round(const float *pc, const uint32_t *cc, const uint32_t *nc,
                                                 uint32_t snd, float sp, uint32_t sc, int own0, int own1, int own2,
                                                 int own3)
{
    constexpr uint32_t NONE = 0xFFFFu;
    int todo = (int)(snd >> 16);
    if (todo == 1) {  // the common chain node: one donor, one step of the rule below
        const uint32_t dn = nc[own0];
        const int dnd = (int)(dn >> 16);
        if (dnd > 1) return FrontNode{1, sp, sc, own0, own1, own2, own3, false};
        const float p = __fadd_rn(sp, pc[own0]);
        const uint32_t c = sc + cc[own0];
        return FrontNode{dnd == 0 ? 0 : 1, p, c, dnd == 0 ? own0 : (int)(dn & NONE), own1, own2, own3, true};
    }
    uint32_t N0 = nc[own0], N1 = nc[own1], N2 = snd, N3 = snd;
    float P0 = pc[own0], P1 = pc[own1], P2 = sp, P3 = sp;
    uint32_t C0 = cc[own0], C1 = cc[own1], C2 = sc, C3 = sc;
    if (todo == 2) {  // two donors: both are absorbed (or not) in slot order; the scan unrolled
        const Two r = two_donors((int)(N0 >> 16), (int)(N1 >> 16), own0, own1, (int)(N0 & NONE), (int)(N1 & NONE));
        float p = sp;
        uint32_t c = sc;
        if (r.a0) { p = __fadd_rn(p, P0); c += C0; }
        if (r.a1) { p = __fadd_rn(p, P1); c += C1; }
        return FrontNode{r.todo, p, c, r.w0, r.w1, own2, own3, r.a0 || r.a1};
    }
    if (todo > 2) { N2 = nc[own2]; P2 = pc[own2]; C2 = cc[own2]; }
    if (todo > 3) { N3 = nc[own3]; P3 = pc[own3]; C3 = cc[own3]; }
    int w0 = own0, w1 = own1, w2 = own2, w3 = own3;
    int q0 = 0, q1 = 1, q2 = 2, q3 = 3;
    bool worked = false;
    float padd = 0.f;
    uint32_t cadd = 0;
    int i = 0;
#pragma unroll
    for (int step = 0; step < 4; ++step) {  // each step moves i up or todo down: todo0 <= 4 steps
        if (i >= todo || i >= 4) break;
        const int q = sel4(i, q0, q1, q2, q3);
        const uint32_t dn = q == 0 ? N0 : (q == 1 ? N1 : (q == 2 ? N2 : N3));
        const float dp = q == 0 ? P0 : (q == 1 ? P1 : (q == 2 ? P2 : P3));
        const uint32_t dc = q == 0 ? C0 : (q == 1 ? C1 : (q == 2 ? C2 : C3));
        const int dnd = (int)(dn >> 16);
        if (dnd <= 1) {
            if (!worked) { padd = sp; cadd = sc; }
            worked = true;
            padd = __fadd_rn(padd, dp);
            cadd += dc;
            if (dnd == 0) {
                --todo;
                if (todo > i && todo < 4) {
                    set4(i, sel4(todo, own0, own1, own2, own3), w0, w1, w2, w3);
                    set4(i, todo, q0, q1, q2, q3);
                }
            } else {
                set4(i, (int)(dn & NONE), w0, w1, w2, w3);
                ++i;
            }
        } else {
            ++i;
        }
    }
    return FrontNode{todo, padd, cadd, w0, w1, w2, w3, worked};
}

// The pointers address the grid's own cells; idb is added to every cell id written (the
// grid's offset in a packed batch).
template <int MODE, int FR>
__device__ __forceinline__ void front_tile(const int32_t *__restrict__ rcv, const float *__restrict__ seed,
                                           Pub *cur_out, Pub *nxt_out, int4 *priv, uint32_t *counts, int *la, int *nla,
                                           int *lf, int *nlf, int *nonlocal, const Grid &g, int tx, int ty, int idb)
{
    using F = Front<FR>;
    constexpr int H = F::H, RW = F::RW, RH = F::RH, NR = F::NR, BS = F::BS, TW = F::TW, TH = F::TH;
    constexpr uint32_t NONE = 0xFFFFu;
    extern __shared__ __align__(16) unsigned char front_sm[];
    __shared__ int rowg[RH], colg[RW];  // global row / column of each region row / column, or -1
    float *pA = reinterpret_cast<float *>(front_sm), *pB = pA + NR;
    uint32_t *cA = reinterpret_cast<uint32_t *>(pB + NR), *cB = cA + NR;
    uint32_t *nA = cB + NR, *nB = nA + NR;  // ndnr << 16 | d0 (local id)
    uint16_t *s1 = reinterpret_cast<uint16_t *>(nB + NR), *s2 = s1 + NR, *s3 = s2 + NR;
    uint8_t *dir = reinterpret_cast<uint8_t *>(s3 + NR);
    const int c0 = tx * TW - H, r0 = ty * TH - H;  // region origin, before any wrap

    for (int k = threadIdx.x; k < RH + RW; k += BS) {
        if (k < RH) {
            int row = r0 + k;
            if (MODE == 2) {
                row %= g.ny;
                if (row < 0) row += g.ny;
            }
            rowg[k] = (row >= 0 && row < g.ny) ? row : -1;
        } else {
            int col = c0 + k - RH;
            if (MODE == 1) {
                col %= g.nx;
                if (col < 0) col += g.nx;
            }
            colg[k - RH] = (col >= 0 && col < g.nx) ? col : -1;
        }
    }
    __syncthreads();
    auto gid = [&](int lr, int lc) -> int {  // lr, lc within the region
        const int r = rowg[lr], c = colg[lc];
        return (r < 0 || c < 0) ? -1 : r * g.nx + c;
    };
    // a neighbour one step outside the region is never a receiver that matters;
    // -2 keeps it from matching any cell
    auto gidn = [&](int lr, int lc) -> int {
        return (lr < 0 || lr >= RH || lc < 0 || lc >= RW) ? -2 : gid(lr, lc);
    };

    // 1. each cell's receiver as a direction: 0-3 neighbour k, 4 itself, 5 other.
    //    A cell on the region's rim may see its receiver as "other"; it lies
    //    beyond every cell whose state the tile needs.
    bool bad = false;
    for (int x = threadIdx.x; x < NR; x += BS) {
        const int lr = x / RW, lc = x - lr * RW;
        const int t = gid(lr, lc);
        uint8_t d = 5;
        float p = 0.f;
        if (t >= 0) {
            const int rt = rcv[t];
            p = seed[t];
            const int row = rowg[lr], col = colg[lc], dt = rt - t;
            if (rt == t) d = 4;
            else if (row > 0 && row < g.ny - 1 && col > 0 && col < g.nx - 1)  // no wrap or edge next to it
                d = dt == -g.nx ? 0 : (dt == -1 ? 1 : (dt == 1 ? 2 : (dt == g.nx ? 3 : 5)));
            else if (rt == gidn(lr - 1, lc)) d = 0;
            else if (rt == gidn(lr, lc - 1)) d = 1;
            else if (rt == gidn(lr, lc + 1)) d = 2;
            else if (rt == gidn(lr + 1, lc)) d = 3;
            const bool own = lr >= H && lr < H + TH && lc >= H && lc < H + TW && r0 + lr < g.ny && c0 + lc < g.nx;
            if (own && d == 5) bad = true;
        }
        dir[x] = d;
        pA[x] = p;
    }
    if (bad) *nonlocal = 1;
    __syncthreads();

    // 2. initial records within 2^FR - 1 of the tile: the donors are the
    //    neighbours whose receiver is this cell, in ascending global index (wrap
    //    partners can come out of order)
    {
        constexpr int D = H - 1, W = TW + 2 * D, HH = TH + 2 * D;
        for (int u = threadIdx.x; u < W * HH; u += BS) {
            const int lr = u / W + (H - D), lc = u % W + (H - D);
            const int x = lr * RW + lc;
            const int row = rowg[lr], col = colg[lc];
            const bool cell = row >= 0 && col >= 0;
            // candidates in local order top, left, right, bottom: the ascending
            // global order unless a wrap sits next to the cell
            int l0 = NONE, l1 = NONE, l2 = NONE, l3 = NONE;
            if (cell) {
                if (dir[x - RW] == 3) l0 = x - RW;
                if (dir[x - 1] == 2) l1 = x - 1;
                if (dir[x + 1] == 1) l2 = x + 1;
                if (dir[x + RW] == 0) l3 = x + RW;
            }
            const int nd = (l0 != (int)NONE) + (l1 != (int)NONE) + (l2 != (int)NONE) + (l3 != (int)NONE);
            if (nd > 1 && ((MODE == 1 && (col == 0 || col == g.nx - 1)) || (MODE == 2 && (row == 0 || row == g.ny - 1)))) {
                auto key = [&](int l) { return l == (int)NONE ? 0x7FFFFFFF : gid(l / RW, l % RW); };
                int k0 = key(l0), k1 = key(l1), k2 = key(l2), k3 = key(l3);
                auto cs = [](int &ka, int &la_, int &kb, int &lb) {
                    if (ka > kb) {
                        int v = ka; ka = kb; kb = v;
                        v = la_; la_ = lb; lb = v;
                    }
                };
                cs(k0, l0, k1, l1); cs(k2, l2, k3, l3); cs(k0, l0, k2, l2); cs(k1, l1, k3, l3); cs(k1, l1, k2, l2);
            } else {
                // drop the gaps, keeping the order
                if (l0 == (int)NONE) { l0 = l1; l1 = l2; l2 = l3; l3 = NONE; }
                if (l0 == (int)NONE) { l0 = l1; l1 = l2; l2 = NONE; }
                if (l0 == (int)NONE) { l0 = l1; l1 = NONE; }
                if (l1 == (int)NONE) { l1 = l2; l2 = l3; l3 = NONE; }
                if (l1 == (int)NONE) { l1 = l2; l2 = NONE; }
                if (l2 == (int)NONE) { l2 = l3; l3 = NONE; }
            }
            nA[x] = ((uint32_t)nd << 16) | (uint32_t)l0;
            cA[x] = cell ? 1u : 0u;
            s1[x] = (uint16_t)l1;
            s2[x] = (uint16_t)l2;
            s3[x] = (uint16_t)l3;
        }
    }
    __syncthreads();

    // 3. rounds 0..FR-2 within 2^FR - 2^(r+1) of the tile
    float *pc = pA, *pn = pB;
    uint32_t *cc = cA, *cn = cB, *nc = nA, *nn = nB;
#pragma unroll
    for (int r = 0; r < FR - 1; ++r) {
        const int D = H - (2 << r), W = TW + 2 * D, HH = TH + 2 * D;
        for (int u = threadIdx.x; u < W * HH; u += BS) {
            const int x = (u / W + (H - D)) * RW + u % W + (H - D);
            const uint32_t snd = nc[x];
            const float sp = pc[x];
            const uint32_t sc = cc[x];
            if ((snd >> 16) == 0) {
                pn[x] = sp; cn[x] = sc; nn[x] = snd;
                continue;
            }
            const FrontNode o = front_round(pc, cc, nc, snd, sp, sc, (int)(snd & NONE), s1[x], s2[x], s3[x]);
            if (!o.worked) {
                pn[x] = sp; cn[x] = sc; nn[x] = snd;
            } else {
                pn[x] = o.p;
                cn[x] = o.c;
                nn[x] = ((uint32_t)o.todo << 16) | (uint32_t)(o.todo > 0 ? o.w0 : (int)(snd & NONE));
                if (o.todo > 1) {
                    s1[x] = (uint16_t)o.w1;
                    s2[x] = (uint16_t)o.w2;
                    s3[x] = (uint16_t)o.w3;
                }
            }
        }
        __syncthreads();
        float *tp = pc; pc = pn; pn = tp;
        uint32_t *tc = cc; cc = cn; cn = tc;
        uint32_t *tn = nc; nc = nn; nn = tn;
    }

    // 4. round FR-1 for the tile's cells, in registers, then the outputs
    auto l2g = [&](int l) -> int {
        if (l == (int)NONE) return -1;
        const int lr = l / RW;
        return gid(lr, l - lr * RW) + idb;
    };
#pragma unroll 1
    for (int k = 0; k < TW * TH / BS; ++k) {
        const int u = k * BS + threadIdx.x;
        const int ir = u / TW, ic = u - ir * TW;
        const int row = ty * TH + ir, col = tx * TW + ic;
        bool act = false, fin = false;
        int t = -1;
        if (row < g.ny && col < g.nx) {
            t = row * g.nx + col;
            const int x = (ir + H) * RW + ic + H;
            const uint32_t snd = nc[x];
            int nd = (int)(snd >> 16);
            float p = pc[x];
            uint32_t c = cc[x];
            int d0 = (int)(snd & NONE), d1 = s1[x], d2 = s2[x], d3 = s3[x];
            if (nd > 0) {
                const FrontNode o = front_round(pc, cc, nc, snd, p, c, d0, d1, d2, d3);
                if (o.worked) {
                    nd = o.todo;
                    p = o.p;
                    c = o.c;
                    if (nd > 0) d0 = o.w0;
                    d1 = o.w1; d2 = o.w2; d3 = o.w3;
                }
            }
            const Pub rec{nd, p, c, nd > 0 ? l2g(d0) : -1};
            cur_out[t] = rec;
            if (nd > 1) priv[t] = make_int4(l2g(d1), nd > 2 ? l2g(d2) : -1, nd > 3 ? l2g(d3) : -1, -1);
            if (nd > 0) {
                act = true;
            } else if (c == 1u) {  // a leaf: it never absorbed a donor
                nxt_out[t] = rec;
                if (counts) counts[t] = 1u;
            } else {
                fin = true;
            }
        }
        block_append2<BS>(act, fin, t + idb, la, nla, lf, nlf);
    }
}

template <int MODE, int FR>
__global__ void __launch_bounds__(Front<FR>::BS) k_acc_front(const int32_t *__restrict__ rcv,
                                                              const float *__restrict__ seed, Pub *cur_out,
                                                              Pub *nxt_out, int4 *priv, uint32_t *counts, int *la,
                                                              int *nla, int *lf, int *nlf, int *nonlocal, Grid g,
                                                              int ntx)
{
    front_tile<MODE, FR>(rcv, seed, cur_out, nxt_out, priv, counts, la, nla, lf, nlf, nonlocal, g, blockIdx.x % ntx,
                         blockIdx.x / ntx, 0);
}

// The front over a ragged batch: items[k] = the batch tile of work item k, whose front
// tile is k - (the first item of that batch tile).
constexpr int BATCH_FR = 3;
__global__ void __launch_bounds__(Front<BATCH_FR>::BS) k_batch_front(BatchAcc b, Pub *cur_out, Pub *nxt_out, int4 *priv,
                                                                     int *la, int *nla, int *lf, int *nlf, int *nonlocal)
{
    using F = Front<BATCH_FR>;
    const int n = b.small && *b.small ? 0 : b.limits[2];
    for (int k = blockIdx.x; k < n; k += gridDim.x) {
        const BatchTile T = b.by_offset[b.items[k]];
        const Grid g{T.nx, T.ny, T.mode, nullptr};
        const int ntx = (T.nx + F::TW - 1) / F::TW, e = k - T.item0, tx = e % ntx, ty = e / ntx;
        const int32_t *rcv = b.rcv + T.off;
        float *Q = b.Q + T.off;
        uint32_t *c = b.counts + T.off;
        const int idb = (int)T.off;
        if (T.mode == 0)
            front_tile<0, BATCH_FR>(rcv, Q, cur_out + T.off, nxt_out + T.off, priv + T.off, c, la, nla, lf, nlf, nonlocal, g,
                                    tx, ty, idb);
        else if (T.mode == 1)
            front_tile<1, BATCH_FR>(rcv, Q, cur_out + T.off, nxt_out + T.off, priv + T.off, c, la, nla, lf, nlf, nonlocal, g,
                                    tx, ty, idb);
        else
            front_tile<2, BATCH_FR>(rcv, Q, cur_out + T.off, nxt_out + T.off, priv + T.off, c, la, nla, lf, nlf, nonlocal, g,
                                    tx, ty, idb);
        __syncthreads();  // the shared buffers are reused by the next item
    }
}

template <int MODE, int FR>
static int l_acc_front(const int32_t *rcv, const float *seed, Pub *cur_out, Pub *nxt_out, int4 *priv,
                       uint32_t *counts, int *la, int *nla, int *lf, int *nlf, int *nonlocal, const Grid &g,
                       cudaStream_t st)
{
    using F = Front<FR>;
    static bool attr = false;
    if (!attr) {
        PFF_CUDA(cudaFuncSetAttribute(k_acc_front<MODE, FR>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)F::SMEM));
        attr = true;
    }
    const int ntx = div_up(g.nx, F::TW), nty = div_up(g.ny, F::TH);
    { k_acc_front<MODE, FR><<<ntx * nty, F::BS, F::SMEM, st>>>(rcv, seed, cur_out, nxt_out, priv, counts, la, nla, lf,
                                                              nlf, nonlocal, g, ntx); count_launch(); }
    return PFF_OK;
}

// Rounds taken by the tile front (0: off).  A tuning switch; both settings give
// identical results.
static int g_front_rounds = 3;

template <int FR>
static int front_dispatch(int mode, const int32_t *rcv, const float *seed, Pub *cur_out, Pub *nxt_out, int4 *priv,
                          uint32_t *counts, int *la, int *nla, int *lf, int *nlf, int *nonlocal, const Grid &g,
                          cudaStream_t st)
{
    switch (mode) {
    case 0: return l_acc_front<0, FR>(rcv, seed, cur_out, nxt_out, priv, counts, la, nla, lf, nlf, nonlocal, g, st);
    case 1: return l_acc_front<1, FR>(rcv, seed, cur_out, nxt_out, priv, counts, la, nla, lf, nlf, nonlocal, g, st);
    default: return l_acc_front<2, FR>(rcv, seed, cur_out, nxt_out, priv, counts, la, nla, lf, nlf, nonlocal, g, st);
    }
}

template <int MODE>
static void l_acc_gather(const int32_t *rcv, Pub *A, Pub *B, int4 *priv, const float *Q, uint32_t *counts, int *list,
                         int *nlist, int *nonlocal, int *overflow, const Grid &g, cudaStream_t st)
{
    dim3 gr(div_up(g.nx, 32), div_up(g.ny, 8));
    { k_acc_gather<MODE, 256><<<gr, 256, 0, st>>>(rcv, A, B, priv, Q, counts, list, nlist, nonlocal, overflow, g); count_launch(); }
}

// Blocks of the cooperative rounds over n nodes: one per 8192 up to one per SM.  More blocks
// make each barrier dearer than the shorter lists save: one per 2048 takes the whole call at
// 700 x 500 from 437 to 453 us, 48 tiles of 32 to 160 from 422 to 432.  Where no grid is given
// the scatter's passes over every node are in the same launch, and one per 2048 is the better:
// 155 against 205 us at 200 x 200, 229 against 246 at 700 x 500.
static int launch_rounds(AccRounds &a, int n, int per_block, cudaStream_t st)
{
    int dev = 0, nsm = 0;
    PFF_CUDA(cudaGetDevice(&dev));
    PFF_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    void *args[] = {&a};
    PFF_CUDA(cudaLaunchCooperativeKernel((void *)k_acc_rounds, std::max(1, std::min(nsm, div_up(n, per_block))), ACC_THREADS,
                                         args, 0, st));
    count_launch();
    return PFF_OK;
}

bool batch_front_takes(int nx, int ny, int mode) { return mode <= 2 && nx >= 3 && ny >= 3 && ceil_log2((long long)nx * ny) + 1 > BATCH_FR; }
int batch_front_items(int nx, int ny)
{
    return div_up(nx, Front<BATCH_FR>::TW) * div_up(ny, Front<BATCH_FR>::TH);
}

// Upstream sums of the batch tiles the front takes, in the reference's f32 order: the
// first rounds tile by tile in shared memory, the others over packed lists.
int launch_batch_accumulate(const BatchAcc &b, cudaStream_t st)
{
    int dev = 0, nsm = 0;
    PFF_CUDA(cudaGetDevice(&dev));
    PFF_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    using F = Front<BATCH_FR>;
    PFF_CUDA(cudaFuncSetAttribute(k_batch_front, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)F::SMEM));
    int *cnt = b.ctr, *nonlocal = b.ctr + 128, *bar = b.ctr + 136;
    constexpr int pa = BATCH_FR & 1;
    Pub *buf[2] = {(Pub *)b.bufA, (Pub *)b.bufB};
    { k_batch_front<<<2 * nsm, F::BS, F::SMEM, st>>>(b, buf[pa], buf[pa ^ 1], (int4 *)b.priv, b.la[pa], cnt + 2 * BATCH_FR,
                                                     b.lf[pa], cnt + 2 * BATCH_FR + 1, nonlocal); count_launch(); }
    AccRounds a{};
    a.rcv = b.rcv;
    a.buf[0] = buf[0]; a.buf[1] = buf[1];
    a.priv = (int4 *)b.priv;
    a.Q = b.Q; a.counts = b.counts;
    for (int k = 0; k < 2; ++k) { a.la[k] = b.la[k]; a.lf[k] = b.lf[k]; }
    a.cnt = cnt; a.nonlocal = nonlocal; a.overflow = nonlocal + 1;
    a.N = (int)b.total; a.first = BATCH_FR; a.bar = bar; a.wait = bar_wait(BAR_ROUNDS);
    a.tiles = b.by_offset; a.ntiles = b.ntiles; a.limits = b.limits; a.status = b.status;
    return launch_rounds(a, (int)b.total, 8192, st);
}

}  // namespace pff

using namespace pff;

extern "C" int pff_rcv2donor(const int32_t *rcv, int32_t *dnr, int32_t *ndnr, int N, void *stream)

{
    clear_error();
    if (N <= 0 || !rcv || !dnr || !ndnr || 4LL * N >= (1LL << 31)) {
        set_error("pff_rcv2donor: bad arguments");
        return PFF_ERR_ARG;
    }
    { k_rcv2donor_scatter<<<div_up(N, 256), 256, 0, S(stream)>>>(rcv, dnr, ndnr, N); count_launch(); }
    { k_sort_donors<<<div_up(N, 256), 256, 0, S(stream)>>>(dnr, ndnr, N); count_launch(); }
    return check_cuda("pff_rcv2donor");
}

extern "C" int pff_rake_compress_accum(int32_t *dnr, int32_t *ndnr, float *p, int32_t *src, int32_t *dnr_,
                                       int32_t *ndnr_, float *p_, int iteration, int N, void *stream)
{
    clear_error();
    if (N <= 0 || !dnr || !ndnr || !p || !src || !dnr_ || !ndnr_ || !p_) {
        set_error("pff_rake_compress_accum: bad arguments");
        return PFF_ERR_ARG;
    }
    { k_rake<false><<<div_up(N, 256), 256, 0, S(stream)>>>(dnr, ndnr, p, src, dnr_, ndnr_, p_, nullptr,
                                                        nullptr, iteration, N, nullptr); count_launch(); }
    return check_cuda("pff_rake_compress_accum");
}

extern "C" int pff_fuse(float *A, const int32_t *src, const float *B, int iteration, int N, void *stream)
{
    clear_error();
    if (N <= 0 || !A || !src || !B) {
        set_error("pff_fuse: bad arguments");
        return PFF_ERR_ARG;
    }
    { k_fuse<float><<<div_up(N, 256), 256, 0, S(stream)>>>(A, src, B, iteration, N); count_launch(); }
    return check_cuda("pff_fuse");
}

extern "C" int pff_accumulate_set_front(int rounds)
{
    clear_error();
    if (rounds < 0 || rounds > 3) {
        set_error("pff_accumulate_set_front: rounds must be 0 (off) to 3");
        return PFF_ERR_ARG;
    }
    g_front_rounds = rounds;
    return PFF_OK;
}

extern "C" size_t pff_accumulate_workspace_bytes(int N)
{
    const size_t n = (size_t)N;
    return Carver::round(16 * n) * 3 + Carver::round(4 * n) * 4 + Carver::round(64 * sizeof(int)) + 4096;
}

extern "C" int pff_accumulate(const int32_t *receivers, float *Q, uint32_t *counts, int N, void *workspace,
                              size_t workspace_bytes, void *stream)
{
    return pff_accumulate_grid(receivers, Q, counts, 0, 0, 0, nullptr, N, workspace, workspace_bytes, stream);
}

extern "C" int pff_accumulate_grid(const int32_t *receivers, float *Q, uint32_t *counts, int nx, int ny, int mode,
                                   const uint8_t *codes, int N, void *workspace, size_t workspace_bytes, void *stream)
{
    clear_error();
    if (nx > 0) {
        PFF_TRY(check_grid(nx, ny, mode, codes));
        if (nx * ny != N) {
            set_error("pff_accumulate_grid: N != nx*ny");
            return PFF_ERR_ARG;
        }
    }
    if (N <= 0 || !receivers || !Q || 4LL * N >= (1LL << 31)) {
        set_error("pff_accumulate: bad arguments");
        return PFF_ERR_ARG;
    }
    if (workspace_bytes < pff_accumulate_workspace_bytes(N) || !workspace) {
        set_error("pff_accumulate: workspace too small (%zu < %zu)", workspace_bytes,
                  pff_accumulate_workspace_bytes(N));
        return PFF_ERR_WORKSPACE;
    }
    cudaStream_t st = S(stream);
    Carver cv(workspace, workspace_bytes);
    Pub *A = cv.take<Pub>(N);
    Pub *B = cv.take<Pub>(N);
    int4 *priv = cv.take<int4>(N);
    int *lA0 = cv.take<int>(N), *lA1 = cv.take<int>(N), *lF0 = cv.take<int>(N), *lF1 = cv.take<int>(N);
    int *ctr = cv.take<int>(256);  // [2*r] active, [2*r+1] finished nodes of round r; flags and the barrier past 128
    const int logn = ceil_log2(N) + 1;  // flowfields.py:272
    const int FR = g_front_rounds;
    const bool front = nx > 0 && mode >= 0 && mode <= 2 && nx >= 3 && ny >= 3 && FR > 0 && logn > FR;
    PFF_CUDA(cudaMemsetAsync(ctr, 0, 256 * sizeof(int), st));
    int *nonlocal = ctr + 128, *overflow = ctr + 129, *bar = ctr + 136;
    Pub *bufs[2] = {A, B};
    int *la[2] = {lA0, lA1}, *lf[2] = {lF0, lF1};
    if (front) {
        Grid g{nx, ny, mode, codes};
        const int pa = FR & 1;
        int *na = ctr + 2 * FR;
        auto run = [&](auto fr) {
            return front_dispatch<decltype(fr)::value>(mode, receivers, Q, bufs[pa], bufs[pa ^ 1], priv, counts,
                                                       la[pa], na, lf[pa], na + 1, nonlocal, g, st);
        };
        PFF_TRY(FR == 1 ? run(std::integral_constant<int, 1>{})
                        : (FR == 2 ? run(std::integral_constant<int, 2>{}) : run(std::integral_constant<int, 3>{})));
    } else if (nx > 0) {
        Grid g{nx, ny, mode, codes};
        PFF_MODE_DISPATCH(mode, l_acc_gather, receivers, A, B, priv, Q, counts, lA0, ctr + 0, nonlocal, overflow, g,
                          st);
    } else if (N >= ACC_WIDE) {
        int dev = 0, nsm = 148;
        PFF_CUDA(cudaGetDevice(&dev));
        PFF_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
        { k_acc_init<<<8 * nsm, 256, 0, st>>>(A, B, priv, Q, counts, N); count_launch(); }
        { k_acc_scatter<<<8 * nsm, 256, 0, st>>>(receivers, A, priv, N, overflow); count_launch(); }
        { k_acc_list0<<<8 * nsm, 256, 0, st>>>(A, B, priv, lA0, ctr, N); count_launch(); }
    } else {
        PFF_CUDA(cudaMemsetAsync(nonlocal, 1, sizeof(int), st));
    }
    // the remaining rounds; receivers that are not D4 neighbours (or no grid given) start
    // again there by the scatter path
    int *host = nullptr, *dptr = nullptr;
    PFF_TRY(pinned_ints(&host, &dptr));
    host[0] = -1;
    AccRounds a{};
    a.rcv = receivers;
    a.buf[0] = A; a.buf[1] = B;
    a.priv = priv;
    a.Q = Q; a.counts = counts;
    for (int k = 0; k < 2; ++k) { a.la[k] = la[k]; a.lf[k] = lf[k]; }
    a.cnt = ctr; a.nonlocal = nonlocal; a.overflow = overflow;
    a.N = N; a.first = front ? FR : 0; a.logn = logn;
    if (!front && N >= ACC_WIDE) {
        int dev = 0, nsm = 148;
        PFF_CUDA(cudaGetDevice(&dev));
        PFF_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
        for (; a.first < ACC_WIDE_ROUNDS; ++a.first) {
            k_acc_round_wide<256><<<5 * nsm, 256, 0, st>>>(a, a.first);
            count_launch();
        }
    }
    a.bar = bar; a.wait = bar_wait(BAR_ROUNDS); a.over_out = dptr;
    PFF_TRY(launch_rounds(a, N, nx > 0 ? 8192 : 2048, st));
    PFF_CUDA(cudaStreamSynchronize(st));
    PFF_TRY(check_cuda("pff_accumulate"));
    const int over = *(volatile int *)host;
    if (over < 0) {
        set_error("pff_accumulate: the rounds did not end");
        return PFF_ERR_NOCONV;
    }
    if (over) {
        set_error("pff_accumulate: a node has more than 4 donors (possible only after jump rerouting); "
                  "the reference's donor slots overflow there and this case is not supported");
        return PFF_ERR_ARG;
    }
    return PFF_OK;
}
