// libpff core: error plumbing, argument checks, and the D4 receiver stencil.
#include <cstdarg>
#include <cstring>
#include <mutex>
#include "pff_internal.h"
#include "pff_div.cuh"

namespace pff {

static thread_local char g_err[512] = {0};
std::atomic<long long> g_launches{0};

void set_error(const char *fmt, ...)
{
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
}
void clear_error() { g_err[0] = 0; }

int check_cuda(const char *where)
{
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_error("%s: %s", where, cudaGetErrorString(e));
        return PFF_ERR_CUDA;
    }
    return PFF_OK;
}

int check_grid(int nx, int ny, int mode, const uint8_t *codes)
{
    if (nx < 2 || ny < 2) {
        set_error("grid must be at least 2x2 (got nx=%d, ny=%d)", nx, ny);
        return PFF_ERR_ARG;
    }
    if ((long long)nx * ny * 4LL >= (1LL << 31)) {
        set_error("grid too large for int32 donor indexing (nx*ny=%lld)", (long long)nx * ny);
        return PFF_ERR_ARG;
    }
    if (mode < 0 || mode > 3) {
        set_error("bound_mode must be 0..3 (got %d)", mode);
        return PFF_ERR_ARG;
    }
    if (mode == 3 && !codes) {
        set_error("custom bound_mode needs a device codes array");
        return PFF_ERR_ARG;
    }
    return PFF_OK;
}

// ---------------------------------------------------------------------------
// Receivers: pyfastflow/flow/receivers.py:31-58.
//
// Each warp walks a 32-column strip down RCV_ROWS rows: the cell's own row and
// the rows above and below stay in registers (one coalesced 128-byte load per
// row), left and right neighbours come from the adjacent lanes by shuffle (the
// two strip-edge lanes load one extra value).  Cells on the grid edge, and the
// custom mode, use the generic neighbour rules with direct loads.

// D4 receiver of cell i from its own and its neighbours' elevations.  A drop can
// only beat the best so far if it exceeds the best drop so far (division by
// dx > 0 is monotone), so the IEEE division -- the costly part -- runs only for
// improving candidates; the comparison is still between rounded quotients, as in
// the reference (strict '>', ties after rounding keep the earlier k).
__device__ __forceinline__ void rcv_pick(float zi, const float (&zn)[4], const int (&jn)[4], float dx, int &r,
                                         float &sr)
{
    float dbest = 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (jn[k] == -1) continue;
        const float d = __fsub_rn(zi, zn[k]);
        if (d > dbest) {
            const float tsr = __fdiv_rn(d, dx);
            if (tsr > sr) { sr = tsr; r = jn[k]; dbest = d; }
        }
    }
}

constexpr int RCV_ROWS = 32;
constexpr int RCV_AHEAD = 4;  // rows loaded per group (RCV_ROWS is a multiple)
constexpr int RCV4_ROWS = 8;   // rows per warp of the 4-column kernel
constexpr int RCV4_AHEAD = 2;  // rows loaded per group there (RCV4_ROWS is a multiple)

template <int MODE>
__global__ void __launch_bounds__(128) k_receivers(const float *__restrict__ z, int32_t *__restrict__ rcv,
                                                   float *__restrict__ grad, Grid g, float dx, int rows)
{
    const int lane = threadIdx.x & 31;
    const int warp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int nstrips = (g.nx + 31) >> 5;
    const int strip = warp % nstrips, band = warp / nstrips;
    const int col = (strip << 5) + lane;
    const int row0 = band * rows;
    if (row0 >= g.ny) return;
    const int row1 = min(row0 + rows, g.ny);
    const bool incol = col < g.nx;
    const int nx = g.nx;
    // register window: above, centre, below (column `col`); rows are loaded in groups
    // of RCV_AHEAD so that several loads per warp are in flight
    float za = 0.f, zc = 0.f;
    if (incol) {
        zc = __ldg(z + (size_t)row0 * nx + col);
        if (row0 > 0) za = __ldg(z + (size_t)(row0 - 1) * nx + col);
    }
    const bool hl = lane == 0 && col > 0 && incol;                                 // loads its left halo
    const bool hr = (lane == 31 || col == nx - 1) && col + 1 < nx && incol;        // loads its right halo
    for (int row = row0; row < row1; row += RCV_AHEAD) {
        float zq[RCV_AHEAD], ql[RCV_AHEAD], qr[RCV_AHEAD];
#pragma unroll
        for (int q = 0; q < RCV_AHEAD; ++q) {
            const int rb = row + 1 + q, rc = row + q;
            zq[q] = (incol && rb < g.ny && rb <= row1) ? __ldg(z + (size_t)rb * nx + col) : 0.f;
            ql[q] = (hl && rc < row1) ? __ldg(z + (size_t)rc * nx + col - 1) : 0.f;
            qr[q] = (hr && rc < row1) ? __ldg(z + (size_t)rc * nx + col + 1) : 0.f;
        }
#pragma unroll
        for (int q = 0; q < RCV_AHEAD; ++q) {
            const int rw = row + q;
            if (rw >= row1) break;
            const int i = rw * nx + col;
            const float zb = zq[q];
            // left/right from the neighbouring lanes; strip-edge lanes use their halo loads
            float zl = __shfl_up_sync(0xffffffffu, zc, 1);
            float zr = __shfl_down_sync(0xffffffffu, zc, 1);
            if (hl) zl = ql[q];
            if (hr) zr = qr[q];
            if (incol) {
                int r = i;
                float sr = 0.f;
                if (MODE != 3 && rw > 0 && rw < g.ny - 1 && col > 0 && col < nx - 1) {
                    const float zn[4] = {za, zl, zr, zb};
                    const int jn[4] = {i - nx, i - 1, i + 1, i + nx};
                    rcv_pick(zc, zn, jn, dx, r, sr);
                } else {
                    int jn[4];
                    float zn[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        jn[k] = neighbour<MODE>(g, i, rw, col, k);
                        zn[k] = jn[k] != -1 ? __ldg(z + jn[k]) : 0.f;
                    }
                    rcv_pick(zc, zn, jn, dx, r, sr);
                }
                rcv[i] = r;
                grad[i] = sr;
            }
            za = zc;
            zc = zb;
        }
    }
}

// The same choice with one division: the reference's sequential strict '>' keeps the
// first direction whose rounded quotient equals the largest rounded quotient, and
// by monotonicity that largest quotient is fl(dmax / dx).  Another direction can
// tie with it after rounding only if its drop lies within a few ulps of dmax, so
// only such near-ties pay a second division.
__device__ __forceinline__ void rcv_pick1(float zi, const float (&zn)[4], const int (&jn)[4], float dx, int &r,
                                          float &sr)
{
    float d[4], dmax = 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        d[k] = jn[k] != -1 ? __fsub_rn(zi, zn[k]) : 0.f;
        if (d[k] > dmax) dmax = d[k];
    }
    if (!(dmax > 0.f)) return;
    const float q = __fdiv_rn(dmax, dx);
    if (!(q > 0.f)) return;
    const unsigned qe = (__float_as_uint(q) >> 23) & 0xffu;
    if (qe == 0u || qe == 255u) {
        // subnormal or infinite quotients: drops far apart can round to the same
        // value, so take the reference's ordered scan with a strict '>' (:43-52)
        float best = 0.f;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (jn[k] == -1) continue;
            const float t = __fdiv_rn(d[k], dx);
            if (t > best) { best = t; r = jn[k]; sr = t; }
        }
        return;
    }
    const float near = __fmul_rn(dmax, 1.0f - 0x1p-21f);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (!(d[k] >= near)) continue;  // also skips invalid directions (d = 0 < near) and NaN
        if (d[k] == dmax || __fdiv_rn(d[k], dx) == q) {
            r = jn[k];
            sr = q;
            return;
        }
    }
}

// rcv_pick1 for an interior cell, whose four neighbours all exist: k = 0 top (-nx),
// 1 left (-1), 2 right (+1), 3 bottom (+nx).
__device__ __forceinline__ void rcv_pick_interior(float zi, float zt, float zl, float zr, float zb, int i, int nx,
                                                  float dx, int &r, float &sr)
{
    const float d0 = __fsub_rn(zi, zt), d1 = __fsub_rn(zi, zl), d2 = __fsub_rn(zi, zr), d3 = __fsub_rn(zi, zb);
    float dmax = 0.f;
    dmax = d0 > dmax ? d0 : dmax;
    dmax = d1 > dmax ? d1 : dmax;
    dmax = d2 > dmax ? d2 : dmax;
    dmax = d3 > dmax ? d3 : dmax;
    if (!(dmax > 0.f)) return;
    const float q = __fdiv_rn(dmax, dx);
    if (!(q > 0.f)) return;
    const unsigned qe = (__float_as_uint(q) >> 23) & 0xffu;
    if (qe == 0u || qe == 255u) {
        // subnormal or infinite quotients: drops far apart can round to the same
        // value, so take the reference's ordered scan with a strict '>' (:43-52)
        const float dk[4] = {d0, d1, d2, d3};
        const int off[4] = {-nx, -1, 1, nx};
        float best = 0.f;
        int kk = -1;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float t = __fdiv_rn(dk[k], dx);
            if (t > best) { best = t; kk = k; }
        }
        if (kk >= 0) { r = i + off[kk]; sr = best; }
        return;
    }
    // the first direction reaching q: an exact maximum, unless an earlier drop ties after
    // rounding (only possible within a few ulps of dmax: the rare slow path below)
    const float near = __fmul_rn(dmax, 1.0f - 0x1p-21f);
    const int first = d0 == dmax ? 0 : d1 == dmax ? 1 : d2 == dmax ? 2 : 3;
    int k = first;
    const bool n0 = d0 >= near && first > 0, n1 = d1 >= near && first > 1, n2 = d2 >= near && first > 2;
    if (n0 | n1 | n2) {
        if (n0 && __fdiv_rn(d0, dx) == q) k = 0;
        else if (n1 && __fdiv_rn(d1, dx) == q) k = 1;
        else if (n2 && __fdiv_rn(d2, dx) == q) k = 2;
    }
    r = i + (k == 0 ? -nx : k == 1 ? -1 : k == 2 ? 1 : nx);
    sr = q;
}

// A cell on the grid's edge (or any cell in custom mode): neighbours through the
// boundary rules.  Out of line, so that the interior path keeps its registers.
template <int MODE>
__device__ __noinline__ void rcv_boundary(const float *__restrict__ z, const Grid &g, int i, int row, int col, float dx,
                                          int *r, float *sr)
{
    int jn[4];
    float zn[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        jn[m] = neighbour<MODE>(g, i, row, col, m);
        zn[m] = jn[m] != -1 ? __ldg(z + jn[m]) : 0.f;
    }
    int rr = i;
    float s = 0.f;
    rcv_pick1(__ldg(z + i), zn, jn, dx, rr, s);
    *r = rr;
    *sr = s;
}

// Four columns per thread: a warp covers a 128-column strip, rows in groups of
// RCV_AHEAD; float4 loads and int4 / float4 stores; left and right neighbours from
// the adjacent lanes.  Needs nx % 4 == 0 (16-byte aligned rows).
template <int MODE>
__global__ void __launch_bounds__(128, 6) k_receivers4(const float *__restrict__ z, int32_t *__restrict__ rcv,
                                                    float *__restrict__ grad, Grid g, float dx)
{
    const int lane = threadIdx.x & 31;
    const int warp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int nx = g.nx, ny = g.ny;
    const int nstrips = (nx + 127) >> 7;
    const int strip = warp % nstrips, band = warp / nstrips;
    const int c0 = (strip << 7) + 4 * lane;  // first of this thread's 4 columns
    const int row0 = band * RCV4_ROWS;
    if (row0 >= ny) return;
    const int row1 = min(row0 + RCV4_ROWS, ny);
    const bool incol = c0 < nx;  // nx % 4 == 0: all 4 columns are in
    const float4 *z4 = reinterpret_cast<const float4 *>(z);
    const int nx4 = nx >> 2;
    const int q0 = c0 >> 2;
    float4 za = make_float4(0.f, 0.f, 0.f, 0.f), zc = za;
    if (incol) {
        zc = __ldg(z4 + (size_t)row0 * nx4 + q0);
        if (row0 > 0) za = __ldg(z4 + (size_t)(row0 - 1) * nx4 + q0);
    }
    const bool hl = lane == 0 && c0 > 0 && incol;                         // left halo from memory
    const bool hr = (lane == 31 || c0 + 4 >= nx) && c0 + 4 < nx && incol;  // right halo from memory
    for (int row = row0; row < row1; row += RCV4_AHEAD) {
        float4 zq[RCV4_AHEAD];
        float ql[RCV4_AHEAD], qr[RCV4_AHEAD];
#pragma unroll
        for (int q = 0; q < RCV4_AHEAD; ++q) {
            const int rb = row + 1 + q, rc = row + q;
            zq[q] = (incol && rb < ny && rb <= row1) ? __ldg(z4 + (size_t)rb * nx4 + q0) : make_float4(0.f, 0.f, 0.f, 0.f);
            ql[q] = (hl && rc < row1) ? __ldg(z + (size_t)rc * nx + c0 - 1) : 0.f;
            qr[q] = (hr && rc < row1) ? __ldg(z + (size_t)rc * nx + c0 + 4) : 0.f;
        }
#pragma unroll
        for (int q = 0; q < RCV4_AHEAD; ++q) {
            const int rw = row + q;
            if (rw >= row1) break;
            const float4 zb = zq[q];
            float zl = __shfl_up_sync(0xffffffffu, zc.w, 1);
            float zr = __shfl_down_sync(0xffffffffu, zc.x, 1);
            if (hl) zl = ql[q];
            if (hr) zr = qr[q];
            if (incol) {
                const float cz[4] = {zc.x, zc.y, zc.z, zc.w};
                const float az[4] = {za.x, za.y, za.z, za.w};
                const float bz[4] = {zb.x, zb.y, zb.z, zb.w};
                int rr[4];
                float ss[4];
                const bool rowin = MODE != 3 && rw > 0 && rw < ny - 1;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int col = c0 + k;
                    const int i = rw * nx + col;
                    int r = i;
                    float sr = 0.f;
                    if (rowin && col > 0 && col < nx - 1) {
                        rcv_pick_interior(cz[k], az[k], k > 0 ? cz[k - 1] : zl, k < 3 ? cz[k + 1] : zr, bz[k], i, nx,
                                          dx, r, sr);
                    } else {
                        rcv_boundary<MODE>(z, g, i, rw, col, dx, &r, &sr);
                    }
                    rr[k] = r;
                    ss[k] = sr;
                }
                const size_t o = (size_t)rw * nx4 + q0;
                reinterpret_cast<int4 *>(rcv)[o] = make_int4(rr[0], rr[1], rr[2], rr[3]);
                reinterpret_cast<float4 *>(grad)[o] = make_float4(ss[0], ss[1], ss[2], ss[3]);
            }
            za = zc;
            zc = zb;
        }
    }
}

// Lean receivers (modes 0-2, nx % 4 == 0): the instruction count per cell is what
// bounds this stencil, so the interior path is written for it.
//
//  * A warp walks a 128-column strip (4 columns per thread) down a band of rows with
//    RL_P rows of loads in flight per thread (a rolling register ring: the load of
//    row r + 1 + RL_P is issued as row r + 1 is consumed).
//  * Drops are shared between neighbours: the left drop of a cell is the negated
//    right drop of the cell before it, the top drop the negated bottom drop of the
//    row above (a - b == -(b - a) exactly in IEEE round-to-nearest).
//  * The choice needs one quotient, fl(dmax / dx) (division by dx > 0 is monotone,
//    so the largest rounded quotient is that of the largest drop).  The reference's
//    strict '>' keeps the first direction whose rounded quotient equals it; a
//    direction can round to it only with a drop within 2^-21 of dmax (relative),
//    so the first direction at or above that bound is the answer when its drop is
//    dmax itself, and anything else (a near tie, or a drop outside the range in
//    which the division below is exact) takes the reference's ordered scan.
//  * The quotient is RN(dmax / dx) by Markstein's correction with a precomputed
//    reciprocal (pff_div.cuh), exact in the range [mlo, mhi] of dmax.
//  * Cells on the grid's edge take the same path: a link that leaves the grid has
//    drop -inf, and the periodic modes' wrapped neighbours come from halo loads of
//    the opposite column (east-west) or row (north-south), with the receiver offset
//    of the wrapped link.  No warp takes a slower path for its edge cells.
constexpr int RL_ROWS = 32;  // rows per warp band, at most
// Band height: up to RL_ROWS rows, fewer on small grids, so that the grid holds
// enough warps to fill every SM (a warp's rows run one after another).
static int rl_rows(const Grid &g)
{
    static int sms = 0;
    if (!sms) {
        int dev = 0, v = 148;
        if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
        sms = v;
    }
    const long long strips = (g.nx + 127) / 128, want = 24LL * sms;  // 24 of the 28 resident warps per SM
    int rows = RL_ROWS;
    while (rows > 4 && strips * ((g.ny + rows - 1) / rows) < want) rows >>= 1;
    return rows;
}
static std::atomic<int> g_rcv_lean{1};  // pff_receivers_set_path

// The reference's ordered scan (receivers.py:43-52) on the four drops of one cell
// (top, left, right, bottom; an invalid link has drop -inf, whose quotient never
// passes '>'): strict '>' on IEEE quotients.  Returns {direction or -1, gradient bits}.
__device__ __noinline__ int2 rcv_scan_dir(float d0, float d1, float d2, float d3, float dx)
{
    const float d[4] = {d0, d1, d2, d3};
    float best = 0.f;
    int kk = -1;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float t = __fdiv_rn(d[k], dx);
        if (t > best) {
            best = t;
            kk = k;
        }
    }
    return make_int2(kk, __float_as_int(best));
}

// Fast choice from the four drops (-inf for an invalid link): the direction (-1: the
// cell is its own receiver) and the gradient; `ok` false when the ordered scan must
// decide instead.
__device__ __forceinline__ int rcv_off_fast(float d0, float d1, float d2, float d3, int ot, int ow, int oe, int ob,
                                            const DivC &c, float &s, bool &ok)
{
    const float m = fmaxf(fmaxf(d0, d1), fmaxf(d2, d3));  // NaN drops are ignored, as by '>'
    const float near = __fmul_rn(m, 1.0f - 0x1p-21f);
    const bool p0 = d0 >= near, p1 = d1 >= near, p2 = d2 >= near;
    const float dsel = p0 ? d0 : (p1 ? d1 : (p2 ? d2 : d3));
    const int off = p0 ? ot : (p1 ? ow : (p2 ? oe : ob));
    const float q = div_markstein(m, c);
    const bool pit = !(m > 0.f);  // pit or flat (or all drops NaN / invalid)
    ok = pit || (dsel == m && m >= c.mlo && m <= c.mhi);
    s = pit ? 0.f : q;
    return pit ? 0 : off;
}

template <int MODE, int RL_P, int MINB>
__global__ void __launch_bounds__(128, MINB) k_receivers_lean(const float *__restrict__ z, int32_t *__restrict__ rcv,
                                                              float *__restrict__ grad, Grid g, DivC c, int rows)
{
    static_assert(MODE >= 0 && MODE <= 2, "custom codes take the generic kernels");
    const int lane = threadIdx.x & 31;
    const int warp = blockIdx.x * 4 + (threadIdx.x >> 5);
    const int nx = g.nx, ny = g.ny, nx4 = nx >> 2;
    const int nstrips = (nx + 127) >> 7;
    const int strip = warp % nstrips, band = warp / nstrips;
    const int c0 = (strip << 7) + 4 * lane;
    const int r0 = band * rows;
    if (r0 >= ny) return;
    const int r1 = min(r0 + rows, ny);
    const bool incol = c0 < nx;
    const int q0 = c0 >> 2;
    const float4 *z4 = reinterpret_cast<const float4 *>(z);
    const float NEG = -__int_as_float(0x7f800000);  // -inf: an invalid link
    // Column neighbours of this thread's first and last cell.  Inside the strip they
    // come from the adjacent lanes; at a strip edge from a halo load; at the grid's
    // east / west edge from the wrapped column (periodic east-west) or nowhere.
    const bool lvalid = c0 > 0 || MODE == 1, rvalid = c0 + 4 < nx || MODE == 1;
    const bool lhalo = incol && lvalid && lane == 0;
    const bool rhalo = incol && rvalid && (lane == 31 || c0 + 4 == nx);
    const int lcol = c0 > 0 ? c0 - 1 : nx - 1, rcol = c0 + 4 < nx ? c0 + 4 : 0;
    // receiver offsets of the first / last cell's west / east links
    const int offl = c0 > 0 ? -1 : nx - 1, offr = c0 + 4 < nx ? 1 : 1 - nx;
    const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);

    float4 za = zero4, zc = zero4;
    float hl = 0.f, hr = 0.f;
    if (incol) {
        zc = __ldg(z4 + (size_t)r0 * nx4 + q0);
        const int ra = r0 > 0 ? r0 - 1 : (MODE == 2 ? ny - 1 : -1);  // the row above (wrapped north-south)
        if (ra >= 0) za = __ldg(z4 + (size_t)ra * nx4 + q0);
    }
    if (lhalo) hl = __ldg(z + (size_t)r0 * nx + lcol);
    if (rhalo) hr = __ldg(z + (size_t)r0 * nx + rcol);
    // rows r0 + 1 ... r0 + RL_P in a rolling ring (the row below each row of the band;
    // below the grid's last row: row 0 in periodic north-south, else nothing)
    float4 ring[RL_P];
    float lring[RL_P], rring[RL_P];
#pragma unroll
    for (int p = 0; p < RL_P; ++p) {
        const int rw = r0 + 1 + p;
        const int rl = rw < ny ? (rw <= r1 ? rw : -1) : (MODE == 2 && rw == ny ? 0 : -1);
        ring[p] = (incol && rl >= 0) ? __ldg(z4 + (size_t)rl * nx4 + q0) : zero4;
        lring[p] = (lhalo && rw < r1) ? __ldg(z + (size_t)rw * nx + lcol) : 0.f;
        rring[p] = (rhalo && rw < r1) ? __ldg(z + (size_t)rw * nx + rcol) : 0.f;
    }
    // bottom drops of the row above: the top drops of this row, negated
    float db0 = __fsub_rn(za.x, zc.x), db1 = __fsub_rn(za.y, zc.y), db2 = __fsub_rn(za.z, zc.z),
          db3 = __fsub_rn(za.w, zc.w);

    for (int rb = r0; rb < r1; rb += RL_P) {
#pragma unroll
        for (int p = 0; p < RL_P; ++p) {
            const int r = rb + p;
            if (r >= r1) break;
            const float4 zb = ring[p];
            const float hlb = lring[p], hrb = rring[p];
            {
                const int rw = r + 1 + RL_P;
                const int rl = rw < ny ? (rw <= r1 ? rw : -1) : (MODE == 2 && rw == ny ? 0 : -1);
                ring[p] = (incol && rl >= 0) ? __ldg(z4 + (size_t)rl * nx4 + q0) : zero4;
                lring[p] = (lhalo && rw < r1) ? __ldg(z + (size_t)rw * nx + lcol) : 0.f;
                rring[p] = (rhalo && rw < r1) ? __ldg(z + (size_t)rw * nx + rcol) : 0.f;
            }
            float zl = __shfl_up_sync(0xffffffffu, zc.w, 1);
            float zr = __shfl_down_sync(0xffffffffu, zc.x, 1);
            if (lhalo) zl = hl;
            if (rhalo) zr = hr;
            const float n0 = __fsub_rn(zc.x, zb.x), n1 = __fsub_rn(zc.y, zb.y), n2 = __fsub_rn(zc.z, zb.z),
                        n3 = __fsub_rn(zc.w, zb.w);  // bottom drops
            // the four cells of this row; tvalid / bvalid: the row has a north / south
            // neighbour row; offt / offb: the receiver offsets of those links
            auto cells = [&](bool tvalid, bool bvalid, int offt, int offb) {
                const float t0 = tvalid ? -db0 : NEG, t1 = tvalid ? -db1 : NEG, t2 = tvalid ? -db2 : NEG,
                            t3 = tvalid ? -db3 : NEG;
                const float b0 = bvalid ? n0 : NEG, b1 = bvalid ? n1 : NEG, b2 = bvalid ? n2 : NEG,
                            b3 = bvalid ? n3 : NEG;
                const float e0 = __fsub_rn(zc.x, zc.y), e1 = __fsub_rn(zc.y, zc.z), e2 = __fsub_rn(zc.z, zc.w);
                const float e3 = rvalid ? __fsub_rn(zc.w, zr) : NEG;  // east drop of the last cell
                const float l0 = lvalid ? __fsub_rn(zc.x, zl) : NEG;  // west drop of the first cell
                float s0, s1, s2, s3;
                bool ok0, ok1, ok2, ok3;
                int o0 = rcv_off_fast(t0, l0, e0, b0, offt, offl, 1, offb, c, s0, ok0);
                int o1 = rcv_off_fast(t1, -e0, e1, b1, offt, -1, 1, offb, c, s1, ok1);
                int o2 = rcv_off_fast(t2, -e1, e2, b2, offt, -1, 1, offb, c, s2, ok2);
                int o3 = rcv_off_fast(t3, -e2, e3, b3, offt, -1, offr, offb, c, s3, ok3);
                if (!(ok0 && ok1 && ok2 && ok3)) {  // rare: near ties or drops outside the exact-division range
                    auto off = [&](int k, int ow, int oe) {
                        return k < 0 ? 0 : (k == 0 ? offt : (k == 1 ? ow : (k == 2 ? oe : offb)));
                    };
                    int2 v;
                    if (!ok0) { v = rcv_scan_dir(t0, l0, e0, b0, c.dx); o0 = off(v.x, offl, 1); s0 = __int_as_float(v.y); }
                    if (!ok1) { v = rcv_scan_dir(t1, -e0, e1, b1, c.dx); o1 = off(v.x, -1, 1); s1 = __int_as_float(v.y); }
                    if (!ok2) { v = rcv_scan_dir(t2, -e1, e2, b2, c.dx); o2 = off(v.x, -1, 1); s2 = __int_as_float(v.y); }
                    if (!ok3) { v = rcv_scan_dir(t3, -e2, e3, b3, c.dx); o3 = off(v.x, -1, offr); s3 = __int_as_float(v.y); }
                }
                const int i0 = r * nx + c0;
                const size_t o = (size_t)r * nx4 + q0;
                reinterpret_cast<int4 *>(rcv)[o] = make_int4(i0 + o0, i0 + 1 + o1, i0 + 2 + o2, i0 + 3 + o3);
                reinterpret_cast<float4 *>(grad)[o] = make_float4(s0, s1, s2, s3);
            };
            if (incol) {
                if (r > 0 && r < ny - 1) cells(true, true, -nx, nx);  // an interior row
                else  // the first or last row (wrapped links in periodic north-south)
                    cells(r > 0 || MODE == 2, r < ny - 1 || MODE == 2, (MODE == 2 && r == 0) ? (ny - 1) * nx : -nx,
                          (MODE == 2 && r == ny - 1) ? -(ny - 1) * nx : nx);
            }
            db0 = n0;
            db1 = n1;
            db2 = n2;
            db3 = n3;
            zc = zb;
            hl = hlb;
            hr = hrb;
        }
    }
}

// Counts the floats m in [mlo, mhi] (every one, by bit pattern) for which the
// Markstein quotient differs from the IEEE division by dx.
__global__ void k_div_selfcheck(DivC c, unsigned lo, unsigned hi, unsigned long long *bad)
{
    unsigned long long nb = 0;
    for (unsigned long long u = lo + (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; u <= hi;
         u += (unsigned long long)gridDim.x * blockDim.x) {
        const float m = __uint_as_float((unsigned)u);
        nb += __float_as_uint(div_markstein(m, c)) != __float_as_uint(__fdiv_rn(m, c.dx));
    }
    if (nb) atomicAdd(bad, nb);
}

template <int MODE>
static void launch_receivers(const float *z, int32_t *rcv, float *grad, const Grid &g, float dx,
                             cudaStream_t st)
{
    const bool vec = g.nx % 4 == 0 && ((uintptr_t)z % 16) == 0 && ((uintptr_t)rcv % 16) == 0 &&
                     ((uintptr_t)grad % 16) == 0;
    if constexpr (MODE != 3) {
        const int lean = g_rcv_lean.load(std::memory_order_relaxed);
        if (vec && lean) {
            const int rows = rl_rows(g);
            const long long warps = (long long)((g.nx + 127) / 128) * ((g.ny + rows - 1) / rows);
            const unsigned nb = (unsigned)div_up(warps, 4);
            const DivC c = make_divc(dx);
            // 2 rows of loads in flight per thread; registers for 7 (path 1) or 8 CTAs per SM
            if (lean == 2)
                PFF_PROBED("k_receivers", st, k_receivers_lean<MODE, 2, 8><<<nb, 128, 0, st>>>(z, rcv, grad, g, c, rows));
            else
                PFF_PROBED("k_receivers", st, k_receivers_lean<MODE, 2, 7><<<nb, 128, 0, st>>>(z, rcv, grad, g, c, rows));
            count_launch();
            return;
        }
    }
    if (vec) {
        const long long warps = (long long)((g.nx + 127) / 128) * ((g.ny + RCV4_ROWS - 1) / RCV4_ROWS);
        PFF_PROBED("k_receivers", st, k_receivers4<MODE><<<div_up(warps, 4), 128, 0, st>>>(z, rcv, grad, g, dx));
        count_launch();
        return;
    }
    // bands of RCV_ROWS rows, shorter while they would leave the GPU with less than 32 warps
    // per SM (1001 x 777 has 800 bands of 32 rows, 30 us; of 4 rows it takes 10 us)
    int rows = RCV_ROWS;
    while (rows > RCV_AHEAD && (long long)((g.nx + 31) / 32) * ((g.ny + rows - 1) / rows) < 148 * 32) rows /= 2;
    const long long warps = (long long)((g.nx + 31) / 32) * ((g.ny + rows - 1) / rows);
    PFF_PROBED("k_receivers", st, k_receivers<MODE><<<div_up(warps, 4), 128, 0, st>>>(z, rcv, grad, g, dx, rows));
    count_launch();
}

// Stochastic receivers (receivers.py:46-47, RAND_RCV): each direction's slope is scaled
// by a uniform number in [0, 1) before the strict '>' selection.  The reference draws
// from Taichi's generator; here u(seed, i, k) is a counter-based draw: SplitMix64
// (Steele, Lea, Flood 2014) of seed and 4*i + k, top 24 bits / 2^24.
__host__ __device__ __forceinline__ unsigned long long splitmix64(unsigned long long x)
{
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}
__device__ __forceinline__ float uniform01(unsigned long long seed, long long i, int k)
{
    const unsigned long long h = splitmix64(seed ^ splitmix64((unsigned long long)(4 * i + k)));
    return (float)(h >> 40) * 0x1p-24f;
}

template <int MODE>
__global__ void __launch_bounds__(256) k_receivers_stochastic(const float *__restrict__ z, int32_t *__restrict__ rcv,
                                                              float *__restrict__ grad, Grid g, float dx,
                                                              unsigned long long seed)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.N()) return;
    const int row = i / g.nx, col = i - row * g.nx;
    const float zi = z[i];
    int r = i;
    float sr = 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int j = neighbour<MODE>(g, i, row, col, k);
        const bool valid = j != -1;
        float tsr = valid ? __fdiv_rn(__fsub_rn(zi, z[j]), dx) : -1.f;
        tsr = __fmul_rn(tsr, uniform01(seed, i, k));
        if (valid && tsr > sr) {
            sr = tsr;
            r = j;
        }
    }
    rcv[i] = r;
    grad[i] = sr;
}

}  // namespace pff

using namespace pff;

extern "C" int pff_compute_receivers_stochastic(const float *z, int32_t *receivers, float *gradient, int nx, int ny,
                                                float dx, int bound_mode, const uint8_t *codes,
                                                unsigned long long seed, void *stream)
{
    clear_error();
    PFF_TRY(check_grid(nx, ny, bound_mode, codes));
    if (!z || !receivers || !gradient) {
        set_error("pff_compute_receivers_stochastic: null pointer");
        return PFF_ERR_ARG;
    }
    Grid g{nx, ny, bound_mode, codes};
    const int N = nx * ny;
    cudaStream_t st = S(stream);
    switch (bound_mode) {
    case 0: { k_receivers_stochastic<0><<<div_up(N, 256), 256, 0, st>>>(z, receivers, gradient, g, dx, seed); count_launch(); } break;
    case 1: { k_receivers_stochastic<1><<<div_up(N, 256), 256, 0, st>>>(z, receivers, gradient, g, dx, seed); count_launch(); } break;
    case 2: { k_receivers_stochastic<2><<<div_up(N, 256), 256, 0, st>>>(z, receivers, gradient, g, dx, seed); count_launch(); } break;
    default: { k_receivers_stochastic<3><<<div_up(N, 256), 256, 0, st>>>(z, receivers, gradient, g, dx, seed); count_launch(); } break;
    }
    return check_cuda("pff_compute_receivers_stochastic");
}

extern "C" int pff_version(void) { return 100; }
extern "C" const char *pff_last_error_string(void) { return g_err; }
namespace pff {

__global__ void k_read_ints(IntReads r, volatile int *dst)
{
    int o = 0;
    for (int a = 0; a < r.k; ++a)
        for (int q = 0; q < r.n[a]; ++q) dst[o++] = r.src[a][q];
    __threadfence_system();
}

// One mapped pinned buffer per host thread and device (256 bytes each, kept
// until the process exits).
int pinned_ints(int **host, int **dptr)
{
    static thread_local int *host_buf[64] = {nullptr};
    static thread_local int *dev_buf[64] = {nullptr};
    int dev = 0;
    PFF_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) {
        set_error("pinned_ints: device %d out of range", dev);
        return PFF_ERR_ARG;
    }
    if (!host_buf[dev]) {
        void *p = nullptr, *d = nullptr;
        PFF_CUDA(cudaHostAlloc(&p, 64 * sizeof(int), cudaHostAllocMapped | cudaHostAllocPortable));
        PFF_CUDA(cudaHostGetDevicePointer(&d, p, 0));
        host_buf[dev] = (int *)p;
        dev_buf[dev] = (int *)d;
    }
    *host = host_buf[dev];
    *dptr = dev_buf[dev];
    return PFF_OK;
}

static thread_local int g_bar_kernels = 0;
static thread_local BarWait g_bar_wait = {0, 2000000};
BarWait bar_wait(int kernel) { return g_bar_kernels & kernel ? g_bar_wait : BarWait{0, 2000000}; }

int read_ints(const IntReads &r, int *out, cudaStream_t st)
{
    if (r.k > 8) {
        set_error("read_ints: %d reads out of range", r.k);
        return PFF_ERR_ARG;
    }
    int total = 0;
    for (int a = 0; a < r.k; ++a) total += r.n[a];
    if (total > 64) {
        set_error("read_ints: %d ints exceed 64", total);
        return PFF_ERR_ARG;
    }
    int *host = nullptr, *dptr = nullptr;
    PFF_TRY(pinned_ints(&host, &dptr));
    { k_read_ints<<<1, 1, 0, st>>>(r, dptr); count_launch(); }
    PFF_CUDA(cudaStreamSynchronize(st));
    PFF_TRY(check_cuda("read_ints"));
    const volatile int *h = host;
    for (int q = 0; q < total; ++q) out[q] = h[q];
    return PFF_OK;
}

// ---- kernel timing probes -------------------------------------------------------
// A probe brackets one kind of launch with two events on the launching stream.
// Armed only on request (benchmarks); launches inside a stream capture are not
// probed (an event recorded there would become a graph node).
namespace {
constexpr int PROBE_NAMES = 24, PROBE_EVENTS = 512;
struct Probe {
    const char *name = nullptr;
    cudaEvent_t a[PROBE_EVENTS], b[PROBE_EVENTS];
    int made = 0, used = 0;
};
std::mutex g_probe_mu;
std::atomic<bool> g_probe_on{false};
Probe g_probes[PROBE_NAMES];
}  // namespace

// A one-thread kernel that keeps the stream busy for about `ns` nanoseconds (bounded
// by the global timer).  Launched before a probed kernel's start event, it lets the
// host enqueue the event and the kernel while the GPU is still busy, so the event
// pair brackets the kernel alone and not a host launch gap.
__global__ void k_probe_pad(unsigned long long ns)
{
    unsigned long long t0;
    asm volatile("mov.u64 %0, %%globaltimer;\n" : "=l"(t0));
    for (int k = 0; k < 100000; ++k) {
        unsigned long long t;
        asm volatile("mov.u64 %0, %%globaltimer;\n" : "=l"(t));
        if (t - t0 >= ns) break;
        __nanosleep(1000);
    }
}

ProbeMark probe_begin(const char *name, cudaStream_t st)
{
    ProbeMark m{-1, -1};
    if (!g_probe_on.load(std::memory_order_relaxed)) return m;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) return m;
    std::lock_guard<std::mutex> lk(g_probe_mu);
    int k = 0;
    while (k < PROBE_NAMES && g_probes[k].name && strcmp(g_probes[k].name, name) != 0) ++k;
    if (k == PROBE_NAMES) return m;
    Probe &p = g_probes[k];
    p.name = name;
    if (p.used == PROBE_EVENTS) return m;
    if (p.used == p.made) {
        if (cudaEventCreate(&p.a[p.made]) != cudaSuccess) return m;
        if (cudaEventCreate(&p.b[p.made]) != cudaSuccess) {
            cudaEventDestroy(p.a[p.made]);
            return m;
        }
        ++p.made;
    }
    k_probe_pad<<<1, 1, 0, st>>>(30000ull);
    if (cudaEventRecord(p.a[p.used], st) != cudaSuccess) return m;
    m.slot = k;
    m.idx = p.used++;
    return m;
}

void probe_end(ProbeMark m, cudaStream_t st)
{
    if (m.slot < 0) return;
    std::lock_guard<std::mutex> lk(g_probe_mu);
    cudaEventRecord(g_probes[m.slot].b[m.idx], st);
}

}  // namespace pff

extern "C" int pff_barrier_test(int kernels, int absent, int limit_us)
{
    clear_error();
    if (kernels < 0 || kernels > 15 || absent < 0 || absent > 1 || (kernels && (limit_us < 1 || limit_us > 2000000))) {
        set_error("pff_barrier_test: bad arguments");
        return PFF_ERR_ARG;
    }
    g_bar_kernels = kernels;
    g_bar_wait = BarWait{absent, (unsigned)limit_us};
    return PFF_OK;
}

extern "C" long long pff_launch_count(void) { return g_launches.load(); }

extern "C" int pff_probe_enable(int on)
{
    clear_error();
    std::lock_guard<std::mutex> lk(g_probe_mu);
    for (auto &p : g_probes) {
        p.name = nullptr;
        p.used = 0;
    }
    g_probe_on.store(on != 0);
    return PFF_OK;
}

extern "C" int pff_probe_read(const char *name, double *total_ms, int *launches)
{
    clear_error();
    if (!name || !total_ms || !launches) {
        set_error("pff_probe_read: bad arguments");
        return PFF_ERR_ARG;
    }
    std::lock_guard<std::mutex> lk(g_probe_mu);
    *total_ms = 0.0;
    *launches = 0;
    for (auto &p : g_probes) {
        if (!p.name || strcmp(p.name, name) != 0) continue;
        for (int q = 0; q < p.used; ++q) {
            PFF_CUDA(cudaEventSynchronize(p.b[q]));
            float ms = 0.f;
            PFF_CUDA(cudaEventElapsedTime(&ms, p.a[q], p.b[q]));
            *total_ms += ms;
        }
        *launches = p.used;
    }
    return PFF_OK;
}

extern "C" int pff_set_device(int device)
{
    clear_error();
    PFF_CUDA(cudaSetDevice(device));
    return PFF_OK;
}

extern "C" int pff_receivers_set_path(int lean)
{
    clear_error();
    return g_rcv_lean.exchange(lean < 0 || lean > 2 ? 1 : lean);
}

extern "C" int pff_receivers_div_selfcheck(float dx, long long *mismatches, long long *checked)
{
    clear_error();
    if (!mismatches || !checked || !(dx > 0.f) || !(dx < 3.0e38f)) {
        set_error("pff_receivers_div_selfcheck: bad arguments");
        return PFF_ERR_ARG;
    }
    const DivC c = make_divc(dx);
    unsigned lo, hi;
    std::memcpy(&lo, &c.mlo, 4);
    std::memcpy(&hi, &c.mhi, 4);
    unsigned long long *d = nullptr;
    PFF_CUDA(cudaMalloc(&d, sizeof(unsigned long long)));
    cudaMemset(d, 0, sizeof(unsigned long long));
    k_div_selfcheck<<<148 * 16, 256>>>(c, lo, hi, d);
    unsigned long long bad = 0;
    cudaError_t e = cudaMemcpy(&bad, d, sizeof(bad), cudaMemcpyDeviceToHost);
    cudaFree(d);
    if (e != cudaSuccess) {
        set_error("pff_receivers_div_selfcheck: %s", cudaGetErrorString(e));
        return PFF_ERR_CUDA;
    }
    *mismatches = (long long)bad;
    *checked = (long long)hi - (long long)lo + 1;
    return PFF_OK;
}

extern "C" int pff_compute_receivers(const float *z, int32_t *receivers, float *gradient, int nx,
                                     int ny, float dx, int bound_mode, const uint8_t *codes,
                                     void *stream)
{
    clear_error();
    PFF_TRY(check_grid(nx, ny, bound_mode, codes));
    if (!z || !receivers || !gradient) {
        set_error("pff_compute_receivers: null pointer");
        return PFF_ERR_ARG;
    }
    Grid g{nx, ny, bound_mode, codes};
    PFF_MODE_DISPATCH(bound_mode, launch_receivers, z, receivers, gradient, g, dx, S(stream));
    return check_cuda("pff_compute_receivers");
}
