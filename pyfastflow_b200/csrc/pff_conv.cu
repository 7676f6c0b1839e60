// libpff convolutions for the GraphFlood warm-start network: BF16 3x3 convolution
// (stride 1, zero padding 1) as an implicit GEMM on the tensor cores with FP32
// accumulation -- forward, data gradient (the forward kernel on flipped,
// transposed weights) and weight gradient -- plus the small ops of a U-Net
// (2x2 average pooling, nearest 2x upsampling into a concatenation slice, ReLU
// backward, bias gradient, masked MSE loss, Adam).  No reference counterpart:
// the reference has no learned component.
//
// Activations are NHWC bf16 rows of `cs` channels; an operand may be a channel
// slice [off, off + C) of a wider row (the U-Net's concatenations), so every
// tensor argument is (pointer, row stride cs, channel offset off).  Weights are
// [Cout][9][Cin] bf16 (k = tap*Cin + ci, tap = kh*3 + kw).
//
// GEMM mapping (forward): M = pixels, N = Cout, K = 9*Cin.  A rows are gathered
// 16 bytes at a time straight from the activations with zero fill for the halo
// (cp.async, 3-stage pipeline), fragments come from XOR-swizzled shared memory
// through ldmatrix, products are mma.sync m16n8k16 bf16 -> f32.
#include <cuda_bf16.h>
#include "pff_internal.h"

namespace pff {

typedef uint16_t bf16_t;  // raw bf16 bits in the C ABI

__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void cp_async16(unsigned dst, const void *src, bool valid)
{
    const int n = valid ? 16 : 0;  // 0 source bytes: the 16 destination bytes are zero-filled
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(n));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

__device__ __forceinline__ void ldsm_x4(unsigned addr, unsigned &r0, unsigned &r1, unsigned &r2, unsigned &r3)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_t(unsigned addr, unsigned &r0, unsigned &r1, unsigned &r2, unsigned &r3)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(addr));
}
__device__ __forceinline__ void mma16816(float (&d)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0,
                                         unsigned b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                 "{%0,%1,%2,%3};\n"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ float bf2f(bf16_t v) { return __uint_as_float((unsigned)v << 16); }
__device__ __forceinline__ bf16_t f2bf(float f)
{
    __nv_bfloat16 b = __float2bfloat16_rn(f);
    return *reinterpret_cast<bf16_t *>(&b);
}

// ---- forward / data-gradient convolution ---------------------------------------------
constexpr int CV_BM = 128, CV_BK = 32, CV_ST = 3, CV_THREADS = 128;

struct ConvArgs {
    const bf16_t *x;
    int csx, offx;
    const bf16_t *w;  // [Cout][9*Cin]
    const float *bias;
    void *y;
    int csy, offy;
    int B, H, W, Cin, Cout;
    int relu, out_f32;
};

// 64-byte rows (4 chunks of 16 B), chunk c of row r stored at c ^ ((r >> 1) & 3)
__device__ __forceinline__ int sw64(int r, int c) { return r * 4 + (c ^ ((r >> 1) & 3)); }

// Rows of CH 16-byte chunks, chunk c of row r stored at c ^ (r & 7) within its group of 8, or at
// c ^ ((r >> 1) & 3) within 4 (CH = 4, 12): ldmatrix reads 8 rows of a chunk without conflicts.
template <int CH>
__device__ __forceinline__ int swr(int r, int c)
{
    return CH == 1 ? r : CH % 8 ? r * CH + (c ^ ((r >> 1) & 3)) : r * CH + (c ^ (r & 7));
}

// bias, ReLU and the store of channels co, co + 1 of pixel p (bf16 pairs, or f32)
__device__ __forceinline__ void conv_store(const ConvArgs &a, long long p, int co, float v0, float v1)
{
    const bool two = co + 1 < a.Cout;
    if (a.bias) {
        v0 += a.bias[co];
        if (two) v1 += a.bias[co + 1];
    }
    if (a.relu) {
        v0 = fmaxf(v0, 0.f);
        v1 = fmaxf(v1, 0.f);
    }
    if (a.out_f32) {
        float *yo = (float *)a.y + p * a.csy + a.offy + co;
        yo[0] = v0;
        if (two) yo[1] = v1;
    } else {
        bf16_t *yo = (bf16_t *)a.y + p * a.csy + a.offy + co;
        if (two)
            *reinterpret_cast<unsigned *>(yo) = (unsigned)f2bf(v0) | ((unsigned)f2bf(v1) << 16);
        else
            yo[0] = f2bf(v0);
    }
}

// BN output channels per CTA: 64 (2 x 2 warps of 64 x 32), or 32 and 16 (4 warps of
// 32 x BN) where Cout is that small.  The U-Net's full-resolution layers have 32 (and the
// head 8) output channels and only 9 to 27 K steps, so half to seven eighths of a 64-wide
// tile was padding, and the pixel decoding in 64-bit divisions cost more than the steps
// (635 us for the 11 such launches of a training step at 16 x 128 x 128; every sum keeps
// its order, so the results are the same).
template <int BN>
__global__ void __launch_bounds__(CV_THREADS) k_conv3x3(ConvArgs a)
{
    constexpr int WN = BN == 64 ? 2 : 1, MI = BN == 64 ? 4 : 2, NJ = BN / WN / 8;
    __shared__ __align__(128) uint4 sA[CV_ST][CV_BM * 4];
    __shared__ __align__(128) uint4 sB[CV_ST][BN * 4];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = warp / WN, wn = warp % WN;
    const long long P = (long long)a.B * a.H * a.W;
    const long long m0 = (long long)blockIdx.x * CV_BM;
    const int n0 = blockIdx.y * BN;
    const int K = 9 * a.Cin;
    const int nk = (K + CV_BK - 1) / CV_BK;

    // this thread's A rows (4) and chunk: rows tid/4 + 32j, chunk tid%4
    const int ac = tid & 3;
    int ay[4], ax[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const long long p = m0 + (tid >> 2) + 32 * j;
        if (P <= 0x7fffffffLL) {  // 32-bit divisions
            const unsigned q = p < P ? (unsigned)p : 0u, t = q / (unsigned)a.W;
            ax[j] = (int)(q - t * (unsigned)a.W);
            ay[j] = (int)(t % (unsigned)a.H);
        } else {
            const long long q = p < P ? p : 0, t = q / a.W;
            ax[j] = (int)(q - t * a.W);
            ay[j] = (int)(t % a.H);
        }
        if (p >= P) ay[j] = -4;  // no row of the image: every tap is padding
    }
    const bf16_t *xrow = a.x + (m0 + (tid >> 2)) * a.csx + a.offx;  // row j is 32 j pixels on
    // the chunk's K position at the next stage to load: k = tap * Cin + ci
    int ltap = ac * 8 / a.Cin, lci = ac * 8 - ltap * a.Cin;
    // B rows: n = tid/4 + 32j, chunk tid%4
    auto load_stage = [&](int st, int kt) {
        const int k = kt * CV_BK + ac * 8;
        const bool kval = k < K;
        const int dy = ltap / 3 - 1, dx = ltap % 3 - 1;
        const bf16_t *xs = xrow + (long long)(dy * a.W + dx) * a.csx + lci;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int r = (tid >> 2) + 32 * j;
            const int yy = ay[j] + dy, xx = ax[j] + dx;
            const bool v = kval && (unsigned)yy < (unsigned)a.H && (unsigned)xx < (unsigned)a.W;
            cp_async16(smem_u32(&sA[st][sw64(r, ac)]), v ? xs + (long long)(32 * j) * a.csx : a.x, v);
        }
#pragma unroll
        for (int j = 0; j < (BN + 31) / 32; ++j) {
            const int r = (tid >> 2) + 32 * j;
            if (BN % 32 && r >= BN) break;
            const int co = n0 + r;
            const bool v = kval && co < a.Cout;
            const bf16_t *src = v ? a.w + (long long)co * K + k : a.w;
            cp_async16(smem_u32(&sB[st][sw64(r, ac)]), src, v);
        }
        for (lci += CV_BK; lci >= a.Cin; lci -= a.Cin) ++ltap;
    };

    float acc[MI][NJ][4];
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[i][j][q] = 0.f;

#pragma unroll
    for (int s = 0; s < CV_ST - 1; ++s) {
        if (s < nk) load_stage(s, s);
        cp_commit();
    }
    for (int kt = 0; kt < nk; ++kt) {
        cp_wait<CV_ST - 2>();
        __syncthreads();
        {  // prefetch stage kt + ST - 1 (its buffer was consumed at iteration kt - 1)
            const int nt = kt + CV_ST - 1;
            if (nt < nk) load_stage(nt % CV_ST, nt);
            cp_commit();
        }
        const int st = kt % CV_ST;
#pragma unroll
        for (int kk = 0; kk < 2; ++kk) {  // two k16 steps per 32-wide stage
            unsigned af[MI][4], bfr[NJ][2];
#pragma unroll
            for (int i = 0; i < MI; ++i) {
                const int r = wm * (16 * MI) + i * 16 + (lane & 15);
                const int c = kk * 2 + (lane >> 4);
                ldsm_x4(smem_u32(&sA[st][sw64(r, c)]), af[i][0], af[i][1], af[i][2], af[i][3]);
            }
#pragma unroll
            for (int j = 0; j < NJ / 2; ++j) {
                const int r = wn * (8 * NJ) + j * 16 + (lane & 7) + ((lane >> 4) << 3);
                const int c = kk * 2 + ((lane >> 3) & 1);
                unsigned r0, r1, r2, r3;
                ldsm_x4(smem_u32(&sB[st][sw64(r, c)]), r0, r1, r2, r3);
                bfr[2 * j][0] = r0;
                bfr[2 * j][1] = r1;
                bfr[2 * j + 1][0] = r2;
                bfr[2 * j + 1][1] = r3;
            }
#pragma unroll
            for (int i = 0; i < MI; ++i)
#pragma unroll
                for (int j = 0; j < NJ; ++j)
                    mma16816(acc[i][j], af[i][0], af[i][1], af[i][2], af[i][3], bfr[j][0], bfr[j][1]);
        }
    }
    cp_wait<0>();

    // epilogue: bias, ReLU, store (bf16 pairs, or f32)
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            const long long p = m0 + wm * (16 * MI) + i * 16 + (lane >> 2) + hf * 8;
            if (p >= P) continue;
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
                const int co = n0 + wn * (8 * NJ) + j * 8 + 2 * (lane & 3);
                if (co >= a.Cout) continue;
                conv_store(a, p, co, acc[i][j][2 * hf], acc[i][j][2 * hf + 1]);
            }
        }
}

// The convolution with 8, 32, 64 or 96 input channels: the im2col form above fetches every
// pixel nine times from L2 and a thread's addresses cost more than its products.  Here a
// CTA keeps the weights of NB output channels in shared memory and walks over tiles of 16
// rows of 16 pixels, double-buffered with their halo; the taps read the tile shifted.  A
// warp takes MI rows of pixels; K steps go through taps and channels in the order of the
// form above, so every sum is the same.  Bound by
// fragment loads (6 per 16 products) and the tensor pipe; 16 x 128 x 128, before and now:
// 96 -> 32 channels 74 and 54 us, 32 -> 96 90 and 56, 32 -> 32 31 and 27, 32 -> 8 27 and 20,
// 8 -> 32 25 and 17 (two taps per K step); 64 -> 32 at 16 x 64 x 64 19 and 15.
constexpr int CT_TW = 16, CT_TH = 16, CT_HW = CT_TW + 2, CT_PITCH = 24;
// 16-byte chunks of a weight row: odd, so that 8 rows lie on 8 bank groups
__host__ __device__ constexpr int ct_wrow(int CC) { return CC == 1 ? 11 : 9 * CC + 1; }
__host__ __device__ constexpr int ct_smem(int CC, int NB) { return 16 * (NB * ct_wrow(CC) + 2 * CT_PITCH * (CT_TH + 2) * CC); }

template <int CC, int NB, int WARPS>
__global__ void __launch_bounds__(32 * WARPS) k_conv3x3_tile(ConvArgs a, int ntx, int nty, int ntiles)
{
    constexpr int MI = CT_TH / WARPS, NJ = NB / 8, THREADS = 32 * WARPS;
    constexpr int WR = ct_wrow(CC), WC = CC == 1 ? 10 : 9 * CC;  // 8 channels: a tenth tap of zeros
    constexpr int ST = CT_PITCH * (CT_TH + 2) * CC;
    extern __shared__ __align__(128) uint4 ct[];
    uint4 *sW = ct, *sX = ct + NB * WR;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n0 = blockIdx.y * NB;
    for (int e = tid; e < NB * WC; e += THREADS) {
        const int n = e / WC, q = e % WC;
        const bool v = n0 + n < a.Cout && q < 9 * CC;
        cp_async16(smem_u32(sW + n * WR + q), v ? a.w + ((long long)(n0 + n) * 9 * CC + q) * 8 : a.w, v);
    }
    auto load_tile = [&](int st, int t) {
        const int tx = t % ntx, u = t / ntx, ty = u % nty, b = u / nty;
        const int y0 = ty * CT_TH - 1, x0 = tx * CT_TW - 1;
        const bf16_t *xb = a.x + (((long long)b * a.H + y0) * a.W + x0) * a.csx + a.offx;
        uint4 *X = sX + st * ST;
        for (int e = tid; e < CT_HW * (CT_TH + 2) * CC; e += THREADS) {
            const int r = e / CC, c = e % CC, y = r / CT_HW, x = r % CT_HW;
            const bool v = (unsigned)(y0 + y) < (unsigned)a.H && (unsigned)(x0 + x) < (unsigned)a.W;
            cp_async16(smem_u32(X + swr<CC>(y * CT_PITCH + x, c)), v ? xb + ((y * a.W + x) * a.csx + c * 8) : a.x, v);
        }
        cp_commit();
    };
    const unsigned wb = smem_u32(sW) + 16 * (((lane & 7) + ((lane >> 4) << 3)) * WR + ((lane >> 3) & 1));
    const unsigned xs = smem_u32(sX);
    int t = blockIdx.x;
    load_tile(0, t);  // the weights' copies are in the same group
    for (int k = 0; t < ntiles; ++k, t += gridDim.x) {
        if (t + (int)gridDim.x < ntiles)
            load_tile((k + 1) & 1, t + gridDim.x);
        else
            cp_commit();
        cp_wait<1>();
        __syncthreads();
        float acc[MI][NJ][4];
#pragma unroll
        for (int i = 0; i < MI; ++i)
#pragma unroll
            for (int j = 0; j < NJ; ++j)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[i][j][q] = 0.f;
        const unsigned xb = xs + 16 * ((k & 1) * ST + warp * MI * CT_PITCH * CC);
        // one K step of 16: A rows at xa, weight chunks from q
        auto step = [&](unsigned xa, int q, bool last) {
            unsigned af[MI][4], bf[NJ][2];
#pragma unroll
            for (int i = 0; i < MI; ++i) {
                ldsm_x4(xa + i * (16 * CT_PITCH * CC), af[i][0], af[i][1], af[i][2], af[i][3]);
                if (last) af[i][2] = af[i][3] = 0;  // past the last tap: 0 times an infinity is no 0
            }
#pragma unroll
            for (int j = 0; j < NJ / 2; ++j)
                ldsm_x4(wb + 16 * (j * 16 * WR + q), bf[2 * j][0], bf[2 * j][1], bf[2 * j + 1][0], bf[2 * j + 1][1]);
#pragma unroll
            for (int i = 0; i < MI; ++i)
#pragma unroll
                for (int j = 0; j < NJ; ++j)
                    mma16816(acc[i][j], af[i][0], af[i][1], af[i][2], af[i][3], bf[j][0], bf[j][1]);
        };
        if constexpr (CC == 1) {  // two taps per step
#pragma unroll
            for (int q = 0; q < 10; q += 2) {
                const int tap = min(q + (lane >> 4), 8);
                step(xb + 16 * (tap / 3 * CT_PITCH + tap % 3 + (lane & 15)), q, q == 8);
            }
        } else {
#pragma unroll 1
            for (int kh = 0; kh < 3; ++kh)
#pragma unroll
                for (int kw = 0; kw < 3; ++kw)
#pragma unroll
                    for (int s = 0; s < CC / 2; ++s)
                        step(xb + 16 * (kh * CT_PITCH * CC + swr<CC>(kw + (lane & 15), 2 * s + (lane >> 4))),
                             (3 * kh + kw) * CC + 2 * s, false);
        }
        __syncthreads();  // the tile's buffer is free for the load after next
        const int tx = t % ntx, u = t / ntx, ty = u % nty, b = u / nty;
#pragma unroll
        for (int i = 0; i < MI; ++i) {
            const int y = ty * CT_TH + warp * MI + i;
            if (y >= a.H) break;
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                const int x = tx * CT_TW + (lane >> 2) + hf * 8;
                if (x >= a.W) continue;
#pragma unroll
                for (int j = 0; j < NJ; ++j) {
                    const int co = n0 + j * 8 + 2 * (lane & 3);
                    if (co < a.Cout)
                        conv_store(a, ((long long)b * a.H + y) * a.W + x, co, acc[i][j][2 * hf], acc[i][j][2 * hf + 1]);
                }
            }
        }
    }
    cp_wait<0>();
}

template <int CC, int NB, int WARPS>
static int launch_conv_tile(const ConvArgs &a, cudaStream_t st)
{
    auto kern = k_conv3x3_tile<CC, NB, WARPS>;
    constexpr int smem = ct_smem(CC, NB), per = 227 * 1024 / (smem + 1024);
    static_assert(per >= 1, "shared memory of an SM");
    PFF_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    const int ntx = (a.W + CT_TW - 1) / CT_TW, nty = (a.H + CT_TH - 1) / CT_TH, nt = a.B * ntx * nty;
    const int ny = (a.Cout + NB - 1) / NB;
    // resident CTAs, each with the same number of tiles but for one
    const int most = std::max(1, 148 * std::min(per, 4) / ny), each = (nt + most - 1) / most;
    kern<<<dim3((nt + each - 1) / each, ny), 32 * WARPS, smem, st>>>(a, ntx, nty, nt);
    count_launch();
    return PFF_OK;
}

template <int CC, int WARPS>
static int launch_conv_tile(const ConvArgs &a, cudaStream_t st)
{
    return a.Cout > 16 ? launch_conv_tile<CC, 32, WARPS>(a, st) : launch_conv_tile<CC, 16, WARPS>(a, st);
}

// wt[ci][tap'][co] = w[co][8 - tap'][ci]: the data gradient of a 3x3 convolution is
// the forward convolution of dy with these weights.
__global__ void k_wflip(const bf16_t *__restrict__ w, bf16_t *wt, int Cin, int Cout)
{
    const long long n = 9LL * Cin * Cout;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        const int co = (int)(e % Cout);
        const long long t = e / Cout;
        const int tp = (int)(t % 9);
        const int ci = (int)(t / 9);
        wt[e] = w[((long long)co * 9 + (8 - tp)) * Cin + ci];
    }
}

// ---- weight gradient --------------------------------------------------------------------
// dw[co][k] += sum_p dy[p][co] * x~[p][k],  x~[p][k] = x[shift(p, tap(k))][ci(k)] (0 outside).
// GEMM M = Cout, N = 9*Cin, reduced over pixels; each CTA reduces one pixel range
// and adds its BM x BN tile into dw with f32 atomics.
constexpr int WG_BK = 32, WG_ST = 3, WG_THREADS = 128;

struct WgradArgs {
    const bf16_t *x;
    int csx, offx;
    const bf16_t *dy;
    int csd, offd;
    float *dw;
    int B, H, W, Cin, Cout;
    long long pchunk;  // pixels per CTA (multiple of WG_BK)
};

// The form for rows whose tiles k_conv3x3_wgrad9 cannot address in 32 bits.  A thread's
// pixels advance by WG_BK per stage: their positions are kept, not divided out.
template <int BM, int BN>
__global__ void __launch_bounds__(WG_THREADS) k_conv3x3_wgrad(WgradArgs a)
{
    constexpr int CA = BM / 8, CB = BN / 8;        // chunks per row
    constexpr int MI = BM / 32, NJ = BN / 16;      // 2 x 2 warps of 16 MI x 8 NJ
    constexpr int NA = WG_BK * CA / WG_THREADS, NB = WG_BK * CB / WG_THREADS;
    static_assert(WG_BK * CA % WG_THREADS == 0 && WG_BK * CB % WG_THREADS == 0, "uniform loads");
    __shared__ __align__(128) uint4 sA[WG_ST][WG_BK * CA];  // [pixel][co]
    __shared__ __align__(128) uint4 sB[WG_ST][WG_BK * CB];  // [pixel][k]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = warp >> 1, wn = warp & 1;
    const long long P = (long long)a.B * a.H * a.W;
    const int K = 9 * a.Cin;
    const int n0 = blockIdx.x * BN, m0 = blockIdx.y * BM;
    const long long pb = (long long)blockIdx.z * a.pchunk;
    const long long pe = min(P, pb + a.pchunk);
    if (pb >= pe) return;
    const int nk = (int)((pe - pb + WG_BK - 1) / WG_BK);
    const int np = (int)(pe - pb);
    // loads: element e = tid + 128 j of the stage, row e / chunks, chunk e % chunks
    int by[NB], bx[NB];           // B elements: image row and column of the next stage's pixel
    int bshift[NB], bcol[NB];     // pixel shift of the tap (dy * 4 + dx + 5), channel or -1
    {
        const unsigned W = (unsigned)a.W, H = (unsigned)a.H;
#pragma unroll
        for (int j = 0; j < NB; ++j) {
            const int e = tid + WG_THREADS * j, r = e / CB, kb = n0 + (e % CB) * 8;
            const int tap = kb < K ? kb / a.Cin : 0;
            bcol[j] = kb < K ? kb - tap * a.Cin : -1;
            bshift[j] = tap;
            const long long p = pb + r, t = p / W;
            bx[j] = (int)(p - t * W);
            by[j] = (int)(t % H);
        }
    }
    auto load_stage = [&](int st, int kt) {
#pragma unroll
        for (int j = 0; j < NA; ++j) {
            const int e = tid + WG_THREADS * j, r = e / CA, c = e % CA, q = kt * WG_BK + r;
            const bool v = q < np && m0 + c * 8 < a.Cout;
            cp_async16(smem_u32(&sA[st][swr<CA>(r, c)]), v ? a.dy + (pb + q) * a.csd + a.offd + m0 + c * 8 : a.dy, v);
        }
#pragma unroll
        for (int j = 0; j < NB; ++j) {
            const int e = tid + WG_THREADS * j, r = e / CB, c = e % CB, q = kt * WG_BK + r;
            const int dy = bshift[j] / 3 - 1, dx = bshift[j] % 3 - 1;
            const bool v = q < np && bcol[j] >= 0 && (unsigned)(by[j] + dy) < (unsigned)a.H &&
                           (unsigned)(bx[j] + dx) < (unsigned)a.W;
            cp_async16(smem_u32(&sB[st][swr<CB>(r, c)]),
                       v ? a.x + (pb + q + dy * a.W + dx) * a.csx + a.offx + bcol[j] : a.x, v);
            for (bx[j] += WG_BK; bx[j] >= a.W; bx[j] -= a.W)
                if (++by[j] == a.H) by[j] = 0;
        }
    };
    float acc[MI][NJ][4];
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[i][j][q] = 0.f;
#pragma unroll
    for (int s = 0; s < WG_ST - 1; ++s) {
        if (s < nk) load_stage(s, s);
        cp_commit();
    }
    for (int kt = 0; kt < nk; ++kt) {
        cp_wait<WG_ST - 2>();
        __syncthreads();
        {
            const int nt = kt + WG_ST - 1;
            if (nt < nk) load_stage(nt % WG_ST, nt);
            cp_commit();
        }
        const int st = kt % WG_ST;
#pragma unroll
        for (int kk = 0; kk < 2; ++kk) {
            unsigned af[MI][4], bfr[NJ][2];
#pragma unroll
            for (int i = 0; i < MI; ++i) {  // A^T from [pixel][co]: trans loads
                const int r = kk * 16 + (lane & 7) + ((lane >> 4) << 3);
                const int c = (wm * 16 * MI + i * 16) / 8 + ((lane >> 3) & 1);
                ldsm_x4_t(smem_u32(&sA[st][swr<CA>(r, c)]), af[i][0], af[i][1], af[i][2], af[i][3]);
            }
#pragma unroll
            for (int j = 0; j < NJ / 2; ++j) {  // B from [pixel][k]: trans loads
                const int r = kk * 16 + (lane & 7) + (((lane >> 3) & 1) << 3);
                const int c = (wn * 8 * NJ + j * 16) / 8 + (lane >> 4);
                unsigned r0, r1, r2, r3;
                ldsm_x4_t(smem_u32(&sB[st][swr<CB>(r, c)]), r0, r1, r2, r3);
                bfr[2 * j][0] = r0;
                bfr[2 * j][1] = r1;
                bfr[2 * j + 1][0] = r2;
                bfr[2 * j + 1][1] = r3;
            }
#pragma unroll
            for (int i = 0; i < MI; ++i)
#pragma unroll
                for (int j = 0; j < NJ; ++j)
                    mma16816(acc[i][j], af[i][0], af[i][1], af[i][2], af[i][3], bfr[j][0], bfr[j][1]);
        }
    }
    cp_wait<0>();
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            const int co = m0 + wm * 16 * MI + i * 16 + (lane >> 2) + hf * 8;
            if (co >= a.Cout) continue;
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
                const int k = n0 + wn * 8 * NJ + j * 8 + 2 * (lane & 3);
                if (k < K) atomicAdd(a.dw + (long long)co * K + k, acc[i][j][2 * hf]);
                if (k + 1 < K) atomicAdd(a.dw + (long long)co * K + k + 1, acc[i][j][2 * hf + 1]);
            }
        }
}

// The weight gradient: all nine taps of a CO x CI
// channel block in one CTA.  With one tile of the GEMM per CTA every pixel's activations
// crossed from L2 once per tap and column tile (24 to 32 products per byte); here a stage
// is a tile of 8 rows of 16 pixels and its halo, which the taps read shifted, at 144
// products per byte (32 x 32) or 230 (64 x 64).  12 warps = 3 tap rows x 4: quadrants of
// 32 x 32 channels, or where the block has fewer, groups that take every 2nd or 4th row
// and meet in shared memory at the end.  A warp keeps three taps' 32 x 32 sums (96
// registers) and loads dy's fragments once for the three.  Bound by the
// mma.sync pipe (active 57 to 65 % of the kernel; L2 11 %); the rest are the first loads, the
// few passes per CTA (4 to 20) and the adds into dw.  At 16 x 128 x 128 (full resolution), old and new: 96 -> 32 channels 117 and
// 50 us, 32 -> 32 39 and 23; at 16 x 32 x 32, 384 -> 128 channels 83 and 45 us.
// Halo rows are 24 pixels apart in shared memory, a multiple of the swizzle's period, so
// that a fragment's address moves by a constant from row to row.
constexpr int W9_TW = 16, W9_HW = W9_TW + 2, W9_PITCH = 24, W9_ST = 3, W9_THREADS = 384;
__host__ __device__ constexpr int w9_rows(int CO, int CI) { return CO * CI == 4096 ? 8 : 16; }
__host__ __device__ constexpr int w9_smem(int CO, int CI)
{
    return W9_ST * 2 * (W9_TW * w9_rows(CO, CI) * CO + W9_PITCH * (w9_rows(CO, CI) + 2) * CI);
}

struct Wgrad9Args {
    const bf16_t *x;
    int csx, offx;
    const bf16_t *dy;
    int csd, offd;
    float *dw;
    int B, H, W, Cin, Cout;
    int ntx, nty, ntiles;  // pixel tiles across, down, in all
    int pair;              // dw takes 8-byte adds
};

template <int CO, int CI>
__global__ void __launch_bounds__(W9_THREADS, 1) k_conv3x3_wgrad9(Wgrad9Args a)
{
    constexpr int CA = CO / 8, CB = CI / 8, QM = CO / 32, Q = QM * (CI / 32), KG = 4 / Q;
    constexpr int TH = w9_rows(CO, CI);
    constexpr int SA = W9_TW * TH * CA, SB = W9_PITCH * (TH + 2) * CB;  // 16-byte chunks of a stage
    extern __shared__ __align__(128) uint4 w9[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int trow = warp % 3, grp = warp / 3, quad = grp % Q, kg = grp / Q;
    const int qm = quad % QM * 32, qn = quad / QM * 32;
    const int m0 = blockIdx.y * CO, n0 = blockIdx.x * CI;
    const int t0 = (int)((long long)a.ntiles * blockIdx.z / gridDim.z);
    const int nt = (int)((long long)a.ntiles * (blockIdx.z + 1) / gridDim.z) - t0;

    // the next tile to load and the next to multiply
    int lx = t0 % a.ntx, ly = t0 / a.ntx % a.nty, lb = t0 / a.ntx / a.nty, cx = lx, cy = ly;
    auto load_stage = [&](int st) {
        const int y0 = ly * TH, x0 = lx * W9_TW;
        const long long at = ((long long)lb * a.H + y0) * a.W + x0;  // the tile's first pixel
        const bf16_t *da = a.dy + at * a.csd + a.offd + m0, *xb = a.x + (at - a.W - 1) * a.csx + a.offx + n0;
        uint4 *A = w9 + st * (SA + SB), *B = A + SA;
#pragma unroll
        for (int j = 0; j < (SA + W9_THREADS - 1) / W9_THREADS; ++j) {
            const int e = tid + W9_THREADS * j, r = e / CA, c = e % CA, y = r / W9_TW, x = r % W9_TW;
            if (SA % W9_THREADS && e >= SA) break;
            const bool v = y0 + y < a.H && x0 + x < a.W && m0 + c * 8 < a.Cout;
            cp_async16(smem_u32(A + swr<CA>(r, c)), v ? da + ((y * a.W + x) * a.csd + c * 8) : a.dy, v);
        }
#pragma unroll
        for (int j = 0; j < (W9_HW * (TH + 2) * CB + W9_THREADS - 1) / W9_THREADS; ++j) {
            const int e = tid + W9_THREADS * j, r = e / CB, c = e % CB, y = r / W9_HW, x = r % W9_HW;
            if (e >= W9_HW * (TH + 2) * CB) break;
            const bool v = (unsigned)(y0 + y - 1) < (unsigned)a.H && (unsigned)(x0 + x - 1) < (unsigned)a.W &&
                           n0 + c * 8 < a.Cin;
            cp_async16(smem_u32(B + swr<CB>(y * W9_PITCH + x, c)), v ? xb + ((y * a.W + x) * a.csx + c * 8) : a.x, v);
        }
        if (++lx == a.ntx) {
            lx = 0;
            if (++ly == a.nty) ly = 0, ++lb;
        }
    };
    float acc[3][2][4][4];
#pragma unroll
    for (int d = 0; d < 3; ++d)
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[d][i][j][q] = 0.f;
#pragma unroll
    for (int s = 0; s < W9_ST - 1; ++s) {
        if (s < nt) load_stage(s);
        cp_commit();
    }
    // fragment addresses in the first stage, at the group's first row
    const int ar = kg * W9_TW + (lane & 7) + ((lane >> 4) << 3), ac = qm / 8 + ((lane >> 3) & 1);
    const int br = (kg + trow) * W9_PITCH + (lane & 7) + (((lane >> 3) & 1) << 3), bc = qn / 8 + (lane >> 4);
    const unsigned s0 = smem_u32(w9);
    unsigned fa[2], fb[3][2];
#pragma unroll
    for (int i = 0; i < 2; ++i) fa[i] = 16 * swr<CA>(ar, ac + 2 * i);
#pragma unroll
    for (int d = 0; d < 3; ++d)
#pragma unroll
        for (int j = 0; j < 2; ++j) fb[d][j] = 16 * (SA + swr<CB>(br + d, bc + 2 * j));
    for (int k = 0; k < nt; ++k) {
        cp_wait<W9_ST - 2>();
        __syncthreads();
        if (k + W9_ST - 1 < nt) load_stage((k + W9_ST - 1) % W9_ST);
        cp_commit();
        const unsigned sk = s0 + k % W9_ST * (16 * (SA + SB));
        const int rows = a.H - cy * TH;  // rows below the image are left out
        // the column right of the image has dy = 0 but the image's last x at its left tap:
        // that x is taken out of the fragments, as 0 times an infinity is no 0
        const int xe = a.W - cx * W9_TW;
        unsigned mask[2];
#pragma unroll
        for (int h = 0; h < 2; ++h)
            mask[h] = xe < W9_TW && (xe >> 1) == (lane & 3) + 4 * h ? (xe & 1 ? 0x0000ffffu : 0xffff0000u) : 0xffffffffu;
        if (++cx == a.ntx) {
            cx = 0;
            if (++cy == a.nty) cy = 0;
        }
        auto row_products = [&](int m) {  // the group's m-th row
            unsigned af[2][4];
#pragma unroll
            for (int i = 0; i < 2; ++i)
                ldsm_x4_t(sk + fa[i] + m * (KG * W9_TW * CA * 16), af[i][0], af[i][1], af[i][2], af[i][3]);
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                unsigned bf[4][2];
#pragma unroll
                for (int j = 0; j < 2; ++j)
                    ldsm_x4_t(sk + fb[d][j] + m * (KG * W9_PITCH * CB * 16), bf[2 * j][0], bf[2 * j][1],
                              bf[2 * j + 1][0], bf[2 * j + 1][1]);
                if (d == 0) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) bf[j][0] &= mask[0], bf[j][1] &= mask[1];
                }
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        mma16816(acc[d][i][j], af[i][0], af[i][1], af[i][2], af[i][3], bf[j][0], bf[j][1]);
            }
        };
        if (rows >= TH) {
#pragma unroll 4
            for (int m = 0; m < TH / KG; ++m) row_products(m);
        } else {
#pragma unroll 1
            for (int m = 0; kg + m * KG < rows; ++m) row_products(m);
        }
    }
    cp_wait<0>();
    if (KG > 1) {  // the row groups' sums, one group at a time (3 Q warps of 96 x 32 floats)
        float *red = reinterpret_cast<float *>(w9) + (trow * Q + quad) * 96 * 32 + lane;
        for (int g = 1; g < KG; ++g) {
            __syncthreads();
            if (kg == g) {
#pragma unroll
                for (int e = 0; e < 96; ++e) red[e * 32] = acc[e / 32][e / 16 % 2][e / 4 % 4][e % 4];
            }
            __syncthreads();
            if (kg == 0) {
#pragma unroll
                for (int e = 0; e < 96; ++e) acc[e / 32][e / 16 % 2][e / 4 % 4][e % 4] += red[e * 32];
            }
        }
        if (kg) return;
    }
    const long long K = 9LL * a.Cin;
#pragma unroll
    for (int d = 0; d < 3; ++d)
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                const int co = m0 + qm + i * 16 + (lane >> 2) + hf * 8;
                if (co >= a.Cout) continue;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int ci = n0 + qn + j * 8 + 2 * (lane & 3);
                    if (ci >= a.Cin) continue;
                    float *o = a.dw + co * K + (3 * trow + d) * a.Cin + ci;
                    const float v0 = acc[d][i][j][2 * hf], v1 = acc[d][i][j][2 * hf + 1];
                    if (a.pair)
                        atomicAdd(reinterpret_cast<float2 *>(o), make_float2(v0, v1));
                    else
                        atomicAdd(o, v0), atomicAdd(o + 1, v1);
                }
            }
}

template <int CO, int CI>
static int launch_wgrad9(Wgrad9Args a, cudaStream_t st)
{
    static_assert(CO * CI == 4096 || w9_smem(CO, CI) >= 3 * 96 * 32 * 4 * (CO * CI / 1024), "room for the groups' sums");
    auto kern = k_conv3x3_wgrad9<CO, CI>;
    PFF_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, w9_smem(CO, CI)));
    const int nb = (a.Cin + CI - 1) / CI, mb = (a.Cout + CO - 1) / CO;
    a.ntx = (a.W + W9_TW - 1) / W9_TW;
    a.nty = (a.H + w9_rows(CO, CI) - 1) / w9_rows(CO, CI);
    a.ntiles = a.B * a.ntx * a.nty;
    // one CTA per SM: as many ranges of pixel tiles as that takes
    const int split = std::max(1, std::min(a.ntiles, 148 / (nb * mb)));
    kern<<<dim3(nb, mb, split), W9_THREADS, w9_smem(CO, CI), st>>>(a);
    count_launch();
    return PFF_OK;
}

// ---- small ops --------------------------------------------------------------------------
#define GRID_STRIDE(e, n) \
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < (n); e += (long long)gridDim.x * blockDim.x)

// db[c] += sum_p dy[p][c]: each block reduces a pixel range per channel
__global__ void k_bias_grad(const bf16_t *__restrict__ dy, int cs, int off, float *db, long long P, int C)
{
    const int c = threadIdx.x % C;
    const int lanes = blockDim.x / C;
    const int l = threadIdx.x / C;
    if (l >= lanes) return;
    float s = 0.f;
    for (long long p = blockIdx.x * (long long)lanes + l; p < P; p += (long long)gridDim.x * lanes)
        s += bf2f(dy[p * cs + off + c]);
    atomicAdd(db + c, s);
}

__global__ void k_relu_bwd(bf16_t *g, int csg, int offg, const bf16_t *__restrict__ y, int csy, int offy, long long P,
                           int C)
{
    GRID_STRIDE(e, P * C)
    {
        const long long p = e / C;
        const int c = (int)(e - p * C);
        if (!(bf2f(y[p * csy + offy + c]) > 0.f)) g[p * csg + offg + c] = 0;
    }
}

// y[b, Y, X] = mean of the 2x2 block of x (H, W even: the fine grid)
__global__ void k_avgpool2(const bf16_t *__restrict__ x, int csx, int offx, bf16_t *y, int csy, int offy, int B, int H,
                           int W, int C)
{
    const int h2 = H / 2, w2 = W / 2;
    GRID_STRIDE(e, (long long)B * h2 * w2 * C)
    {
        const int c = (int)(e % C);
        const long long q = e / C;
        const int X = (int)(q % w2);
        const long long t = q / w2;
        const int Y = (int)(t % h2);
        const long long b = t / h2;
        const long long p00 = (b * H + 2 * Y) * W + 2 * X;
        const float s = bf2f(x[p00 * csx + offx + c]) + bf2f(x[(p00 + 1) * csx + offx + c]) +
                        bf2f(x[(p00 + W) * csx + offx + c]) + bf2f(x[(p00 + W + 1) * csx + offx + c]);
        y[q * csy + offy + c] = f2bf(0.25f * s);
    }
}

// dx[fine] (+)= dy[coarse] / 4
__global__ void k_avgpool2_bwd(const bf16_t *__restrict__ dy, int csd, int offd, bf16_t *dx, int csx, int offx, int B,
                               int H, int W, int C, int accumulate)
{
    const int h2 = H / 2, w2 = W / 2;
    GRID_STRIDE(e, (long long)B * H * W * C)
    {
        const int c = (int)(e % C);
        const long long p = e / C;
        const int x = (int)(p % W);
        const long long t = p / W;
        const int y = (int)(t % H);
        const long long b = t / H;
        const long long q = (b * h2 + y / 2) * w2 + x / 2;
        float v = 0.25f * bf2f(dy[q * csd + offd + c]);
        bf16_t *o = dx + p * csx + offx + c;
        if (accumulate) v += bf2f(*o);
        *o = f2bf(v);
    }
}

// y[fine] = x[coarse] (nearest), H, W: the coarse grid
__global__ void k_upsample2(const bf16_t *__restrict__ x, int csx, int offx, bf16_t *y, int csy, int offy, int B, int H,
                            int W, int C)
{
    const int H2 = 2 * H, W2 = 2 * W;
    GRID_STRIDE(e, (long long)B * H2 * W2 * C)
    {
        const int c = (int)(e % C);
        const long long p = e / C;
        const int X = (int)(p % W2);
        const long long t = p / W2;
        const int Y = (int)(t % H2);
        const long long b = t / H2;
        y[p * csy + offy + c] = x[((b * H + Y / 2) * W + X / 2) * csx + offx + c];
    }
}

// dx[coarse] = sum of dy over the 2x2 block
__global__ void k_upsample2_bwd(const bf16_t *__restrict__ dy, int csd, int offd, bf16_t *dx, int csx, int offx, int B,
                                int H, int W, int C)
{
    const int W2 = 2 * W;
    GRID_STRIDE(e, (long long)B * H * W * C)
    {
        const int c = (int)(e % C);
        const long long q = e / C;
        const int X = (int)(q % W);
        const long long t = q / W;
        const int Y = (int)(t % H);
        const long long b = t / H;
        const long long p00 = (b * 2 * H + 2 * Y) * W2 + 2 * X;
        const float s = bf2f(dy[p00 * csd + offd + c]) + bf2f(dy[(p00 + 1) * csd + offd + c]) +
                        bf2f(dy[(p00 + W2) * csd + offd + c]) + bf2f(dy[(p00 + W2 + 1) * csd + offd + c]);
        dx[q * csx + offx + c] = f2bf(s);
    }
}

// ---- the same ops on 8 channels (16 bytes) per thread ----------------------------------
// Where C, the row strides, the offsets and the addresses are multiples of 8 channels.  The
// one-channel forms moved 2 bytes per load and divided 64-bit indices: 305 us for the ten
// launches of a training step at 16 x 128 x 128, whose bytes take 30 us.
struct Row8 {
    float f[8];
};
__device__ __forceinline__ Row8 load8(const bf16_t *p)
{
    const uint4 v = *reinterpret_cast<const uint4 *>(p);
    const unsigned w[4] = {v.x, v.y, v.z, v.w};
    Row8 r;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        r.f[2 * k] = __uint_as_float(w[k] << 16);
        r.f[2 * k + 1] = __uint_as_float(w[k] & 0xffff0000u);
    }
    return r;
}
__device__ __forceinline__ void store8(bf16_t *p, const Row8 &r)
{
    unsigned w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) w[k] = (unsigned)f2bf(r.f[2 * k]) | ((unsigned)f2bf(r.f[2 * k + 1]) << 16);
    *reinterpret_cast<uint4 *>(p) = make_uint4(w[0], w[1], w[2], w[3]);
}

// OP 0: average pooling (h, w the coarse grid), 1: its data gradient (h, w the fine grid),
// 2: nearest upsampling (h, w the fine grid), 3: its data gradient (h, w the coarse grid).
// n = pixels of the h x w grid times C / 8, below 2^31.
template <int OP>
__global__ void __launch_bounds__(256) k_resample8(const bf16_t *__restrict__ x, int csx, int offx, bf16_t *y, int csy,
                                                   int offy, int h, int w, int cg, unsigned n, int accumulate)
{
    for (unsigned e = blockIdx.x * 256u + threadIdx.x; e < n; e += gridDim.x * 256u) {
        const unsigned q = e / (unsigned)cg, c = (e - q * (unsigned)cg) * 8;
        const unsigned t = q / (unsigned)w, X = q - t * (unsigned)w;
        bf16_t *o = y + (long long)q * csy + offy + c;
        if (OP == 0 || OP == 3) {  // sources on the fine grid: 2 x 2 block (rows t = b * h + Y)
            const long long p00 = (long long)t * 2 * (2 * w) + 2 * X;
            const bf16_t *s = x + p00 * csx + offx + c;
            const Row8 a0 = load8(s), a1 = load8(s + csx), a2 = load8(s + (long long)2 * w * csx),
                       a3 = load8(s + ((long long)2 * w + 1) * csx);
            Row8 r;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const float v = a0.f[k] + a1.f[k] + a2.f[k] + a3.f[k];
                r.f[k] = OP == 0 ? 0.25f * v : v;
            }
            store8(o, r);
        } else {  // source on the coarse grid: row t / 2 (fine rows of an image are even in number)
            const long long p = (long long)(t / 2) * (w / 2) + X / 2;
            const bf16_t *s = x + p * csx + offx + c;
            if (OP == 2) {
                *reinterpret_cast<uint4 *>(o) = *reinterpret_cast<const uint4 *>(s);
            } else {
                Row8 r = load8(s);
#pragma unroll
                for (int k = 0; k < 8; ++k) r.f[k] = 0.25f * r.f[k];
                if (accumulate) {
                    const Row8 g = load8(o);
#pragma unroll
                    for (int k = 0; k < 8; ++k) r.f[k] += g.f[k];
                }
                store8(o, r);
            }
        }
    }
}

// g = 0 where the layer's output y is not positive (y may be null: no ReLU), and
// db[c] += sum_p g[p][c], in one pass of 16-byte loads; the sums collect per thread, then
// per block, then by one atomic per block and channel.  As two passes of 2-byte loads these
// took 516 us of a training step at 16 x 128 x 128.
__global__ void __launch_bounds__(256) k_relu_bias_bwd(bf16_t *g, int csg, int offg, const bf16_t *__restrict__ y, int csy,
                                                       int offy, float *db, long long P, int C)
{
    __shared__ float sm[256][9];  // 9: rows of threads with the same channels fall in different banks
    const int cg = C / 8, rows = 256 / cg, c = threadIdx.x % cg * 8, r = threadIdx.x / cg;
    Row8 s;
#pragma unroll
    for (int k = 0; k < 8; ++k) s.f[k] = 0.f;
    if (r < rows)
        for (long long p = (long long)blockIdx.x * rows + r; p < P; p += (long long)gridDim.x * rows) {
            bf16_t *gp = g + p * csg + offg + c;
            uint4 gv = *reinterpret_cast<const uint4 *>(gp);
            if (y) {
                const Row8 yv = load8(y + p * csy + offy + c);
                unsigned *w = reinterpret_cast<unsigned *>(&gv);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if (!(yv.f[2 * k] > 0.f)) w[k] &= 0xffff0000u;
                    if (!(yv.f[2 * k + 1] > 0.f)) w[k] &= 0x0000ffffu;
                }
                *reinterpret_cast<uint4 *>(gp) = gv;
            }
            const unsigned w[4] = {gv.x, gv.y, gv.z, gv.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                s.f[2 * k] += __uint_as_float(w[k] << 16);
                s.f[2 * k + 1] += __uint_as_float(w[k] & 0xffff0000u);
            }
        }
#pragma unroll
    for (int k = 0; k < 8; ++k) sm[threadIdx.x][k] = s.f[k];
    __syncthreads();
    for (int e = threadIdx.x; e < C; e += 256) {
        float t = 0.f;
        for (int q = 0; q < rows; ++q) t += sm[q * cg + e / 8][e % 8];
        atomicAdd(db + e, t);
    }
}

static bool rows8(const void *p, int cs, int off, int C)
{
    return ((uintptr_t)p & 15) == 0 && cs % 8 == 0 && off % 8 == 0 && C % 8 == 0;
}

// loss += sum_p w_p (pred_p - t_p)^2 * scale; dpred[p][0] = 2 w_p (pred_p - t_p) * scale (bf16),
// the other channels of the dpred row zeroed.
__global__ void k_mse(const float *__restrict__ pred, int csp, const float *__restrict__ tgt,
                      const float *__restrict__ wgt, long long P, bf16_t *dpred, int csd, float scale, float *loss)
{
    float s = 0.f;
    GRID_STRIDE(p, P)
    {
        const float w = wgt ? wgt[p] : 1.f;
        const float d = pred[p * csp] - tgt[p];
        s += w * d * d;
        bf16_t *o = dpred + p * csd;
        o[0] = f2bf(2.f * w * d * scale);
        for (int c = 1; c < csd; ++c) o[c] = 0;
    }
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(loss, s * scale);
}

// Adam (decoupled weight decay); writes the bf16 copy of the parameters if asked
__global__ void k_adam(float *p, const float *__restrict__ g, float *m, float *v, bf16_t *pb, long long n, float lr,
                       float b1, float b2, float eps, float bc1, float bc2, float wd)
{
    GRID_STRIDE(e, n)
    {
        const float gi = g[e];
        const float mi = b1 * m[e] + (1.f - b1) * gi;
        const float vi = b2 * v[e] + (1.f - b2) * gi * gi;
        m[e] = mi;
        v[e] = vi;
        float pi = p[e] * (1.f - lr * wd);
        pi -= lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
        p[e] = pi;
        if (pb) pb[e] = f2bf(pi);
    }
}

__global__ void k_f32_to_bf16(const float *__restrict__ s, bf16_t *d, long long n)
{
    GRID_STRIDE(e, n) d[e] = f2bf(s[e]);
}

static int grid_for(long long n, int threads = 256)
{
    long long b = (n + threads - 1) / threads;
    return (int)std::max<long long>(1, std::min<long long>(b, 148LL * 16));
}

// the tcgen05 forward (pff_conv_tc.cu)
int conv_path();
bool conv_tc_supported(int H, int W, int Cin, int Cout, int csx, int offx, int csy, int offy, int out_f32, int *BW,
                       int *BH);
int conv3x3_tc(const bf16_t *x, int csx, int offx, const bf16_t *w, const float *bias, void *y, int csy, int offy,
               int B, int H, int W, int Cin, int Cout, int relu, int out_f32, cudaStream_t st);

static int check_slice(const char *who, int cs, int off, int C)
{
    if (cs <= 0 || off < 0 || C <= 0 || off + C > cs) {
        set_error("%s: channel slice [%d, %d) outside rows of %d", who, off, off + C, cs);
        return PFF_ERR_ARG;
    }
    return PFF_OK;
}

}  // namespace pff

using namespace pff;

extern "C" int pff_conv3x3_fwd(const bf16_t *x, int csx, int offx, const bf16_t *w, const float *bias, void *y,
                               int csy, int offy, int B, int H, int W, int Cin, int Cout, int relu, int out_f32,
                               void *stream)
{
    clear_error();
    if (!x || !w || !y || B <= 0 || H <= 0 || W <= 0 || Cin <= 0 || Cout <= 0 || Cin % 8 || csx % 8 || offx % 8) {
        set_error("pff_conv3x3_fwd: bad arguments (Cin, row stride and offset must be multiples of 8)");
        return PFF_ERR_ARG;
    }
    PFF_TRY(check_slice("pff_conv3x3_fwd input", csx, offx, Cin));
    PFF_TRY(check_slice("pff_conv3x3_fwd output", csy, offy, Cout));
    if (!out_f32 && ((Cout % 2 && Cout != 1) || csy % 2 || offy % 2)) {
        set_error("pff_conv3x3_fwd: bf16 output needs even Cout, row stride and offset");
        return PFF_ERR_ARG;
    }
    const int path = conv_path();
    int bw, bh;
    const bool tc_ok = conv_tc_supported(H, W, Cin, Cout, csx, offx, csy, offy, out_f32, &bw, &bh);
    if (path == 2 || (path == 0 && tc_ok))
        return conv3x3_tc(x, csx, offx, w, bias, y, csy, offy, B, H, W, Cin, Cout, relu, out_f32, S(stream));
    ConvArgs a{x, csx, offx, w, bias, y, csy, offy, B, H, W, Cin, Cout, relu, out_f32};
    const long long P = (long long)B * H * W;
    // whole tiles of 8, 32, 64 or 96 channels fit shared memory twice beside the weights; other counts,
    // and rows beyond 32-bit offsets within a tile, take the im2col form
    if ((Cin == 8 || (Cin % 32 == 0 && Cin <= 96)) && Cout <= 1 << 20 && P < (1LL << 30) && (20LL * W + 32) * csx < (1LL << 31)) {
        const int rc = Cin == 8 ? launch_conv_tile<1, 4>(a, S(stream))
                     : Cin == 32 ? launch_conv_tile<4, 4>(a, S(stream))
                     : Cin == 64 ? launch_conv_tile<8, 8>(a, S(stream)) : launch_conv_tile<12, 8>(a, S(stream));
        if (rc != PFF_OK) return rc;
        return check_cuda("pff_conv3x3_fwd");
    }
    const int bn = Cout > 32 ? 64 : (Cout > 16 ? 32 : 16);
    dim3 grid((unsigned)((P + CV_BM - 1) / CV_BM), (unsigned)((Cout + bn - 1) / bn));
    if (bn == 64) k_conv3x3<64><<<grid, CV_THREADS, 0, S(stream)>>>(a);
    else if (bn == 32) k_conv3x3<32><<<grid, CV_THREADS, 0, S(stream)>>>(a);
    else k_conv3x3<16><<<grid, CV_THREADS, 0, S(stream)>>>(a);
    count_launch();
    return check_cuda("pff_conv3x3_fwd");
}

extern "C" int pff_conv3x3_wflip(const bf16_t *w, bf16_t *wt, int Cin, int Cout, void *stream)
{
    clear_error();
    if (!w || !wt || Cin <= 0 || Cout <= 0) {
        set_error("pff_conv3x3_wflip: bad arguments");
        return PFF_ERR_ARG;
    }
    const long long n = 9LL * Cin * Cout;
    { k_wflip<<<grid_for(n), 256, 0, S(stream)>>>(w, wt, Cin, Cout); count_launch(); }
    return check_cuda("pff_conv3x3_wflip");
}

extern "C" int pff_conv3x3_wgrad(const bf16_t *x, int csx, int offx, const bf16_t *dy, int csd, int offd, float *dw,
                                 int B, int H, int W, int Cin, int Cout, void *stream)
{
    clear_error();
    if (!x || !dy || !dw || B <= 0 || H <= 0 || W <= 0 || Cin % 8 || Cout % 8 || Cin <= 0 || Cout <= 0 || csx % 8 ||
        offx % 8 || csd % 8 || offd % 8) {
        set_error("pff_conv3x3_wgrad: bad arguments (channels, strides, offsets multiples of 8)");
        return PFF_ERR_ARG;
    }
    PFF_TRY(check_slice("pff_conv3x3_wgrad input", csx, offx, Cin));
    PFF_TRY(check_slice("pff_conv3x3_wgrad dy", csd, offd, Cout));
    const long long P = (long long)B * H * W;
    // always, where a tile's offsets and the number of tiles fit 32 bits (also with 8 channels on
    // one side, three quarters of a block padding: 8 -> 32 at 16 x 128 x 128 23 us against 31,
    // 32 -> 8 22 against 39)
    if (Cin <= 32768 && Cout <= 32768 && P < (1LL << 30) &&
        (20LL * W + 32) * std::max(csx, csd) < (1LL << 31)) {
        Wgrad9Args a{x, csx, offx, dy, csd, offd, dw, B, H, W, Cin, Cout, 0, 0, 0, ((uintptr_t)dw & 7) == 0};
        // channel blocks of 64 where at most 31 of the last one's are padding
        const bool co64 = (Cout + 31) / 32 % 2 == 0, ci64 = (Cin + 31) / 32 % 2 == 0;
        const int rc = co64 ? ci64 ? launch_wgrad9<64, 64>(a, S(stream)) : launch_wgrad9<64, 32>(a, S(stream))
                            : ci64 ? launch_wgrad9<32, 64>(a, S(stream)) : launch_wgrad9<32, 32>(a, S(stream));
        if (rc != PFF_OK) return rc;
        return check_cuda("pff_conv3x3_wgrad");
    }
    const int K = 9 * Cin;
    constexpr int bm = 64, bn = 64;
    const int tiles = ((K + bn - 1) / bn) * ((Cout + bm - 1) / bm);
    // enough pixel chunks for ~4 CTAs per SM, each at least 512 pixels
    long long chunks = std::max<long long>(1, (148LL * 4 + tiles - 1) / tiles);
    long long pchunk = (P + chunks - 1) / chunks;
    pchunk = std::max<long long>(512, (pchunk + WG_BK - 1) / WG_BK * WG_BK);
    chunks = (P + pchunk - 1) / pchunk;
    if (pchunk > 0x7fffffffLL - WG_BK) {
        set_error("pff_conv3x3_wgrad: too many pixels");
        return PFF_ERR_ARG;
    }
    WgradArgs a{x, csx, offx, dy, csd, offd, dw, B, H, W, Cin, Cout, pchunk};
    dim3 grid((unsigned)((K + bn - 1) / bn), (unsigned)((Cout + bm - 1) / bm), (unsigned)chunks);
    k_conv3x3_wgrad<bm, bn><<<grid, WG_THREADS, 0, S(stream)>>>(a);
    count_launch();
    return check_cuda("pff_conv3x3_wgrad");
}

extern "C" int pff_bias_grad(const bf16_t *dy, int cs, int off, float *db, long long P, int C, void *stream)
{
    clear_error();
    if (!dy || !db || P <= 0 || C <= 0 || C > 256) {
        set_error("pff_bias_grad: bad arguments (1 <= C <= 256)");
        return PFF_ERR_ARG;
    }
    PFF_TRY(check_slice("pff_bias_grad", cs, off, C));
    const int lanes = std::max(1, 256 / C);
    const int blocks = (int)std::min<long long>(1184, (P + lanes - 1) / lanes);
    { k_bias_grad<<<blocks, lanes * C, 0, S(stream)>>>(dy, cs, off, db, P, C); count_launch(); }
    return check_cuda("pff_bias_grad");
}

extern "C" int pff_relu_bwd(bf16_t *g, int csg, int offg, const bf16_t *y, int csy, int offy, long long P, int C,
                            void *stream)
{
    clear_error();
    if (!g || !y || P <= 0) {
        set_error("pff_relu_bwd: bad arguments");
        return PFF_ERR_ARG;
    }
    PFF_TRY(check_slice("pff_relu_bwd g", csg, offg, C));
    PFF_TRY(check_slice("pff_relu_bwd y", csy, offy, C));
    { k_relu_bwd<<<grid_for(P * C), 256, 0, S(stream)>>>(g, csg, offg, y, csy, offy, P, C); count_launch(); }
    return check_cuda("pff_relu_bwd");
}

extern "C" int pff_relu_bias_bwd(bf16_t *g, int csg, int offg, const bf16_t *y, int csy, int offy, float *db,
                                 long long P, int C, void *stream)
{
    clear_error();
    if (!g || !db || P <= 0 || C <= 0 || C > 256) {
        set_error("pff_relu_bias_bwd: bad arguments (1 <= C <= 256)");
        return PFF_ERR_ARG;
    }
    PFF_TRY(check_slice("pff_relu_bias_bwd g", csg, offg, C));
    if (y) PFF_TRY(check_slice("pff_relu_bias_bwd y", csy, offy, C));
    if (rows8(g, csg, offg, C) && (!y || rows8(y, csy, offy, C))) {
        const int rows = 256 / (C / 8);
        const int blocks = (int)std::min<long long>(148 * 6, (P + 4 * rows - 1) / (4 * rows));
        k_relu_bias_bwd<<<blocks, 256, 0, S(stream)>>>(g, csg, offg, y, csy, offy, db, P, C);
        count_launch();
        return check_cuda("pff_relu_bias_bwd");
    }
    if (y) PFF_TRY(pff_relu_bwd(g, csg, offg, y, csy, offy, P, C, stream));
    return pff_bias_grad(g, csg, offg, db, P, C, stream);
}

extern "C" int pff_avgpool2(const bf16_t *x, int csx, int offx, bf16_t *y, int csy, int offy, int B, int H, int W,
                            int C, void *stream)
{
    clear_error();
    if (!x || !y || B <= 0 || H < 2 || W < 2 || H % 2 || W % 2) {
        set_error("pff_avgpool2: bad arguments (even H, W)");
        return PFF_ERR_ARG;
    }
    PFF_TRY(check_slice("pff_avgpool2 x", csx, offx, C));
    PFF_TRY(check_slice("pff_avgpool2 y", csy, offy, C));
    const long long n = (long long)B * (H / 2) * (W / 2) * C;
    if (rows8(x, csx, offx, C) && rows8(y, csy, offy, C) && n / 8 < (1LL << 31)) {
        k_resample8<0><<<grid_for(n / 8), 256, 0, S(stream)>>>(x, csx, offx, y, csy, offy, H / 2, W / 2, C / 8, (unsigned)(n / 8), 0);
        count_launch();
    } else
    { k_avgpool2<<<grid_for(n), 256, 0, S(stream)>>>(x, csx, offx, y, csy, offy, B, H, W, C); count_launch(); }
    return check_cuda("pff_avgpool2");
}

extern "C" int pff_avgpool2_bwd(const bf16_t *dy, int csd, int offd, bf16_t *dx, int csx, int offx, int B, int H,
                                int W, int C, int accumulate, void *stream)
{
    clear_error();
    if (!dy || !dx || B <= 0 || H < 2 || W < 2 || H % 2 || W % 2) {
        set_error("pff_avgpool2_bwd: bad arguments (even H, W)");
        return PFF_ERR_ARG;
    }
    PFF_TRY(check_slice("pff_avgpool2_bwd dy", csd, offd, C));
    PFF_TRY(check_slice("pff_avgpool2_bwd dx", csx, offx, C));
    const long long n = (long long)B * H * W * C;
    if (rows8(dy, csd, offd, C) && rows8(dx, csx, offx, C) && n / 8 < (1LL << 31)) {
        k_resample8<1><<<grid_for(n / 8), 256, 0, S(stream)>>>(dy, csd, offd, dx, csx, offx, H, W, C / 8, (unsigned)(n / 8),
                                                             accumulate);
        count_launch();
    } else
    {
        k_avgpool2_bwd<<<grid_for(n), 256, 0, S(stream)>>>(dy, csd, offd, dx, csx, offx, B, H, W, C, accumulate);
        count_launch();
    }
    return check_cuda("pff_avgpool2_bwd");
}

extern "C" int pff_upsample2(const bf16_t *x, int csx, int offx, bf16_t *y, int csy, int offy, int B, int H, int W,
                             int C, void *stream)
{
    clear_error();
    if (!x || !y || B <= 0 || H <= 0 || W <= 0) {
        set_error("pff_upsample2: bad arguments");
        return PFF_ERR_ARG;
    }
    PFF_TRY(check_slice("pff_upsample2 x", csx, offx, C));
    PFF_TRY(check_slice("pff_upsample2 y", csy, offy, C));
    const long long n = (long long)B * 4 * H * W * C;
    if (rows8(x, csx, offx, C) && rows8(y, csy, offy, C) && n / 8 < (1LL << 31)) {
        k_resample8<2><<<grid_for(n / 8), 256, 0, S(stream)>>>(x, csx, offx, y, csy, offy, 2 * H, 2 * W, C / 8, (unsigned)(n / 8), 0);
        count_launch();
    } else
    { k_upsample2<<<grid_for(n), 256, 0, S(stream)>>>(x, csx, offx, y, csy, offy, B, H, W, C); count_launch(); }
    return check_cuda("pff_upsample2");
}

extern "C" int pff_upsample2_bwd(const bf16_t *dy, int csd, int offd, bf16_t *dx, int csx, int offx, int B, int H,
                                 int W, int C, void *stream)
{
    clear_error();
    if (!dy || !dx || B <= 0 || H <= 0 || W <= 0) {
        set_error("pff_upsample2_bwd: bad arguments");
        return PFF_ERR_ARG;
    }
    PFF_TRY(check_slice("pff_upsample2_bwd dy", csd, offd, C));
    PFF_TRY(check_slice("pff_upsample2_bwd dx", csx, offx, C));
    const long long n = (long long)B * H * W * C;
    if (rows8(dy, csd, offd, C) && rows8(dx, csx, offx, C) && n / 8 < (1LL << 31)) {
        k_resample8<3><<<grid_for(n / 8), 256, 0, S(stream)>>>(dy, csd, offd, dx, csx, offx, H, W, C / 8, (unsigned)(n / 8), 0);
        count_launch();
    } else
    { k_upsample2_bwd<<<grid_for(n), 256, 0, S(stream)>>>(dy, csd, offd, dx, csx, offx, B, H, W, C); count_launch(); }
    return check_cuda("pff_upsample2_bwd");
}

extern "C" int pff_mse_loss(const float *pred, int csp, const float *target, const float *weight, long long P,
                            bf16_t *dpred, int csd, float scale, float *loss, void *stream)
{
    clear_error();
    if (!pred || !target || !dpred || !loss || P <= 0 || csp <= 0 || csd <= 0) {
        set_error("pff_mse_loss: bad arguments");
        return PFF_ERR_ARG;
    }
    { k_mse<<<grid_for(P), 256, 0, S(stream)>>>(pred, csp, target, weight, P, dpred, csd, scale, loss); count_launch(); }
    return check_cuda("pff_mse_loss");
}

extern "C" int pff_adam(float *p, const float *g, float *m, float *v, bf16_t *p_bf16, long long n, float lr, float b1,
                        float b2, float eps, int step, float weight_decay, void *stream)
{
    clear_error();
    if (!p || !g || !m || !v || n <= 0 || step < 1) {
        set_error("pff_adam: bad arguments");
        return PFF_ERR_ARG;
    }
    const float bc1 = 1.f - powf(b1, (float)step), bc2 = 1.f - powf(b2, (float)step);
    {
        k_adam<<<grid_for(n), 256, 0, S(stream)>>>(p, g, m, v, p_bf16, n, lr, b1, b2, eps, bc1, bc2, weight_decay);
        count_launch();
    }
    return check_cuda("pff_adam");
}

extern "C" int pff_f32_to_bf16(const float *src, bf16_t *dst, long long n, void *stream)
{
    clear_error();
    if (!src || !dst || n <= 0) {
        set_error("pff_f32_to_bf16: bad arguments");
        return PFF_ERR_ARG;
    }
    { k_f32_to_bf16<<<grid_for(n), 256, 0, S(stream)>>>(src, dst, n); count_launch(); }
    return check_cuda("pff_f32_to_bf16");
}
