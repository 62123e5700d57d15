// mlp.cu -- the learned warm start's network and its training on the GPU.
//
// An MLP, 40 -> 128 -> 128 -> 16 with ReLU, maps the statistics of a locus
// pair (r, n), or of one sequence at a target column (the dual form's start),
// to a starting point (the inputs are built in warmstart.cu).
//
// Inference, and the forward pass of training, is one fused tcgen05 kernel
// (k_mlp_tc): BF16 weights and activations, FP32 accumulators in TMEM, all
// three layers of a 128-row tile without leaving the SM.  The backward pass
// (k_mlp_bwd) is one fused FP32 kernel on the FP32 master weights from the
// saved FP32 activations (mixed-precision training), and one more kernel adds
// its partial sums and takes the Adam step.  sdca_mlp_grad takes the FP32
// forward (tiled products, k_mm), the exact derivative the CPU oracle checks.  The parameter blob (MLP_* offsets in
// engine.h) holds the input normalisation, the FP32 weights and the output
// scale; the BF16 weight image is made from it (k_mlp_pack).
//
// SuperDCA has no learned component: its solver starts every locus from
// zero (SuperDCA/include/plmDCA.hpp:298).  The warm start only moves the
// starting point of a strictly convex problem.
#include <algorithm>
#include <cstdint>
#include <cstring>
#include <random>
#include <string>
#include <vector>

#include "engine.h"
#include <cuda_bf16.h>

#include "kernels_common.cuh"
#include "superdca_gb300.h"
#include "tcgen05.cuh"

namespace sdca {
namespace {

constexpr int TM = 64, TN = 64, TK = 16;

// C[M x N] = A[M x K] . B[N x K]^T + bias, with ReLU when asked
__global__ void __launch_bounds__(256)
k_mm(int M, int N, int K, const float *__restrict__ A, const float *__restrict__ B, float *__restrict__ C,
     const float *__restrict__ bias, int relu)
{
    __shared__ float sA[TK][TM + 4];
    __shared__ float sB[TK][TN + 4];
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int m0 = blockIdx.y * TM, n0 = blockIdx.x * TN;
    float acc[4][4] = {};
    for (int k0 = 0; k0 < K; k0 += TK) {
        for (int e = threadIdx.x; e < TM * TK; e += 256) {
            const int kk = e % TK, mm = e / TK, m = m0 + mm, k = k0 + kk;
            sA[kk][mm] = m < M && k < K ? A[(int64_t)m * K + k] : 0.f;
        }
        for (int e = threadIdx.x; e < TN * TK; e += 256) {
            const int kk = e % TK, nn = e / TK, n = n0 + nn, k = k0 + kk;
            sB[kk][nn] = n < N && k < K ? B[(int64_t)n * K + k] : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < TK; ++kk) {
            float a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = sA[kk][ty + 16 * i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = sB[kk][tx + 16 * j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = m0 + ty + 16 * i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx + 16 * j;
            if (n >= N) continue;
            float v = acc[i][j] + bias[n];
            C[(int64_t)m * N + n] = relu ? fmaxf(v, 0.f) : v;
        }
    }
}

void mm(cudaStream_t st, int M, int N, int K, const float *A, const float *B, float *C, const float *bias, int relu)
{
    // rows in pieces that keep grid.y within its limit
    const int rows = std::min(M, 65535 * TM);
    for (int m0 = 0; m0 < M; m0 += rows) {
        const int mr = std::min(rows, M - m0);
        dim3 grid((N + TN - 1) / TN, (mr + TM - 1) / TM);
        k_mm<<<grid, 256, 0, st>>>(mr, N, K, A + (int64_t)m0 * K, B, C + (int64_t)m0 * N, bias, relu);
    }
}

// (x - mean) * scale, row-major M x MLP_IN
__global__ void k_normalise(int64_t M, const float *__restrict__ X, const float *__restrict__ p,
                            float *__restrict__ Xn)
{
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= M * MLP_IN) return;
    const int c = (int)(t % MLP_IN);
    Xn[t] = (X[t] - p[MLP_IN_MEAN + c]) * p[MLP_IN_SCALE + c];
}

// ---- the fused backward (FP32)
//
// From the outputs, targets and saved activations of M rows to the gradient
// of every weight: one CTA takes tiles of up to 64 rows, holds W2 and W3 and
// the tile's h1, h2, inputs and output gradient in shared memory, and keeps
// its sums of the three weight gradients in registers (92 per thread) over
// all its tiles.  h2 becomes d2 = (dout W3) masked, and h1 becomes d1 = (d2
// W2) masked, in place.  Each CTA writes its sums once; k_mlp_reduce adds the
// CTAs' up.  FP32 multiply-adds bound it (0.7 GFLOP at 8192 rows, some 10 us
// on all SMs).  As separate tiled products C = op(A) op(B) split along the
// rows, the three weight gradients ran on 4 to 16 CTAs and took 617 us each at 8192
// rows (1.9 ms of a 2 ms step); this kernel takes 32 us, the reduction and
// Adam 8, the forward 19.
constexpr int BW_THREADS = 256, BW_ROWS = 64;
constexpr int MLP_NPAR = MLP_TRAIN_END - MLP_W1;                 // trained parameters, W1 .. b3
constexpr int BW_W2 = 0, BW_W3 = BW_W2 + MLP_H * MLP_H, BW_H1 = BW_W3 + MLP_OUT * MLP_H, BW_H2 = BW_H1 + BW_ROWS * MLP_H,
              BW_X = BW_H2 + BW_ROWS * MLP_H, BW_D = BW_X + BW_ROWS * MLP_IN, BW_FLOATS = BW_D + BW_ROWS * MLP_OUT;
constexpr int BW_SMEM = BW_FLOATS * 4;
static_assert(MLP_H == 128 && MLP_OUT == 16 && MLP_IN == 40, "thread tiles of k_mlp_bwd");

__device__ __forceinline__ void fma4(float (&c)[4], float a, float4 b)
{
    c[0] = fmaf(a, b.x, c[0]);
    c[1] = fmaf(a, b.y, c[1]);
    c[2] = fmaf(a, b.z, c[2]);
    c[3] = fmaf(a, b.w, c[3]);
}

// idx (may be null): row m of the batch is row idx[m] of X and T.  tile_rows:
// rows per tile (a multiple of 4, at most BW_ROWS).  part[blockIdx.x]: this
// CTA's sums; loss += the mean squared error.
__global__ void __launch_bounds__(BW_THREADS, 1)
k_mlp_bwd(int64_t M, int tile_rows, const int32_t *__restrict__ idx, const float *__restrict__ X,
          const float *__restrict__ T, const float *__restrict__ p, const float *__restrict__ out,
          const float *__restrict__ h1, const float *__restrict__ h2, float *__restrict__ part,
          double *__restrict__ loss)
{
    extern __shared__ __align__(16) float sm[];
    float4 *const s4 = reinterpret_cast<float4 *>(sm);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, tx = t & 15, ty = t >> 4;
    static_assert(MLP_W2 % 4 == 0 && MLP_W3 % 4 == 0 && MLP_IN_MEAN % 4 == 0 && MLP_IN_SCALE % 4 == 0, "float4 loads of the blob");
#pragma unroll 8
    for (int e = t; e < MLP_H * MLP_H / 4; e += BW_THREADS) s4[BW_W2 / 4 + e] = reinterpret_cast<const float4 *>(p + MLP_W2)[e];
#pragma unroll
    for (int e = t; e < MLP_OUT * MLP_H / 4; e += BW_THREADS) s4[BW_W3 / 4 + e] = reinterpret_cast<const float4 *>(p + MLP_W3)[e];
    float g2[8][2][4] = {};   // W2: rows 4 ty + (0..3) and 64 + .., columns 4 tx + (0..3) and 64 + ..
    float g1[4][5] = {};      // W1: rows 4 (t / 8) + .., columns 5 (t % 8) + ..
    float g3[2][4] = {};      // W3: rows 2 warp + .., columns 4 lane + ..
    float gb = 0.f, gb3 = 0.f;   // b2[t] (t < 128) or b1[t - 128]; b3[t] (t < 16)
    double ls = 0.0;
    const float inv = 2.f / (float)M;
    const int64_t tiles = (M + tile_rows - 1) / tile_rows;
    for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int64_t m0 = tile * tile_rows;
        const int R = (int)min((int64_t)tile_rows, M - m0);
        __syncthreads();   // (the tile before is used up)
        // (16-byte loads: a row of X is ten of them, of T and the outputs four)
        for (int e = t; e < R * (MLP_OUT / 4); e += BW_THREADS) {
            const int m = e >> 2, o = e & 3;
            const int64_t row = idx ? (int64_t)idx[m0 + m] : m0 + m;
            const float4 y = reinterpret_cast<const float4 *>(out)[(m0 + m) * (MLP_OUT / 4) + o];
            const float4 w = reinterpret_cast<const float4 *>(T)[row * (MLP_OUT / 4) + o];
            const float4 r = make_float4(y.x - w.x, y.y - w.y, y.z - w.z, y.w - w.w);
            s4[BW_D / 4 + e] = make_float4(inv * r.x, inv * r.y, inv * r.z, inv * r.w);
            ls += (double)r.x * r.x + (double)r.y * r.y + (double)r.z * r.z + (double)r.w * r.w;
        }
#pragma unroll 3
        for (int e = t; e < R * (MLP_IN / 4); e += BW_THREADS) {
            const int m = e / (MLP_IN / 4), c = e % (MLP_IN / 4);
            const int64_t row = idx ? (int64_t)idx[m0 + m] : m0 + m;
            const float4 x = reinterpret_cast<const float4 *>(X)[row * (MLP_IN / 4) + c];
            const float4 mu = reinterpret_cast<const float4 *>(p + MLP_IN_MEAN)[c],
                         sc = reinterpret_cast<const float4 *>(p + MLP_IN_SCALE)[c];
            s4[BW_X / 4 + e] = make_float4((x.x - mu.x) * sc.x, (x.y - mu.y) * sc.y, (x.z - mu.z) * sc.z, (x.w - mu.w) * sc.w);
        }
#pragma unroll 4
        for (int e = t; e < R * (MLP_H / 4); e += BW_THREADS) {
            s4[BW_H1 / 4 + e] = reinterpret_cast<const float4 *>(h1 + m0 * MLP_H)[e];
            s4[BW_H2 / 4 + e] = reinterpret_cast<const float4 *>(h2 + m0 * MLP_H)[e];
        }
        __syncthreads();
        // W3 gradient: dout^T h2
        for (int m = 0; m < R; ++m) {
            const float4 h = s4[BW_H2 / 4 + m * (MLP_H / 4) + lane];
            fma4(g3[0], sm[BW_D + m * MLP_OUT + 2 * warp], h);
            fma4(g3[1], sm[BW_D + m * MLP_OUT + 2 * warp + 1], h);
        }
        if (t < MLP_OUT)
            for (int m = 0; m < R; ++m) gb3 += sm[BW_D + m * MLP_OUT + t];
        __syncthreads();
        // d2 = (dout W3) where h2 > 0, in place of h2: 8 rows per warp at a time
        for (int r0 = 8 * warp; r0 < R; r0 += 64) {
            float d[8][4] = {};
#pragma unroll 4
            for (int o = 0; o < MLP_OUT; ++o) {
                const float4 w = s4[BW_W3 / 4 + o * (MLP_H / 4) + lane];
#pragma unroll
                for (int k = 0; k < 8; ++k) fma4(d[k], sm[BW_D + (r0 + k) * MLP_OUT + o], w);
            }
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                if (r0 + k >= R) break;
                float4 &h = s4[BW_H2 / 4 + (r0 + k) * (MLP_H / 4) + lane];
                h = make_float4(h.x > 0.f ? d[k][0] : 0.f, h.y > 0.f ? d[k][1] : 0.f, h.z > 0.f ? d[k][2] : 0.f,
                                h.w > 0.f ? d[k][3] : 0.f);
            }
        }
        __syncthreads();
        // W2 gradient: d2^T h1
#pragma unroll 2
        for (int m = 0; m < R; ++m) {
            const float4 a0 = s4[BW_H2 / 4 + m * 32 + ty], a1 = s4[BW_H2 / 4 + m * 32 + 16 + ty];
            const float4 b0 = s4[BW_H1 / 4 + m * 32 + tx], b1 = s4[BW_H1 / 4 + m * 32 + 16 + tx];
            const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                fma4(g2[i][0], a[i], b0);
                fma4(g2[i][1], a[i], b1);
            }
        }
        if (t < MLP_H)
            for (int m = 0; m < R; ++m) gb += sm[BW_H2 + m * MLP_H + t];
        __syncthreads();
        // d1 = (d2 W2) where h1 > 0, in place of h1: rows 4 ty + .., columns as above
        if (4 * ty < R) {
            float d[4][2][4] = {};
#pragma unroll 2
            for (int j = 0; j < MLP_H; j += 4) {
                float4 a[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) a[i] = s4[BW_H2 / 4 + (4 * ty + i) * 32 + j / 4];
#pragma unroll
                for (int jj = 0; jj < 4; ++jj) {
                    const float4 b0 = s4[BW_W2 / 4 + (j + jj) * 32 + tx], b1 = s4[BW_W2 / 4 + (j + jj) * 32 + 16 + tx];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float v = jj == 0 ? a[i].x : jj == 1 ? a[i].y : jj == 2 ? a[i].z : a[i].w;
                        fma4(d[i][0], v, b0);
                        fma4(d[i][1], v, b1);
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    if (4 * ty + i >= R) break;
                    float4 &h = s4[BW_H1 / 4 + (4 * ty + i) * 32 + 16 * hh + tx];
                    h = make_float4(h.x > 0.f ? d[i][hh][0] : 0.f, h.y > 0.f ? d[i][hh][1] : 0.f,
                                    h.z > 0.f ? d[i][hh][2] : 0.f, h.w > 0.f ? d[i][hh][3] : 0.f);
                }
        }
        __syncthreads();
        // W1 gradient: d1^T x
        {
            const int k4 = t >> 3, c0 = 5 * (t & 7);
#pragma unroll 2
            for (int m = 0; m < R; ++m) {
                const float4 a = s4[BW_H1 / 4 + m * 32 + k4];
#pragma unroll
                for (int c = 0; c < 5; ++c) {
                    const float x = sm[BW_X + m * MLP_IN + c0 + c];
                    g1[0][c] = fmaf(a.x, x, g1[0][c]);
                    g1[1][c] = fmaf(a.y, x, g1[1][c]);
                    g1[2][c] = fmaf(a.z, x, g1[2][c]);
                    g1[3][c] = fmaf(a.w, x, g1[3][c]);
                }
            }
        }
        if (t >= MLP_H)
            for (int m = 0; m < R; ++m) gb += sm[BW_H1 + m * MLP_H + t - MLP_H];
    }
    float *o = part + (int64_t)blockIdx.x * MLP_NPAR - MLP_W1;   // (blob offsets)
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
            const int r = 4 * ty + (i & 3) + 64 * (i >> 2), c = 4 * tx + 64 * hh;
#pragma unroll
            for (int k = 0; k < 4; ++k) o[MLP_W2 + r * MLP_H + c + k] = g2[i][hh][k];
        }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int c = 0; c < 5; ++c) o[MLP_W1 + (4 * (t >> 3) + i) * MLP_IN + 5 * (t & 7) + c] = g1[i][c];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int k = 0; k < 4; ++k) o[MLP_W3 + (2 * warp + i) * MLP_H + 4 * lane + k] = g3[i][k];
    o[t < MLP_H ? MLP_B2 + t : MLP_B1 + t - MLP_H] = gb;
    if (t < MLP_OUT) o[MLP_B3 + t] = gb3;
    ls = warp_sum(ls);
    __shared__ double red[BW_THREADS / 32];
    if (lane == 0) red[warp] = ls;
    __syncthreads();
    if (t == 0) {
        double v = 0.0;
        for (int k = 0; k < BW_THREADS / 32; ++k) v += red[k];
        atomicAdd(loss, v / (double)M);
    }
}

// The parameter's place in the BF16 weight image, -1 for a bias
__device__ __forceinline__ int wb_place(int e)
{
    if (e < MLP_B1) return (e - MLP_W1) / MLP_IN * 64 + (e - MLP_W1) % MLP_IN;
    if (e >= MLP_W2 && e < MLP_B2) return MLP_H * 64 + e - MLP_W2;
    if (e >= MLP_W3 && e < MLP_B3) return MLP_H * 64 + MLP_H * MLP_H + e - MLP_W3;
    return -1;
}

// The gradient of a parameter is the sum of the CTAs' partial sums (RD_SEG
// threads share them out); written to g, or (g null) an Adam step on p and
// the parameter's entry of the BF16 image.
constexpr int RD_PAR = 32, RD_SEG = 8;

__global__ void __launch_bounds__(RD_PAR * RD_SEG)
k_mlp_reduce(int blocks, const float *__restrict__ part, float *__restrict__ g, float *__restrict__ p,
             float *__restrict__ m1, float *__restrict__ m2, __nv_bfloat16 *__restrict__ wb, float lr, float b1,
             float b2, float eps, float c1, float c2)
{
    __shared__ float red[RD_SEG][RD_PAR];
    const int k = threadIdx.x % RD_PAR, seg = threadIdx.x / RD_PAR, i = blockIdx.x * RD_PAR + k;
    float s = 0.f;
    if (i < MLP_NPAR) {
#pragma unroll 8
        for (int b = seg; b < blocks; b += RD_SEG) s += part[(int64_t)b * MLP_NPAR + i];
    }
    red[seg][k] = s;
    __syncthreads();
    if (seg != 0 || i >= MLP_NPAR) return;
    float gi = 0.f;
#pragma unroll
    for (int q = 0; q < RD_SEG; ++q) gi += red[q][k];
    const int e = MLP_W1 + i;
    if (g) {
        g[e] = gi;
        return;
    }
    const float a = b1 * m1[e] + (1.f - b1) * gi;
    const float b = b2 * m2[e] + (1.f - b2) * gi * gi;
    m1[e] = a;
    m2[e] = b;
    const float v = p[e] - lr * (a / c1) / (sqrtf(b / c2) + eps);
    p[e] = v;
    const int place = wb_place(e);
    if (place >= 0) wb[place] = __float2bfloat16_rn(v);
}

// ---- the fused tensor-core forward (BF16 weights, FP32 accumulators)
//
// One CTA of 128 threads owns the three BF16 weight matrices in shared
// memory (128-byte swizzled K-major tiles: W1 128 x 64 with the 40 inputs
// zero-padded, W2 128 x 128 as two 64-column atoms, W3 16 x 128 likewise)
// and walks 128-row tiles of the input.  Per tile: thread r normalises row
// r, rounds it to BF16 into the A tile; one thread issues the layer's
// tcgen05.mma (M128, K16 steps) into TMEM and commits to an mbarrier; every
// thread reads its row's accumulators back (tcgen05.ld, TMEM lane = row),
// adds the bias, applies ReLU and writes the next layer's BF16 A tile.
// Layer 3 (N = 16) writes the outputs.  Row m of the input is row idx[m] of X
// when idx is given.  h1, h2 (optional) receive the FP32
// activations for the backward pass.
constexpr int MT_THREADS = 128;
constexpr int MT_K1 = 64;                                       // layer-1 K, padded
constexpr int MT_W1_ELEMS = MLP_H * MT_K1, MT_W2_ELEMS = MLP_H * MLP_H, MT_W3_ELEMS = MLP_OUT * MLP_H;
constexpr int MT_WB_ELEMS = MT_W1_ELEMS + MT_W2_ELEMS + MT_W3_ELEMS;   // BF16 weight image
constexpr uint32_t MT_SW1 = 0, MT_SW2 = 16384, MT_SW3 = 49152, MT_SA1 = 53248, MT_SA2 = 69632;
constexpr uint32_t MT_SBAR = 102400;
constexpr int MT_SMEM = (int)MT_SBAR + 64 + 1024;
constexpr uint32_t MT_TMEM_COLS = 256;                          // layer 1/3 at 0, layer 2 at 128
// kind::f16 instruction descriptor: D = F32, A = B = BF16, K-major, M = 128
constexpr uint32_t mt_idesc(int n) { return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | (8u << 24); }
static_assert(MLP_IN <= MT_K1 && MLP_H == 128 && MLP_OUT == 16, "tile shapes of k_mlp_tc");
static_assert(MT_WB_ELEMS == MLP_WB_ELEMS, "weight image size");
static_assert(MT_SW2 - MT_SW1 == 2 * MT_W1_ELEMS && MT_SW3 - MT_SW2 == 2 * MT_W2_ELEMS &&
              MT_SA1 - MT_SW3 == 2 * MT_W3_ELEMS && MT_SBAR - MT_SA2 == 2 * 128 * 128,
              "shared-memory map");

__device__ __forceinline__ void mt_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}

__device__ __forceinline__ uint32_t bf2(float a, float b)
{
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&v);
}

// rows x (64 * atoms) BF16, row-major in global -> 128-byte swizzled atoms
__device__ void mt_stage_weights(const __nv_bfloat16 *__restrict__ w, int rows, int atoms, uint32_t dst)
{
    for (int e = threadIdx.x; e < rows * atoms * 8; e += blockDim.x) {
        const int c = e & 7, r = (e >> 3) % rows, a = (e >> 3) / rows;
        const uint4 v = *reinterpret_cast<const uint4 *>(w + (int64_t)r * 64 * atoms + a * 64 + c * 8);
        tc::st_shared_v4(tc::sw128(dst + (uint32_t)(a * rows * 128), r, c), v);
    }
}

// 32 accumulator columns of this thread's row: + bias, ReLU, into the BF16 A
// tile (4 chunks of 8 at column c0) and, when given, the FP32 activations
__device__ __forceinline__ void mt_hidden(const float (&v)[32], const float *__restrict__ bias, int c0, uint32_t a2,
                                         int r, float *__restrict__ h)
{
    float x[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) x[j] = fmaxf(v[j] + bias[c0 + j], 0.f);
    if (h) {
#pragma unroll
        for (int j = 0; j < 32; j += 4)
            *reinterpret_cast<float4 *>(h + c0 + j) = make_float4(x[j], x[j + 1], x[j + 2], x[j + 3]);
    }
    const int atom = c0 >> 6;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int c = ((c0 & 63) >> 3) + q;
        tc::st_shared_v4(tc::sw128(a2 + (uint32_t)(atom * 16384), r, c),
                         make_uint4(bf2(x[8 * q], x[8 * q + 1]), bf2(x[8 * q + 2], x[8 * q + 3]),
                                    bf2(x[8 * q + 4], x[8 * q + 5]), bf2(x[8 * q + 6], x[8 * q + 7])));
    }
}

__global__ void __launch_bounds__(MT_THREADS, 2)
k_mlp_tc(int64_t M, const int32_t *__restrict__ idx, const float *__restrict__ X, const float *__restrict__ p,
         const __nv_bfloat16 *__restrict__ wb, float *__restrict__ out, float *__restrict__ h1, float *__restrict__ h2, int *__restrict__ err)
{
    extern __shared__ uint8_t smem_raw[];
    const uint32_t s0 = tc::smem_u32(smem_raw);
    const uint32_t sb = (s0 + 1023u) & ~1023u;
    uint8_t *const sg = smem_raw + (sb - s0);
    const uint32_t bar = sb + MT_SBAR, slot = bar + 8;
    const int t = threadIdx.x, warp = t >> 5;
    if (t == 0) {
        tc::mbar_init(bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot),
                     "r"(MT_TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    mt_stage_weights(wb, MLP_H, 1, sb + MT_SW1);
    mt_stage_weights(wb + MT_W1_ELEMS, MLP_H, 2, sb + MT_SW2);
    mt_stage_weights(wb + MT_W1_ELEMS + MT_W2_ELEMS, MLP_OUT, 2, sb + MT_SW3);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *reinterpret_cast<const uint32_t *>(sg + MT_SBAR + 8);
    const uint32_t lanes = (uint32_t)(warp * 32) << 16;
    const float *b1 = p + MLP_B1, *b2 = p + MLP_B2, *b3 = p + MLP_B3;
    uint32_t phase = 0;
    bool failed = false;
    // one layer: MMAs by thread 0, commit, bounded wait by every thread
    auto layer = [&](uint32_t d, uint32_t a, uint32_t w, int atoms, int a_stride, int w_stride, int n) -> bool {
        // the A tile's generic-proxy stores and this thread's TMEM reads come
        // before the MMAs that read the tile and overwrite the accumulators
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        if (t == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (int at = 0; at < atoms; ++at)
#pragma unroll
                for (int kk = 0; kk < 4; ++kk)
                    mt_mma(tmem + d, tc::smem_desc_sw128(a + (uint32_t)(at * a_stride + kk * 32)),
                           tc::smem_desc_sw128(w + (uint32_t)(at * w_stride + kk * 32)), mt_idesc(n),
                           (at > 0 || kk > 0) ? 1u : 0u);
            tc::mma_commit(bar);
        }
        const bool ok = tc::mbar_wait(bar, phase);
        phase ^= 1u;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        return __syncthreads_and(ok ? 1 : 0) != 0;
    };
    const int64_t tiles = (M + 127) / 128;
    for (int64_t tile = blockIdx.x; tile < tiles && !failed; tile += gridDim.x) {
        const int64_t row = tile * 128 + t;
        const bool live = row < M;
        {
            // input row -> normalised BF16, K padded to 64
            float x[MT_K1];
#pragma unroll
            for (int k = 0; k < MT_K1; ++k) x[k] = 0.f;
            if (live) {
                const float *xr = X + (idx ? (int64_t)idx[row] : row) * MLP_IN;
#pragma unroll
                for (int k = 0; k < MLP_IN; k += 4) {
                    const float4 v = *reinterpret_cast<const float4 *>(xr + k);
                    x[k] = (v.x - p[MLP_IN_MEAN + k]) * p[MLP_IN_SCALE + k];
                    x[k + 1] = (v.y - p[MLP_IN_MEAN + k + 1]) * p[MLP_IN_SCALE + k + 1];
                    x[k + 2] = (v.z - p[MLP_IN_MEAN + k + 2]) * p[MLP_IN_SCALE + k + 2];
                    x[k + 3] = (v.w - p[MLP_IN_MEAN + k + 3]) * p[MLP_IN_SCALE + k + 3];
                }
            }
#pragma unroll
            for (int c = 0; c < 8; ++c)
                tc::st_shared_v4(tc::sw128(sb + MT_SA1, t, c),
                                 make_uint4(bf2(x[8 * c], x[8 * c + 1]), bf2(x[8 * c + 2], x[8 * c + 3]),
                                            bf2(x[8 * c + 4], x[8 * c + 5]), bf2(x[8 * c + 6], x[8 * c + 7])));
        }
        if (!layer(0, sb + MT_SA1, sb + MT_SW1, 1, 0, 0, MLP_H)) { failed = true; break; }
#pragma unroll 1
        for (int c0 = 0; c0 < MLP_H; c0 += 32) {
            float v[32];
            tc::tmem_ld32(tmem + lanes + (uint32_t)c0, v);
            mt_hidden(v, b1, c0, sb + MT_SA2, t, live && h1 ? h1 + row * MLP_H : nullptr);
        }
        if (!layer(128, sb + MT_SA2, sb + MT_SW2, 2, 16384, 16384, MLP_H)) { failed = true; break; }
        // layer-2 activations replace layer-1's in the A tile (the MMA that read them is complete)
#pragma unroll 1
        for (int c0 = 0; c0 < MLP_H; c0 += 32) {
            float v[32];
            tc::tmem_ld32(tmem + lanes + (uint32_t)(128 + c0), v);
            mt_hidden(v, b2, c0, sb + MT_SA2, t, live && h2 ? h2 + row * MLP_H : nullptr);
        }
        if (!layer(0, sb + MT_SA2, sb + MT_SW3, 2, 16384, 2048, MLP_OUT)) { failed = true; break; }
        float v0[8], v1[8];
        tc::tmem_ld8(tmem + lanes, v0);
        tc::tmem_ld8(tmem + lanes + 8u, v1);
        if (live) {
            float4 *o = reinterpret_cast<float4 *>(out + row * MLP_OUT);
            o[0] = make_float4(v0[0] + b3[0], v0[1] + b3[1], v0[2] + b3[2], v0[3] + b3[3]);
            o[1] = make_float4(v0[4] + b3[4], v0[5] + b3[5], v0[6] + b3[6], v0[7] + b3[7]);
            o[2] = make_float4(v1[0] + b3[8], v1[1] + b3[9], v1[2] + b3[10], v1[3] + b3[11]);
            o[3] = make_float4(v1[4] + b3[12], v1[5] + b3[13], v1[6] + b3[14], v1[7] + b3[15]);
        }
        // the next tile overwrites the A tiles and layer 1's accumulators
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
    }
    if (failed && t == 0 && err) atomicExch(err, 1);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(MT_TMEM_COLS)
                     : "memory");
    }
}

// FP32 weights of the blob -> the BF16 image k_mlp_tc reads (W1 zero-padded to 64 inputs)
__global__ void k_mlp_pack(const float *__restrict__ p, __nv_bfloat16 *__restrict__ wb)
{
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < MT_WB_ELEMS; e += gridDim.x * blockDim.x) {
        float v;
        if (e < MT_W1_ELEMS) {
            const int r = e / MT_K1, k = e % MT_K1;
            v = k < MLP_IN ? p[MLP_W1 + r * MLP_IN + k] : 0.f;
        } else if (e < MT_W1_ELEMS + MT_W2_ELEMS) {
            v = p[MLP_W2 + (e - MT_W1_ELEMS)];
        } else {
            v = p[MLP_W3 + (e - MT_W1_ELEMS - MT_W2_ELEMS)];
        }
        wb[e] = __float2bfloat16_rn(v);
    }
}

struct Dev {
    std::vector<void *> ptrs;
    bool ok = true;
    ~Dev() { for (void *q : ptrs) cudaFree(q); }
    template <typename T> T *alloc(size_t n)
    {
        void *q = nullptr;
        if (cudaMalloc(&q, sizeof(T) * std::max<size_t>(n, 1)) != cudaSuccess) {
            ok = false;
            return nullptr;
        }
        ptrs.push_back(q);
        return (T *)q;
    }
};

struct Scratch {
    float *h1, *h2, *out;
};

// forward over M normalised rows; activations kept for the backward
void forward(cudaStream_t st, const float *p, const float *Xn, int64_t M, const Scratch &s)
{
    mm(st, (int)M, MLP_H, MLP_IN, Xn, p + MLP_W1, s.h1, p + MLP_B1, 1);
    mm(st, (int)M, MLP_H, MLP_H, s.h1, p + MLP_W2, s.h2, p + MLP_B2, 1);
    mm(st, (int)M, MLP_OUT, MLP_H, s.h2, p + MLP_W3, s.out, p + MLP_B3, 0);
}

// CTAs of the backward over M rows and their tiles' rows: every SM one tile
// of up to 64 rows, then further tiles
int bwd_tile_rows(int64_t M) { return (int)std::min<int64_t>(BW_ROWS, ((M + 151) / 152 + 7) / 8 * 8); }
int bwd_blocks(int64_t M)
{
    const int64_t r = bwd_tile_rows(M);
    return (int)std::min<int64_t>(152, (M + r - 1) / r);
}

// A kernel's limit of dynamic shared memory, which belongs to the current
// device: raised by every call that launches it (a host call of about a
// microsecond), so that each device of a process has it and every call that
// cannot raise it says so.
template <typename Kernel> cudaError_t allow_smem(Kernel *k, int bytes)
{
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) cudaGetLastError();   // (reported by the call, not left pending)
    return e;
}

// the gradient's partial sums (bwd_blocks(M) x MLP_NPAR) and the loss (after
// allow_smem)
void backward(cudaStream_t st, const float *p, const int32_t *idx, const float *X, const float *T, int64_t M,
              const Scratch &s, float *part, double *loss)
{
    k_mlp_bwd<<<bwd_blocks(M), BW_THREADS, BW_SMEM, st>>>(M, bwd_tile_rows(M), idx, X, T, p, s.out, s.h1, s.h2, part, loss);
}

thread_local std::string t_err;

int mfail(const std::string &m)
{
    t_err = m;
    return SDCA_E_CUDA;
}

#define MK(call)                                                                       \
    do {                                                                               \
        cudaError_t e_ = (call);                                                       \
        if (e_ != cudaSuccess) return mfail(std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)

int check_blob(const float *params)
{
    if (!params) return SDCA_E_ARG;
    // version 1 (per-pair start) and 2 (the dual form's per-sequence start) share the network
    if (params[MLP_VERSION] != (float)MLP_BLOB_VERSION && params[MLP_VERSION] != (float)MLP_BLOB_VERSION_DUAL)
        return SDCA_E_ARG;
    return SDCA_OK;
}

} // namespace

void mlp_pack(const float *p_dev, void *wb, cudaStream_t st)
{
    k_mlp_pack<<<(MT_WB_ELEMS + 255) / 256, 256, 0, st>>>(p_dev, static_cast<__nv_bfloat16 *>(wb));
}

namespace {

// the fused forward over M rows (after allow_smem): outputs, and the FP32
// activations when h1, h2 are given
void mt_forward(const float *p_dev, const void *wb, const int32_t *idx, const float *X, int64_t M, float *out,
                float *h1, float *h2, int *err, cudaStream_t st)
{
    if (M <= 0) return;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 152;
    const int64_t tiles = (M + 127) / 128;
    const unsigned grid = (unsigned)std::min<int64_t>(tiles, 2 * (int64_t)sms);
    k_mlp_tc<<<grid, MT_THREADS, MT_SMEM, st>>>(M, idx, X, p_dev, static_cast<const __nv_bfloat16 *>(wb), out, h1, h2,
                                                  err);
}

} // namespace

cudaError_t mlp_infer(const float *p_dev, const void *wb, const float *X, int64_t M, float *out, int *err,
                      cudaStream_t st)
{
    const cudaError_t e = allow_smem(k_mlp_tc, MT_SMEM);
    if (e == cudaSuccess) mt_forward(p_dev, wb, nullptr, X, M, out, nullptr, nullptr, err, st);
    return e;
}

} // namespace sdca

using namespace sdca;

extern "C" {

int sdca_mlp_blob_size(void) { return MLP_BLOB_SIZE; }

int sdca_mlp_grad(const float *params, const float *X, const float *T, int64_t M, double *loss, float *grad)
{
    if (check_blob(params) || !X || !T || M < 1 || !loss || !grad) return SDCA_E_ARG;
    cudaStream_t st = 0;
    Dev d;
    float *p = d.alloc<float>(MLP_BLOB_SIZE), *x = d.alloc<float>(M * MLP_IN), *xn = d.alloc<float>(M * MLP_IN);
    float *t = d.alloc<float>(M * MLP_OUT), *h1 = d.alloc<float>(M * MLP_H), *h2 = d.alloc<float>(M * MLP_H);
    float *out = d.alloc<float>(M * MLP_OUT), *g = d.alloc<float>(MLP_BLOB_SIZE);
    float *part = d.alloc<float>((size_t)bwd_blocks(M) * MLP_NPAR);
    double *l = d.alloc<double>(1);
    if (!d.ok) return mfail("device allocation failed"), SDCA_E_NOMEM;
    MK(allow_smem(k_mlp_bwd, BW_SMEM));
    MK(cudaMemcpy(p, params, sizeof(float) * MLP_BLOB_SIZE, cudaMemcpyHostToDevice));
    MK(cudaMemcpy(x, X, sizeof(float) * M * MLP_IN, cudaMemcpyHostToDevice));
    MK(cudaMemcpy(t, T, sizeof(float) * M * MLP_OUT, cudaMemcpyHostToDevice));
    MK(cudaMemset(g, 0, sizeof(float) * MLP_BLOB_SIZE));
    MK(cudaMemset(l, 0, sizeof(double)));
    k_normalise<<<(unsigned)((M * MLP_IN + 255) / 256), 256, 0, st>>>(M, x, p, xn);
    const Scratch s{h1, h2, out};
    forward(st, p, xn, M, s);
    backward(st, p, nullptr, x, t, M, s, part, l);
    k_mlp_reduce<<<(MLP_NPAR + RD_PAR - 1) / RD_PAR, RD_PAR * RD_SEG, 0, st>>>(
        bwd_blocks(M), part, g, nullptr, nullptr, nullptr, nullptr, 0.f, 0.f, 0.f, 0.f, 1.f, 1.f);
    MK(cudaGetLastError());
    MK(cudaMemcpy(grad, g, sizeof(float) * MLP_BLOB_SIZE, cudaMemcpyDeviceToHost));
    MK(cudaMemcpy(loss, l, sizeof(double), cudaMemcpyDeviceToHost));
    return SDCA_OK;
}

int sdca_mlp_predict(const float *params, const float *X, int64_t M, float *out)
{
    if (check_blob(params) || !X || M < 1 || !out) return SDCA_E_ARG;
    Dev d;
    float *p = d.alloc<float>(MLP_BLOB_SIZE), *x = d.alloc<float>(M * MLP_IN), *o = d.alloc<float>(M * MLP_OUT);
    __nv_bfloat16 *wb = d.alloc<__nv_bfloat16>(MT_WB_ELEMS);
    int *err = d.alloc<int>(1);
    if (!d.ok) return mfail("device allocation failed"), SDCA_E_NOMEM;
    MK(cudaMemcpy(p, params, sizeof(float) * MLP_BLOB_SIZE, cudaMemcpyHostToDevice));
    MK(cudaMemcpy(x, X, sizeof(float) * M * MLP_IN, cudaMemcpyHostToDevice));
    MK(cudaMemset(err, 0, sizeof(int)));
    mlp_pack(p, wb, 0);
    MK(mlp_infer(p, wb, x, M, o, err, 0));
    MK(cudaGetLastError());
    int e = 0;
    MK(cudaMemcpy(&e, err, sizeof(int), cudaMemcpyDeviceToHost));
    if (e) return mfail("tensor-core forward: a pipeline wait gave up");
    MK(cudaMemcpy(out, o, sizeof(float) * M * MLP_OUT, cudaMemcpyDeviceToHost));
    return SDCA_OK;
}

int sdca_mlp_train(float *params, const float *X, const float *T, int64_t M, int epochs, int batch, float lr,
                   uint64_t seed, double *losses)
{
    if (check_blob(params) || !X || !T || M < 1 || epochs < 1 || batch < 1 || !(lr > 0.f)) return SDCA_E_ARG;
    cudaStream_t st = 0;
    const int64_t Bm = std::min<int64_t>(batch, M);
    Dev d;
    float *p = d.alloc<float>(MLP_BLOB_SIZE), *x = d.alloc<float>(M * MLP_IN), *t = d.alloc<float>(M * MLP_OUT);
    float *h1 = d.alloc<float>(Bm * MLP_H), *h2 = d.alloc<float>(Bm * MLP_H), *out = d.alloc<float>(Bm * MLP_OUT);
    float *part = d.alloc<float>((size_t)bwd_blocks(Bm) * MLP_NPAR);
    float *m1 = d.alloc<float>(MLP_BLOB_SIZE), *m2 = d.alloc<float>(MLP_BLOB_SIZE);
    int32_t *perm_d = d.alloc<int32_t>(M);
    double *l = d.alloc<double>(1);
    __nv_bfloat16 *wb = d.alloc<__nv_bfloat16>(MT_WB_ELEMS);
    int *err = d.alloc<int>(1);
    if (!d.ok) return mfail("device allocation failed"), SDCA_E_NOMEM;
    MK(allow_smem(k_mlp_tc, MT_SMEM));
    MK(allow_smem(k_mlp_bwd, BW_SMEM));
    MK(cudaMemset(err, 0, sizeof(int)));
    MK(cudaMemcpy(p, params, sizeof(float) * MLP_BLOB_SIZE, cudaMemcpyHostToDevice));
    MK(cudaMemcpy(x, X, sizeof(float) * M * MLP_IN, cudaMemcpyHostToDevice));
    MK(cudaMemcpy(t, T, sizeof(float) * M * MLP_OUT, cudaMemcpyHostToDevice));
    MK(cudaMemset(m1, 0, sizeof(float) * MLP_BLOB_SIZE));
    MK(cudaMemset(m2, 0, sizeof(float) * MLP_BLOB_SIZE));
    mlp_pack(p, wb, st);   // (the weights' entries follow every step; the padding stays zero)
    std::mt19937_64 rng(seed);
    std::vector<int32_t> perm((size_t)M);
    const float b1 = 0.9f, b2 = 0.999f;
    float c1 = 1.f, c2 = 1.f;
    const Scratch s{h1, h2, out};
    for (int ep = 0; ep < epochs; ++ep) {
        for (int64_t i = 0; i < M; ++i) perm[i] = (int32_t)i;
        std::shuffle(perm.begin(), perm.end(), rng);
        MK(cudaMemcpy(perm_d, perm.data(), sizeof(int32_t) * M, cudaMemcpyHostToDevice));
        MK(cudaMemset(l, 0, sizeof(double)));
        int64_t nb = 0;
        for (int64_t b0 = 0; b0 + Bm <= M; b0 += Bm, ++nb) {
            // forward on the tensor cores (BF16 image of the current weights),
            // backward in FP32 from its saved activations, Adam
            mt_forward(p, wb, perm_d + b0, x, Bm, out, h1, h2, err, st);
            backward(st, p, perm_d + b0, x, t, Bm, s, part, l);
            c1 *= b1;
            c2 *= b2;
            k_mlp_reduce<<<(MLP_NPAR + RD_PAR - 1) / RD_PAR, RD_PAR * RD_SEG, 0, st>>>(
                bwd_blocks(Bm), part, nullptr, p, m1, m2, wb, lr, b1, b2, 1e-8f, 1.f - c1, 1.f - c2);
        }
        MK(cudaGetLastError());
        int e = 0;
        MK(cudaMemcpy(&e, err, sizeof(int), cudaMemcpyDeviceToHost));
        if (e) return mfail("tensor-core forward: a pipeline wait gave up");
        double lsum = 0.0;
        MK(cudaMemcpy(&lsum, l, sizeof(double), cudaMemcpyDeviceToHost));
        if (losses) losses[ep] = nb ? lsum / (double)nb : 0.0;
    }
    MK(cudaMemcpy(params, p, sizeof(float) * MLP_BLOB_SIZE, cudaMemcpyDeviceToHost));
    return SDCA_OK;
}

const char *sdca_mlp_last_error(void) { return t_err.c_str(); }

} // extern "C"
