// kernels_gather.cu -- the plain contraction form: FP32 gather (forward) and
// masked accumulation (backward) on CUDA cores.
//
// forward   u_b[i][a] = sum_n v_b[n][X_in][a]                 (X one-hot . v_J)
// backward  g_b[n][s][a] = sum_{i: X_in = s} R_b[i][a] + 2 lambda_J x_b[n][s][a]
//
// These are SuperDCA's block gather (SuperDCA/include/plmDCA_objective.hpp:86-121,
// Coupling_matrix_view.hpp:59-86) and gradient scatter (plmDCA_objective.hpp:
// 153-190, Coupling_matrix_view.hpp:88-111) for a batch of target loci that
// share one alignment read.  Both are bound by shared-memory / FP32 issue
// (one 16-byte shared load or 16 FMAs per (sequence, locus, slot)).
#include <algorithm>

#include <cuda_pipeline_primitives.h>

#include "engine.h"
#include "kernels_common.cuh"

namespace sdca {

namespace {

constexpr int FWD_THREADS = 256;  // sequences per CTA
constexpr int FWD_G = 8;          // slots per CTA
constexpr int FWD_SUB = 32;       // loci per shared-memory sub-tile

__global__ void __launch_bounds__(FWD_THREADS)
k_fwd_gather(const uint8_t *__restrict__ X, int64_t Lx, int N, int L, int64_t LC,
             const int32_t *__restrict__ list, int nlist, const float *__restrict__ vecs,
             int64_t Dp, float4 *__restrict__ partial, int Bmax, int64_t Nx)
{
    __shared__ float4 sJ[FWD_G][FWD_SUB][Q];
    const int i = blockIdx.x * FWD_THREADS + threadIdx.x;
    const int c = blockIdx.z;
    const int64_t n_begin = (int64_t)c * LC;
    const int64_t n_end = min((int64_t)L, n_begin + LC);
    int slot[FWD_G];
#pragma unroll
    for (int g = 0; g < FWD_G; ++g) {
        const int k = blockIdx.y * FWD_G + g;
        slot[g] = k < nlist ? list[k] : -1;
    }
    float4 acc[FWD_G];
#pragma unroll
    for (int g = 0; g < FWD_G; ++g) acc[g] = make_float4(0.f, 0.f, 0.f, 0.f);

    for (int64_t n0 = n_begin; n0 < n_end; n0 += FWD_SUB) {
        for (int k = threadIdx.x; k < FWD_G * FWD_SUB * Q; k += FWD_THREADS) {
            const int g = k / (FWD_SUB * Q), rem = k % (FWD_SUB * Q);
            const int nl = rem / Q, s = rem % Q;
            const int64_t n = n0 + nl;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (slot[g] >= 0 && n < n_end)
                v = reinterpret_cast<const float4 *>(vecs + (int64_t)slot[g] * Dp)[n * Q + s];
            sJ[g][nl][s] = v;
        }
        __syncthreads();
        if (i < N) {
            const uint4 *xp = reinterpret_cast<const uint4 *>(X + (int64_t)i * Lx + n0);
            const uint4 w0 = xp[0], w1 = xp[1];
            const uint32_t words[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
            for (int wd = 0; wd < 8; ++wd) {
#pragma unroll
                for (int bt = 0; bt < 4; ++bt) {
                    const int nl = wd * 4 + bt;
                    const int s = (words[wd] >> (8 * bt)) & 0x3;
#pragma unroll
                    for (int g = 0; g < FWD_G; ++g) {
                        const float4 j = sJ[g][nl][s];
                        acc[g].x += j.x;
                        acc[g].y += j.y;
                        acc[g].z += j.z;
                        acc[g].w += j.w;
                    }
                }
            }
        }
        __syncthreads();
    }
    if (i < N) {
#pragma unroll
        for (int g = 0; g < FWD_G; ++g)
            if (slot[g] >= 0) partial[((int64_t)c * Bmax + slot[g]) * Nx + i] = acc[g];
    }
}

// Logits at a stored point, for the start of a locus and for the objective a
// converged locus reports.  The sequences of an alignment share most of their
// states, so rounding errors of long FP32 locus sums are correlated across
// sequences and add up over the N terms of the objective; here FP32 sums run
// over 64-locus stretches only and the stretches accumulate in FP64.
constexpr int EX_G = 4;

__global__ void __launch_bounds__(FWD_THREADS)
k_fwd_gather_exact(const uint8_t *__restrict__ X, int64_t Lx, int N, int L, int64_t LC,
                   const int32_t *__restrict__ list, int nlist, const float *__restrict__ vecs,
                   int64_t Dp, double4 *__restrict__ partial, int Bmax, int64_t Nx)
{
    __shared__ float4 sJ[EX_G][FWD_SUB][Q];
    const int i = blockIdx.x * FWD_THREADS + threadIdx.x;
    const int c = blockIdx.z;
    const int64_t n_begin = (int64_t)c * LC;
    const int64_t n_end = min((int64_t)L, n_begin + LC);
    int slot[EX_G];
#pragma unroll
    for (int g = 0; g < EX_G; ++g) {
        const int k = blockIdx.y * EX_G + g;
        slot[g] = k < nlist ? list[k] : -1;
    }
    float4 acc[EX_G];
    double a64[EX_G][4];
#pragma unroll
    for (int g = 0; g < EX_G; ++g) {
        acc[g] = make_float4(0.f, 0.f, 0.f, 0.f);
        a64[g][0] = a64[g][1] = a64[g][2] = a64[g][3] = 0.0;
    }
    int sub = 0;
    for (int64_t n0 = n_begin; n0 < n_end; n0 += FWD_SUB, ++sub) {
        for (int k = threadIdx.x; k < EX_G * FWD_SUB * Q; k += FWD_THREADS) {
            const int g = k / (FWD_SUB * Q), rem = k % (FWD_SUB * Q);
            const int nl = rem / Q, s = rem % Q;
            const int64_t n = n0 + nl;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (slot[g] >= 0 && n < n_end)
                v = reinterpret_cast<const float4 *>(vecs + (int64_t)slot[g] * Dp)[n * Q + s];
            sJ[g][nl][s] = v;
        }
        __syncthreads();
        if (i < N) {
            const uint4 *xp = reinterpret_cast<const uint4 *>(X + (int64_t)i * Lx + n0);
            const uint4 w0 = xp[0], w1 = xp[1];
            const uint32_t words[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
            for (int wd = 0; wd < 8; ++wd) {
#pragma unroll
                for (int bt = 0; bt < 4; ++bt) {
                    const int nl = wd * 4 + bt;
                    const int s = (words[wd] >> (8 * bt)) & 0x3;
#pragma unroll
                    for (int g = 0; g < EX_G; ++g) {
                        const float4 j = sJ[g][nl][s];
                        acc[g].x += j.x;
                        acc[g].y += j.y;
                        acc[g].z += j.z;
                        acc[g].w += j.w;
                    }
                }
            }
            if (sub & 1) {
#pragma unroll
                for (int g = 0; g < EX_G; ++g) {
                    a64[g][0] += acc[g].x; a64[g][1] += acc[g].y;
                    a64[g][2] += acc[g].z; a64[g][3] += acc[g].w;
                    acc[g] = make_float4(0.f, 0.f, 0.f, 0.f);
                }
            }
        }
        __syncthreads();
    }
    if (i < N) {
#pragma unroll
        for (int g = 0; g < EX_G; ++g)
            if (slot[g] >= 0)
                partial[((int64_t)c * Bmax + slot[g]) * Nx + i] =
                    make_double4(a64[g][0] + acc[g].x, a64[g][1] + acc[g].y, a64[g][2] + acc[g].z,
                                 a64[g][3] + acc[g].w);
    }
}

__global__ void k_reduce_partial64(const double4 *__restrict__ partial, int C, int Bmax, int64_t Nx,
                                   int N, const int32_t *__restrict__ list,
                                   const float *__restrict__ vecs, int64_t Dp, int64_t hoff,
                                   double *__restrict__ out_d)
{
    const int b = list[blockIdx.y];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    const float *h = vecs + (int64_t)b * Dp + hoff;
    double s0 = h[0], s1 = h[1], s2 = h[2], s3 = h[3];
    for (int c = 0; c < C; ++c) {
        const double4 p = partial[((int64_t)c * Bmax + b) * Nx + i];
        s0 += p.x; s1 += p.y; s2 += p.z; s3 += p.w;
    }
    const int64_t o = (int64_t)b * Nx + i;
    out_d[o * 4 + 0] = s0; out_d[o * 4 + 1] = s1;
    out_d[o * 4 + 2] = s2; out_d[o * 4 + 3] = s3;
}

// Sums the partial slices into u (float) or logits (double).  With R given,
// also reduces sum_i R_i . u_i per slot into acc[ACC_DG0]: the slope at
// step 0 of the line the next search walks, from the same numbers the
// trial steps will use.
__global__ void k_reduce_partial(const float4 *__restrict__ partial, int C, int Bmax, int64_t Nx,
                                 int N, const int32_t *__restrict__ list,
                                 const float *__restrict__ vecs, int64_t Dp, int64_t hoff,
                                 int add_h, float4 *__restrict__ out_f, double *__restrict__ out_d,
                                 const float4 *__restrict__ R, double *__restrict__ acc)
{
    const int b = list[blockIdx.y];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (R) {
        // every thread of the block takes part in the reduction
        double ru = 0.0;
        if (i < N) {
            double t[4] = {0, 0, 0, 0};
            if (add_h) {
                const float *h = vecs + (int64_t)b * Dp + hoff;
                t[0] = h[0]; t[1] = h[1]; t[2] = h[2]; t[3] = h[3];
            }
            for (int c = 0; c < C; ++c) {
                const float4 p = partial[((int64_t)c * Bmax + b) * Nx + i];
                t[0] += p.x; t[1] += p.y; t[2] += p.z; t[3] += p.w;
            }
            const float4 uf = make_float4((float)t[0], (float)t[1], (float)t[2], (float)t[3]);
            out_f[(int64_t)b * Nx + i] = uf;
            const float4 r = R[(int64_t)b * Nx + i];
            ru = (double)r.x * uf.x + (double)r.y * uf.y + (double)r.z * uf.z + (double)r.w * uf.w;
        }
        double v[1] = {ru};
        const int idx[1] = {ACC_DG0};
        block_sum_atomic<1>(v, acc + (int64_t)b * NACC, idx);
        return;
    }
    if (i >= N) return;
    double s0 = 0, s1 = 0, s2 = 0, s3 = 0;
    if (add_h) {
        const float *h = vecs + (int64_t)b * Dp + hoff;
        s0 = h[0]; s1 = h[1]; s2 = h[2]; s3 = h[3];
    }
    for (int c = 0; c < C; ++c) {
        const float4 p = partial[((int64_t)c * Bmax + b) * Nx + i];
        s0 += p.x; s1 += p.y; s2 += p.z; s3 += p.w;
    }
    const int64_t o = (int64_t)b * Nx + i;
    if (out_f) out_f[o] = make_float4((float)s0, (float)s1, (float)s2, (float)s3);
    if (out_d) {
        out_d[o * 4 + 0] = s0; out_d[o * 4 + 1] = s1;
        out_d[o * 4 + 2] = s2; out_d[o * 4 + 3] = s3;
    }
}

constexpr int BWD_THREADS = 128;  // loci per CTA (one slot)
constexpr int BG_THREADS = 64;    // loci per CTA (k_bwd_gather)
constexpr int BWD_G = 2;          // slots per CTA (k_bwd_gather)
constexpr int BWD_SUB = 64;       // sequences per shared-memory sub-tile

// a[s][.] += r for the state s of one sequence, as 16 multiply-adds by 0 or 1
// in pairs: one FFMA2 does two of them in one issue slot
__device__ __forceinline__ void add_by_state(int s, float4 r, float2 (&a)[QQ / 2])
{
    const float2 lo = make_float2(r.x, r.y), hi = make_float2(r.z, r.w);
#pragma unroll
    for (int t = 0; t < Q; ++t) {
        const float m = s == t ? 1.f : 0.f;
        a[2 * t] = __ffma2_rn(make_float2(m, m), lo, a[2 * t]);
        a[2 * t + 1] = __ffma2_rn(make_float2(m, m), hi, a[2 * t + 1]);
    }
}

__device__ __forceinline__ void unpack(const float2 (&a)[QQ / 2], float (&c)[QQ])
{
#pragma unroll
    for (int k = 0; k < QQ / 2; ++k) {
        c[2 * k] = a[k].x;
        c[2 * k + 1] = a[k].y;
    }
}

// Bound by FP32 multiply-adds: 16 per (sequence, locus, slot), 0.11 ms for 64
// slots of 1000 x 4001 at two clocks per pair and warp.  0.18 ms: that pipe
// is busy 60 % of the time.  Single multiply-adds, four slots a thread and
// blocks of 128 loci (110 registers, three or four blocks per SM) took 0.30,
// the same in pairs 0.21; two slots a thread leave room for twice the warps,
// and the next sub-tile's residuals are on their way while one is summed.
__global__ void __launch_bounds__(BG_THREADS, 14)
k_bwd_gather(const uint8_t *__restrict__ XT, int64_t Nx, int N, int L,
             const SlotDev *__restrict__ sd, const int32_t *__restrict__ list, int nlist,
             const float4 *__restrict__ R, const float *__restrict__ wa, float *__restrict__ gpool,
             void *__restrict__ Ypool, const void *__restrict__ Spool, int hist_bf16, int m,
             int64_t Dp, double lambda_J, double *__restrict__ acc)
{
    __shared__ float4 sR[2][BWD_G][BWD_SUB];
    const int n = blockIdx.x * BG_THREADS + threadIdx.x;
    int slot[BWD_G];
#pragma unroll
    for (int g = 0; g < BWD_G; ++g) {
        const int k = blockIdx.y * BWD_G + g;
        slot[g] = k < nlist ? list[k] : -1;
    }
    float2 a2[BWD_G][QQ / 2];
#pragma unroll
    for (int g = 0; g < BWD_G; ++g)
#pragma unroll
        for (int k = 0; k < QQ / 2; ++k) a2[g][k] = make_float2(0.f, 0.f);

    static_assert(BG_THREADS == BWD_SUB, "a thread stages one sequence per slot");
    auto stage = [&](int i0, int buf) {
        const int i = i0 + threadIdx.x;
#pragma unroll
        for (int g = 0; g < BWD_G; ++g) {
            const bool ok = slot[g] >= 0 && i < N;   // (else zeros)
            __pipeline_memcpy_async(&sR[buf][g][threadIdx.x], ok ? R + (int64_t)slot[g] * Nx + i : R, 16, ok ? 0 : 16);
        }
        __pipeline_commit();
    };
    stage(0, 0);
    for (int i0 = 0, buf = 0; i0 < N; i0 += BWD_SUB, buf ^= 1) {
        if (i0 + BWD_SUB < N) stage(i0 + BWD_SUB, buf ^ 1);
        else __pipeline_commit();
        uint4 xw[BWD_SUB / 16];
        if (n < L)
#pragma unroll
            for (int q4 = 0; q4 < BWD_SUB / 16; ++q4) xw[q4] = reinterpret_cast<const uint4 *>(XT + (int64_t)n * Nx + i0)[q4];
        __pipeline_wait_prior(1);
        __syncthreads();
        if (n < L) {
#pragma unroll
            for (int q4 = 0; q4 < BWD_SUB / 16; ++q4) {
                const uint32_t words[4] = {xw[q4].x, xw[q4].y, xw[q4].z, xw[q4].w};
#pragma unroll
                for (int wd = 0; wd < 4; ++wd)
#pragma unroll
                    for (int bt = 0; bt < 4; ++bt) {
                        const int s = (words[wd] >> (8 * bt)) & 0x3;
#pragma unroll
                        for (int g = 0; g < BWD_G; ++g) add_by_state(s, sR[buf][g][q4 * 16 + wd * 4 + bt], a2[g]);
                    }
            }
        }
        __syncthreads();
    }

    // epilogue: + 2 lambda_J x, zero the J_rr block, push y, reductions
    const float l2 = (float)(2.0 * lambda_J);
#pragma unroll
    for (int g = 0; g < BWD_G; ++g) {
        if (slot[g] < 0) continue;  // uniform across the block
        const int b = slot[g];
        GradRed red;
        float a[QQ];
        unpack(a2[g], a);
        if (n < L) grad_locus(sd[b], b, n, a, wa, gpool, Ypool, Spool, hist_bf16, m, Dp, l2, red);
        double v[5] = {red.g2, red.x2, red.sy, red.yy, red.ss};
        const int idx[5] = {ACC_G2, ACC_X2J, ACC_SY, ACC_YY, ACC_SS};
        block_sum_atomic<5>(v, acc + (int64_t)b * NACC, idx);
        const float wm = warp_max(red.gmax);
        if ((threadIdx.x & 31) == 0 && wm > 0.f) atomic_max_nonneg(acc + (int64_t)b * NACC + ACC_GMAX, (double)wm);
    }
}

// The tensor-core backward leaves X^T R (scaled back) in the new-gradient
// buffer; this adds the L2 part and does the same bookkeeping.
__global__ void __launch_bounds__(BWD_THREADS)
k_grad_finalize(int L, const SlotDev *__restrict__ sd, const int32_t *__restrict__ list,
                const float *__restrict__ wa, float *__restrict__ gpool, void *__restrict__ Ypool,
                const void *__restrict__ Spool, int hist_bf16, int m, int64_t Dp, double lambda_J,
                double *__restrict__ acc)
{
    const int b = list[blockIdx.y];
    const SlotDev &S = sd[b];
    const float l2 = (float)(2.0 * lambda_J);
    GradRed red;
    for (int64_t n = (int64_t)blockIdx.x * BWD_THREADS + threadIdx.x; n < L; n += (int64_t)gridDim.x * BWD_THREADS) {
        const float4 *gr = reinterpret_cast<const float4 *>(gpool + (int64_t)(2 * b + 1 - S.gcur) * Dp + n * QQ);
        float c[16];
#pragma unroll
        for (int k4 = 0; k4 < 4; ++k4) {
            const float4 v = gr[k4];
            c[4 * k4] = v.x; c[4 * k4 + 1] = v.y; c[4 * k4 + 2] = v.z; c[4 * k4 + 3] = v.w;
        }
        grad_locus(S, b, n, c, wa, gpool, Ypool, Spool, hist_bf16, m, Dp, l2, red);
    }
    double v[5] = {red.g2, red.x2, red.sy, red.yy, red.ss};
    const int idx[5] = {ACC_G2, ACC_X2J, ACC_SY, ACC_YY, ACC_SS};
    block_sum_atomic<5>(v, acc + (int64_t)b * NACC, idx);
    const float wm = warp_max(red.gmax);
    if ((threadIdx.x & 31) == 0 && wm > 0.f) atomic_max_nonneg(acc + (int64_t)b * NACC + ACC_GMAX, (double)wm);
}

// ---- one evaluation (sdca_eval): the same sums as the batch kernels above and
// k_trial, for one point.  The batch kernels' groups of four slots did four
// times the work for one, and the point and the gradient were converted on
// the host between the reference's layout and this one, in 64-bit steps over
// 16 L values each way: 4.7 ms at 3000 x 94,000, where the passes here take
// 0.44 ms (0.22 logits, 0.19 gradient) and the call 0.8.

// the point from the reference's layout (double) into the engine's (FP32,
// J_rr = 0, padding 0); the sums start at zero
__global__ void __launch_bounds__(256)
k_eval_point(const double *__restrict__ x, int64_t L, int64_t Dp, int64_t r, float *__restrict__ wa,
             double *__restrict__ acc)
{
    if (blockIdx.x == 0 && threadIdx.x < NACC) acc[threadIdx.x] = 0.0;
    const int64_t t = (int64_t)blockIdx.x * 256 + threadIdx.x;   // a row of four: locus n, state s
    if (4 * t >= Dp) return;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (t < Q * L) {
        const int64_t n = t / Q, s = t % Q, b = n / 16, e = b < L / 16 ? 16 : L % 16;
        if (n != r) {
            const double *p = x + b * 16 * QQ + (s * e + n % 16) * Q;
            v = make_float4((float)p[0], (float)p[1], (float)p[2], (float)p[3]);
        }
    } else if (t == Q * L) {
        const double *p = x + QQ * L;
        v = make_float4((float)p[0], (float)p[1], (float)p[2], (float)p[3]);
    }
    reinterpret_cast<float4 *>(wa)[t] = v;
}

// Partial logits of k_fwd_gather_exact (FP32 over the same 64-locus
// stretches, FP64 across), one slot.  A block takes 256 sequences and one of
// the `parts` shares of a locus chunk's stretches, so that some eight blocks
// per SM cover the latency of the shared-memory row each (sequence, locus)
// reads; those reads bound it.
constexpr int EF_STR = 64;

__global__ void __launch_bounds__(FWD_THREADS)
k_eval_fwd(const uint8_t *__restrict__ X, int64_t Lx, int N, int L, int64_t LC, int parts, const float *__restrict__ wa,
           double *__restrict__ partial, int64_t Nx)
{
    __shared__ float4 sJ[EF_STR][Q];
    const int t = threadIdx.x, i = blockIdx.x * FWD_THREADS + t, c = blockIdx.y / parts, part = blockIdx.y % parts;
    const int64_t n_begin = (int64_t)c * LC, n_end = min((int64_t)L, n_begin + LC);
    const int64_t str = (n_end - n_begin + EF_STR - 1) / EF_STR;
    const int64_t k0 = str * part / parts, k1 = str * (part + 1) / parts;
    double a0 = 0, a1 = 0, a2 = 0, a3 = 0;
    for (int64_t k = k0; k < k1; ++k) {
        const int64_t n0 = n_begin + k * EF_STR, e = n0 * Q + t;   // EF_STR x Q rows, one per thread
        const float4 row = e < n_end * Q ? reinterpret_cast<const float4 *>(wa)[e] : make_float4(0.f, 0.f, 0.f, 0.f);
        uint4 w[4];
        if (i < N) {
            const uint4 *xp = reinterpret_cast<const uint4 *>(X + (int64_t)i * Lx + n0);
            w[0] = xp[0];
            w[1] = xp[1];
            // (a chunk may end half way through a stretch, at the row's end)
            const bool more = n0 + 32 < n_end;
            w[2] = more ? xp[2] : make_uint4(0u, 0u, 0u, 0u);
            w[3] = more ? xp[3] : make_uint4(0u, 0u, 0u, 0u);
        }
        __syncthreads();
        sJ[t / Q][t % Q] = row;
        __syncthreads();
        if (i < N) {
            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint32_t words[4] = {w[q].x, w[q].y, w[q].z, w[q].w};
#pragma unroll
                for (int wd = 0; wd < 4; ++wd)
#pragma unroll
                    for (int bt = 0; bt < 4; ++bt) {
                        const float4 j = sJ[q * 16 + wd * 4 + bt][(words[wd] >> (8 * bt)) & 0x3];
                        acc.x += j.x;
                        acc.y += j.y;
                        acc.z += j.z;
                        acc.w += j.w;
                    }
            }
            a0 += acc.x;
            a1 += acc.y;
            a2 += acc.z;
            a3 += acc.w;
        }
    }
    if (i < N) {
        double2 *o = reinterpret_cast<double2 *>(partial + ((int64_t)blockIdx.y * Nx + i) * Q);
        o[0] = make_double2(a0, a1);
        o[1] = make_double2(a2, a3);
    }
}

// logits from the chunks' partial sums, objective and node beliefs (k_trial
// at step 0); eight threads share a sequence's chunks
constexpr int EB_SHARE = 8;

__global__ void __launch_bounds__(FWD_THREADS)
k_eval_beliefs(const double *__restrict__ partial, int C, int64_t Nx, int N, const float *__restrict__ h,
               const uint8_t *__restrict__ rstate, const double *__restrict__ w, float4 *__restrict__ R,
               double *__restrict__ acc)
{
    const int i = (blockIdx.x * FWD_THREADS + threadIdx.x) / EB_SHARE, k = threadIdx.x % EB_SHARE;
    double f = 0, rs[4] = {0, 0, 0, 0}, l[4] = {0, 0, 0, 0};
    if (i < N)
#pragma unroll 4
        for (int c = k; c < C; c += EB_SHARE) {
            const double2 *p = reinterpret_cast<const double2 *>(partial + ((int64_t)c * Nx + i) * Q);
            const double2 u = p[0], v = p[1];
            l[0] += u.x;
            l[1] += u.y;
            l[2] += v.x;
            l[3] += v.y;
        }
#pragma unroll
    for (int o = EB_SHARE / 2; o > 0; o >>= 1)
#pragma unroll
        for (int a = 0; a < 4; ++a) l[a] += __shfl_xor_sync(0xffffffffu, l[a], o);
    if (i < N && k == 0) {
#pragma unroll
        for (int a = 0; a < 4; ++a) l[a] += (double)h[a];
        const double mx = fmax(fmax(l[0], l[1]), fmax(l[2], l[3]));
        double e[4], z = 0;
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            e[a] = exp(l[a] - mx);
            z += e[a];
        }
        const int sr = rstate[i] & 3;
        const double wi = w[i];
        f = wi * (mx + log(z) - (sr == 0 ? l[0] : sr == 1 ? l[1] : sr == 2 ? l[2] : l[3]));
#pragma unroll
        for (int a = 0; a < 4; ++a) rs[a] = wi * (e[a] / z) - (a == sr ? wi : 0.0);
        R[i] = make_float4((float)rs[0], (float)rs[1], (float)rs[2], (float)rs[3]);
    }
    double v[5] = {f, rs[0], rs[1], rs[2], rs[3]};
    const int idx[5] = {ACC_F, ACC_RS0, ACC_RS1, ACC_RS2, ACC_RS3};
    block_sum_atomic<5>(v, acc, idx);
}

// the gradient of k_bwd_gather and k_hpart, one slot, into the reference's
// layout (double, values of FP32), and the L2 sums
__global__ void __launch_bounds__(BWD_THREADS)
k_eval_bwd(const uint8_t *__restrict__ XT, int64_t Nx, int N, int L, int64_t r, const float4 *__restrict__ R,
           const float *__restrict__ wa, double lambda_J, double lambda_h, double *__restrict__ g,
           double *__restrict__ acc)
{
    __shared__ float4 sR[BWD_SUB];
    const int n = blockIdx.x * BWD_THREADS + threadIdx.x;
    float2 a2[QQ / 2];
#pragma unroll
    for (int k = 0; k < QQ / 2; ++k) a2[k] = make_float2(0.f, 0.f);
    for (int i0 = 0; i0 < N; i0 += BWD_SUB) {
        __syncthreads();
        if (threadIdx.x < BWD_SUB) sR[threadIdx.x] = i0 + threadIdx.x < N ? R[i0 + threadIdx.x] : make_float4(0.f, 0.f, 0.f, 0.f);
        uint4 w[BWD_SUB / 16];
        if (n < L)
#pragma unroll
            for (int q4 = 0; q4 < BWD_SUB / 16; ++q4) w[q4] = reinterpret_cast<const uint4 *>(XT + (int64_t)n * Nx + i0)[q4];
        __syncthreads();
        if (n < L) {
#pragma unroll
            for (int q4 = 0; q4 < BWD_SUB / 16; ++q4) {
                const uint32_t words[4] = {w[q4].x, w[q4].y, w[q4].z, w[q4].w};
#pragma unroll
                for (int wd = 0; wd < 4; ++wd)
#pragma unroll
                    for (int bt = 0; bt < 4; ++bt) {
                        const int s = (words[wd] >> (8 * bt)) & 0x3;
                        add_by_state(s, sR[q4 * 16 + wd * 4 + bt], a2);
                    }
            }
        }
    }
    float a[QQ];
    unpack(a2, a);
    const float l2 = (float)(2.0 * lambda_J);
    float x2 = 0.f;
    if (n < L) {
        const int64_t b = n / 16, e = b < L / 16 ? 16 : L % 16;
        const float4 *x4 = reinterpret_cast<const float4 *>(wa + (int64_t)n * QQ);
        const bool zero = n == r;
#pragma unroll
        for (int s = 0; s < Q; ++s) {
            const float4 xv = x4[s];
            x2 += dot4(xv, xv);
            if (g) {
                double *o = g + b * 16 * QQ + (s * e + n % 16) * Q;
                o[0] = zero ? 0.f : a[4 * s + 0] + l2 * xv.x;
                o[1] = zero ? 0.f : a[4 * s + 1] + l2 * xv.y;
                o[2] = zero ? 0.f : a[4 * s + 2] + l2 * xv.z;
                o[3] = zero ? 0.f : a[4 * s + 3] + l2 * xv.w;
            }
        }
    }
    double v[1] = {x2};
    const int idx[1] = {ACC_X2J};
    block_sum_atomic<1>(v, acc, idx);
    if (blockIdx.x == 0 && threadIdx.x < Q) {
        const double x = wa[(int64_t)QQ * L + threadIdx.x];
        if (g) g[(int64_t)QQ * L + threadIdx.x] = (float)(acc[ACC_RS0 + threadIdx.x] + 2.0 * lambda_h * x);
        atomicAdd(acc + ACC_X2H, x * x);
    }
}

} // namespace

void launch_fwd_gather(const Problem &P, const uint8_t *X, const int32_t *list, int n,
                       const float *vecs, float *partial, cudaStream_t st)
{
    if (n <= 0) return;
    dim3 grid((unsigned)((P.N + FWD_THREADS - 1) / FWD_THREADS), (unsigned)((n + FWD_G - 1) / FWD_G),
              (unsigned)P.Cg);
    k_fwd_gather<<<grid, FWD_THREADS, 0, st>>>(X, P.Lx, (int)P.N, (int)P.L, P.LC, list, n, vecs, P.Dp,
                                               reinterpret_cast<float4 *>(partial), P.Bmax, P.Nx);
}

void launch_fwd_exact(const Problem &P, const uint8_t *X, const int32_t *list, int n, const float *vecs,
                      double *partial64, double *lbase, cudaStream_t st)
{
    if (n <= 0) return;
    dim3 grid((unsigned)((P.N + FWD_THREADS - 1) / FWD_THREADS), (unsigned)((n + EX_G - 1) / EX_G),
              (unsigned)P.Cg);
    k_fwd_gather_exact<<<grid, FWD_THREADS, 0, st>>>(X, P.Lx, (int)P.N, (int)P.L, P.LC, list, n, vecs, P.Dp,
                                                     reinterpret_cast<double4 *>(partial64), P.Bmax, P.Nx);
    dim3 g2((unsigned)((P.N + 255) / 256), (unsigned)n);
    k_reduce_partial64<<<g2, 256, 0, st>>>(reinterpret_cast<const double4 *>(partial64), (int)P.Cg, P.Bmax,
                                           P.Nx, (int)P.N, list, vecs, P.Dp, QQ * P.L, lbase);
}

void launch_reduce_partial(const Problem &P, const int32_t *list, int n, const float *partial,
                           const float *vecs, int add_h, float *out_f, double *out_d,
                           cudaStream_t st, int C, const float *R, double *acc)
{
    if (n <= 0) return;
    dim3 grid((unsigned)((P.N + 255) / 256), (unsigned)n);
    k_reduce_partial<<<grid, 256, 0, st>>>(reinterpret_cast<const float4 *>(partial), C > 0 ? C : (int)P.Cg,
                                           P.Bmax, P.Nx, (int)P.N, list, vecs, P.Dp, QQ * P.L, add_h,
                                           reinterpret_cast<float4 *>(out_f), out_d,
                                           reinterpret_cast<const float4 *>(R), acc);
}

// One evaluation at the point xg (reference layout, on the device; room for
// 2 Dp floats, which then hold the partial logits and, when want_g, the
// gradient): acc (NACC) receives the objective's data part, the
// residual sums and the L2 sums.  partial64: room for the Cg chunks' partial
// logits, where xg has none.
void launch_eval(const Problem &P, const uint8_t *X, const uint8_t *XT, int64_t r, double *xg, bool want_g,
                 const uint8_t *rstate, const double *w, float *wa, double *partial64, float *R, double *acc, cudaStream_t st)
{
    k_eval_point<<<(unsigned)((P.Dp / 4 + 255) / 256), 256, 0, st>>>(xg, P.L, P.Dp, r, wa, acc);
    const int64_t seq_tiles = (P.N + FWD_THREADS - 1) / FWD_THREADS;
    // shares of a chunk: some eight blocks per SM, at least one stretch each
    const int64_t room = P.Dp / (P.Nx * Q) / P.Cg;   // (Dp doubles)
    const int64_t parts = std::min({room, std::max<int64_t>(1, 8 * 152 / (seq_tiles * P.Cg)), (P.LC + EF_STR - 1) / EF_STR});
    const int slices = (int)(P.Cg * std::max<int64_t>(1, parts));
    double *part = parts >= 1 ? xg : partial64;
    k_eval_fwd<<<dim3((unsigned)seq_tiles, (unsigned)slices), FWD_THREADS, 0, st>>>(
        X, P.Lx, (int)P.N, (int)P.L, P.LC, (int)(slices / P.Cg), wa, part, P.Nx);
    k_eval_beliefs<<<(unsigned)((P.N * EB_SHARE + FWD_THREADS - 1) / FWD_THREADS), FWD_THREADS, 0, st>>>(
        part, slices, P.Nx, (int)P.N, wa + QQ * P.L, rstate, w, reinterpret_cast<float4 *>(R), acc);
    k_eval_bwd<<<(unsigned)((P.L + BWD_THREADS - 1) / BWD_THREADS), BWD_THREADS, 0, st>>>(
        XT, P.Nx, (int)P.N, (int)P.L, r, reinterpret_cast<const float4 *>(R), wa, P.lambda_J, P.lambda_h,
        want_g ? xg : nullptr, acc);
}

void launch_grad_finalize(const Problem &P, const SlotDev *sd, const int32_t *list, int n,
                          const float *wa, float *gpool, void *Ypool, const void *Spool, int hist_bf16,
                          double *acc, cudaStream_t st)
{
    if (n <= 0) return;
    const int64_t need = (P.L + BWD_THREADS - 1) / BWD_THREADS;
    dim3 grid((unsigned)(need < 512 ? need : 512), (unsigned)n);
    k_grad_finalize<<<grid, BWD_THREADS, 0, st>>>((int)P.L, sd, list, wa, gpool, Ypool, Spool, hist_bf16,
                                                   P.ring, P.Dp, P.lambda_J, acc);
}

void launch_bwd_gather(const Problem &P, const uint8_t *XT, const SlotDev *sd,
                       const int32_t *list, int n, const float *R, const float *wa,
                       float *gpool, void *Ypool, const void *Spool, int hist_bf16,
                       double *acc, cudaStream_t st)
{
    if (n <= 0) return;
    dim3 grid((unsigned)((P.L + BG_THREADS - 1) / BG_THREADS), (unsigned)((n + BWD_G - 1) / BWD_G));
    k_bwd_gather<<<grid, BG_THREADS, 0, st>>>(XT, P.Nx, (int)P.N, (int)P.L, sd, list, n,
                                               reinterpret_cast<const float4 *>(R), wa, gpool, Ypool,
                                               Spool, hist_bf16, P.ring, P.Dp, P.lambda_J, acc);
}

} // namespace sdca
