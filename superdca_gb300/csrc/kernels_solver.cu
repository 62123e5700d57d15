// kernels_solver.cu -- per-slot solver kernels shared by every contraction
// form: line-search trials, iterate update, L-BFGS history and direction,
// and coupling scores.
//
// Line-search trials never run a contraction.  The logits of sequence i are
// affine in the step along d: l_i(stp) = lbase_i + stp * u_i with
// u_i = X_i . d_J + d_h, so a trial needs O(N q) work per slot.  This is
// exactly SuperDCA's objective along the search line (plmDCA_objective.hpp:
// 126-151 for the pseudo-likelihood part; the L2 part is a quadratic in stp
// from x.d and d.d).
#include <algorithm>
#include <new>

#include <cooperative_groups.h>

#include "engine.h"
#include "exp_log64.h"
#include "kernels_common.cuh"

namespace sdca {

namespace {

// base logits (FP64)
__device__ __forceinline__ double4 load4(const double *v, int64_t o)
{
    const double2 a = reinterpret_cast<const double2 *>(v + o * 4)[0];
    const double2 b = reinterpret_cast<const double2 *>(v + o * 4)[1];
    return make_double4(a.x, a.y, b.x, b.y);
}

constexpr int SEARCH_WARPS = 15, SEARCH_THREADS = 32 * SEARCH_WARPS;   // evaluating; one more searches
constexpr int SEARCH_CLUSTER = 8;
constexpr int SEARCH_K = 6;   // sums of a trial: f, slope, R per state

// order of doubles as 64-bit integers (comparisons are FP64 work too)
__device__ __forceinline__ bool above_eq(double a, double b)
{
    const long long x = __double_as_longlong(a), y = __double_as_longlong(b);
    const long long kx = x ^ ((x >> 63) & 0x7fffffffffffffffll), ky = y ^ ((y >> 63) & 0x7fffffffffffffffll);
    return kx >= ky;
}

// One sequence at logits l, state sr, weight w: adds w (lse - l[sr]) to f and
// gives the residuals w (p - [a = sr]).  The largest logit's exponential is 1,
// so three are left.
__device__ __forceinline__ void belief(const double (&l)[4], int sr, double w, const ExpTab *E, const LogTab *G,
                                       double &f, double (&r)[4])
{
    const bool a = above_eq(l[0], l[1]), b = above_eq(l[2], l[3]);
    const double M0 = a ? l[0] : l[1], M1 = b ? l[2] : l[3];
    const bool c = above_eq(M0, M1);
    const double mx = c ? M0 : M1;
    const double dn0 = (a ? l[1] : l[0]) - mx, dn1 = (b ? l[3] : l[2]) - mx, dm = (c ? M1 : M0) - mx;
    const double en0 = exp64(dn0, E), en1 = exp64(dn1, E), em = exp64(dm, E);
    // (an infinite largest logit leaves no belief)
    const double one = (__double2hiint(mx) & 0x7ff00000) == 0x7ff00000 ? __longlong_as_double(0x7ff8000000000000ll) : 1.0;
    const double z = (one + em) + (en0 + en1);
    const double dM0 = c ? 0.0 : dm, dM1 = c ? dm : 0.0;
    const double d[4] = {a ? dM0 : dn0, a ? dn0 : dM0, b ? dM1 : dn1, b ? dn1 : dM1};
    const double ds = sr & 2 ? (sr & 1 ? d[3] : d[2]) : (sr & 1 ? d[1] : d[0]);
    f = fma(w, log64(z, G) - ds, f);
    const double rz = w * rcp64(z);
    const double pm = em * rz, pn0 = en0 * rz, pn1 = en1 * rz;
    const double pM0 = c ? rz : pm, pM1 = c ? pm : rz;
    r[0] = a ? pM0 : pn0;
    r[1] = a ? pn0 : pM0;
    r[2] = b ? pM1 : pn1;
    r[3] = b ? pn1 : pM1;
    const double rs = (sr & 2 ? (sr & 1 ? r[3] : r[2]) : (sr & 1 ? r[1] : r[0])) - w;
#pragma unroll
    for (int k = 0; k < 4; ++k) r[k] = k == sr ? rs : r[k];
}

// Line searches, one per cluster: every trial evaluates the slot's sequences
// at lbase + stp u (FP64), the blocks exchange their sums through distributed
// shared memory, and each block's last warp runs the same search step on the
// same numbers, so that one cluster barrier per trial is enough.  While a
// trial runs that warp works out what the step needs besides its values (L2
// part, reciprocal).  Without SLOT_F_SEARCH one evaluation at S.stp.  The R,
// sums and step left behind are the last trial's.
//
// Bound by FP64 issue: 84 instructions per sequence and trial at one in 64
// clocks per quarter of an SM (95 % of that while all slots search), and by
// the serial part of a trial, some 9 us, for the last slots.  64 slots of
// 3000 sequences: 46 us for one evaluation (83 with CUDA's exp, log and
// divisions), 43 per trial, 18 for a lone slot's; a launch, a copy back and a
// search step on the host per trial took another 35 each.  Solves of 64 loci:
// 3000 x 10,000 376 -> 257 ms (tensor-core form), 1000 x 4001 115 -> 94 (plain).
__global__ void __launch_bounds__(SEARCH_THREADS + 32, 2)
k_search(const SlotDev *__restrict__ sd, const int32_t *__restrict__ list, int N, int64_t Nx, double lambda_J,
         double lambda_h, const double *__restrict__ lbase, const float4 *__restrict__ u,
         const uint8_t *__restrict__ rstate, const double *__restrict__ w, float4 *__restrict__ R,
         double *__restrict__ acc)
{
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    __shared__ ExpTab sE[EXP_N];
    __shared__ LogTab sG[LOG_N];
    __shared__ double warp_part[SEARCH_WARPS + 1][8];   // (a zero row)
    __shared__ double parts[2][SEARCH_CLUSTER][8];   // the blocks' sums, by parity of the trial
    __shared__ __align__(16) unsigned char mt_raw[sizeof(MoreThuente)];
    __shared__ double s_stp;
    __shared__ int s_more;
    const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const bool searcher = wid == SEARCH_WARPS;
    for (int k = tid; k < EXP_N; k += blockDim.x) sE[k] = kExpTab[k];
    for (int k = tid; k < LOG_N; k += blockDim.x) sG[k] = kLogTab[k];
    const int b = list[blockIdx.x / C];
    const SlotDev &S = sd[b];
    const bool use_u = S.flags & SLOT_F_USE_U;
    double *A = acc + (int64_t)b * NACC;
    MoreThuente &mt = *reinterpret_cast<MoreThuente *>(mt_raw);   // the searcher's lane 0
    bool search = S.flags & SLOT_F_SEARCH;
    int outcome = LS_MET, trials = 0;
    if (searcher && lane == 0) {
        double stp = S.stp;
        if (search) {
            new (mt_raw) MoreThuente();
            // slope of the search line at 0 from the numbers the trials use
            const double dg0 = A[ACC_DG0] + S.l2.slope(lambda_J, lambda_h, 0.0);
            if (mt.start(S.f0, dg0, S.alpha) == MoreThuente::NEED_EVAL) {
                stp = mt.stp;
            } else {
                outcome = LS_NO_DESCENT;
                search = false;
                stp = 0.0;
            }
        }
        s_stp = stp;
    }
    if (searcher && lane < 8) warp_part[SEARCH_WARPS][lane] = 0;
    const int64_t o0 = (int64_t)b * Nx;
    cl.sync();   // (every block runs before its shared memory is written)
    for (int par = 0;; par ^= 1) {
        const double stp = s_stp;
        double l2f = 0, l2g = 0;
        if (searcher) {
            if (lane == 0 && search) {
                mt.ahead();
                l2f = S.l2.value(lambda_J, lambda_h, stp);
                l2g = S.l2.slope(lambda_J, lambda_h, stp);
            }
        } else {
            double v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
            for (int i = rank * SEARCH_THREADS + tid; i < N; i += C * SEARCH_THREADS) {
                const double4 lb = load4(lbase, o0 + i);
                const float4 uf = use_u ? u[o0 + i] : make_float4(0.f, 0.f, 0.f, 0.f);
                const double4 uu = make_double4(uf.x, uf.y, uf.z, uf.w);
                const double l[4] = {fma(stp, uu.x, lb.x), fma(stp, uu.y, lb.y), fma(stp, uu.z, lb.z),
                                     fma(stp, uu.w, lb.w)};
                double r[4];
                belief(l, rstate[o0 + i], w[i], sE, sG, v[0], r);
                v[1] += r[0] * uu.x + r[1] * uu.y + r[2] * uu.z + r[3] * uu.w;
                v[2] += r[0]; v[3] += r[1]; v[4] += r[2]; v[5] += r[3];
                R[o0 + i] = make_float4((float)r[0], (float)r[1], (float)r[2], (float)r[3]);
            }
            // six sums over the warp by halving what each lane keeps: 4, 2 and
            // 1 values, then two plain steps; lane 4 k holds value k (bits
            // of k: lane bits 16, 8, 4)
#pragma unroll
            for (int s = 0, h = 4; s < 3; ++s, h >>= 1) {
                const int bit = 16 >> s;
#pragma unroll
                for (int k = 0; k < h; ++k) {
                    const double give = lane & bit ? v[k] : v[k + h], keep = lane & bit ? v[k + h] : v[k];
                    v[k] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
                }
            }
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
            if ((lane & 3) == 0) warp_part[wid][lane >> 2] = v[0];
        }
        __syncthreads();
        const int k8 = lane & 7, g8 = lane >> 3;   // the searcher's lane: value, and one of four groups of rows
        auto groups = [](double t) {
            t += __shfl_xor_sync(0xffffffffu, t, 8);
            return t + __shfl_xor_sync(0xffffffffu, t, 16);
        };
        if (searcher) {
            double t = warp_part[g8][k8];
#pragma unroll
            for (int k = 4; k < SEARCH_WARPS + 1; k += 4) t += warp_part[g8 + k][k8];
            t = groups(t);
            for (int k = g8; k < C; k += 4) cl.map_shared_rank(&parts[par][rank][0], k)[k8] = t;
        }
        cl.sync();
        if (searcher) {
            double t = 0;
            for (int k = g8; k < C; k += 4) t += parts[par][k][k8];
            t = groups(t);
            const double fd = __shfl_sync(0xffffffffu, t, 0), dd = __shfl_sync(0xffffffffu, t, 1);
            int more = 0;
            if (lane == 0 && search) {
                ++trials;
                const double f = fd + l2f, dg = dd + l2g;
                if (!isfinite(f) || !isfinite(dg)) {
                    outcome = LS_NOT_FINITE;
                } else if (mt.feed(f, dg) == MoreThuente::DONE) {
                    outcome = mt.info == 1 ? LS_MET : LS_ENDED;
                } else {
                    more = 1;
                    s_stp = mt.stp;
                }
            }
            if (lane == 0) s_more = more;
            more = __shfl_sync(0xffffffffu, more, 0);
            if (!more && rank == 0) {
                if (lane < SEARCH_K) A[ACC_F + lane] = t;
                if (lane == 0) {
                    A[ACC_STP] = stp;
                    A[ACC_TRIALS] = trials;
                    A[ACC_LS] = outcome;
                }
            }
        }
        __syncthreads();
        if (!s_more) return;
    }
}

// Loci enter slots (who: slot, locus), starting from zero.  One launch for
// all of them: as five memsets, a copy and an upload per slot it was the
// host's time between two rounds, some 16 us per locus.
__device__ __forceinline__ void zero_span(void *p, int64_t bytes)
{
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < bytes / 16; k += (int64_t)gridDim.x * blockDim.x)
        reinterpret_cast<uint4 *>(p)[k] = make_uint4(0, 0, 0, 0);
}

__global__ void __launch_bounds__(256)
k_slots_begin(const int2 *__restrict__ who, int64_t Nx, int64_t Dp, const uint8_t *__restrict__ states,
              uint8_t *__restrict__ rstate, float *__restrict__ wa, float *__restrict__ d, double *__restrict__ lbase,
              float2 *__restrict__ dv, int64_t dv_slot, DualCtl *__restrict__ ctl)
{
    const int64_t b = who[blockIdx.y].x, r = who[blockIdx.y].y;
    zero_span(wa + b * Dp, Dp * 4);
    if (d) zero_span(d + b * Dp, Dp * 4);
    zero_span(lbase + b * Nx * 4, Nx * 32);
    if (dv) zero_span(dv + b * dv_slot, dv_slot * 8);
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < Nx / 16; k += (int64_t)gridDim.x * blockDim.x)
        reinterpret_cast<uint4 *>(rstate + b * Nx)[k] = reinterpret_cast<const uint4 *>(states + r * Nx)[k];
    if (ctl && blockIdx.x == 0) {
        static_assert(sizeof(DualCtl) % 8 == 0, "zeroed in words");
        for (unsigned k = threadIdx.x; k < sizeof(DualCtl) / 8; k += blockDim.x)
            reinterpret_cast<unsigned long long *>(ctl + b)[k] = 0;
        __syncthreads();
        if (threadIdx.x == 0) {
            ctl[b].phase = DC_EVAL0;
            ctl[b].ring_new = -1;
            ctl[b].last_check = -1000;
        }
    }
}

// x <- x + stp d; with a history push, s = x_new - x_old goes to ring_new.
__global__ void k_accept(const SlotDev *__restrict__ sd, const int32_t *__restrict__ list,
                         int64_t Dp, int m, float *__restrict__ wa, const float *__restrict__ d,
                         void *__restrict__ Spool, int hist_bf16)
{
    const int b = list[blockIdx.y];
    const SlotDev &S = sd[b];
    const float stp = (float)S.stp;
    const bool push = (S.flags & SLOT_F_PUSH) && S.ring_new >= 0;
    for (int64_t e = 4 * ((int64_t)blockIdx.x * blockDim.x + threadIdx.x); e < Dp;
         e += 4 * (int64_t)gridDim.x * blockDim.x) {
        float4 *xp = reinterpret_cast<float4 *>(wa + (int64_t)b * Dp + e);
        const float4 x = *xp;
        const float4 dv = *reinterpret_cast<const float4 *>(d + (int64_t)b * Dp + e);
        float4 xn;
        xn.x = fmaf(stp, dv.x, x.x);
        xn.y = fmaf(stp, dv.y, x.y);
        xn.z = fmaf(stp, dv.z, x.z);
        xn.w = fmaf(stp, dv.w, x.w);
        if (push)
            store_hist4(Spool, ((int64_t)b * m + S.ring_new) * Dp + e,
                        make_float4(xn.x - x.x, xn.y - x.y, xn.z - x.z, xn.w - x.w), hist_bf16);
        *xp = xn;
    }
}

__global__ void k_lbase_update(const SlotDev *__restrict__ sd, const int32_t *__restrict__ list,
                               int N, int64_t Nx, double *__restrict__ lbase,
                               const float4 *__restrict__ u)
{
    const int b = list[blockIdx.y];
    const double stp = sd[b].stp;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N || stp == 0.0) return;
    const int64_t o = (int64_t)b * Nx + i;
    const float4 uu = u[o];
    double *lb = lbase + o * 4;
    lb[0] += stp * uu.x;
    lb[1] += stp * uu.y;
    lb[2] += stp * uu.z;
    lb[3] += stp * uu.w;
}

// gradient of h_r: sum_i R_i + 2 lambda_h h (plmDCA_objective.hpp:149,198)
__global__ void k_hpart(const SlotDev *__restrict__ sd, const int32_t *__restrict__ list,
                        int64_t L, int64_t Dp, int m, double lambda_h, const float *__restrict__ wa,
                        float *__restrict__ gpool, void *__restrict__ Ypool,
                        const void *__restrict__ Spool, int hist_bf16, double *__restrict__ acc)
{
    const int b = list[blockIdx.x];
    if (threadIdx.x != 0) return;
    const SlotDev &S = sd[b];
    const int64_t hoff = QQ * L;
    const float *x = wa + (int64_t)b * Dp + hoff;
    float *gn = gpool + (int64_t)(2 * b + 1 - S.gcur) * Dp + hoff;
    const float *go = gpool + (int64_t)(2 * b + S.gcur) * Dp + hoff;
    const bool push = (S.flags & SLOT_F_PUSH) && S.ring_new >= 0;
    double g2 = 0, x2 = 0, sy = 0, yy = 0, ss = 0, gmax = 0;
    float4 gv, yv;
    float *gp = &gv.x, *yp = &yv.x;
    for (int a = 0; a < 4; ++a) {
        const double g = S.rs[a] + 2.0 * lambda_h * (double)x[a];
        gp[a] = (float)g;
        gn[a] = gp[a];
        g2 += (double)gp[a] * gp[a];
        x2 += (double)x[a] * x[a];
        gmax = fmax(gmax, fabs((double)gp[a]));
        yp[a] = gp[a] - go[a];
    }
    if (push) {
        const int64_t off = ((int64_t)b * m + S.ring_new) * Dp + hoff;
        yv = store_hist4(Ypool, off, yv, hist_bf16);
        const float4 sv = load_hist4(Spool, off, hist_bf16);
        sy = (double)dot4(sv, yv);
        yy = (double)dot4(yv, yv);
        ss = (double)dot4(sv, sv);
    }
    double *A = acc + (int64_t)b * NACC;
    atomicAdd(A + ACC_G2, g2);
    atomicAdd(A + ACC_X2H, x2);
    if (push) {
        atomicAdd(A + ACC_SY, sy);
        atomicAdd(A + ACC_YY, yy);
        atomicAdd(A + ACC_SS, ss);
    }
    if (gmax > 0) atomic_max_nonneg(A + ACC_GMAX, gmax);
}

constexpr int DOT_THREADS = 256;
constexpr int DOT_U = 4;  // float4 groups per thread per tile: 16 KB runs per stream per block

// dots[b] = [S_j.g | Y_j.g | S_j.y_new | Y_j.y_new], j over the history.
// Blocks walk tiles of DOT_THREADS x DOT_U float4 groups; within a tile g and
// y_new stay in registers while the history vectors stream through one at a
// time, so every stream is read in long contiguous runs.
__global__ void __launch_bounds__(DOT_THREADS)
k_hist_dots(const SlotDev *__restrict__ sd, const int32_t *__restrict__ list, int64_t Dp, int m,
            const float *__restrict__ gpool, const void *__restrict__ Spool,
            const void *__restrict__ Ypool, int hist_bf16, double *__restrict__ dots)
{
    const int b = list[blockIdx.y];
    const SlotDev &S = sd[b];
    const int nh = S.nhist;
    const float4 *g4 = reinterpret_cast<const float4 *>(gpool + (int64_t)(2 * b + S.gcur) * Dp);
    const bool has_new = S.ring_new >= 0;
    const int64_t ybase = ((int64_t)b * m + (has_new ? S.ring_new : 0)) * Dp;
    const int64_t nv4 = Dp / 4, tile = (int64_t)DOT_THREADS * DOT_U;
    float aSg[MAXHIST], aYg[MAXHIST], aSy[MAXHIST], aYy[MAXHIST];
#pragma unroll
    for (int j = 0; j < MAXHIST; ++j) aSg[j] = aYg[j] = aSy[j] = aYy[j] = 0.f;
    for (int64_t tb = (int64_t)blockIdx.x * tile; tb < nv4; tb += (int64_t)gridDim.x * tile) {
        float4 gv[DOT_U], yn[DOT_U];
#pragma unroll
        for (int u = 0; u < DOT_U; ++u) {
            const int64_t v = tb + u * DOT_THREADS + threadIdx.x;
            const bool ok = v < nv4;
            gv[u] = ok ? g4[v] : make_float4(0.f, 0.f, 0.f, 0.f);
            yn[u] = (ok && has_new) ? load_hist4(Ypool, ybase + 4 * v, hist_bf16) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int j = 0; j < MAXHIST; ++j) {
            if (j < nh) {
                const int64_t base = ((int64_t)b * m + S.ring[j]) * Dp;
                float4 sv[DOT_U], yv[DOT_U];
#pragma unroll
                for (int u = 0; u < DOT_U; ++u) {
                    const int64_t v = tb + u * DOT_THREADS + threadIdx.x;
                    const bool ok = v < nv4;
                    sv[u] = ok ? load_hist4(Spool, base + 4 * v, hist_bf16) : make_float4(0.f, 0.f, 0.f, 0.f);
                    yv[u] = ok ? load_hist4(Ypool, base + 4 * v, hist_bf16) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
#pragma unroll
                for (int u = 0; u < DOT_U; ++u) {
                    aSg[j] += dot4(sv[u], gv[u]);
                    aYg[j] += dot4(yv[u], gv[u]);
                    aSy[j] += dot4(sv[u], yn[u]);
                    aYy[j] += dot4(yv[u], yn[u]);
                }
            }
        }
    }
    float v[4 * MAXHIST];
    int idx[4 * MAXHIST];
#pragma unroll
    for (int j = 0; j < MAXHIST; ++j) {
        v[j] = aSg[j];
        v[MAXHIST + j] = aYg[j];
        v[2 * MAXHIST + j] = aSy[j];
        v[3 * MAXHIST + j] = aYy[j];
    }
#pragma unroll
    for (int k = 0; k < 4 * MAXHIST; ++k) idx[k] = k;
    block_sum_atomic_f<4 * MAXHIST>(v, dots + (int64_t)b * 4 * MAXHIST, idx);
}

// d = coef_g g + sum_j (coefS_j s_j + coefY_j y_j), J_rr block zero;
// reductions g.d, d.d and x.d split into the J and h parts, and max|d|.
// Same tiling as k_hist_dots: d and g of a tile stay in registers while the
// history streams through.
__global__ void __launch_bounds__(DOT_THREADS)
k_direction(const SlotDev *__restrict__ sd, const int32_t *__restrict__ list, int64_t L,
            int64_t Dp, int m, const float *__restrict__ gpool, const void *__restrict__ Spool,
            const void *__restrict__ Ypool, int hist_bf16, const float *__restrict__ wa,
            float *__restrict__ d, double *__restrict__ acc)
{
    const int b = list[blockIdx.y];
    const SlotDev &S = sd[b];
    const int nh = S.nhist;
    const float4 *g4 = reinterpret_cast<const float4 *>(gpool + (int64_t)(2 * b + S.gcur) * Dp);
    const float4 *x4 = reinterpret_cast<const float4 *>(wa + (int64_t)b * Dp);
    float4 *d4 = reinterpret_cast<float4 *>(d + (int64_t)b * Dp);
    const float cg = (float)S.coef_g;
    const int64_t hoff4 = QQ * L / 4;
    const int64_t rlo4 = (int64_t)S.locus * QQ / 4, rhi4 = rlo4 + QQ / 4;
    const int64_t nv4 = Dp / 4, tile = (int64_t)DOT_THREADS * DOT_U;
    float gd = 0.f, ddJ = 0.f, ddH = 0.f, xdJ = 0.f, xdH = 0.f, dmax = 0.f;
    for (int64_t tb = (int64_t)blockIdx.x * tile; tb < nv4; tb += (int64_t)gridDim.x * tile) {
        float4 gv[DOT_U], dv[DOT_U];
#pragma unroll
        for (int u = 0; u < DOT_U; ++u) {
            const int64_t v = tb + u * DOT_THREADS + threadIdx.x;
            gv[u] = v < nv4 ? g4[v] : make_float4(0.f, 0.f, 0.f, 0.f);
            dv[u] = make_float4(cg * gv[u].x, cg * gv[u].y, cg * gv[u].z, cg * gv[u].w);
        }
#pragma unroll
        for (int j = 0; j < MAXHIST; ++j) {
            if (j < nh) {
                const int64_t base = ((int64_t)b * m + S.ring[j]) * Dp;
                const float cs = (float)S.coefS[j], cy = (float)S.coefY[j];
                float4 sv[DOT_U], yv[DOT_U];
#pragma unroll
                for (int u = 0; u < DOT_U; ++u) {
                    const int64_t v = tb + u * DOT_THREADS + threadIdx.x;
                    const bool ok = v < nv4;
                    sv[u] = ok ? load_hist4(Spool, base + 4 * v, hist_bf16) : make_float4(0.f, 0.f, 0.f, 0.f);
                    yv[u] = ok ? load_hist4(Ypool, base + 4 * v, hist_bf16) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
#pragma unroll
                for (int u = 0; u < DOT_U; ++u) {
                    dv[u].x += cs * sv[u].x + cy * yv[u].x;
                    dv[u].y += cs * sv[u].y + cy * yv[u].y;
                    dv[u].z += cs * sv[u].z + cy * yv[u].z;
                    dv[u].w += cs * sv[u].w + cy * yv[u].w;
                }
            }
        }
#pragma unroll
        for (int u = 0; u < DOT_U; ++u) {
            const int64_t v = tb + u * DOT_THREADS + threadIdx.x;
            if (v >= nv4) continue;
            if (v >= rlo4 && v < rhi4) dv[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            d4[v] = dv[u];
            const float4 xv = x4[v];
            gd += dot4(gv[u], dv[u]);
            dmax = fmaxf(dmax, fmaxf(fmaxf(fabsf(dv[u].x), fabsf(dv[u].y)), fmaxf(fabsf(dv[u].z), fabsf(dv[u].w))));
            if (v < hoff4) {
                ddJ += dot4(dv[u], dv[u]);
                xdJ += dot4(xv, dv[u]);
            } else {
                ddH += dot4(dv[u], dv[u]);
                xdH += dot4(xv, dv[u]);
            }
        }
    }
    float v[5] = {gd, ddJ, ddH, xdJ, xdH};
    const int idx[5] = {ACC_GD, ACC_DDJ, ACC_DDH, ACC_XDJ, ACC_XDH};
    block_sum_atomic_f<5>(v, acc + (int64_t)b * NACC, idx);
    const float wm = warp_max(dmax);
    if ((threadIdx.x & 31) == 0 && wm > 0.f) atomic_max_nonneg(acc + (int64_t)b * NACC + ACC_DMAX, (double)wm);
}

// S[r][n] = || gauge(M) ||_F without GAP, M = J_rn (transposed for n < r):
// SuperDCA/include/plmDCA.hpp:378-393, plmDCA_utility.hpp:57-83,
// Matrix_math.hpp:166-213.  G[i][j] = ((M[i][j] - rowmean(M)[j]) -
// colmean(M)[i]) + mean(rowmean(M)), evaluated in FP64 like the reference.
__global__ void k_score(const SlotDev *__restrict__ sd, const int32_t *__restrict__ list,
                        int64_t L, int64_t Dp, const float *__restrict__ wa, int gap,
                        float *__restrict__ rows)
{
    const int k = blockIdx.y;
    const int b = list[k];
    const int64_t r = sd[b].locus;
    const int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= L) return;
    float *row = rows + (int64_t)k * L;
    if (n == r) {
        row[n] = __int_as_float(0x7fc00000);
        return;
    }
    const float4 *jp = reinterpret_cast<const float4 *>(wa + (int64_t)b * Dp + n * QQ);
    // single precision: the block is stored in FP32 and the score is written
    // as FP32 (GB300's FP64 rate is a small fraction of its FP32 rate)
    float J[4][4];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        const float4 v = jp[s];
        const float t[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            if (n < r) J[a][s] = t[a];
            else J[s][a] = t[a];
        }
    }
    float rm[4], cm[4], gm = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float t = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) t = t + J[i][j];
        rm[i] = t * 0.25f;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        float t = 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) t = t + J[i][j];
        cm[j] = t * 0.25f;
    }
    {
        float t = 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) t += rm[i];
        gm = t * 0.25f;
    }
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if (i == gap) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (j == gap) continue;
            const float gij = ((J[i][j] - rm[j]) - cm[i]) + gm;
            sum = fmaf(gij, gij, sum);
        }
    }
    row[n] = sqrtf(sum);
}

// blocks per slot for the D-length passes: at most `cap`, so that every
// thread streams many float4 before the per-block reduction
unsigned dgrid(int64_t Dp, int threads, int64_t cap = 256)
{
    const int64_t need = (Dp / 4 + threads - 1) / threads;
    return (unsigned)(need < cap ? need : cap);
}

} // namespace

void launch_slots_begin(const Problem &P, const int2 *who, int n, const uint8_t *states, uint8_t *rstate, float *wa,
                        float *d, double *lbase, float2 *dv, int64_t dv_slot, DualCtl *ctl, cudaStream_t st)
{
    if (n <= 0) return;
    // (Nx, Dp and the vectors are multiples of 64 elements)
    const int64_t words = (std::max(P.Dp * 4, dv ? dv_slot * 8 : 0) / 16 + 255) / 256;
    k_slots_begin<<<dim3((unsigned)std::min<int64_t>(words, 64), (unsigned)n), 256, 0, st>>>(
        who, P.Nx, P.Dp, states, rstate, wa, d, lbase, dv, dv_slot, ctl);
}

// One cluster per slot, its blocks sharing the slot's sequences: as many as
// there are SMs for, while each evaluating thread still has a sequence.  Two
// blocks per SM, which would let a slot that ends early leave its SM to the
// other, took longer (54 us for 46 above: the blocks do not spread evenly; with
// clusters of eight and blocks of 256 threads some SMs stay empty, 57).
void launch_search(const Problem &P, const SlotDev *sd, const int32_t *list, int n,
                   const double *lbase, const float *u, const uint8_t *rstate, const double *w,
                   float *R, double *acc, cudaStream_t st)
{
    if (n <= 0) return;
    int c = 1;
    while (c < SEARCH_CLUSTER && (int64_t)c * SEARCH_THREADS < P.N && (int64_t)2 * c * n <= 152) c *= 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)c * n);
    cfg.blockDim = dim3(SEARCH_THREADS + 32);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)c;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, k_search, sd, list, (int)P.N, P.Nx, P.lambda_J, P.lambda_h, lbase,
                       reinterpret_cast<const float4 *>(u), rstate, w, reinterpret_cast<float4 *>(R), acc);
}

void launch_accept(const Problem &P, const SlotDev *sd, const int32_t *list, int n, float *wa,
                   const float *d, void *Spool, int hist_bf16, cudaStream_t st)
{
    if (n <= 0) return;
    dim3 grid(dgrid(P.Dp, 256), (unsigned)n);
    k_accept<<<grid, 256, 0, st>>>(sd, list, P.Dp, P.ring, wa, d, Spool, hist_bf16);
}

void launch_lbase_update(const Problem &P, const SlotDev *sd, const int32_t *list, int n,
                         double *lbase, const float *u, cudaStream_t st)
{
    if (n <= 0) return;
    dim3 grid((unsigned)((P.N + 255) / 256), (unsigned)n);
    k_lbase_update<<<grid, 256, 0, st>>>(sd, list, (int)P.N, P.Nx, lbase,
                                         reinterpret_cast<const float4 *>(u));
}

void launch_hpart(const Problem &P, const SlotDev *sd, const int32_t *list, int n,
                  const float *wa, float *gpool, void *Ypool, const void *Spool, int hist_bf16,
                  double *acc, cudaStream_t st)
{
    if (n <= 0) return;
    k_hpart<<<n, 32, 0, st>>>(sd, list, P.L, P.Dp, P.ring, P.lambda_h, wa, gpool, Ypool, Spool,
                              hist_bf16, acc);
}

void launch_hist_dots(const Problem &P, const SlotDev *sd, const int32_t *list, int n,
                      const float *gpool, const void *Spool, const void *Ypool, int hist_bf16,
                      double *dots, cudaStream_t st)
{
    if (n <= 0) return;
    // enough blocks for about two waves in total, each thread streaming
    // hundreds of float4 before the block reduction
    const int64_t per_slot = std::max<int64_t>(4, std::min<int64_t>(64, (4 * 152 + n - 1) / n));
    dim3 grid(dgrid(P.Dp, DOT_THREADS * DOT_U, per_slot), (unsigned)n);
    k_hist_dots<<<grid, DOT_THREADS, 0, st>>>(sd, list, P.Dp, P.ring, gpool, Spool, Ypool, hist_bf16,
                                              dots);
}

void launch_direction(const Problem &P, const SlotDev *sd, const int32_t *list, int n,
                      const float *gpool, const void *Spool, const void *Ypool, int hist_bf16,
                      const float *wa, float *d, double *acc, cudaStream_t st)
{
    if (n <= 0) return;
    const int64_t per_slot = std::max<int64_t>(4, std::min<int64_t>(128, (4 * 152 + n - 1) / n));
    dim3 grid(dgrid(P.Dp, DOT_THREADS * DOT_U, per_slot), (unsigned)n);
    k_direction<<<grid, DOT_THREADS, 0, st>>>(sd, list, P.L, P.Dp, P.ring, gpool, Spool, Ypool,
                                              hist_bf16, wa, d, acc);
}

void launch_score(const Problem &P, const SlotDev *sd, const int32_t *list, int n,
                  const float *wa, int gap, float *rows, cudaStream_t st)
{
    if (n <= 0) return;
    dim3 grid((unsigned)((P.L + 127) / 128), (unsigned)n);
    k_score<<<grid, 128, 0, st>>>(sd, list, P.L, P.Dp, wa, gap, rows);
}

} // namespace sdca
