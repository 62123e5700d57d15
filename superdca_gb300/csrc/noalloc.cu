// noalloc.cu -- one objective evaluation that allocates no memory.
//
// sdca_eval needs a handle, and a handle allocates device memory for the
// alignment and the solver state.  Some callers cannot let a library
// allocate: host programs that own all device memory through their own
// allocator (a framework's caching allocator, or an embedded runtime with a
// fixed memory budget) and forbid libraries from calling cudaMalloc or
// cudaFree behind their back.  sdca_eval_noalloc serves them: the caller
// passes device pointers for every input and output, and the intermediate
// values (per-sequence node beliefs, per-block partial sums and an error
// word) live in one file-scope __device__ array of fixed size, SCRATCH_BYTES
// below, which every GPU that loads this library holds until the process
// exits; the caller's g holds partial logits until the gradient is written,
// unless it overlaps x or the weights (an evaluation in place).
//
// The array is shared by every call: two calls whose kernels overlap on the
// GPU (different streams, or different host threads) race on it.  Each call
// writes every scratch element it reads before reading it, and the error
// word is returned to zero by the last kernel of every call, so nothing needs
// clearing between calls.
//
// The array's device address is looked up with cudaGetSymbolAddress once per
// CUDA context (the first call made while that context is current), and
// cached under the context's unique id; a context created anew (for example
// after cudaDeviceReset) has a new id, so its first call looks the address up
// again.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <mutex>
#include <utility>
#include <vector>

#include "../../include/superdca_gb300.h"

namespace {

constexpr int NA_THREADS = 256, NG_THREADS = 448;   // per block: most passes, the gradient's
constexpr int NA_MAX_BLOCKS = (int)((SDCA_NOALLOC_MAX_LOCI + NA_THREADS - 1) / NA_THREADS);  // partial-sum slots
constexpr int64_t NA_MAX_SEQS = SDCA_NOALLOC_MAX_SEQS;
// node beliefs (N x 4 doubles) + per-block partials (5 doubles per block,
// two passes) + one error word (8 bytes)
constexpr size_t NA_ERR_OFFSET = (size_t)NA_MAX_SEQS * 4 + (size_t)2 * NA_MAX_BLOCKS * 8;   // in doubles
constexpr size_t SCRATCH_BYTES = (NA_ERR_OFFSET + 1) * sizeof(double);

__device__ __align__(256) unsigned char g_na_scratch[SCRATCH_BYTES];

// scratch address per CUDA context, keyed by the context's unique id
std::mutex g_na_mu;
std::vector<std::pair<unsigned long long, double *>> g_na_ptr;

// The current context's unique id (cuCtxGetCurrent + cuCtxGetId, reached
// through the runtime's driver entry points, so no link to libcuda).
bool current_context_id(unsigned long long *id)
{
    using get_current_fn = int (*)(void **);
    using get_id_fn = int (*)(void *, unsigned long long *);
    static get_current_fn get_current = nullptr;
    static get_id_fn get_id = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_current = reinterpret_cast<get_current_fn>(p);
        p = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_id = reinterpret_cast<get_id_fn>(p);
        cudaGetLastError();
    });
    if (!get_current || !get_id) return false;
    void *ctx = nullptr;
    if (get_current(&ctx) != 0 || !ctx) return false;
    return get_id(ctx, id) == 0;
}

// Position of J_r[n][s][a] in SuperDCA's parameter layout: 16-locus blocks,
// STATES order inside a block (SuperDCA/include/Matrix_kernel_access_order.hpp:
// 28-34, Coupling_matrix_view.hpp:156-168).
__device__ __forceinline__ int64_t na_index(int64_t L, int64_t n, int s, int a)
{
    const int64_t b = n / 16, p = n % 16, nfull = L / 16;
    const int64_t e = b < nfull ? 16 : L % 16;
    return b * 256 + ((int64_t)s * e + p) * 4 + a;
}

__device__ __forceinline__ double na_warp_sum(double v)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// block sum of K values (at most NG_THREADS threads); thread 0 gets the totals
template <int K>
__device__ __forceinline__ void na_block_sum(double (&v)[K])
{
    __shared__ double red[NG_THREADS / 32][K];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int k = 0; k < K; ++k) v[k] = na_warp_sum(v[k]);
    if (lane == 0)
        for (int k = 0; k < K; ++k) red[w][k] = v[k];
    __syncthreads();
    if (threadIdx.x == 0)
        for (int k = 0; k < K; ++k) {
            double t = 0.0;
            for (int j = 0; j < (int)blockDim.x / 32; ++j) t += red[j][k];
            v[k] = t;
        }
}

// ---- The contractions.  Both are sums of FP64 rows chosen by the states, and
// GB300 adds two FP64 values per cycle and SM, so the additions are the bound
// (2 x 4 N L of them: 0.56 ms at 616 x 65,563), and tables cut their number:
// the sums over a few loci (or sequences) are formed once for every
// combination and looked up.  One thread per sequence, and then one per
// locus, took 26 ms and 0.5 ms there; these passes take 0.15 ms (logits), 0.02
// (beliefs) and 0.29 (gradient), FP64 additions still the bound.

constexpr int NA_QUADS = 4;                       // locus quads per step: 16 loci
constexpr int NA_STEP = 4 * NA_QUADS;
constexpr int NA_MAX_SPT = 4;                     // sequences per thread of the logits pass, at most

// The 16 codes of a sequence's loci n0 .. n0 + 15 as four words (codes past
// the end of the row are 0); any code >= 4 sets bad.  Words are read whole
// where they lie in the array, whatever the row's alignment.
__device__ __forceinline__ void na_codes(const uint8_t *__restrict__ states, int64_t total, int64_t at, int live,
                                         uint32_t (&c)[NA_QUADS], uint32_t &bad)
{
    const uint8_t *p = states + at;
    const uintptr_t lo = reinterpret_cast<uintptr_t>(p) & ~(uintptr_t)3, first = reinterpret_cast<uintptr_t>(states);
    if (lo >= first && lo + 4 * (NA_QUADS + 1) <= first + (uintptr_t)total) {
        const uint32_t *w = reinterpret_cast<const uint32_t *>(lo);
        const uint32_t sh = 8u * (uint32_t)(reinterpret_cast<uintptr_t>(p) - lo);
        uint32_t v[NA_QUADS + 1];
#pragma unroll
        for (int k = 0; k <= NA_QUADS; ++k) v[k] = w[k];
#pragma unroll
        for (int k = 0; k < NA_QUADS; ++k) c[k] = __funnelshift_r(v[k], v[k + 1], sh);
    } else {
#pragma unroll
        for (int k = 0; k < NA_QUADS; ++k) {
            c[k] = 0u;
            for (int q = 0; q < 4; ++q)
                if (4 * k + q < live) c[k] |= (uint32_t)p[4 * k + q] << (8 * q);
        }
    }
#pragma unroll
    for (int k = 0; k < NA_QUADS; ++k) {
        const int left = live - 4 * k;   // live codes of this word
        if (left < 4) c[k] &= left <= 0 ? 0u : (1u << (8 * left)) - 1u;
        bad |= c[k] & 0xFCFCFCFCu;
        c[k] &= 0x03030303u;
    }
}

// pass 1: partial logits of every sequence over this block's steps of 16 loci
// (plmDCA_objective.hpp:86-121), into part[blockIdx.x][i][a].  A step forms
// the sums of every combination of states of four loci (256 rows, from pairs)
// four times over, then each sequence adds one row per quad: 1152 additions
// for the table of a quad and 4 per sequence, instead of 16 per sequence.
template <int SPT>
__global__ void __launch_bounds__(NA_THREADS)
k_na_logits(const uint8_t *__restrict__ states, int64_t N, int64_t L, int64_t r, const double *__restrict__ x,
            double *__restrict__ part, double *__restrict__ scratch)
{
    __shared__ __align__(16) double2 quad[NA_QUADS][256][2];
    __shared__ __align__(16) double2 pair[2 * NA_QUADS][16][2];
    const int t = threadIdx.x;
    const int64_t i0 = (int64_t)blockIdx.y * NA_THREADS * SPT + t;
    const int64_t steps = (L + NA_STEP - 1) / NA_STEP;
    const int64_t s0 = steps * blockIdx.x / gridDim.x, s1 = steps * (blockIdx.x + 1) / gridDim.x;
    double l[SPT][4] = {};
    uint32_t bad = 0u;
    for (int64_t st = s0; st < s1; ++st) {
        const int64_t n0 = st * NA_STEP;
        const int live = (int)min((int64_t)NA_STEP, L - n0);
        uint32_t c[SPT][NA_QUADS];
#pragma unroll
        for (int k = 0; k < SPT; ++k) {
            const int64_t i = i0 + (int64_t)k * NA_THREADS;
            if (i < N) na_codes(states, N * L, i * L + n0, live, c[k], bad);
        }
        // sums of two loci: 8 pairs x 16 combinations x 4
#pragma unroll
        for (int v = t; v < 2 * NA_QUADS * 64; v += NA_THREADS) {
            const int pr = v >> 6, cmb = (v >> 2) & 15, a = v & 3;
            const int64_t n1 = n0 + 2 * pr, n2 = n1 + 1;
            const double x1 = n1 < L && n1 != r ? x[na_index(L, n1, cmb & 3, a)] : 0.0;
            const double x2 = n2 < L && n2 != r ? x[na_index(L, n2, cmb >> 2, a)] : 0.0;
            reinterpret_cast<double *>(&pair[pr][cmb][0])[a] = x1 + x2;
        }
        __syncthreads();   // (the rows of the step before are used up too)
#pragma unroll
        for (int v = t; v < NA_QUADS * 512; v += NA_THREADS) {
            const int qd = v >> 9, cmb = (v >> 1) & 255, h = v & 1;
            const double2 u = pair[2 * qd][cmb & 15][h], w = pair[2 * qd + 1][cmb >> 4][h];
            quad[qd][cmb][h] = make_double2(u.x + w.x, u.y + w.y);
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < SPT; ++k) {
            if (i0 + (int64_t)k * NA_THREADS >= N) break;
#pragma unroll
            for (int qd = 0; qd < NA_QUADS; ++qd) {
                const int cmb = (int)((c[k][qd] * 0x01041040u) >> 24);   // c0 + 4 c1 + 16 c2 + 64 c3
                const double2 u = quad[qd][cmb][0], w = quad[qd][cmb][1];
                l[k][0] += u.x;
                l[k][1] += u.y;
                l[k][2] += w.x;
                l[k][3] += w.y;
            }
        }
    }
    if (bad) atomicOr(reinterpret_cast<unsigned long long *>(scratch + NA_ERR_OFFSET), 1ull);
#pragma unroll
    for (int k = 0; k < SPT; ++k) {
        const int64_t i = i0 + (int64_t)k * NA_THREADS;
        if (i < N)
#pragma unroll
            for (int a = 0; a < 4; ++a) part[((int64_t)blockIdx.x * N + i) * 4 + a] = l[k][a];
    }
}

// pass 2, one warp per sequence: the logits from their partial sums,
// objective term and node beliefs (plmDCA_objective.hpp:126-151).  part may be
// nb itself: a warp reads its sequence's logits, of which the first slice's
// lie where it writes the beliefs afterwards.
__global__ void __launch_bounds__(NA_THREADS)
k_na_beliefs(const uint8_t *__restrict__ states, int64_t N, int64_t L, int64_t r, const double *__restrict__ w,
             const double *__restrict__ x, int slices, const double *part, double *nb,
             double *__restrict__ scratch)
{
    double *sums = scratch + NA_MAX_SEQS * 4;     // blocks x 8
    const int lane = threadIdx.x & 31;
    const double *h = x + 16 * L;
    double v[5] = {0, 0, 0, 0, 0};
    for (int64_t i = (int64_t)blockIdx.x * (NA_THREADS / 32) + (threadIdx.x >> 5); i < N;
         i += (int64_t)gridDim.x * (NA_THREADS / 32)) {
        double l[4] = {0, 0, 0, 0};
#pragma unroll 4
        for (int s = lane; s < slices; s += 32)
#pragma unroll
            for (int a = 0; a < 4; ++a) l[a] += part[((int64_t)s * N + i) * 4 + a];
#pragma unroll
        for (int a = 0; a < 4; ++a) l[a] = na_warp_sum(l[a]) + h[a];
        const double mx = fmax(fmax(l[0], l[1]), fmax(l[2], l[3]));
        // one exponential per lane
        const double la = lane == 0 ? l[0] : lane == 1 ? l[1] : lane == 2 ? l[2] : l[3];
        const double ea = exp(la - mx);
        double e[4], z = 0.0;
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            e[a] = __shfl_sync(0xffffffffu, ea, a);
            z += e[a];
        }
        const int sr = states[i * L + r] & 3;
        const double wi = w[i];
        if (lane == 0) v[0] += wi * ((mx + log(z)) - (sr == 0 ? l[0] : sr == 1 ? l[1] : sr == 2 ? l[2] : l[3]));
        if (lane < 4) nb[i * 4 + lane] = wi * (ea / z) - (lane == sr ? wi : 0.0);
        const double bel = lane < 4 ? wi * (ea / z) - (lane == sr ? wi : 0.0) : 0.0;
#pragma unroll
        for (int a = 0; a < 4; ++a)
            if (lane == a) v[1 + a] += bel;
    }
    na_block_sum<5>(v);
    if (threadIdx.x == 0)
        for (int k = 0; k < 5; ++k) sums[blockIdx.x * 8 + k] = v[k];
}

// pass 3: the gradient's contraction, X^T of the node beliefs, one locus per
// thread (plmDCA_objective.hpp:153-190).  For eight sequences at a time the
// beliefs' sums over all 256 subsets are formed once per block (32 sequences
// a step, from subsets of four); a locus then adds, for each state, the row
// of the subset that has it: 2 additions per (sequence, locus) and entry a
// step cost 16 per thread for its table.  blockIdx.y: share of the sequences;
// with one share the gradient (and the L2 part of the objective, plmDCA_
// objective.hpp:192-244) is finished here, else part[y] holds the sums.
constexpr int NG_LOCI = 1, NG_SEQS = 32, NG_SETS = NG_SEQS / 8;

__global__ void __launch_bounds__(NG_THREADS)
k_na_gradient(const uint8_t *__restrict__ states, int64_t N, int64_t L, int64_t r, double lambda_J,
              const double *x, double *g, double *__restrict__ part, const double *__restrict__ nb,
              double *__restrict__ scratch)
{
    __shared__ __align__(16) double2 set[NG_SETS][256][2];
    __shared__ __align__(16) double2 half[2 * NG_SETS][16][2];
    const int t = threadIdx.x;
    const int64_t n0 = (int64_t)blockIdx.x * NG_THREADS * NG_LOCI + t;
    const int64_t steps = (N + NG_SEQS - 1) / NG_SEQS;
    const int64_t s0 = steps * blockIdx.y / gridDim.y, s1 = steps * (blockIdx.y + 1) / gridDim.y;
    double c[NG_LOCI][4][4] = {};
    for (int64_t st = s0; st < s1; ++st) {
        const int64_t i0 = st * NG_SEQS;
        // the eight subsets' masks of this thread's loci: byte s of m[set] has
        // bit k when sequence i0 + 8 set + k has state s
        uint32_t m[NG_LOCI][NG_SETS];
#pragma unroll
        for (int q = 0; q < NG_LOCI; ++q) {
            const int64_t n = n0 + (int64_t)q * NG_THREADS;
#pragma unroll
            for (int e = 0; e < NG_SETS; ++e) {
                uint32_t v = 0u;
                if (n < L) {
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const int64_t i = i0 + 8 * e + k;
                        if (i < N) v |= (1u << k) << (8 * (states[i * L + n] & 3));
                    }
                }
                m[q][e] = v;
            }
        }
        // sums over the subsets of four sequences: 8 halves x 16 x 4
        for (int v = t; v < 2 * NG_SETS * 64; v += NG_THREADS) {
            const int hf = v >> 6, mask = (v >> 2) & 15, a = v & 3;
            double u = 0.0;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int64_t i = i0 + 4 * hf + k;
                if ((mask >> k & 1) && i < N) u += nb[i * 4 + a];
            }
            reinterpret_cast<double *>(&half[hf][mask][0])[a] = u;
        }
        __syncthreads();   // (the rows of the step before are used up too)
        for (int v = t; v < NG_SETS * 512; v += NG_THREADS) {
            const int e = v >> 9, mask = (v >> 1) & 255, hh = v & 1;
            const double2 u = half[2 * e][mask & 15][hh], w = half[2 * e + 1][mask >> 4][hh];
            set[e][mask][hh] = make_double2(u.x + w.x, u.y + w.y);
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < NG_LOCI; ++q)
#pragma unroll
            for (int e = 0; e < NG_SETS; ++e)
#pragma unroll
                for (int s = 0; s < 4; ++s) {
                    const int mask = m[q][e] >> (8 * s) & 255;
                    const double2 u = set[e][mask][0], w = set[e][mask][1];
                    c[q][s][0] += u.x;
                    c[q][s][1] += u.y;
                    c[q][s][2] += w.x;
                    c[q][s][3] += w.y;
                }
    }
    double v[1] = {0.0};
#pragma unroll
    for (int q = 0; q < NG_LOCI; ++q) {
        const int64_t n = n0 + (int64_t)q * NG_THREADS;
        if (n >= L) continue;
        // (g may be x: this thread's entries are read before it writes any)
        double xv[4][4] = {};
        if (!part && n != r) {
#pragma unroll
            for (int s = 0; s < 4; ++s)
#pragma unroll
                for (int a = 0; a < 4; ++a) xv[s][a] = x[na_index(L, n, s, a)];
        }
#pragma unroll
        for (int s = 0; s < 4; ++s)
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                const int64_t o = na_index(L, n, s, a);
                if (part) {
                    part[(int64_t)blockIdx.y * 16 * L + o] = c[q][s][a];
                } else if (n == r) {
                    g[o] = 0.0;
                } else {
                    g[o] = c[q][s][a] + 2.0 * lambda_J * xv[s][a];
                    v[0] += lambda_J * xv[s][a] * xv[s][a];
                }
            }
    }
    if (part) return;
    na_block_sum<1>(v);
    if (t == 0) scratch[NA_MAX_SEQS * 4 + (size_t)NA_MAX_BLOCKS * 8 + blockIdx.x * 8] = v[0];
}

// the gradient from its shares, and the L2 part of the objective
__global__ void __launch_bounds__(NA_THREADS)
k_na_gradient_sum(int64_t L, int64_t r, double lambda_J, int shares, const double *__restrict__ part,
                  const double *x, double *g, double *__restrict__ scratch)
{
    double v[1] = {0.0};
    for (int64_t e = (int64_t)blockIdx.x * NA_THREADS + threadIdx.x; e < 16 * L; e += (int64_t)gridDim.x * NA_THREADS) {
        // the locus of entry e: 16-locus blocks, [s][locus][a] inside
        const int64_t b = e / 256, width = b < L / 16 ? 16 : L % 16, n = b * 16 + (e - b * 256) / 4 % width;
        const double xv = x[e];   // (g may be x)
        double u = 0.0;
        for (int k = 0; k < shares; ++k) u += part[(int64_t)k * 16 * L + e];
        if (n == r) {
            g[e] = 0.0;
        } else {
            g[e] = u + 2.0 * lambda_J * xv;
            v[0] += lambda_J * xv * xv;
        }
    }
    na_block_sum<1>(v);
    if (threadIdx.x == 0) scratch[NA_MAX_SEQS * 4 + (size_t)NA_MAX_BLOCKS * 8 + blockIdx.x * 8] = v[0];
}

// pass 4, one block: totals, h gradient and the h part of the objective.
// A state code >= 4 seen by pass 1 makes f and the h gradient NaN; the
// error word is returned to zero for the next call.
__global__ void k_na_total(int64_t L, int nb1, int nb2, double lambda_h, const double *x, double *f, double *g,
                           double *__restrict__ scratch)
{
    const double *p1 = scratch + NA_MAX_SEQS * 4;
    const double *p2 = p1 + (size_t)NA_MAX_BLOCKS * 8;
    double v[6] = {0, 0, 0, 0, 0, 0};
    for (int b = threadIdx.x; b < nb1; b += NA_THREADS)
        for (int k = 0; k < 5; ++k) v[k] += p1[b * 8 + k];
    for (int b = threadIdx.x; b < nb2; b += NA_THREADS) v[5] += p2[b * 8];
    na_block_sum<6>(v);
    if (threadIdx.x == 0) {
        unsigned long long *err = reinterpret_cast<unsigned long long *>(scratch + NA_ERR_OFFSET);
        const bool bad = *err != 0ull;
        *err = 0ull;
        double fv = v[0] + v[5];
        for (int a = 0; a < 4; ++a) {
            const double h = x[16 * L + a];   // (g may be x)
            fv += lambda_h * h * h;
            g[16 * L + a] = bad ? nan("") : v[1 + a] + 2.0 * lambda_h * h;
        }
        *f = bad ? nan("") : fv;
    }
}

} // namespace

extern "C" int sdca_eval_noalloc(const uint8_t *states, int64_t n_seqs, int64_t n_loci,
                                 const double *weights, double lambda_h, double lambda_J, uint32_t r,
                                 const double *x, double *f, double *g, void *stream)
{
    // every rejection happens before any work is queued
    if (!states || !weights || !x || !f || !g) return SDCA_E_ARG;
    if (n_seqs < 1 || n_loci < 2 || (int64_t)r >= n_loci) return SDCA_E_ARG;
    if (n_seqs > NA_MAX_SEQS || n_loci > SDCA_NOALLOC_MAX_LOCI) return SDCA_E_ARG;
    // an error left pending by the caller's earlier work is theirs: report
    // it without consuming it, and queue nothing
    if (cudaPeekAtLastError() != cudaSuccess) return SDCA_E_CUDA;
    double *scratch = nullptr;
    {
        std::lock_guard<std::mutex> lk(g_na_mu);
        unsigned long long id = 0;
        bool have_id = current_context_id(&id);
        if (have_id)
            for (const auto &e : g_na_ptr)
                if (e.first == id) scratch = e.second;
        if (!scratch) {
            void *p = nullptr;
            const cudaError_t e = cudaGetSymbolAddress(&p, g_na_scratch);   // makes the context current
            if (e != cudaSuccess) {
                cudaGetLastError();
                return SDCA_E_CUDA;
            }
            scratch = static_cast<double *>(p);
            if (!have_id) have_id = current_context_id(&id);
            if (have_id && g_na_ptr.size() < 256) g_na_ptr.emplace_back(id, scratch);
        }
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    double *nb = scratch;
    // Logits: slices of the loci x blocks of up to 1024 sequences, three blocks
    // per SM.  The slices' sums (4 n_seqs doubles each) go to g, whose values
    // overwrite them afterwards; where g has no room for two, one slice goes
    // to the beliefs' own place.  A g that overlaps x or the weights must not
    // be written before these have been read: then as many slices as the
    // scratch array holds, the first in the beliefs' place.
    const auto apart = [](const double *a, int64_t na, const double *b, int64_t nb_) {
        const uintptr_t a0 = reinterpret_cast<uintptr_t>(a), b0 = reinterpret_cast<uintptr_t>(b);
        return a0 + 8 * (uintptr_t)na <= b0 || b0 + 8 * (uintptr_t)nb_ <= a0;
    };
    const int64_t params = 16 * n_loci + 4;
    const bool in_g = apart(g, params, x, params) && apart(g, params, weights, n_seqs);
    const int spt = (int)std::min<int64_t>(NA_MAX_SPT, (n_seqs + NA_THREADS - 1) / NA_THREADS);
    const int64_t seq_blocks = (n_seqs + (int64_t)NA_THREADS * spt - 1) / ((int64_t)NA_THREADS * spt);
    const int64_t steps = (n_loci + NA_STEP - 1) / NA_STEP;
    const int64_t fit = in_g ? params / (4 * n_seqs) : NA_MAX_SEQS / n_seqs;
    int64_t slices = std::min({std::max<int64_t>(1, 456 / seq_blocks), steps, fit});
    double *part = in_g ? g : nb;
    if (slices < 2) {
        slices = 1;
        part = nb;
    }
    const dim3 gl((unsigned)slices, (unsigned)seq_blocks);
    switch (spt) {
    case 1: k_na_logits<1><<<gl, NA_THREADS, 0, st>>>(states, n_seqs, n_loci, r, x, part, scratch); break;
    case 2: k_na_logits<2><<<gl, NA_THREADS, 0, st>>>(states, n_seqs, n_loci, r, x, part, scratch); break;
    case 3: k_na_logits<3><<<gl, NA_THREADS, 0, st>>>(states, n_seqs, n_loci, r, x, part, scratch); break;
    default: k_na_logits<4><<<gl, NA_THREADS, 0, st>>>(states, n_seqs, n_loci, r, x, part, scratch); break;
    }
    const int nb1 = (int)std::min<int64_t>(NA_MAX_BLOCKS, (n_seqs + NA_THREADS / 32 - 1) / (NA_THREADS / 32));
    k_na_beliefs<<<nb1, NA_THREADS, 0, st>>>(states, n_seqs, n_loci, r, weights, x, (int)slices, part, nb, scratch);
    // Gradient: 448 loci per block; with few loci the sequences are shared
    // out too, as far as the scratch array behind the beliefs holds the
    // shares' sums (16 n_loci doubles each).
    const int64_t gx = (n_loci + NG_THREADS * NG_LOCI - 1) / (NG_THREADS * NG_LOCI);
    const int64_t room = (NA_MAX_SEQS * 4 - 4 * n_seqs) / (16 * n_loci);
    int64_t shares = std::min({152 / gx, (n_seqs + NG_SEQS - 1) / NG_SEQS, room});
    int nb2 = (int)gx;
    if (shares < 2) {
        k_na_gradient<<<dim3((unsigned)gx, 1), NG_THREADS, 0, st>>>(states, n_seqs, n_loci, r, lambda_J, x, g, nullptr, nb,
                                                                    scratch);
    } else {
        double *gp = scratch + 4 * n_seqs;
        k_na_gradient<<<dim3((unsigned)gx, (unsigned)shares), NG_THREADS, 0, st>>>(states, n_seqs, n_loci, r, lambda_J, x,
                                                                                   g, gp, nb, scratch);
        nb2 = (int)std::min<int64_t>(NA_MAX_BLOCKS, (16 * n_loci + NA_THREADS - 1) / NA_THREADS);
        k_na_gradient_sum<<<nb2, NA_THREADS, 0, st>>>(n_loci, r, lambda_J, (int)shares, gp, x, g, scratch);
    }
    k_na_total<<<1, NA_THREADS, 0, st>>>(n_loci, nb1, nb2, lambda_h, x, f, g, scratch);
    return cudaGetLastError() == cudaSuccess ? SDCA_OK : SDCA_E_CUDA;
}
