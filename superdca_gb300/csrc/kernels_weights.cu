// kernels_weights.cu -- sequence reweighting on the GPU.
//
// SuperDCA's calculate_weights (SuperDCA/include/plmDCA_optimizer_parameters.hpp:
// 39-98) gives sequence i the weight mult_i / (mult_i + sum of mult_j over
// the other sequences j with identity (L - d_ij) / L >= threshold), d_ij
// the number of loci whose states differ.  That is N^2/2 Hamming distances
// over L loci (4.5 million pairs x 94,000 loci at 3000 x 94,000).
//
// Here the states are packed as two bit planes, 32 loci in the low and high
// word of a 64-bit value; a pair differs at the bits of
// (lo ^ lo') | (hi ^ hi').  Counting those bits is what costs: the population
// count runs at 16 per cycle and SM, an eighth of the logic operations.  So
// two words at a time go through a carry-save adder with the pair's running
// parity word, and only the carries are counted, half as many: 3 logic
// operations and half a count per 32 loci and pair (two counts and ten other
// operations before, on packed pairs of bits).  A CTA owns a square block of
// the lower triangle of the pair matrix, streams both sequence blocks through
// shared memory 32 words at a time and keeps R x R pairs per thread in
// registers.  All pairs of 3000 x 94,000: 2.8 ms (7.7 before).
// Distances are exact integers and the identity test is the reference's
// double comparison, so the weights are bit-identical.
#include <cstdint>

#include "engine.h"
#include "kernels_common.cuh"

namespace sdca {
namespace {

constexpr int WCH = 32;     // words per shared-memory chunk
constexpr int WROW = WCH + 2;   // row stride: 16-byte reads of 8 rows fall in distinct banks

// bit k of byte b of a 4-byte word of states, for b = 0..3, as 4 bits
__device__ __forceinline__ uint32_t plane4(uint32_t w, int k)
{
    return (((w >> k) & 0x01010101u) * 0x08040201u) >> 24 & 15u;
}

// states [N][ld] u8 (ld a multiple of 32, zero past the last locus) -> packed
// [N][W] words of 32 loci, planes in the low and high halves
__global__ void k_pack2(const uint8_t *__restrict__ X, int64_t ld, int N, int64_t W, uint2 *__restrict__ packed)
{
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (int64_t)N * W) return;
    const int64_t i = t / W, w = t - i * W;
    uint32_t lo = 0, hi = 0;
    if (w * 32 < ld) {
        const uint4 *row = reinterpret_cast<const uint4 *>(X + i * ld + w * 32);
        const uint4 u = row[0], v = row[1];
        const uint32_t c[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            lo |= plane4(c[k], 0) << (4 * k);
            hi |= plane4(c[k], 1) << (4 * k);
        }
    }
    packed[t] = make_uint2(lo, hi);
}

// DIST: write base + sign d of every pair (both orders, rows of ld values)
// instead of adding to the neighbour sums of the pairs with d <= d_max
template <bool DIST, int R>
__global__ void __launch_bounds__(256)
k_pair_neighbours(const uint2 *__restrict__ packed, int N, int64_t W, int d_max, const double *__restrict__ mult,
                  double *__restrict__ nbr, int base, int sign, int64_t ld, int32_t *__restrict__ dist)
{
    constexpr int WT = 16 * R;   // sequences per tile side
    // lower-triangle tile index -> (ti, tj) with tj <= ti
    const int64_t tid = blockIdx.x;
    int ti = (int)((sqrt(8.0 * (double)tid + 1.0) - 1.0) / 2.0);
    while ((int64_t)ti * (ti + 1) / 2 > tid) --ti;
    while ((int64_t)(ti + 1) * (ti + 2) / 2 <= tid) ++ti;
    const int tj = (int)(tid - (int64_t)ti * (ti + 1) / 2);
    const int i0 = ti * WT, j0 = tj * WT;

    __shared__ __align__(16) uint2 sa[WT][WROW];
    __shared__ __align__(16) uint2 sb[WT][WROW];
    // 16 x 16 threads, R x R pairs each; rows interleaved by 16
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    uint32_t one[R][R];   // parity of each bit so far
    int d[R][R];          // carries counted, each worth 2
#pragma unroll
    for (int a = 0; a < R; ++a)
#pragma unroll
        for (int b = 0; b < R; ++b) {
            one[a][b] = 0u;
            d[a][b] = 0;
        }

    // (W is even: 16-byte loads of two words)
    for (int64_t w0 = 0; w0 < W; w0 += WCH) {
#pragma unroll
        for (int k = threadIdx.x; k < WT * (WCH / 2); k += 256) {
            const int r = k / (WCH / 2), c = 2 * (k % (WCH / 2));
            const int64_t w = w0 + c;
            const int ia = i0 + r, jb = j0 + r;
            const uint4 z = make_uint4(0u, 0u, 0u, 0u);
            *reinterpret_cast<uint4 *>(&sa[r][c]) =
                (ia < N && w < W) ? *reinterpret_cast<const uint4 *>(packed + (int64_t)ia * W + w) : z;
            *reinterpret_cast<uint4 *>(&sb[r][c]) =
                (jb < N && w < W) ? *reinterpret_cast<const uint4 *>(packed + (int64_t)jb * W + w) : z;
        }
        __syncthreads();
#pragma unroll 2
        for (int c = 0; c < WCH; c += 2) {
            uint4 av[R], bv[R];
#pragma unroll
            for (int a = 0; a < R; ++a) av[a] = *reinterpret_cast<const uint4 *>(&sa[ty + 16 * a][c]);
#pragma unroll
            for (int b = 0; b < R; ++b) bv[b] = *reinterpret_cast<const uint4 *>(&sb[tx + 16 * b][c]);
#pragma unroll
            for (int a = 0; a < R; ++a)
#pragma unroll
                for (int b = 0; b < R; ++b) {
                    const uint32_t x = (av[a].x ^ bv[b].x) | (av[a].y ^ bv[b].y);
                    const uint32_t y = (av[a].z ^ bv[b].z) | (av[a].w ^ bv[b].w);
                    const uint32_t o = one[a][b];
                    d[a][b] += __popc((o & x) | (o & y) | (x & y));
                    one[a][b] = o ^ x ^ y;
                }
        }
        __syncthreads();
    }
#pragma unroll
    for (int a = 0; a < R; ++a)
#pragma unroll
        for (int b = 0; b < R; ++b) d[a][b] = 2 * d[a][b] + __popc(one[a][b]);
    if (DIST) {
#pragma unroll
        for (int a = 0; a < R; ++a) {
            const int i = i0 + ty + 16 * a;
            if (i >= N) continue;
#pragma unroll
            for (int b = 0; b < R; ++b) {
                const int j = j0 + tx + 16 * b;
                if (j > i) continue;
                const int v = base + sign * d[a][b];
                dist[(int64_t)i * ld + j] = v;
                dist[(int64_t)j * ld + i] = v;
            }
        }
        return;
    }
    // neighbours' multiplicities, summed over the warp's 16 x 2 threads of a
    // row (column) before the atomics; most blocks have no neighbours
    bool near[R][R], any = false;
#pragma unroll
    for (int a = 0; a < R; ++a)
#pragma unroll
        for (int b = 0; b < R; ++b) {
            const int i = i0 + ty + 16 * a, j = j0 + tx + 16 * b;
            near[a][b] = i < N && j < i && d[a][b] <= d_max;   // pairs j < i, as the reference loops
            any = any || near[a][b];
        }
    if (!__any_sync(0xffffffffu, any)) return;
#pragma unroll
    for (int a = 0; a < R; ++a) {
        double v = 0.0;
#pragma unroll
        for (int b = 0; b < R; ++b)
            if (near[a][b]) v += mult ? mult[j0 + tx + 16 * b] : 1.0;
        for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (tx == 0 && v != 0.0) atomicAdd(nbr + i0 + ty + 16 * a, v);
    }
#pragma unroll
    for (int b = 0; b < R; ++b) {
        double v = 0.0;
#pragma unroll
        for (int a = 0; a < R; ++a)
            if (near[a][b]) v += mult ? mult[i0 + ty + 16 * a] : 1.0;
        v += __shfl_xor_sync(0xffffffffu, v, 16);
        if ((threadIdx.x & 16) == 0 && v != 0.0) atomicAdd(nbr + j0 + tx + 16 * b, v);
    }
}

// Pair blocks of 64 x 64 sequences, or of 32 x 32 when those would leave SMs
// idle (1000 x 4001: 136 blocks against 528, 25 us a pass instead of 57 to 85 with the larger ones and a count for every word).
template <bool DIST>
void launch_pairs(const uint64_t *packed, int N, int64_t W, int d_max, const double *mult, double *nbr, int base, int sign,
                  int64_t ld, int32_t *dist, cudaStream_t st)
{
    const uint2 *p = reinterpret_cast<const uint2 *>(packed);
    const int64_t nt = (N + 63) / 64, nt2 = (N + 31) / 32;
    const int64_t tiles = nt * (nt + 1) / 2, tiles2 = nt2 * (nt2 + 1) / 2;
    if (tiles >= 2 * 152)
        k_pair_neighbours<DIST, 4><<<(unsigned)tiles, 256, 0, st>>>(p, N, W, d_max, mult, nbr, base, sign, ld, dist);
    else
        k_pair_neighbours<DIST, 2><<<(unsigned)tiles2, 256, 0, st>>>(p, N, W, d_max, mult, nbr, base, sign, ld, dist);
}

// The largest distance whose identity (L - d) / L reaches the threshold by
// the reference's double comparison (the quotient falls as d grows), -1 if
// none does: the kernel compares integers instead of dividing for each pair.
int largest_distance(int L, double threshold)
{
    int lo = -1, hi = L;   // lo reaches it (or is -1), everything above hi does not
    while (lo < hi) {
        const int d = lo + (hi - lo + 1) / 2;
        if ((double)(L - d) / (double)L >= threshold) lo = d;
        else hi = d - 1;
    }
    return lo;
}

void launch_pack(const uint8_t *X, int64_t ld, int N, int64_t W, uint64_t *packed, cudaStream_t st)
{
    const int64_t total = (int64_t)N * W;
    k_pack2<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(X, ld, N, W, reinterpret_cast<uint2 *>(packed));
}

} // namespace

// words of 32 loci per packed sequence (even, for 16-byte loads)
int64_t packed_words(int64_t L) { return (L + 63) / 64 * 2; }

void launch_weights(const uint8_t *X, int64_t ld, int N, int L, uint64_t *packed, double threshold,
                    const double *mult, double *nbr, cudaStream_t st)
{
    const int64_t W = packed_words(L);
    launch_pack(X, ld, N, W, packed, st);
    launch_pairs<false>(packed, N, W, largest_distance(L, threshold), mult, nbr, 0, 0, 0, nullptr, st);
}

// the full N x N matrix of differing-locus counts (diagonal 0)
void launch_distances(const uint8_t *X, int64_t ld, int N, int L, uint64_t *packed, int32_t *dist, cudaStream_t st)
{
    const int64_t W = packed_words(L);
    launch_pack(X, ld, N, W, packed, st);
    launch_pairs<true>(packed, N, W, 0, nullptr, nullptr, 0, 1, N, dist, st);
}

// the N x N agreement counts L - d in rows of ld values
void launch_agreements(const uint8_t *X, int64_t ldx, int N, int L, uint64_t *packed, int32_t *K, int64_t ld,
                       cudaStream_t st)
{
    const int64_t W = packed_words(L);
    launch_pack(X, ldx, N, W, packed, st);
    launch_pairs<true>(packed, N, W, 0, nullptr, nullptr, L, -1, ld, K, st);
}

} // namespace sdca
