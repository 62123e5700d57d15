// kdig.cuh -- the digit layout of the exact K rho product (k_kdig in
// kernels_tc.cu), which the residual quantiser (kernels_dual.cu) writes.
#pragma once

#include <cstdint>

#include <cuda_fp16.h>

namespace sdca {
namespace tc {

constexpr int KD_KDIG = 3, KD_RDIG = 3;      // digits of K and of rho
constexpr int KD_S = 17;                     // slots per tile
constexpr int KD_C = 3;                      // product columns per slot (the fourth follows)
constexpr int KD_PS = 52;                    // rows (accumulator columns) from one plane to the next
constexpr int KD_NB = 160;                   // rho rows of a tile: accumulator columns per K digit
constexpr int KD_RBASE = 640, KD_RHALF = 320;

} // namespace tc

// Sequence j of list position P: the first three columns of rho_q as fp16
// balanced base-640 digits, plane p of column c in row 52 p + 3 (P % 17) + c
// of tile P / 17.
__device__ __forceinline__ void kd_digits(int P, int64_t j, int64_t Nx, int4 q, __half *__restrict__ Rd)
{
    using namespace tc;
    const int64_t row0 = (int64_t)(P / KD_S) * KD_NB + (P % KD_S) * KD_C;
    const int qq[KD_C] = {q.x, q.y, q.z};
#pragma unroll
    for (int c = 0; c < KD_C; ++c) {
        int v = qq[c];
#pragma unroll
        for (int p = 0; p < KD_RDIG; ++p) {
            int d = v;
            if (p < KD_RDIG - 1) {
                // |v| < 2^28: shifted by a multiple of the base to be positive
                constexpr int UP = (1 << 28) / KD_RBASE;
                const unsigned t = (unsigned)(v + KD_RHALF) + (unsigned)(UP * KD_RBASE);
                const unsigned qt = t / KD_RBASE;
                d = (int)(t - qt * KD_RBASE) - KD_RHALF;
                v = (int)qt - UP;
            }
            Rd[(row0 + p * KD_PS + c) * Nx + j] = __int2half_rn(d);
        }
    }
}

} // namespace sdca
