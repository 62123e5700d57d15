// quotient.h -- FP64 quotients from one reciprocal.
#pragma once

#include <math.h>

#ifdef __CUDACC__
#define SDCA_HD_Q __host__ __device__
#else
#define SDCA_HD_Q
#endif

namespace sdca {

// v / z from rz = 1 / z correctly rounded: a first quotient and the
// correction by its remainder (Markstein, IBM J. Res. Dev. 34(1), 1990).
// Three operations where a division on GB300 is a long chain of FP64
// instructions, for quotients that share a divisor.  For z in [1, 4] it
// gave the bits of the division for every pair tried with |v| >= 2^-960
// (tests/test_quotient.py has the hardest kinds).  Below that the remainder
// underflows and the result may be one unit in the last place off: a softmax
// weight that small does not reach an FP32 residual or an FP64 sum over
// sequences.
SDCA_HD_Q inline double quotient_by(double v, double z, double rz)
{
    const double q = v * rz;
    return fma(fma(-q, z, v), rz, q);
}

} // namespace sdca
