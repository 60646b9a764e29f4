// A correctly rounded quotient from a stored reciprocal. Plain C++ besides the qualifiers, so that it can be checked against
// division on the host and on the GPU.
#pragma once

#include <cmath>

#if defined(__CUDACC__)
#define SLOSH_HD __host__ __device__ __forceinline__
#else
#define SLOSH_HD inline
#endif

namespace slosh {

SLOSH_HD float exact_fma(float a, float b, float c) {
#if defined(__CUDA_ARCH__)
    return __fmaf_rn(a, b, c);
#else
    return fmaf(a, b, c);
#endif
}
// a / d correctly rounded, rc = the correctly rounded 1 / d (Markstein's theorem, IBM J. Res. Dev. 34 (1), 1990: a
// faithful quotient corrected once by its exact remainder times rc is the rounded quotient; the first correction makes
// the product faithful). Five dependent operations where the division takes about 200 cycles. The remainders are exact
// only away from the ends of the exponent range: outside [1e-25, 1e25] the division itself. d: 1e-5 to 1e5.
SLOSH_HD float div_by(float a, float d, float rc) {
    const float m = fabsf(a);
    if (!(m >= 1e-25f && m <= 1e25f)) return a == 0.0f ? a * rc : a / d;
    float q = a * rc;
    q = exact_fma(exact_fma(-q, d, a), rc, q);
    return exact_fma(exact_fma(-q, d, a), rc, q);
}

}  // namespace slosh
