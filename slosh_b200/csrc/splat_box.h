// The voxels that a particle's kernel visits along one axis of the density field. Plain C++ besides the qualifiers,
// so that the arithmetic can be checked on the host for positions that no tank produces (infinite, NaN, far away).
#pragma once

#include <cmath>

#if defined(__CUDACC__)
#define SLOSH_HD __host__ __device__ __forceinline__
#else
#define SLOSH_HD inline
#endif

namespace slosh {

// Rounded down and up to an integer; the GPU's conversions saturate (NaN: 0).
SLOSH_HD int splat_floor(float x) {
#if defined(__CUDA_ARCH__)
    return __float2int_rd(x);
#else
    return x != x ? 0 : (x >= 2147483648.0f ? 2147483647 : (x < -2147483648.0f ? -2147483647 - 1 : int(floorf(x))));
#endif
}
SLOSH_HD int splat_ceil(float x) {
#if defined(__CUDA_ARCH__)
    return __float2int_ru(x);
#else
    return x != x ? 0 : (x >= 2147483648.0f ? 2147483647 : (x < -2147483648.0f ? -2147483647 - 1 : int(ceilf(x))));
#endif
}

struct SplatSpan {
    int lo, hi;  // empty when lo > hi
};
// c: the particle in voxels; rr: the kernel's radius; n: voxels of the axis. The reference's span reaches one voxel beyond
// the kernel on each side; where the kernel is whole (not cut by the footprint) those, more than 1e-3 radii outside, fail
// the distance test and are left out. An empty span is left as it is: of a far or infinite position it may end at the
// largest or smallest integer, which one voxel more would wrap, turning the span into one of 2^32 voxels.
SLOSH_HD SplatSpan splat_span(float c, float rr, int n, bool whole) {
    SplatSpan s;
    s.lo = splat_floor(c - rr - 0.5f);
    s.hi = splat_ceil(c + rr - 0.5f);
    s.lo = s.lo > 0 ? s.lo : 0;
    s.hi = s.hi < n - 1 ? s.hi : n - 1;
    if (whole && s.lo <= s.hi) {
        const float far = rr * 1.001f;  // the test squares this same difference times 1 / rr
        const int up = (float(s.lo) + 0.5f) - c < -far ? 1 : 0, down = (float(s.hi) + 0.5f) - c > far ? 1 : 0;
        s.lo += up;
        s.hi -= down;
    }
    return s;
}

}  // namespace slosh
