// Where a particle's stencils lie on one axis of G2P's shared-memory tile. Plain C++ besides the qualifiers, so that the
// arithmetic can be checked on the host for positions that no tank produces (infinite, far away).
#pragma once

#if defined(__CUDACC__)
#define SLOSH_HD __host__ __device__ __forceinline__
#else
#define SLOSH_HD inline
#endif

namespace slosh {

// b0, b1: the first nodes of the stencils for a face on the axis and beside it (b1 is b0 or b0 - 1; saturated integers for
// far positions); the tile has the n nodes from o on, o + n below 2^30. True when both stencils' nodes lie in the tile; local
// then holds the first nodes' places in it. The differences are taken modulo 2^32, where b0's of any node outside the tile is
// at least n - 1.
SLOSH_HD bool tile_axis(int b0, int b1, int o, int n, int (&local)[2]) {
    local[0] = int(unsigned(b0) - unsigned(o));
    local[1] = int(unsigned(b1) - unsigned(o));
    return local[1] >= 0 && unsigned(local[0]) < unsigned(n - 1);  // the stencil beside starts no later and ends no later
}

}  // namespace slosh
