// Where a particle's stencils lie on one axis of G2P's shared-memory tile. Plain C++ besides the qualifiers, so that the
// arithmetic can be checked on the host for positions that no tank produces (infinite, far away).
#pragma once

#if defined(__CUDACC__)
#define SLOSH_HD __host__ __device__ __forceinline__
#else
#define SLOSH_HD inline
#endif

namespace slosh {

// The place of node b in a tile that starts at node o, modulo 2^32: of a far position b has saturated, and b - o may wrap.
SLOSH_HD int tile_place(int b, int o) { return int(unsigned(b) - unsigned(o)); }
// Whether both stencils' nodes lie in the tile of n nodes; l0, l1: the places of the first nodes of the stencils for a face on
// the axis and beside it, which are nodes b and b, or b and b - 1 within +-2^30 (farther out half a cell changes no float). With
// o + n below 2^30 a place that wraps comes out above every n, which fails the second test.
SLOSH_HD bool tile_holds(int l0, int l1, int n) { return l1 >= 0 && l0 < n - 1; }

}  // namespace slosh
