// Headless liquid surface from the particles (sm_100a): density splat, field resolve and surface nets,
// written into device buffers (no window, swapchain or graphics API).
//
// Reference: PLUG/Shaders/Private/SloshSurface.usf -- DensitySplatCS (:54-100), FieldResolveCS (:109-149),
// SampleField/FieldGradient (:154-165), SurfaceNetsVerticesCS (:330-399), SurfaceNetsFacesCS (:401-458),
// SurfaceNetsArgsCS (:460-470); ellipsoids from AnisoComputeCS (SloshRender.usf:281-376) in sphere mode
// (AnisoStrength 0: centre = particle position, axes = splat radius along x, y and z); parameters as
// BuildDensityField / FillFieldParameters set them (PLUG/Source/SloshRender/Private/SloshRenderer.cpp:118-170).
//
// Same arithmetic as the reference; deliberate differences, identical in the CPU restatement:
//   * vertices and quads are numbered in cell order (flags, exclusive scan, write), not in the order in which
//     atomic counters hand out slots, so the mesh is deterministic;
//   * the field gradient of a vertex normal samples the f16 field by exact FP32 trilinear interpolation with
//     clamped addressing (the reference uses the texture unit's filter);
//   * normalize(v) is v / sqrt(dot(v, v)); positions are in sim metres (voxel centre v at v + 0.5 voxels).
#include <cuda_fp16.h>

#include "kernels.h"
#include "splat_box.h"

namespace slosh {

namespace {

constexpr float FIELD_W_FIXED = 1024.0f, FIELD_X_FIXED = 256.0f;
constexpr uint32_t FIELD_MOMENTS = 5u, NO_VERTEX = 0xFFFFFFFFu;
constexpr int SURF_THREADS = 256;

__device__ __forceinline__ uint32_t voxel_index(const SurfaceDev& s, int3 v) { return uint32_t(v.x + s.dim.x * (v.y + s.dim.y * v.z)); }
__device__ __forceinline__ uint32_t field_brick(const SurfaceDev& s, int3 v) {
    const int bx = min(max(v.x >> 3, 0), s.bdim.x - 1), by = min(max(v.y >> 3, 0), s.bdim.y - 1), bz = min(max(v.z >> 3, 0), s.bdim.z - 1);
    return uint32_t(bx + s.bdim.x * (by + s.bdim.y * bz));
}
__device__ __forceinline__ uint32_t cell_of(const SurfaceDev& s, int3 c) {
    return uint32_t(c.x + (s.dim.x - 1) * (c.y + (s.dim.y - 1) * c.z));
}
__device__ __forceinline__ int3 cell_coord(const SurfaceDev& s, uint32_t i) {
    const uint32_t cx = uint32_t(s.dim.x - 1), cy = uint32_t(s.dim.y - 1);
    return make_int3(int(i % cx), int((i / cx) % cy), int(i / (cx * cy)));
}
__device__ __forceinline__ float field_at(const SurfaceDev& s, int3 v) {
    return __half2float(__ushort_as_half(s.field[voxel_index(s, v)]));
}
__device__ __forceinline__ float dot3f(float3 a, float3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }

// ---- DensitySplatCS ------------------------------------------------------------------------------------------
// Five fixed-point moments (weight, weighted offset to the particle, weighted radius) per voxel of a particle's
// kernel: integer sums, exact in any order. The kernel is a sphere, so the squared distance in kernel radii separates
// into one square per axis: q2 = (x^2 + y^2) + z^2, the reference's three dot products with their zero terms left
// out (adding a zero changes no bit of a square); a row of voxels with y^2 + z^2 >= 1 has no voxel inside, because
// rounding is monotonic.
// One CTA takes PER x 256 consecutive (spatially sorted) particles, adds their moments into a shared-memory tile
// over the bounding box of their kernels and adds each non-zero tile word to global memory once. A box larger than
// the tile is visited in slabs of whole z planes (every particle adds the rows of its kernel that lie in the slab);
// more than SPLAT_MAX_SLABS slabs (particles in no spatial order) add straight to global memory.
// Bound by the global atomics before (7.2 voxels x 5 moments a particle at the default kernel), by issue now; a slab
// more costs a second walk over the particles, which is why a box of several tiles still takes them. Measured for
// 8.2 M particles in 160^3 voxels, the default kernel: 1,857 us with global atomics, 529 with the tile, 467 with the
// voxels taken from a mask, about 375 with the 27 tests of a small kernel from nine squares. A field with its mesh:
// 2,349 -> 632 us there, 366 -> 182 us for 64 x 64 x 48 voxels and 0.7 M particles. 4 CTAs per SM (64 registers);
// 1 particle per thread (at this size) or a tile of 1,536 voxels took 655 us, 4 per thread in CTAs of 128 took 706, chunks of 2,048
// and 4,096 particles (before the small kernel's form) 904 and 953 against 726: too few warps in flight.
constexpr int SPLAT_THREADS = 256;
constexpr int SPLAT_CTAS = 4;  // per SM
constexpr int SPLAT_TILE = 2048;                               // voxels: 40 KB
constexpr int SPLAT_SMEM = SPLAT_TILE * int(FIELD_MOMENTS) * 4;
template <int PER> constexpr int SPLAT_MAX_SLABS = PER == 1 ? 4 : 8;

struct SplatKernel {
    float3 c;  // the particle in voxels
    int3 lo, hi;
};
struct SplatShape {
    float w, reach;  // 1 / kernel radius (voxels) as the reference forms it, and the radius clamped to the footprint
    bool whole;      // neither the footprint nor the smallest radius cuts the kernel
    bool three;      // whole, and at most 3 voxels an axis
    bool small;      // every moment is below 2^22: rounded by adding 1.5 x 2^23 instead of converted
};
__device__ __forceinline__ SplatShape splat_shape(const SurfaceDev& s) {
    const float u = s.splat_radius * (s.support * s.inv_voxel);
    const float aa = fmaxf(u * u, 1e-8f);
    SplatShape h;
    h.w = u / aa;
    h.reach = fminf(sqrtf(aa), s.max_footprint);
    h.whole = u * u >= 1e-8f && sqrtf(aa) <= s.max_footprint;  // w = 1 / reach
    h.three = h.whole && 2.0f * 1.002f * h.reach < 3.0f;  // the cut box spans less than 3 voxels
    h.small = fabsf(s.radius_voxels) < 8192.0f;
    return h;
}
// The voxels a particle visits (splat_span): 2-3 voxels an axis instead of the reference's 4-5 at the default kernel.
__device__ __forceinline__ SplatKernel splat_kernel(const SurfaceDev& s, const SplatShape& h, float4 a) {
    SplatKernel k;
    k.c = make_float3(a.x * s.inv_voxel, a.y * s.inv_voxel, a.z * s.inv_voxel);
    const SplatSpan x = splat_span(k.c.x, h.reach, s.dim.x, h.whole), y = splat_span(k.c.y, h.reach, s.dim.y, h.whole),
                    z = splat_span(k.c.z, h.reach, s.dim.z, h.whole);
    k.lo = make_int3(x.lo, y.lo, z.lo);
    k.hi = make_int3(x.hi, y.hi, z.hi);
    return k;
}
// x rounded to the nearest integer (ties to even) for |x| < 2^22, and cut to an integer for 0 <= x < 2^22: the sum
// with a power of two leaves the integer in the low mantissa bits. The conversion instruction gives the same value at
// a quarter of the issue rate of an addition.
__device__ __forceinline__ int32_t small_rn(float x) { return __float_as_int(x + 12582912.0f) - 0x4B400000; }
__device__ __forceinline__ int32_t small_rz(float x) { return __float_as_int(__fadd_rz(x, 8388608.0f)) - 0x4B000000; }
__device__ __forceinline__ void splat_moments(const SurfaceDev& s, const SplatShape& h, float dx, float dy, float dz, float q2, int32_t m[5]) {
    float wk = 1.0f - q2;
    wk = wk * wk * wk;
    const float wx = wk * FIELD_X_FIXED;  // a power of two: dx wx is the reference's (dx wk) scaled, bit for bit
    if (h.small) {
        m[0] = small_rz(wk * FIELD_W_FIXED + 0.5f);
        m[1] = small_rn(-(dx * wx));
        m[2] = small_rn(-(dy * wx));
        m[3] = small_rn(-(dz * wx));
        m[4] = small_rn(s.radius_voxels * wx);
    } else {
        m[0] = __float2int_rz(wk * FIELD_W_FIXED + 0.5f);
        m[1] = __float2int_rn(-(dx * wx));
        m[2] = __float2int_rn(-(dy * wx));
        m[3] = __float2int_rn(-(dz * wx));
        m[4] = __float2int_rn(s.radius_voxels * wx);
    }
}
// splat_voxels for a kernel of at most 3 voxels an axis (SplatShape::three): the 27 tests are sums of nine squares
// computed once; a voxel past the box, or outside [z0, z1], gets a square of 2.
template <class Add>
__device__ __forceinline__ void splat_voxels3(const SurfaceDev& s, const SplatShape& h, const SplatKernel& k, int z0, int z1, Add add) {
    const float w = h.w;
    float dx[3], dy[3], dz[3], xx[3], yy[3], zz[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        dx[j] = (float(k.lo.x + j) + 0.5f) - k.c.x;
        dy[j] = (float(k.lo.y + j) + 0.5f) - k.c.y;
        dz[j] = (float(k.lo.z + j) + 0.5f) - k.c.z;
        const float qx = dx[j] * w, qy = dy[j] * w, qz = dz[j] * w;
        xx[j] = k.lo.x + j <= k.hi.x ? qx * qx : 2.0f;
        yy[j] = k.lo.y + j <= k.hi.y ? qy * qy : 2.0f;
        zz[j] = k.lo.z + j <= k.hi.z && k.lo.z + j >= z0 && k.lo.z + j <= z1 ? qz * qz : 2.0f;
    }
    uint32_t mask = 0u;
#pragma unroll
    for (int y = 0; y < 3; ++y)
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            const float xy = xx[x] + yy[y];
#pragma unroll
            for (int z = 0; z < 3; ++z)
                if (xy + zz[z] < 1.0f) mask |= 1u << (x + 3 * y + 9 * z);
        }
    while (mask != 0u) {
        const uint32_t b = uint32_t(__ffs(int(mask))) - 1u;
        mask &= mask - 1u;
        const uint32_t bz = (b * 57u) >> 9, r = b - 9u * bz, by = (r * 11u) >> 5, bx = r - 3u * by;  // exact for b < 27
        const float ex = bx == 0u ? dx[0] : (bx == 1u ? dx[1] : dx[2]);
        const float ey = by == 0u ? dy[0] : (by == 1u ? dy[1] : dy[2]);
        const float ez = bz == 0u ? dz[0] : (bz == 1u ? dz[1] : dz[2]);
        const float qx = ex * w, qy = ey * w, qz = ez * w;
        int32_t m[5];
        splat_moments(s, h, ex, ey, ez, (qx * qx + qy * qy) + qz * qz, m);
        add(k.lo.x + int(bx), k.lo.y + int(by), k.lo.z + int(bz), m);
    }
}
// add(x, y, z, moments) for every voxel of the kernel whose z lies in [z0, z1]. Up to 32 voxels of the box at a time
// (whole z planes of it) are tested first and the voxels inside then taken from the bits of the mask: the lanes of a
// warp walk their 7 or so voxels side by side, where the nested loops ran the moments for each of the box's voxels in
// which any lane had one.
template <class Add>
__device__ __forceinline__ void splat_voxels(const SurfaceDev& s, const SplatShape& h, const SplatKernel& k, int z0, int z1, Add add) {
    if (h.three) {
        splat_voxels3(s, h, k, z0, z1, add);
        return;
    }
    const float w = h.w;
    const int nx = k.hi.x - k.lo.x + 1, ny = k.hi.y - k.lo.y + 1, per = nx * ny;
    const int zb = max(k.lo.z, z0), ze = min(k.hi.z, z1);
    if (per <= 32) {
        const int group = 32 / per;
        const uint32_t inv_per = 65536u / uint32_t(per) + 1u, inv_nx = 65536u / uint32_t(nx) + 1u;  // exact for bits < 32
        for (int z = zb; z <= ze; z += group) {
            uint32_t mask = 0u;
            int bit = 0;
            for (int g = z; g < z + group && g <= ze; ++g) {
                const float dz = (float(g) + 0.5f) - k.c.z, qz = dz * w, zz = qz * qz;
                for (int y = k.lo.y; y <= k.hi.y; ++y) {
                    const float dy = (float(y) + 0.5f) - k.c.y, qy = dy * w, yy = qy * qy;
                    for (int x = k.lo.x; x <= k.hi.x; ++x, ++bit) {
                        const float dx = (float(x) + 0.5f) - k.c.x, qx = dx * w;
                        if ((qx * qx + yy) + zz < 1.0f) mask |= 1u << bit;
                    }
                }
            }
            while (mask != 0u) {
                const uint32_t b = uint32_t(__ffs(int(mask))) - 1u;
                mask &= mask - 1u;
                const uint32_t bz = (b * inv_per) >> 16, r = b - bz * uint32_t(per), by = (r * inv_nx) >> 16, bx = r - by * uint32_t(nx);
                const int x = k.lo.x + int(bx), y = k.lo.y + int(by), zv = z + int(bz);
                const float dx = (float(x) + 0.5f) - k.c.x, dy = (float(y) + 0.5f) - k.c.y, dz = (float(zv) + 0.5f) - k.c.z;
                const float qx = dx * w, qy = dy * w, qz = dz * w;
                int32_t m[5];
                splat_moments(s, h, dx, dy, dz, (qx * qx + qy * qy) + qz * qz, m);
                add(x, y, zv, m);
            }
        }
        return;
    }
    for (int z = zb; z <= ze; ++z) {
        const float dz = (float(z) + 0.5f) - k.c.z, qz = dz * w, zz = qz * qz;
        for (int y = k.lo.y; y <= k.hi.y; ++y) {
            const float dy = (float(y) + 0.5f) - k.c.y, qy = dy * w, yy = qy * qy;
            if (yy + zz >= 1.0f) continue;
            for (int x = k.lo.x; x <= k.hi.x; ++x) {
                const float dx = (float(x) + 0.5f) - k.c.x, qx = dx * w;
                const float q2 = (qx * qx + yy) + zz;
                if (!(q2 < 1.0f)) continue;
                int32_t m[5];
                splat_moments(s, h, dx, dy, dz, q2, m);
                add(x, y, z, m);
            }
        }
    }
}
// PER: particles per thread. 2 (a CTA's 512 are about one 4^3 sort key of 8 a cell) for many; 1 while all of those CTAs run at
// once, where a second particle, or a fifth slab, is only a longer chain. A field alone, us with global atomics, with 2 per
// thread, with 1 (and 8 slabs): 2,000 records all over 64^3 voxels, smoothing 6, 224, 348, 199; 20,000 in a sorted sheet, 96^3
// voxels, smoothing 3, 143, 276, 104 (165); 100,000 sorted, 64^3 voxels, smoothing 6, 762, 347, 243 (240).
template <int PER>
__global__ void __launch_bounds__(SPLAT_THREADS, SPLAT_CTAS) k_density_splat(SurfaceDev s, const slosh_particle_t* __restrict__ particles, uint32_t n) {
    extern __shared__ int32_t splat_tile[];  // [5][SPLAT_TILE]
    __shared__ int s_box[6];
    const int big = 0x7FFFFFFF;
    if (threadIdx.x < 3) { s_box[threadIdx.x] = big; s_box[3 + threadIdx.x] = -big; }
    __syncthreads();
    const SplatShape shape = splat_shape(s);
    constexpr int CHUNK = SPLAT_THREADS * PER;
    SplatKernel kern[PER];
    bool live[PER];
    int3 mn = make_int3(big, big, big), mx = make_int3(-big, -big, -big);
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        // lanes 8 PER records apart: neighbouring records share a cell, and lanes adding to one voxel take turns
        const uint32_t i = blockIdx.x * uint32_t(CHUNK) + (threadIdx.x & 31u) * uint32_t(CHUNK / 32) + (threadIdx.x >> 5) * uint32_t(PER) + uint32_t(j);
        const float4 a = i < n ? __ldg(reinterpret_cast<const float4*>(particles + i)) : make_float4(0.0f, 0.0f, 0.0f, -1.0f);
        kern[j] = splat_kernel(s, shape, a);
        // a removed particle's ellipsoid is all zeros: skipped; a kernel outside the field touches no voxel
        live[j] = !is_dead_age(a.w) && kern[j].lo.x <= kern[j].hi.x && kern[j].lo.y <= kern[j].hi.y && kern[j].lo.z <= kern[j].hi.z;
        if (live[j]) {
            mn = make_int3(min(mn.x, kern[j].lo.x), min(mn.y, kern[j].lo.y), min(mn.z, kern[j].lo.z));
            mx = make_int3(max(mx.x, kern[j].hi.x), max(mx.y, kern[j].hi.y), max(mx.z, kern[j].hi.z));
        }
    }
    mn.x = __reduce_min_sync(0xFFFFFFFFu, mn.x); mn.y = __reduce_min_sync(0xFFFFFFFFu, mn.y); mn.z = __reduce_min_sync(0xFFFFFFFFu, mn.z);
    mx.x = __reduce_max_sync(0xFFFFFFFFu, mx.x); mx.y = __reduce_max_sync(0xFFFFFFFFu, mx.y); mx.z = __reduce_max_sync(0xFFFFFFFFu, mx.z);
    if ((threadIdx.x & 31) == 0 && mn.x <= mx.x) {
        atomicMin(s_box + 0, mn.x); atomicMin(s_box + 1, mn.y); atomicMin(s_box + 2, mn.z);
        atomicMax(s_box + 3, mx.x); atomicMax(s_box + 4, mx.y); atomicMax(s_box + 5, mx.z);
    }
    __syncthreads();
    if (s_box[0] == big) return;  // no live particle in this CTA (uniform)
    const int3 o = make_int3(s_box[0], s_box[1], s_box[2]);
    const int3 e = make_int3(s_box[3] - o.x + 1, s_box[4] - o.y + 1, s_box[5] - o.z + 1);
    const long long plane = (long long)e.x * e.y;
    const int rows = plane <= SPLAT_TILE ? int(SPLAT_TILE / plane) : 0;  // z planes of a slab
    if (rows == 0 || e.z > rows * SPLAT_MAX_SLABS<PER>) {
#pragma unroll
        for (int j = 0; j < PER; ++j)
            if (live[j])
                splat_voxels(s, shape, kern[j], kern[j].lo.z, kern[j].hi.z, [&](int x, int y, int z, const int32_t* m) {
                    int32_t* acc = s.accum + voxel_index(s, make_int3(x, y, z)) * FIELD_MOMENTS;
#pragma unroll
                    for (int q = 0; q < 5; ++q) atomicAdd(acc + q, m[q]);
                });
        return;
    }
    const uint32_t pl = uint32_t(plane);
    for (int z0 = 0; z0 < e.z; z0 += rows) {
        const int nz = min(rows, e.z - z0);
        const uint32_t nodes = pl * uint32_t(nz);
        for (uint32_t t = threadIdx.x; t < nodes; t += SPLAT_THREADS) {
#pragma unroll
            for (int q = 0; q < 5; ++q) splat_tile[q * SPLAT_TILE + t] = 0;
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < PER; ++j)
            if (live[j])
                splat_voxels(s, shape, kern[j], o.z + z0, o.z + z0 + nz - 1, [&](int x, int y, int z, const int32_t* m) {
                    int32_t* acc = splat_tile + (x - o.x) + e.x * (y - o.y) + int(pl) * (z - o.z - z0);
#pragma unroll
                    for (int q = 0; q < 5; ++q) atomicAdd(acc + q * SPLAT_TILE, m[q]);
                });
        __syncthreads();
        for (uint32_t t = threadIdx.x; t < nodes; t += SPLAT_THREADS) {
            int32_t m[5];
            int any = 0;
#pragma unroll
            for (int q = 0; q < 5; ++q) {
                m[q] = splat_tile[q * SPLAT_TILE + t];
                any |= m[q];
            }
            if (any == 0) continue;
            const uint32_t tz = t / pl, r = t - tz * pl, ty = r / uint32_t(e.x), tx = r - ty * uint32_t(e.x);
            int32_t* acc = s.accum + voxel_index(s, make_int3(o.x + int(tx), o.y + int(ty), o.z + z0 + int(tz))) * FIELD_MOMENTS;
#pragma unroll
            for (int q = 0; q < 5; ++q)
                if (m[q] != 0) atomicAdd(acc + q, m[q]);
        }
        __syncthreads();
    }
}

// ---- FieldResolveCS: fixed point -> f16 field (Zhu & Bridson surface) + dilated brick occupancy ---------------
// Bound by the read of the moments (20 bytes a voxel). The occupancy is a flag that only ever becomes 1, so a voxel
// stores it where it is not seen set yet instead of adding it atomically, once per distinct brick that its
// neighbourhood of one voxel reaches (its own, unless it lies on a face of its brick): with 8 atomics a voxel of
// liquid the pass took 193 us for 160^3 voxels, 36 now.
__global__ void __launch_bounds__(SURF_THREADS) k_field_resolve(SurfaceDev s) {
    const uint32_t i = blockIdx.x * SURF_THREADS + threadIdx.x;
    const uint32_t nv = uint32_t(s.dim.x) * uint32_t(s.dim.y) * uint32_t(s.dim.z);
    if (i >= nv) return;
    const int3 v = make_int3(int(i % uint32_t(s.dim.x)), int((i / uint32_t(s.dim.x)) % uint32_t(s.dim.y)), int(i / uint32_t(s.dim.x * s.dim.y)));
    const int32_t* acc = s.accum + i * FIELD_MOMENTS;
    const float w = float(acc[0]) / FIELD_W_FIXED;
    float f = 0.0f;
    if (w > 1e-3f) {
        const float den = FIELD_X_FIXED * w;
        const float3 mo = make_float3(float(acc[1]) / den, float(acc[2]) / den, float(acc[3]) / den);
        const float rbar = fmaxf(float(acc[4]) / den, 1e-3f);
        const float phi = sqrtf(dot3f(mo, mo)) - rbar;
        f = saturatef(0.5f - 0.5f * phi / rbar);
    }
    s.field[i] = __half_as_ushort(__float2half_rn(f));
    if (f <= 0.0f) return;
    // a voxel on a brick's face reaches the brick beyond it; the neighbour outside the field is not marked
    const int ix = v.x & 7, iy = v.y & 7, iz = v.z & 7;
    const int ox = ix == 0 ? -1 : (ix == 7 ? 1 : 0), oy = iy == 0 ? -1 : (iy == 7 ? 1 : 0), oz = iz == 0 ? -1 : (iz == 7 ? 1 : 0);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        if (((k & 1) && ox == 0) || ((k & 2) && oy == 0) || ((k & 4) && oz == 0)) continue;
        const int3 nb = make_int3(v.x + ((k & 1) ? ox : 0), v.y + ((k & 2) ? oy : 0), v.z + ((k & 4) ? oz : 0));
        if (nb.x < 0 || nb.y < 0 || nb.z < 0 || nb.x >= s.dim.x || nb.y >= s.dim.y || nb.z >= s.dim.z) continue;
        uint32_t* flag = s.bricks + field_brick(s, nb);
        if (*flag == 0u) *flag = 1u;
    }
}

// The 8 corner values of a cell and their inside mask (corner k at c + (k & 1, (k >> 1) & 1, k >> 2)).
__device__ __forceinline__ uint32_t cell_corners(const SurfaceDev& s, int3 c, float fc[8]) {
    uint32_t mask = 0u;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        fc[k] = field_at(s, make_int3(c.x + (k & 1), c.y + ((k >> 1) & 1), c.z + (k >> 2)));
        mask |= (fc[k] >= s.iso ? 1u : 0u) << k;
    }
    return mask;
}

// ---- SurfaceNetsVerticesCS, split: flags -> scan -> vertices in cell order -----------------------------------
__global__ void __launch_bounds__(SURF_THREADS) k_sn_vertex_flags(SurfaceDev s, uint32_t ncells) {
    const uint32_t i = blockIdx.x * SURF_THREADS + threadIdx.x;
    if (i >= ncells) return;
    const int3 c = cell_coord(s, i);
    uint32_t flag = 0u;
    if (s.bricks[field_brick(s, c)] != 0u) {
        float fc[8];
        const uint32_t mask = cell_corners(s, c, fc);
        flag = (mask != 0u && mask != 0xFFu) ? 1u : 0u;
    }
    s.vflag[i] = flag;
}

// Exact trilinear sample of the f16 field at Pv (voxel units; voxel v's centre at v + 0.5), clamped edges.
__device__ float sample_field(const SurfaceDev& s, float3 pv) {
    const float x = pv.x - 0.5f, y = pv.y - 0.5f, z = pv.z - 0.5f;
    const float fx0 = floorf(x), fy0 = floorf(y), fz0 = floorf(z);
    const float tx = x - fx0, ty = y - fy0, tz = z - fz0;
    const int x0 = int(fx0), y0 = int(fy0), z0 = int(fz0);
    const int xs[2] = {min(max(x0, 0), s.dim.x - 1), min(max(x0 + 1, 0), s.dim.x - 1)};
    const int ys[2] = {min(max(y0, 0), s.dim.y - 1), min(max(y0 + 1, 0), s.dim.y - 1)};
    const int zs[2] = {min(max(z0, 0), s.dim.z - 1), min(max(z0 + 1, 0), s.dim.z - 1)};
    float cz[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        float cy[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const float a = field_at(s, make_int3(xs[0], ys[j], zs[k])), b = field_at(s, make_int3(xs[1], ys[j], zs[k]));
            cy[j] = a + tx * (b - a);
        }
        cz[k] = cy[0] + ty * (cy[1] - cy[0]);
    }
    return cz[0] + tz * (cz[1] - cz[0]);
}
__device__ __forceinline__ float3 normalize_div(float3 v) {
    const float l = sqrtf(dot3f(v, v));
    return make_float3(v.x / l, v.y / l, v.z / l);
}

__global__ void __launch_bounds__(SURF_THREADS) k_sn_vertices(SurfaceDev s, uint32_t ncells) {
    const uint32_t i = blockIdx.x * SURF_THREADS + threadIdx.x;
    if (i >= ncells) return;
    uint32_t vi = s.vflag[i] ? s.vbase[i] : NO_VERTEX;
    if (vi != NO_VERTEX && vi >= s.max_vertices) vi = NO_VERTEX;
    s.cell_vertex[i] = vi;
    if (vi == NO_VERTEX) return;
    const int3 c = cell_coord(s, i);
    float fc[8];
    const uint32_t mask = cell_corners(s, c, fc);
    float sx = 0.0f, sy = 0.0f, sz = 0.0f, count = 0.0f;
#pragma unroll
    for (int a = 0; a < 8; ++a)
#pragma unroll
        for (int bit = 1; bit <= 4; bit <<= 1) {
            if (a & bit) continue;
            const int b = a | bit;
            if (((mask >> a) & 1u) == ((mask >> b) & 1u)) continue;
            const float t = saturatef((s.iso - fc[a]) / (fc[b] - fc[a]));
            // lerp between corners whose coordinates are 0 or 1: the moving coordinate is t or 1 - t
            const float px = (a & 1) == (b & 1) ? float(a & 1) : ((b & 1) ? t : 1.0f - t);
            const float py = ((a >> 1) & 1) == ((b >> 1) & 1) ? float((a >> 1) & 1) : (((b >> 1) & 1) ? t : 1.0f - t);
            const float pz = (a >> 2) == (b >> 2) ? float(a >> 2) : ((b >> 2) ? t : 1.0f - t);
            sx = sx + px;
            sy = sy + py;
            sz = sz + pz;
            count = count + 1.0f;
        }
    const float3 pv = make_float3((float(c.x) + 0.5f) + sx / count, (float(c.y) + 0.5f) + sy / count, (float(c.z) + 0.5f) + sz / count);
    s.positions[3u * vi + 0u] = pv.x * s.voxel;
    s.positions[3u * vi + 1u] = pv.y * s.voxel;
    s.positions[3u * vi + 2u] = pv.z * s.voxel;
    const float3 g = make_float3(sample_field(s, make_float3(pv.x + 1.0f, pv.y, pv.z)) - sample_field(s, make_float3(pv.x - 1.0f, pv.y, pv.z)),
                                 sample_field(s, make_float3(pv.x, pv.y + 1.0f, pv.z)) - sample_field(s, make_float3(pv.x, pv.y - 1.0f, pv.z)),
                                 sample_field(s, make_float3(pv.x, pv.y, pv.z + 1.0f)) - sample_field(s, make_float3(pv.x, pv.y, pv.z - 1.0f)));
    float3 nrm = make_float3(0.0f, 0.0f, 1.0f);
    if (sqrtf(dot3f(g, g)) > 1e-8f) {
        const float3 ng = normalize_div(g);
        nrm = make_float3(-ng.x, -ng.y, -ng.z);
    }
    const float3 ref = fabsf(nrm.z) < 0.9f ? make_float3(0.0f, 0.0f, 1.0f) : make_float3(1.0f, 0.0f, 0.0f);
    const float3 tx = normalize_div(cross3(nrm, ref));
    s.normals[3u * vi + 0u] = nrm.x;
    s.normals[3u * vi + 1u] = nrm.y;
    s.normals[3u * vi + 2u] = nrm.z;
    s.tangents[3u * vi + 0u] = tx.x;
    s.tangents[3u * vi + 1u] = tx.y;
    s.tangents[3u * vi + 2u] = tx.z;
}

// ---- SurfaceNetsFacesCS, split: quad counts -> scan -> quads in cell order ------------------------------------
// Quads of cell c: for each axis whose edge from voxel c to c + e crosses the level, the four cells around
// the edge (c, c - eu, c - eu - ev, c - ev) when all exist and carry a vertex. emit(axis, in0, v00, v10, v11, v01).
template <class Emit>
__device__ __forceinline__ void cell_quads(const SurfaceDev& s, int3 c, Emit emit) {
    if (s.bricks[field_brick(s, c)] == 0u) return;
    const bool in0 = field_at(s, c) >= s.iso;
#pragma unroll
    for (int axis = 0; axis < 3; ++axis) {
        const int3 e = make_int3(axis == 0, axis == 1, axis == 2);
        const bool in1 = field_at(s, make_int3(c.x + e.x, c.y + e.y, c.z + e.z)) >= s.iso;
        if (in0 == in1) continue;
        const int3 eu = make_int3(axis == 2, axis == 0, axis == 1), ev = make_int3(axis == 1, axis == 2, axis == 0);
        const int3 c10 = make_int3(c.x - eu.x, c.y - eu.y, c.z - eu.z);
        const int3 c11 = make_int3(c.x - eu.x - ev.x, c.y - eu.y - ev.y, c.z - eu.z - ev.z);
        const int3 c01 = make_int3(c.x - ev.x, c.y - ev.y, c.z - ev.z);
        if (c11.x < 0 || c11.y < 0 || c11.z < 0) continue;
        const uint32_t v00 = s.cell_vertex[cell_of(s, c)], v10 = s.cell_vertex[cell_of(s, c10)];
        const uint32_t v11 = s.cell_vertex[cell_of(s, c11)], v01 = s.cell_vertex[cell_of(s, c01)];
        if (v00 == NO_VERTEX || v10 == NO_VERTEX || v11 == NO_VERTEX || v01 == NO_VERTEX) continue;
        emit(in0, v00, v10, v11, v01);
    }
}
__global__ void __launch_bounds__(SURF_THREADS) k_sn_quad_counts(SurfaceDev s, uint32_t ncells) {
    const uint32_t i = blockIdx.x * SURF_THREADS + threadIdx.x;
    if (i >= ncells) return;
    uint32_t count = 0u;
    cell_quads(s, cell_coord(s, i), [&](bool, uint32_t, uint32_t, uint32_t, uint32_t) { ++count; });
    s.qflag[i] = count;
}
__global__ void __launch_bounds__(SURF_THREADS) k_sn_faces(SurfaceDev s, uint32_t ncells) {
    const uint32_t i = blockIdx.x * SURF_THREADS + threadIdx.x;
    if (i >= ncells) return;
    uint32_t q = s.qbase[i];
    cell_quads(s, cell_coord(s, i), [&](bool in0, uint32_t v00, uint32_t v10, uint32_t v11, uint32_t v01) {
        const uint32_t base = 6u * q++;
        if (base + 6u > s.max_indices) return;
        uint32_t* o = s.indices + base;
        // winding faces away from the inside voxel
        if (in0) { o[0] = v00; o[1] = v11; o[2] = v10; o[3] = v00; o[4] = v01; o[5] = v11; }
        else { o[0] = v00; o[1] = v10; o[2] = v11; o[3] = v00; o[4] = v11; o[5] = v01; }
    });
}
// Counters: [0] vertices requested, [1] indices requested (SurfaceNetsArgsCS clamps and rounds on the host).
__global__ void k_sn_totals(SurfaceDev s, uint32_t ncells) {
    s.counters[0] = s.vbase[ncells - 1u] + s.vflag[ncells - 1u];
    s.counters[1] = 6u * (s.qbase[ncells - 1u] + s.qflag[ncells - 1u]);
}

int blocks_of(uint64_t n) { return int((n + SURF_THREADS - 1) / SURF_THREADS); }

}  // namespace

int launch_surface(const SurfaceDev& s, const slosh_particle_t* particles, uint32_t n, bool mesh, int num_sms, cudaStream_t st) {
    const uint64_t nv = uint64_t(s.dim.x) * uint64_t(s.dim.y) * uint64_t(s.dim.z);
    const uint64_t nb = uint64_t(s.bdim.x) * uint64_t(s.bdim.y) * uint64_t(s.bdim.z);
    int launches = 0;
    cudaMemsetAsync(s.accum, 0, nv * FIELD_MOMENTS * 4, st);
    cudaMemsetAsync(s.bricks, 0, nb * 4, st);
    cudaMemsetAsync(s.counters, 0, 8, st);
    if (n > 0) {
        const bool few = n <= uint32_t(num_sms * SPLAT_CTAS * SPLAT_THREADS);
        const uint32_t chunk = SPLAT_THREADS * (few ? 1u : 2u);
        auto kernel = few ? k_density_splat<1> : k_density_splat<2>;
        // room for four CTAs' tiles per SM
        cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        kernel<<<int((uint64_t(n) + chunk - 1u) / chunk), SPLAT_THREADS, SPLAT_SMEM, st>>>(s, particles, n);
        ++launches;
    }
    k_field_resolve<<<blocks_of(nv), SURF_THREADS, 0, st>>>(s);
    ++launches;
    if (!mesh) return launches;
    const uint32_t nc = uint32_t(s.dim.x - 1) * uint32_t(s.dim.y - 1) * uint32_t(s.dim.z - 1);
    if (nc == 0) return launches;
    k_sn_vertex_flags<<<blocks_of(nc), SURF_THREADS, 0, st>>>(s, nc);
    launches += 1 + launch_exclusive_scan(s.vflag, s.vbase, nc, s.scan_tmp, st);
    k_sn_vertices<<<blocks_of(nc), SURF_THREADS, 0, st>>>(s, nc);
    k_sn_quad_counts<<<blocks_of(nc), SURF_THREADS, 0, st>>>(s, nc);
    launches += 2 + launch_exclusive_scan(s.qflag, s.qbase, nc, s.scan_tmp, st);
    k_sn_faces<<<blocks_of(nc), SURF_THREADS, 0, st>>>(s, nc);
    k_sn_totals<<<1, 1, 0, st>>>(s, nc);
    return launches + 2;
}

}  // namespace slosh
