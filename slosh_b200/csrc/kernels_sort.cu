// Spatial sort of particles by 4^3 block key with compaction of dead slots (sm_100a).
//
// Reference: PLUG/Shaders/Private/SloshSort.usf (SortKey :36-47, SortCountCS :65-76, scans :78-132,
// SortScatterCS :134-146, SortWriteCountCS :149-154) and AddSpatialSort, SloshProxy.cpp:1022-1087.
//
// The reference ranks particles inside a key with an atomic counter, so its permutation depends on
// thread timing. This sort is stable: it orders by key and, inside a key, by source slot -- the order
// the reference produces when its atomics resolve in ascending thread order. It is an LSD radix sort of
// (key, slot) pairs whose digits split the key's bits evenly into the fewest passes of at most 10 bits (two
// for 2^18 keys); each pass is reduce-then-scan:
//   upsweep   per 4096-item tile, a shared-memory histogram of the digit (the first pass's by k_keys);
//   scan      each tile's first output position of each digit: up to SORT_SMALL_TILES tiles every scatter CTA
//             adds the whole histogram up for itself, beyond that an exclusive scan in digit-major order;
//   scatter   each warp ranks its 512 contiguous items in order (warp match + per-warp counters), the
//             per-warp counters are prefixed across warps, and items go to tile base + rank.
// One tile (n <= 4096) is sorted by one CTA in shared memory. The key offsets (and counts) are lower bounds in the
// sorted keys, found beside the gather of the records. No step waits on another CTA.
// A small sort is bound by its launches and their dependent loads: 3,001 records took 10 launches and 47 us with the
// three-kernel scans and 8-bit digits, 200,003 records 15 launches and 83 us; now 2 launches and 12 us, 5 and 39 us.
// 20.6 M records (2^18 keys): 1.22 ms with 3 passes of 8 bits and atomic counts, 0.80 ms with two of 10 and 9 bits.
#include <algorithm>

#include "kernels.h"

namespace slosh {

namespace {

constexpr int SORT_THREADS = 256;
constexpr int SORT_WARPS = SORT_THREADS / 32;
constexpr int SORT_ROUNDS = 16;                      // items per lane
constexpr int SORT_TILE = SORT_THREADS * SORT_ROUNDS;  // 4096 items per tile
constexpr int WARP_ITEMS = 32 * SORT_ROUNDS;           // 512 contiguous items per warp
constexpr int SCAN_THREADS = 256;
constexpr int SCAN_ITEMS = 16;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;

__device__ __forceinline__ uint32_t sort_key_of(const Dev& d, float4 a, int3 sdim, uint32_t num_keys) {
    if (is_dead_age(a.w)) return num_keys - 1u;
    const int cx = clampi(int(floorf(a.x * d.inv_h)), 0, d.grid.x - 1);
    const int cy = clampi(int(floorf(a.y * d.inv_h)), 0, d.grid.y - 1);
    const int cz = clampi(int(floorf(a.z * d.inv_h)), 0, d.grid.z - 1);
    const uint32_t k = uint32_t((cx >> 2) + sdim.x * ((cy >> 2) + sdim.y * (cz >> 2)));
    return min(k, num_keys - 2u);
}

__device__ __forceinline__ uint32_t tile_item(uint32_t tile, int r) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    return tile * uint32_t(SORT_TILE) + uint32_t(warp * WARP_ITEMS + r * 32 + lane);
}

constexpr int SORT_MAX_BITS = 10;                     // bits of a digit: 8 warps' counters of 1024 digits in 16 KB
constexpr uint32_t SORT_SMALL_TILES = 64;             // tiles whose histograms every scatter CTA adds up itself

// A tile's histogram of one digit: tile-major rows for few tiles (read whole by every scatter CTA), else digit-major
// (scanned).
__device__ __forceinline__ void store_hist(const uint32_t* hist, uint32_t* tile_hist, uint32_t num_tiles, uint32_t bins, bool small) {
    for (uint32_t d = threadIdx.x; d < bins; d += SORT_THREADS)
        tile_hist[small ? blockIdx.x * bins + d : d * num_tiles + blockIdx.x] = hist[d];
}
// Keys and the first digit's tile histogram.
__global__ void __launch_bounds__(SORT_THREADS) k_keys(Dev d, const slosh_particle_t* __restrict__ particles, uint32_t n,
                                                       uint32_t* __restrict__ keys, uint32_t* __restrict__ tile_hist,
                                                       uint32_t num_tiles, uint32_t bins, bool small, int3 sdim, uint32_t num_keys) {
    pdl_entry();
    __shared__ uint32_t hist[1 << SORT_MAX_BITS];
    for (uint32_t t = threadIdx.x; t < bins; t += SORT_THREADS) hist[t] = 0u;
    __syncthreads();
    const uint32_t tile = blockIdx.x;
#pragma unroll 8
    for (int r = 0; r < SORT_ROUNDS; ++r) {
        const uint32_t i = tile_item(tile, r);
        if (i < n) {
            const uint32_t key = sort_key_of(d, __ldg(reinterpret_cast<const float4*>(particles + i)), sdim, num_keys);
            keys[i] = key;
            atomicAdd(hist + (key & (bins - 1u)), 1u);
        }
    }
    __syncthreads();
    store_hist(hist, tile_hist, num_tiles, bins, small);
}

__global__ void __launch_bounds__(SORT_THREADS) k_upsweep(const uint32_t* keys, uint32_t n, uint32_t* __restrict__ tile_hist,
                                                          uint32_t num_tiles, uint32_t bins, bool small, uint32_t shift) {
    pdl_entry();
    __shared__ uint32_t hist[1 << SORT_MAX_BITS];
    for (uint32_t t = threadIdx.x; t < bins; t += SORT_THREADS) hist[t] = 0u;
    __syncthreads();
    const uint32_t tile = blockIdx.x;
#pragma unroll 8
    for (int r = 0; r < SORT_ROUNDS; ++r) {
        const uint32_t i = tile_item(tile, r);
        if (i < n) atomicAdd(hist + ((keys[i] >> shift) & (bins - 1u)), 1u);
    }
    __syncthreads();
    store_hist(hist, tile_hist, num_tiles, bins, small);
}

__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t* s_warp, uint32_t* total);

// Stable scatter of one digit. vals_in == nullptr means the identity (source slot = item index). tile_hist holds the
// tiles' histograms (small) or their scan.
__global__ void __launch_bounds__(SORT_THREADS) k_scatter(const uint32_t* keys_in, const uint32_t* vals_in, uint32_t* keys_out,
                                                          uint32_t* vals_out, uint32_t n, const uint32_t* tile_hist, uint32_t num_tiles,
                                                          uint32_t bins, bool small, uint32_t shift) {
    pdl_entry();
    __shared__ uint16_t whist[SORT_WARPS][1 << SORT_MAX_BITS];  // a warp's counts, then its first place in the tile
    __shared__ uint32_t first[1 << SORT_MAX_BITS];              // the tile's first output position
    __shared__ uint32_t total[1 << SORT_MAX_BITS];
    __shared__ uint32_t s_warp[33];
    const uint32_t tile = blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t lt_mask = (1u << lane) - 1u;
    uint32_t key[SORT_ROUNDS], val[SORT_ROUNDS], rank[SORT_ROUNDS];
#pragma unroll
    for (int r = 0; r < SORT_ROUNDS; ++r) {
        const uint32_t i = tile_item(tile, r);
        key[r] = i < n ? keys_in[i] : 0u;
        val[r] = i < n ? (vals_in ? vals_in[i] : i) : 0u;
    }
    for (uint32_t t = threadIdx.x; t < bins; t += SORT_THREADS) first[t] = total[t] = 0u;
#pragma unroll
    for (int w = 0; w < SORT_WARPS; ++w)
        for (uint32_t t = threadIdx.x; t < bins; t += SORT_THREADS) whist[w][t] = 0u;
    __syncthreads();
    if (small) {
        const uint32_t words = num_tiles * bins;
#pragma unroll 8
        for (uint32_t t = threadIdx.x; t < words; t += SORT_THREADS) {
            const uint32_t v = tile_hist[t], dgt = t & (bins - 1u);
            if (v != 0u) {
                atomicAdd(total + dgt, v);
                if (t < tile * bins) atomicAdd(first + dgt, v);
            }
        }
    } else {
        for (uint32_t t = threadIdx.x; t < bins; t += SORT_THREADS) first[t] = tile_hist[t * num_tiles + tile];
    }
#pragma unroll
    for (int r = 0; r < SORT_ROUNDS; ++r) {
        const bool valid = tile_item(tile, r) < n;
        const uint32_t digit = valid ? ((key[r] >> shift) & (bins - 1u)) : 0xFFFFFFFFu;
        const uint32_t peers = __match_any_sync(0xFFFFFFFFu, digit);
        uint32_t before = 0u;
        if (valid) before = whist[warp][digit];
        __syncwarp();
        if (valid && lane == __ffs(int(peers)) - 1) whist[warp][digit] = uint16_t(before + uint32_t(__popc(peers)));
        __syncwarp();
        rank[r] = valid ? before + uint32_t(__popc(peers & lt_mask)) : 0xFFFFFFFFu;
    }
    __syncthreads();
    if (small) {  // the digits' exclusive scan: thread t takes the digits from t * per
        const uint32_t per = (bins + SORT_THREADS - 1u) / SORT_THREADS, d0 = threadIdx.x * per;
        uint32_t v = 0u;
        for (uint32_t j = 0; j < per; ++j)
            if (d0 + j < bins) v += total[d0 + j];
        uint32_t all;
        uint32_t run = block_excl_scan(v, s_warp, &all);
        for (uint32_t j = 0; j < per; ++j)
            if (d0 + j < bins) {
                first[d0 + j] += run;
                run += total[d0 + j];
            }
    }
    for (uint32_t dgt = threadIdx.x; dgt < bins; dgt += SORT_THREADS) {
        uint32_t run = 0u;
#pragma unroll
        for (int w = 0; w < SORT_WARPS; ++w) {
            const uint32_t t = whist[w][dgt];
            whist[w][dgt] = uint16_t(run);
            run += t;
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < SORT_ROUNDS; ++r) {
        if (rank[r] == 0xFFFFFFFFu) continue;
        const uint32_t dgt = (key[r] >> shift) & (bins - 1u);
        const uint32_t dst = first[dgt] + whist[warp][dgt] + rank[r];
        keys_out[dst] = key[r];
        vals_out[dst] = val[r];
    }
}

// The whole radix sort of one tile by one CTA of 1024 threads, 4 items each, in shared memory; 8-bit digits.
constexpr int TILE_THREADS = 1024, TILE_WARPS = TILE_THREADS / 32, TILE_ROUNDS = SORT_TILE / TILE_THREADS;
__global__ void __launch_bounds__(TILE_THREADS) k_sort_tile(Dev d, const slosh_particle_t* __restrict__ particles, uint32_t n,
                                                            uint32_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out, int bits,
                                                            int3 sdim, uint32_t num_keys) {
    pdl_entry();
    __shared__ uint16_t whist[TILE_WARPS][256];
    __shared__ uint32_t s_keys[SORT_TILE];
    __shared__ uint16_t s_vals[SORT_TILE];
    __shared__ uint32_t s_warp[33];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t lt_mask = (1u << lane) - 1u;
    uint32_t key[TILE_ROUNDS], val[TILE_ROUNDS], rank[TILE_ROUNDS];
    auto item = [&](int r) { return uint32_t(warp * 32 * TILE_ROUNDS + r * 32 + lane); };
#pragma unroll
    for (int r = 0; r < TILE_ROUNDS; ++r) {
        const uint32_t i = item(r);
        key[r] = i < n ? sort_key_of(d, __ldg(reinterpret_cast<const float4*>(particles + i)), sdim, num_keys) : 0u;
        val[r] = i;
    }
    for (int shift = 0; shift < bits || shift == 0; shift += 8) {
        for (uint32_t t = threadIdx.x; t < uint32_t(TILE_WARPS) * 128u; t += TILE_THREADS) reinterpret_cast<uint32_t*>(&whist[0][0])[t] = 0u;
        __syncthreads();
#pragma unroll
        for (int r = 0; r < TILE_ROUNDS; ++r) {
            const bool valid = item(r) < n;
            const uint32_t digit = valid ? ((key[r] >> shift) & 0xFFu) : 0xFFFFFFFFu;
            const uint32_t peers = __match_any_sync(0xFFFFFFFFu, digit);
            uint32_t before = 0u;
            if (valid) before = whist[warp][digit];
            __syncwarp();
            if (valid && lane == __ffs(int(peers)) - 1) whist[warp][digit] = uint16_t(before + uint32_t(__popc(peers)));
            __syncwarp();
            rank[r] = before + uint32_t(__popc(peers & lt_mask));
        }
        __syncthreads();
        uint32_t sum = 0u;
        if (threadIdx.x < 256u) {
#pragma unroll 8
            for (int w = 0; w < TILE_WARPS; ++w) sum += whist[w][threadIdx.x];
        }
        uint32_t all;
        uint32_t run = block_excl_scan(sum, s_warp, &all);
        if (threadIdx.x < 256u) {
#pragma unroll 8
            for (int w = 0; w < TILE_WARPS; ++w) {
                const uint32_t t = whist[w][threadIdx.x];
                whist[w][threadIdx.x] = uint16_t(run);
                run += t;
            }
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < TILE_ROUNDS; ++r) {
            if (item(r) >= n) continue;
            const uint32_t dst = whist[warp][(key[r] >> shift) & 0xFFu] + rank[r];
            s_keys[dst] = key[r];
            s_vals[dst] = uint16_t(val[r]);
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < TILE_ROUNDS; ++r) {
            const uint32_t i = item(r);
            if (i >= n) continue;
            key[r] = s_keys[i];
            val[r] = s_vals[i];
        }
    }
#pragma unroll
    for (int r = 0; r < TILE_ROUNDS; ++r) {
        const uint32_t i = item(r);
        if (i >= n) continue;
        keys_out[i] = key[r];
        vals_out[i] = val[r];
    }
}

// Gather of the 48-byte records in sorted order (perm keeps the source slot of every output), and for thread k < num_keys
// the key's offset: the number of sorted keys below k. The last key is the dead records', so its offset is the live count.
// counts may be null.
__device__ __forceinline__ uint32_t lower_bound_key(const uint32_t* keys, uint32_t n, uint32_t k) {
    uint32_t lo = 0u, hi = n;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (keys[mid] < k) lo = mid + 1u;
        else hi = mid;
    }
    return lo;
}
__global__ void __launch_bounds__(256) k_gather(const slosh_particle_t* __restrict__ in, slosh_particle_t* __restrict__ out, const uint32_t* keys,
                                                const uint32_t* vals, uint32_t* __restrict__ perm, uint32_t n,
                                                uint32_t* __restrict__ offsets, uint32_t* __restrict__ counts, uint32_t num_keys,
                                                uint32_t* __restrict__ pc) {
    pdl_entry();
    const uint32_t j = blockIdx.x * 256u + threadIdx.x;
    if (j < n) {
        const uint32_t src = vals[j];
        const float4* s = reinterpret_cast<const float4*>(in + src);
        float4* o = reinterpret_cast<float4*>(out + j);
        const float4 a = __ldg(s), b = __ldg(s + 1), c = __ldg(s + 2);
        o[0] = a;
        o[1] = b;
        o[2] = c;
        perm[j] = src;
    }
    if ((j & ~31u) >= num_keys) return;
    const uint32_t at = lower_bound_key(keys, n, min(j, num_keys));
    if (j < num_keys) {
        offsets[j] = at;
        if (j == num_keys - 1u) pc[0] = at;
    }
    if (counts) {  // warp-uniform; the next lane's offset, the last lane's by another search
        uint32_t next = __shfl_down_sync(0xFFFFFFFFu, at, 1);
        if ((j & 31u) == 31u || j + 1u >= num_keys) next = j + 1u < num_keys ? lower_bound_key(keys, n, j + 1u) : n;
        if (j < num_keys) counts[j] = next - at;
    }
}

// ---- exclusive scan of u32 (three kernels, in place allowed) ----------------------------------------
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t* s_warp, uint32_t* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, off);
        if (lane >= off) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        const int nw = blockDim.x / 32;
        uint32_t w = lane < nw ? s_warp[lane] : 0u;
        uint32_t ws = w;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, ws, off);
            if (lane >= off) ws += y;
        }
        if (lane < nw) s_warp[lane] = ws - w;
        if (lane == 31) s_warp[32] = ws;
    }
    __syncthreads();
    const uint32_t ex = s_warp[warp] + x - v;
    *total = s_warp[32];
    __syncthreads();
    return ex;
}

// A thread's SCAN_ITEMS consecutive words as four 16-byte accesses where the tile is whole and both arrays start on 16
// bytes (a caller's offset array may not), else word by word: the words of a warp's threads are 64 bytes apart, so
// word accesses touch 16 lines each (4.1 M words: k_scan_down 25.9 us, 8.8 in
// 16-byte accesses).
__device__ __forceinline__ bool scan_vec(const uint32_t* in, const uint32_t* out, uint32_t base, uint32_t n) {
    return ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15u) == 0u && base + uint32_t(SCAN_ITEMS) <= n;
}
__device__ __forceinline__ void scan_load(const uint32_t* in, uint32_t base, uint32_t n, bool vec, uint32_t (&v)[SCAN_ITEMS]) {
    if (vec) {
#pragma unroll
        for (int k = 0; k < SCAN_ITEMS / 4; ++k) {
            const uint4 q = reinterpret_cast<const uint4*>(in + base)[k];
            v[4 * k] = q.x; v[4 * k + 1] = q.y; v[4 * k + 2] = q.z; v[4 * k + 3] = q.w;
        }
    } else {
#pragma unroll
        for (int k = 0; k < SCAN_ITEMS; ++k) v[k] = base + uint32_t(k) < n ? in[base + uint32_t(k)] : 0u;
    }
}
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_reduce(const uint32_t* __restrict__ in, uint32_t n, uint32_t* __restrict__ sums) {
    __shared__ uint32_t s_warp[33];
    const uint32_t base = blockIdx.x * uint32_t(SCAN_TILE) + threadIdx.x * uint32_t(SCAN_ITEMS);
    uint32_t vals[SCAN_ITEMS];
    scan_load(in, base, n, scan_vec(in, in, base, n), vals);
    uint32_t v = 0u;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) v += vals[k];
    uint32_t total;
    block_excl_scan(v, s_warp, &total);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}
__global__ void __launch_bounds__(1024) k_scan_sums(uint32_t* sums, uint32_t nb) {
    __shared__ uint32_t s_warp[33];
    const uint32_t per = (nb + blockDim.x - 1u) / blockDim.x;
    const uint32_t b0 = min(threadIdx.x * per, nb), b1 = min(b0 + per, nb);
    uint32_t v = 0u;
    for (uint32_t b = b0; b < b1; ++b) v += sums[b];
    uint32_t total;
    uint32_t run = block_excl_scan(v, s_warp, &total);
    for (uint32_t b = b0; b < b1; ++b) {
        const uint32_t t = sums[b];
        sums[b] = run;
        run += t;
    }
}
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_down(const uint32_t* in, uint32_t* out, uint32_t n, const uint32_t* __restrict__ sums) {
    __shared__ uint32_t s_warp[33];
    const uint32_t base = blockIdx.x * uint32_t(SCAN_TILE) + threadIdx.x * uint32_t(SCAN_ITEMS);
    uint32_t vals[SCAN_ITEMS];
    const bool vec = scan_vec(in, out, base, n);
    scan_load(in, base, n, vec, vals);
    uint32_t v = 0u;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) v += vals[k];
    uint32_t total;
    uint32_t run = block_excl_scan(v, s_warp, &total) + sums[blockIdx.x];
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        const uint32_t t = vals[k];
        vals[k] = run;
        run += t;
    }
    if (vec) {
#pragma unroll
        for (int k = 0; k < SCAN_ITEMS / 4; ++k)
            reinterpret_cast<uint4*>(out + base)[k] = make_uint4(vals[4 * k], vals[4 * k + 1], vals[4 * k + 2], vals[4 * k + 3]);
    } else {
#pragma unroll
        for (int k = 0; k < SCAN_ITEMS; ++k)
            if (base + uint32_t(k) < n) out[base + uint32_t(k)] = vals[k];
    }
}

int exclusive_scan(const uint32_t* in, uint32_t* out, uint32_t n, uint32_t* tmp, cudaStream_t s) {
    const uint32_t nb = (n + uint32_t(SCAN_TILE) - 1u) / uint32_t(SCAN_TILE);
    if (nb == 0) return 0;
    k_scan_reduce<<<nb, SCAN_THREADS, 0, s>>>(in, n, tmp);
    k_scan_sums<<<1, 1024, 0, s>>>(tmp, nb);
    k_scan_down<<<nb, SCAN_THREADS, 0, s>>>(in, out, n, tmp);
    return 3;
}

}  // namespace

int launch_exclusive_scan(const uint32_t* in, uint32_t* out, uint32_t n, uint32_t* tmp, cudaStream_t s) {
    return exclusive_scan(in, out, n, tmp, s);
}
size_t exclusive_scan_tmp_size(uint32_t n) { return (size_t(n) + SCAN_TILE - 1) / SCAN_TILE + 1; }

int3 sort_brick_dim(int3 g) { return make_int3((g.x + 3) / 4, (g.y + 3) / 4, (g.z + 3) / 4); }

// Block sums of the largest scan: the tiles' histograms, at most a quarter word per particle and a row.
size_t sort_scan_tmp_size(uint32_t capacity) {
    return (size_t(capacity) / 4 + (size_t(1) << SORT_MAX_BITS) + SCAN_TILE - 1) / SCAN_TILE + 1;
}

int launch_sort(const Dev& d, const SortBuffers& b, const slosh_particle_t* in, slosh_particle_t* out, uint32_t n,
                uint32_t num_keys, int3 sdim, cudaStream_t s) {
    int launches = 0;
    uint32_t bits = 0;
    while ((1u << bits) < num_keys && bits < 32) ++bits;  // keys are < num_keys
    const uint32_t num_tiles = (n + uint32_t(SORT_TILE) - 1u) / uint32_t(SORT_TILE);
    int cur = 0;
    if (num_tiles == 1u) {
        launch_k(k_sort_tile, 1, TILE_THREADS, 0, s, d, in, n, b.keys[0], b.vals[0], int(bits), sdim, num_keys);
        ++launches;
    } else if (num_tiles > 1u) {
        const int passes = std::max(1, int((bits + SORT_MAX_BITS - 1) / SORT_MAX_BITS));
        const bool small = num_tiles <= SORT_SMALL_TILES;
        uint32_t* hist = b.perm;  // 2^10 words a tile of 4096 fit the permutation, which only the gather writes
        uint32_t shift = 0;
        for (int pass = 0; pass < passes; ++pass) {
            const uint32_t width = (bits - shift + uint32_t(passes - pass) - 1u) / uint32_t(passes - pass);
            const uint32_t bins = 1u << std::max(width, 1u);
            if (pass == 0) launch_k(k_keys, num_tiles, SORT_THREADS, 0, s, d, in, n, b.keys[0], hist, num_tiles, bins, small, sdim, num_keys);
            else launch_k(k_upsweep, num_tiles, SORT_THREADS, 0, s, b.keys[cur], n, hist, num_tiles, bins, small, shift);
            ++launches;
            if (!small) launches += exclusive_scan(hist, hist, bins * num_tiles, b.scan_tmp, s);
            launch_k(k_scatter, num_tiles, SORT_THREADS, 0, s, b.keys[cur], pass == 0 ? nullptr : b.vals[cur], b.keys[cur ^ 1], b.vals[cur ^ 1],
                     n, hist, num_tiles, bins, small, shift);
            ++launches;
            cur ^= 1;
            shift += width;
        }
    }
    launch_k(k_gather, (std::max(n, num_keys) + 255u) / 256u, 256, 0, s, in, out, b.keys[cur], b.vals[cur], b.perm, n, b.offsets, b.counts,
             num_keys, b.particle_count);
    return launches + 1;
}

}  // namespace slosh
