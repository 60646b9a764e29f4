// A whole MGPCG solve in one thread-block cluster (included by kernels_mg.cu, inside its namespace).
//
// A small tank's passes take 3-9 us each as launches: a kernel boundary, the chain of dependent loads that starts every
// pass (active count, neighbour slots, words, values) and the last CTA's reduction, not bandwidth; an iteration of a
// 64x64x48 tank is 11 of them. And as graphs with a conditional loop the solves of many tanks run almost one after another.
// Here one cluster of up to 16 CTAs runs the solve's setup and all of its iterations. Its CTAs are scheduled together and
// wait only for one another in hardware cluster barriers, so solves of many tanks run side by side on their own streams.
//
// Resident form (at most CL_WARPS bricks per CTA, 240 for 16 CTAs): a warp owns one active brick, whose z, search direction,
// residual, diagonal and cells of levels 1-3 lie in its block of shared memory; its lanes hold the cells of the launched
// passes' half-row quads, so the dot products' canonical order is the lanes' own. A pass copies the cells of one colour of
// one array that touch the brick's faces from the neighbours' blocks (distributed shared memory), computes from shared
// memory and ends in a cluster barrier. Level `tail` and below are CTA 0's, which owns no bricks and whose tail image stays
// in place for the solve; the restriction writes into it and the prolongation reads from it through distributed shared
// memory too. Each warp sends its dot-product partial to every CTA, and every CTA adds the partials for itself in the
// canonical order: all take the same alpha, beta and stopping decision. Global memory is touched by the setup, the update of
// p and the final statistics only.
// Streamed form (more bricks than that): the launched kernels' bodies over global memory between cluster barriers.
// Both give the launched form's bits.
//
// Used while the resident form holds the bricks that the tank is expected to have (mg_solve_cluster). What bounds a pass now is its chain of
// barrier (0.3-0.5 us), distributed-shared-memory copy and sweep, 1.5-3 us for level 0; the tail is 9 of 35 us of an iteration of
// a 64x64x48 tank (150 active bricks), which took 70 us as launches: its frame 1,034 -> 690 us; 24 tanks of 70-288 active bricks
// stepped together 36.0 -> 16.2 to 16.4 ms.
#pragma once

constexpr int CL_THREADS = 512;  // 128 registers; a spilled value would come from L2 after every barrier (its acquire empties the L1)
constexpr int CL_WARPS = CL_THREADS / 32;

__device__ __forceinline__ uint32_t cl_mapa(uint32_t local, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
    return r;
}
__device__ __forceinline__ float dsm_ld(uint32_t a) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ float4 dsm_ld4(uint32_t a) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void dsm_st(uint32_t a, float v) { asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory"); }
__device__ __forceinline__ void dsm_st(uint32_t a, double v) { asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory"); }

// A warp's brick in shared memory. Words are those of the level arrays, 0 for cells outside the level.
struct __align__(16) ResBrick {
    float z[2][BRICK_CELLS / 2];  // by colour
    float d[2][BRICK_CELLS / 2];
    float r[2][BRICK_CELLS / 2], dg[2][BRICK_CELLS / 2], rc[2][BRICK_CELLS / 2];  // residual, diagonal + epsilon, its reciprocal
    uint8_t word[2][BRICK_CELLS / 2];  // stencil words
    float halo[256];         // the face neighbours' cells of one colour of the array a pass reads (res_pull)
    float halo1[6 * 16];     // their level-1 cells likewise (side 4)
    float x1[64], b1[64], res[64];
    float x2[8], b2[8];
    float x3[2], b3[2];
    uint16_t w1[64], w2[8], w3[8];
};
constexpr size_t CL_BLOCKS = size_t(CL_WARPS) * sizeof(ResBrick);
constexpr size_t CL_SCRATCH = size_t(CL_WARPS) * (BRICK_CELLS * 5u);  // streamed form, per warp: 512 floats and 512 bytes (restrict0)
constexpr uint32_t CL_PARTIALS = 16u * CL_WARPS;  // entries of a dot product in the resident form

struct ClSolve {
    float* p;
    const float* div;
    uint32_t limit, tol_mode;
    double tol;
    int coarse, tail;
    uint32_t setup, tail_bytes;
};

// The canonical reduction (final_reduce) by every CTA; all threads get the sum. Groups of 32 lanes that hold no partial
// are left out: they would add 0.0.
__device__ __forceinline__ double cl_reduce(const double* partials, uint32_t n, double* s_w32) {
    const uint32_t lane = threadIdx.x & 31u, groups = min(32u, max(1u, (n + 31u) / 32u));
    __syncthreads();  // the previous sum has been read
    for (uint32_t g = threadIdx.x >> 5; g < groups; g += CL_WARPS) {
        double v = 0.0;
        for (uint32_t e = g * 32u + lane; e < n; e += 1024u) v = v + partials[e];
        v = warp_fold(v);
        if (lane == 0) s_w32[g] = v;
    }
    __syncthreads();
    double total = s_w32[0];
    for (uint32_t g = 1; g < groups; ++g) total = total + s_w32[g];
    return total;
}

// The solve's setup: coarse types, stencil words, neighbour slots, the tail's lists and image.
__device__ __forceinline__ void cl_setup(const Dev& d, const MGState& m, int tail, uint32_t* s_warp) {
    const int nl = m.num_levels, top = min(3, nl - 1);
    for (int l = 1; l <= top; ++l)
        for (uint32_t i = pass_thread<true>(); i < m.lv[l].cells; i += gridDim.x * blockDim.x) m.lv[l].type[i] = 0u;
    cluster_barrier();
    build_types_fp13<true>(d, m, top);
    cluster_barrier();
    for (int l = top; l < nl - 1; ++l) {
        const MGLevel F = m.lv[l], C = m.lv[l + 1];
        for (uint32_t i = pass_thread<true>(); i < C.cells; i += gridDim.x * blockDim.x) build_type_cell(d, F, C, 0, i, coord3(i, C.dim));
        cluster_barrier();
    }
    level_words_fp13<true>(d, m, top);
    for (int l = top + 1; l < nl; ++l)
        for (uint32_t i = pass_thread<true>(); i < m.lv[l].cells; i += gridDim.x * blockDim.x) level_word_cell(m.lv[l], i, coord3(i, m.lv[l].dim));
    pcg_words<true>(d, m);
    cluster_barrier();
    if (blockIdx.x == 0u) {
        tail_lists(m, tail, s_warp);
        __syncthreads();
    }
}

// State of a solve that every thread holds.
struct ClState {
    double rho, rho_prev, dq, rr, bb, rz;
    uint32_t it;
    bool converged;
};

template <bool FLEX>
__device__ __forceinline__ ClState cl_streamed(const Dev& d, const MGState& m, const ClSolve& a, unsigned char* s_tail, double (*s_sum)[32]) {
    const uint32_t warp = threadIdx.x >> 5;
    float* scratch = reinterpret_cast<float*>(s_tail + a.tail_bytes + warp * (BRICK_CELLS * 5u));
    uint8_t* scratch_b = reinterpret_cast<uint8_t*>(scratch + BRICK_CELLS);
    const int tail = a.tail, sweeps = max(m.sweeps, 1);
    const bool relaxed = m.smooth_weight != 1.0f;
    const uint32_t active = d.active_bricks[0], cap = d.num_pool_bricks;
    auto no_store = [](double, double) {};
    double rho = m.scalars[0], rho_prev = 0.0, dq = 0.0, rz = 0.0, rr, bb;
    uint32_t it = 0u;
    bool converged;
    pcg_init<true>(d, m, a.p, a.div, no_store);
    cluster_barrier();
    rr = cl_reduce(m.partials, active, s_sum[0]);
    bb = cl_reduce(m.partials + cap, active, s_sum[1]);
    converged = a.tol_mode != 0u && (bb > 0.0 ? sqrt(rr / bb) : 0.0) <= a.tol;
    bool run = a.limit > 0u && !converged, image = true;
    while (run) {
        const float vs = coarse_scale(m, rr), ivs = 1.0f / vs;
        auto sweep = [&](int l, uint32_t parity) {
            const MGLevel L = m.lv[l];
            const uint32_t want = parity == 0u ? CW_RED : 0u;
            if (l <= 2) for_footprint_colour<true>(d, L, l, parity, [&](uint32_t i, int3) { smooth_fp_cell(L, i, want); });
            else for_footprint<true>(d, L, l, [&](uint32_t i, int3) { smooth_fp_cell(L, i, want); });
            cluster_barrier();
        };
        smooth0_black<true>(d, m);
        cluster_barrier();
        for (int k = 1; k < sweeps; ++k) {
            smooth0_red<false, false, true>(d, m, ivs);
            cluster_barrier();
            smooth0_black<true>(d, m);
            cluster_barrier();
        }
        for (int l = 0; l < tail; ++l) {
            if (l == 0) {
                restrict0<true>(d, m, vs, scratch, scratch_b);
            } else {
                const MGLevel F = m.lv[l], C = m.lv[l + 1];
                for_footprint<true>(d, C, l + 1, [&](uint32_t ci, int3 c) { restrict_fp_cell(F, C, ci, c, m.restrict_scale); });
            }
            cluster_barrier();
            if (l + 1 < tail) {
                sweep(l + 1, 1u);
                for (int k = 1; k < sweeps; ++k) {
                    sweep(l + 1, 0u);
                    sweep(l + 1, 1u);
                }
            }
        }
        if (blockIdx.x == 0u) vcycle_tail_body<false>(m, tail, a.coarse, s_tail, image);
        image = false;
        cluster_barrier();
        for (int l = tail - 1; l >= 1; --l) {
            const MGLevel F = m.lv[l], C = m.lv[l + 1];
            if (l <= 2) for_footprint_colour<true>(d, F, l, 1u, [&](uint32_t i, int3 c) { prolong_smooth_fp_cell(F, C, i, c); });
            else for_footprint<true>(d, F, l, [&](uint32_t i, int3 c) { prolong_smooth_fp_cell(F, C, i, c); });
            cluster_barrier();
            for (int k = 1; k < sweeps; ++k) {
                sweep(l, 0u);
                sweep(l, 1u);
            }
            sweep(l, 0u);
        }
        prolong_smooth0<true>(d, m, ivs, scratch);
        cluster_barrier();
        for (int k = 1; k < sweeps; ++k) {
            if (k == 1 && relaxed) smooth0_red<false, true, true>(d, m, ivs);
            else smooth0_red<false, false, true>(d, m, ivs);
            cluster_barrier();
            smooth0_black<true>(d, m);
            cluster_barrier();
        }
        if (sweeps == 1 && relaxed) smooth0_red<true, true, true>(d, m, ivs);
        else smooth0_red<true, false, true>(d, m, ivs);
        cluster_barrier();
        rho_prev = rho;
        rho = cl_reduce(m.partials, active, s_sum[0]);
        // into the other half of the partials: a slower CTA may still be reading rho's
        apply_a<true>(d, m, it, pcg_beta(it == 0u, FLEX, rho, rz, rho_prev), no_store, cap);
        cluster_barrier();
        dq = cl_reduce(m.partials + cap, active, s_sum[1]);
        if (FLEX) cluster_barrier();  // UpdatePR writes both halves
        update_pr<FLEX, true>(d, m, a.p, it, ratio_f(rho, dq), no_store);
        cluster_barrier();
        rr = cl_reduce(m.partials, active, s_sum[0]);
        if (FLEX) rz = cl_reduce(m.partials + cap, active, s_sum[1]);
        ++it;
        converged = a.tol_mode != 0u && (bb > 0.0 ? sqrt(rr / bb) : 0.0) <= a.tol;
        run = it < a.limit && !converged;
    }
    return {rho, rho_prev, dq, rr, bb, rz, it, converged};
}

// ---- the resident form ----------------------------------------------------------------------------------------
// Level 0 is kept by colour: cell (x, y, z) is entry (x >> 1) + 4 y + 32 z of its colour's 256, so a sweep's six
// neighbours are entries of the other colour's array: its own row's, +-4 and +-32. In round k lane t has the entries
// 2 h and 2 h + 1 of row y in plane z (h, y, z as in geo_of) of both colours, the cells 4 h .. 4 h + 3 of the row; which
// of them are red is the same in every round: x = 4 h + 2 jj + off, off = o for red and 1 - o for black cells.
struct ResWarp {
    ResBrick* B;
    uint32_t nb[6];       // cluster addresses of the face neighbours' blocks (0: no active brick there)
    uint32_t tail_sm;     // cluster address of CTA 0's tail
    int3 bc;              // brick coordinates
    uint32_t lane, base;  // first pool cell
    uint32_t o;           // off of the lane's red cells
    bool mine;            // the warp has a brick
    float q[2][4][2];     // by colour, round, jj: A d
};
#define RES_OFF(field) uint32_t(offsetof(ResBrick, field))

// The stencil words of entries i and i + 1 of a colour, in the low two bytes.
__device__ __forceinline__ uint32_t res_words(const ResWarp& W, uint32_t colour, uint32_t i) {
    return *reinterpret_cast<const uint16_t*>(W.B->word[colour] + i);
}
__device__ __forceinline__ uint32_t res_entry(const Geo& g) { return 2u * g.h + 4u * g.y + 32u * g.z; }

// Copies the face neighbours' cells of one colour of a level-0 array (at `off` of their blocks) into the warp's halo:
// words 0-63 the z faces (x >> 1) + 4 y, 64-127 the y faces (x >> 1) + 4 z, 128-255 the x faces y + 8 z.
__device__ __forceinline__ void res_pull(const ResWarp& W, uint32_t off, uint32_t colour) {
    const uint32_t t = W.lane, s = t >> 3, i = t & 7u;
    const uint32_t a4 = s == 0u ? W.nb[4] : (s == 1u ? W.nb[5] : (s == 2u ? W.nb[2] : W.nb[3]));
    const uint32_t src = s == 0u ? 224u + 4u * i : (s == 1u ? 4u * i : (s == 2u ? 28u + 32u * i : 32u * i));
    const uint32_t z = t >> 2, y0 = 2u * (t & 3u) + ((colour + 1u + z) & 1u), y1 = 2u * (t & 3u) + ((colour + z) & 1u);
    off += 1024u * colour;
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float x0 = 0.0f, x1 = 0.0f;
    if (a4) v = dsm_ld4(a4 + off + 4u * src);
    if (W.nb[0]) x0 = dsm_ld(W.nb[0] + off + 4u * (3u + 4u * y0 + 32u * z));
    if (W.nb[1]) x1 = dsm_ld(W.nb[1] + off + 4u * (4u * y1 + 32u * z));
    float* h = W.B->halo;
    __syncwarp();  // the last pull's values have been used
    *reinterpret_cast<float4*>(h + 4u * t) = v;
    h[128u + y0 + 8u * z] = x0;
    h[192u + y1 + 8u * z] = x1;
    __syncwarp();
}
// The six neighbours of the lane's two cells of a colour in round k, from the other colour's array F and its halo.
struct Nb2 {
    float n[2][6];
};
__device__ __forceinline__ float2 ld2(const float* p) { return *reinterpret_cast<const float2*>(p); }
__device__ __forceinline__ void st2(float* p, float a, float b) { *reinterpret_cast<float2*>(p) = make_float2(a, b); }
__device__ __forceinline__ Nb2 res_nbrs(const ResWarp& W, const float* F, const Geo& g, uint32_t off) {
    const float* h = W.B->halo;
    const uint32_t i = res_entry(g);
    const float2 c = ld2(F + i);
    const float e = off == 0u ? (g.h ? F[i - 1u] : h[128u + g.y + 8u * g.z]) : (g.h ? h[192u + g.y + 8u * g.z] : F[i + 2u]);
    const float2 ym = ld2(g.y > 0u ? F + i - 4u : h + 64u + 2u * g.h + 4u * g.z);
    const float2 yp = ld2(g.y < 7u ? F + i + 4u : h + 96u + 2u * g.h + 4u * g.z);
    const float2 zm = ld2(g.z > 0u ? F + i - 32u : h + 2u * g.h + 4u * g.y);
    const float2 zp = ld2(g.z < 7u ? F + i + 32u : h + 32u + 2u * g.h + 4u * g.y);
    Nb2 r;
    r.n[0][0] = off ? c.x : e;   r.n[0][1] = off ? c.y : c.x;
    r.n[1][0] = off ? c.y : c.x; r.n[1][1] = off ? e : c.y;
    r.n[0][2] = ym.x; r.n[0][3] = yp.x; r.n[0][4] = zm.x; r.n[0][5] = zp.x;
    r.n[1][2] = ym.y; r.n[1][3] = yp.y; r.n[1][4] = zm.y; r.n[1][5] = zp.y;
    return r;
}
__device__ __forceinline__ uint32_t res_off(const ResWarp& W, uint32_t colour) { return colour == 0u ? W.o : 1u - W.o; }
// Adds a lane's four values of a round in x order: red[0], black[0], red[1], black[1], or black first.
__device__ __forceinline__ double res_add(const ResWarp& W, double acc, const double (&red)[2], const double (&black)[2]) {
#pragma unroll
    for (int jj = 0; jj < 2; ++jj) {
        acc = acc + (W.o ? black[jj] : red[jj]);
        acc = acc + (W.o ? red[jj] : black[jj]);
    }
    return acc;
}

// One colour of level 0 (0 red, 1 black). PROLONGED: the values start from the cell's prolonged value (see load_sweep).
template <uint32_t COLOUR, bool PROLONGED>
__device__ __forceinline__ void res_sweep0(const MGState& m, ResWarp& W, float ivs) {
    if (!W.mine) return;
    res_pull(W, RES_OFF(z), 1u - COLOUR);
    const uint32_t off = res_off(W, COLOUR);
    const bool relax = m.smooth_weight != 1.0f;
#pragma unroll 1
    for (uint32_t k = 0; k < 4u; ++k) {
        const Geo g = geo_of(0u, W.lane, k);
        const Nb2 nb = res_nbrs(W, W.B->z[1u - COLOUR], g, off);
        const uint32_t i = res_entry(g);
        const uint32_t ws = res_words(W, COLOUR, i);
        float* zc = W.B->z[COLOUR] + i;
        const float2 zo = ld2(zc), rc = ld2(W.B->rc[COLOUR] + i), dg = ld2(W.B->dg[COLOUR] + i), r = ld2(W.B->r[COLOUR] + i);
        float out[2] = {zo.x, zo.y};
#pragma unroll
        for (uint32_t jj = 0; jj < 2u; ++jj) {
            const uint32_t w = (ws >> (8u * jj)) & 0xFFu;
            if (!(w & W_FLUID)) continue;
            const float val = div_by((jj ? r.y : r.x) + nb_sum(nb.n[jj], w), jj ? dg.y : dg.x, jj ? rc.y : rc.x);
            float from = out[jj];
            if (PROLONGED && relax) from = from + W.B->x1[2u * g.h + jj + 4u * (g.y >> 1) + 16u * (g.z >> 1)] * ivs;
            out[jj] = relax0(m, from, val);
        }
        st2(zc, out[0], out[1]);
    }
    __syncwarp();
}
// The lane's part of r.z, after the sweeps (its own cells).
__device__ __forceinline__ double res_dot_rz(const ResWarp& W) {
    double acc = 0.0;
    if (!W.mine) return acc;
#pragma unroll 1
    for (uint32_t k = 0; k < 4u; ++k) {
        const Geo g = geo_of(0u, W.lane, k);
        double v[2][2];
#pragma unroll
        for (uint32_t c = 0; c < 2u; ++c) {
            const uint32_t i = res_entry(g);
            const uint32_t ws = res_words(W, c, i);
            const float2 z = ld2(W.B->z[c] + i), r = ld2(W.B->r[c] + i);
#pragma unroll
            for (uint32_t jj = 0; jj < 2u; ++jj)
                v[c][jj] = ((ws >> (8u * jj)) & W_FLUID) ? double((jj ? r.y : r.x) * (jj ? z.y : z.x)) : 0.0;
        }
        acc = res_add(W, acc, v[0], v[1]);
    }
    return acc;
}
// k_prolong_smooth0: the black sweep over the red neighbours' prolonged values.
__device__ __forceinline__ void res_prolong0(const MGState& m, ResWarp& W, float ivs) {
    if (!W.mine) return;
    float v1[3];
#pragma unroll
    for (uint32_t s = 0; s < 3u; ++s) {  // 6 faces x 16 level-1 cells, in pairs of faces
        const uint32_t hi = W.lane >> 4, i = W.lane & 15u, u = i & 3u, v = i >> 2;
        const uint32_t a = hi ? W.nb[2 * s + 1] : W.nb[2 * s];
        const uint32_t f = hi ? 0u : 3u;
        const uint32_t l = s == 0u ? f + 4u * u + 16u * v : (s == 1u ? u + 4u * f + 16u * v : u + 4u * v + 16u * f);
        v1[s] = a ? dsm_ld(a + RES_OFF(x1) + 4u * l) : 0.0f;
    }
#pragma unroll
    for (uint32_t s = 0; s < 3u; ++s) W.B->halo1[32u * s + W.lane] = v1[s];
    res_pull(W, RES_OFF(z), 0u);
    const float* x1 = W.B->x1;
    const float* h1 = W.B->halo1;
    const uint32_t off = res_off(W, 1u);
#pragma unroll 1
    for (uint32_t k = 0; k < 4u; ++k) {
        const Geo g = geo_of(0u, W.lane, k);
        const Nb2 nb = res_nbrs(W, W.B->z[0], g, off);
        const uint32_t i = res_entry(g);
        const uint32_t ws = res_words(W, 1u, i);
        float* zc = W.B->z[1] + i;
        const float2 zo = ld2(zc), rc = ld2(W.B->rc[1] + i), dg = ld2(W.B->dg[1] + i), r = ld2(W.B->r[1] + i);
        float out[2] = {zo.x, zo.y};
        const uint32_t cy = g.y >> 1, cz = g.z >> 1;
#pragma unroll
        for (uint32_t jj = 0; jj < 2u; ++jj) {
            const uint32_t w = (ws >> (8u * jj)) & 0xFFu;
            if (!(w & W_FLUID)) continue;
            const uint32_t cx = 2u * g.h + jj, p = cx + 4u * cy + 16u * cz;
            const float own = x1[p];
            float c[6];
            c[0] = off ? own : (cx > 0u ? x1[p - 1u] : h1[cy + 4u * cz]);
            c[1] = !off ? own : (cx < 3u ? x1[p + 1u] : h1[16u + cy + 4u * cz]);
            c[2] = (g.y & 1u) ? own : (cy > 0u ? x1[p - 4u] : h1[32u + cx + 4u * cz]);
            c[3] = !(g.y & 1u) ? own : (cy < 3u ? x1[p + 4u] : h1[48u + cx + 4u * cz]);
            c[4] = (g.z & 1u) ? own : (cz > 0u ? x1[p - 16u] : h1[64u + cx + 4u * cy]);
            c[5] = !(g.z & 1u) ? own : (cz < 3u ? x1[p + 16u] : h1[80u + cx + 4u * cy]);
            float sum = 0.0f;
#pragma unroll
            for (int b = 0; b < 6; ++b)
                if ((w >> b) & 1u) sum = sum + (nb.n[jj][b] + c[b] * ivs);
            out[jj] = relax0(m, out[jj] + own * ivs, div_by((jj ? r.y : r.x) + sum, jj ? dg.y : dg.x, jj ? rc.y : rc.x));
        }
        st2(zc, out[0], out[1]);
    }
}

// Levels 1-3 of the brick: side S = 8 >> l, cells x + S (y + S z).
template <int S> __device__ __forceinline__ float* res_x(ResBrick* B) { return S == 4 ? B->x1 : (S == 2 ? B->x2 : B->x3); }
template <int S> __device__ __forceinline__ float* res_b(ResBrick* B) { return S == 4 ? B->b1 : (S == 2 ? B->b2 : B->b3); }
template <int S> __device__ __forceinline__ uint16_t* res_w(ResBrick* B) { return S == 4 ? B->w1 : (S == 2 ? B->w2 : B->w3); }
template <int S> __device__ __forceinline__ uint32_t res_x_off() { return S == 4 ? RES_OFF(x1) : (S == 2 ? RES_OFF(x2) : RES_OFF(x3)); }
// x of neighbour n of cell (x, y, z) of the level, read where bit n of w says it is fluid.
template <int S>
__device__ __forceinline__ float res_nbr(const ResWarp& W, uint32_t w, int x, int y, int z, int n) {
    if (!((w >> n) & 1u)) return 0.0f;
    const int a = n >> 1, v = a == 0 ? x : (a == 1 ? y : z), st = a == 0 ? 1 : (a == 1 ? S : S * S), l = x + S * (y + S * z);
    if ((n & 1) ? v < S - 1 : v > 0) return res_x<S>(W.B)[(n & 1) ? l + st : l - st];
    return dsm_ld(W.nb[n] + res_x_off<S>() + 4u * uint32_t((n & 1) ? l - (S - 1) * st : l + (S - 1) * st));
}
// Cell j (one of S^3 / 2) of a colour; a single cell (S = 1) has the colour of its brick.
template <int S>
__device__ __forceinline__ bool res_colour(const ResWarp& W, uint32_t parity, int& x, int& y, int& z) {
    if (S == 1) {
        x = y = z = 0;
        return W.lane == 0u && (uint32_t(W.bc.x + W.bc.y + W.bc.z) & 1u) == parity;
    }
    constexpr uint32_t half = S > 1 ? S / 2 : 1;
    if (W.lane >= half * S * S) return false;
    y = int((W.lane / half) % S);
    z = int(W.lane / (half * S));
    x = int(2u * (W.lane % half) + (uint32_t(y + z + int(parity)) & 1u));
    return true;
}
template <int S>
__device__ __forceinline__ void res_sweep(const ResWarp& W, uint32_t prec, uint32_t parity) {
    int x, y, z;
    if (!W.mine || !res_colour<S>(W, parity, x, y, z)) return;
    const int l = x + S * (y + S * z);
    const uint32_t w = res_w<S>(W.B)[l];
    if (!(w & CW_FLUID)) return;
    float v[6], sum = 0.0f;
#pragma unroll
    for (int n = 0; n < 6; ++n) v[n] = res_nbr<S>(W, w, x, y, z, n);
#pragma unroll
    for (int n = 0; n < 6; ++n)
        if ((w >> n) & 1u) sum = sum + v[n];
    res_x<S>(W.B)[l] = q_prec((res_b<S>(W.B)[l] + sum) / word_diag(w), prec);
}
// Stores b and the red-initialised x of coarse cell lc (side S) of the brick: in its block, or in CTA 0's tail when the
// level is the tail's. sum: the fluid children's residuals times the restriction's scale.
template <int S>
__device__ __forceinline__ void res_put_coarse(const MGState& m, const ResWarp& W, int level, int tail, uint32_t lc, float bb) {
    const uint32_t cw = res_w<S>(W.B)[lc], prec = m.lv[level].prec;
    const bool fluid = (cw & CW_FLUID) != 0u;
    const float b = fluid ? q_prec(bb, prec) : 0.0f, x = fluid && (cw & CW_RED) ? q_prec(bb / word_diag(cw), prec) : 0.0f;
    if (level < tail) {
        res_b<S>(W.B)[lc] = b;
        res_x<S>(W.B)[lc] = x;
        return;
    }
    const int3 c = make_int3(W.bc.x * S + int(lc % S), W.bc.y * S + int((lc / S) % S), W.bc.z * S + int(lc / (S * S)));
    if (!inside3(c, m.lv[level].dim)) return;
    const uint32_t ci = lin3(c, m.lv[level].dim);
    dsm_st(W.tail_sm + 4u * ci, x);                                        // level tail's x, then its b, come first
    dsm_st(W.tail_sm + 4u * (tail_pad4(m.lv[level].cells) + ci), b);
}
// k_restrict0: the residuals stay with their lanes; the lane with even y and z of a coarse cell takes its 8 children's from
// the lanes t ^ 2 (y), t ^ 16 (z) and t ^ 18 and adds the fluid ones in child order.
__device__ __forceinline__ void res_restrict0(const MGState& m, ResWarp& W, int tail, float vs) {
    if (!W.mine) return;
    float res[2][4][2];
    uint32_t fl4 = 0u;  // fluid bits: 4 k + 2 c + jj
#pragma unroll
    for (uint32_t c = 0; c < 2u; ++c) {
        res_pull(W, RES_OFF(z), 1u - c);
        const uint32_t off = res_off(W, c);
#pragma unroll
        for (uint32_t k = 0; k < 4u; ++k) {
            const Geo g = geo_of(0u, W.lane, k);
            const Nb2 nb = res_nbrs(W, W.B->z[1u - c], g, off);
            const uint32_t i = res_entry(g);
            const float2 z = ld2(W.B->z[c] + i), r = ld2(W.B->r[c] + i), dg = ld2(W.B->dg[c] + i);
            const uint32_t ws = res_words(W, c, i);
#pragma unroll
            for (uint32_t jj = 0; jj < 2u; ++jj)
                res[c][k][jj] = (jj ? r.y : r.x) - ((jj ? dg.y : dg.x) * (jj ? z.y : z.x) - nb_sum(nb.n[jj], (ws >> (8u * jj)) & 0xFFu));
            fl4 |= (((ws & W_FLUID) ? 1u : 0u) | ((ws & (W_FLUID << 8)) ? 2u : 0u)) << (4u * k + 2u * c);
            asm volatile("" ::: "memory");  // one round's loads at a time: hoisted, they spill
        }
    }
#pragma unroll
    for (uint32_t k = 0; k < 4u; ++k) {
        const Geo g = geo_of(0u, W.lane, k);
        float mine[4];  // x order
        uint32_t fl = 0u;
#pragma unroll
        for (uint32_t jj = 0; jj < 2u; ++jj) {
            const uint32_t fr = (fl4 >> (4u * k + jj)) & 1u, fb = (fl4 >> (4u * k + 2u + jj)) & 1u;
            mine[2 * jj] = W.o ? res[1][k][jj] : res[0][k][jj];
            mine[2 * jj + 1] = W.o ? res[0][k][jj] : res[1][k][jj];
            fl |= ((W.o ? fb : fr) | ((W.o ? fr : fb) << 1)) << (2u * jj);
        }
        const uint32_t from[3] = {2u, 16u, 18u};
        float ro[3][4];
        uint32_t fo[3];
#pragma unroll
        for (int s = 0; s < 3; ++s) {
            fo[s] = __shfl_xor_sync(0xFFFFFFFFu, fl, int(from[s]));
#pragma unroll
            for (int j = 0; j < 4; ++j) ro[s][j] = __shfl_xor_sync(0xFFFFFFFFu, mine[j], int(from[s]));
        }
        if ((W.lane & 18u) == 0u) {
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                float sum = 0.0f;
#pragma unroll
                for (int o = 0; o < 8; ++o) {
                    const int j = 2 * c + (o & 1), s = (o >> 1) - 1;
                    const uint32_t f = s < 0 ? fl : fo[s < 0 ? 0 : s];
                    if ((f >> j) & 1u) sum = sum + (s < 0 ? mine[j] : ro[s < 0 ? 0 : s][j]);
                }
                res_put_coarse<4>(m, W, 1, tail, 2u * g.h + uint32_t(c) + 4u * (g.y >> 1) + 16u * k, (m.restrict_scale * sum) * vs);
            }
        }
    }
}
// k_restrict_fp from level l (side S) to l + 1: residuals of the brick's cells through shared memory.
template <int S>
__device__ __forceinline__ void res_restrict(const MGState& m, const ResWarp& W, int l, int tail) {
    if (!W.mine) return;
    constexpr uint32_t CELLS = S * S * S;
    for (uint32_t i = W.lane; i < CELLS; i += 32u) {
        const uint32_t w = res_w<S>(W.B)[i];
        if (!(w & CW_FLUID)) continue;
        const int x = int(i % S), y = int((i / S) % S), z = int(i / (S * S));
        float v[6], sum = 0.0f;
#pragma unroll
        for (int n = 0; n < 6; ++n) v[n] = res_nbr<S>(W, w, x, y, z, n);
#pragma unroll
        for (int n = 0; n < 6; ++n)
            if ((w >> n) & 1u) sum = sum + v[n];
        W.B->res[i] = res_b<S>(W.B)[i] - (word_diag(w) * res_x<S>(W.B)[i] - sum);
    }
    __syncwarp();
    constexpr int H = S / 2;
    if (W.lane < uint32_t(H * H * H)) {
        const int cx = int(W.lane) % H, cy = (int(W.lane) / H) % H, cz = int(W.lane) / (H * H);
        float sum = 0.0f;
#pragma unroll
        for (int o = 0; o < 8; ++o) {
            const uint32_t i = uint32_t((2 * cx + (o & 1)) + S * ((2 * cy + ((o >> 1) & 1)) + S * (2 * cz + ((o >> 2) & 1))));
            if (res_w<S>(W.B)[i] & CW_FLUID) sum = sum + W.B->res[i];
        }
        res_put_coarse<H>(m, W, l + 1, tail, W.lane, m.restrict_scale * sum);
    }
}
// k_prolong_smooth_fp from level l + 1 to level l (side S): the black sweep over the neighbours' prolonged values. A
// parent that is not fluid has x = 0, which adds nothing.
template <int S>
__device__ __forceinline__ void res_prolong(const MGState& m, const ResWarp& W, int l, int tail) {
    int x, y, z;
    if (!W.mine || !res_colour<S>(W, 1u, x, y, z)) return;
    const int i = x + S * (y + S * z);
    const uint32_t w = res_w<S>(W.B)[i], prec = m.lv[l].prec;
    if (!(w & CW_FLUID)) return;
    constexpr int H = S / 2 > 0 ? S / 2 : 1;
    float v[6], c[6], sum = 0.0f;
#pragma unroll
    for (int n = 0; n < 6; ++n) {
        v[n] = res_nbr<S>(W, w, x, y, z, n);
        c[n] = 0.0f;
        if (!((w >> n) & 1u)) continue;
        const int3 o = nbr_off(n);
        const int nx = x + o.x, ny = y + o.y, nz = z + o.z;  // may lie in the face neighbour
        if (l + 1 == tail) {
            const int3 pc = make_int3((W.bc.x * S + nx) >> 1, (W.bc.y * S + ny) >> 1, (W.bc.z * S + nz) >> 1);
            c[n] = dsm_ld(W.tail_sm + 4u * lin3(pc, m.lv[tail].dim));
        } else {
            const bool out = nx < 0 || ny < 0 || nz < 0 || nx >= S || ny >= S || nz >= S;
            const uint32_t p = uint32_t(((nx & (S - 1)) >> 1) + H * (((ny & (S - 1)) >> 1) + H * ((nz & (S - 1)) >> 1)));
            c[n] = out ? dsm_ld(W.nb[n] + res_x_off<H>() + 4u * p) : res_x<H>(W.B)[p];
        }
    }
#pragma unroll
    for (int n = 0; n < 6; ++n)
        if ((w >> n) & 1u) sum = sum + q_prec(v[n] + c[n], prec);
    res_x<S>(W.B)[i] = q_prec((res_b<S>(W.B)[i] + sum) / word_diag(w), prec);
}
// A level's call with its side.
#define RES_LEVEL(l, call)            \
    do {                              \
        if ((l) == 1) call(4);        \
        else if ((l) == 2) call(2);   \
        else call(1);                 \
    } while (0)

template <bool FLEX>
__device__ __forceinline__ ClState cl_resident(const Dev& d, const MGState& m, const ClSolve& a, unsigned char* s_tail, double (*s_sum)[32],
                                               double (*s_part)[CL_PARTIALS], uint32_t* s_active, SLevel* s_levels, float* s_dt) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, rank = blockIdx.x;
    const uint32_t active = d.active_bricks[0], others = gridDim.x - 1u, per = (active + others - 1u) / others;
    const uint32_t e = (rank - 1u) * per + warp;  // CTA 0 has the tail, no bricks
    const int tail = a.tail, sweeps = max(m.sweeps, 1);
    const uint32_t blocks_sm = uint32_t(__cvta_generic_to_shared(s_tail));
    ResWarp W;
    W.lane = lane;
    W.mine = rank > 0u && warp < per && e < active;
    W.B = reinterpret_cast<ResBrick*>(s_tail) + warp;
    W.tail_sm = cl_mapa(uint32_t(__cvta_generic_to_shared(s_tail)), 0u);
    for (uint32_t i = threadIdx.x; i < active; i += CL_THREADS) s_active[i] = d.active_bricks[1u + i];
    __syncthreads();
    const uint32_t part_sm = uint32_t(__cvta_generic_to_shared(&s_part[0][0]));
    // dot product `which`: every CTA gets the brick's partial
    auto send = [&](uint32_t which, double lane_sum) {
        if (!W.mine) return;
        const double t = __shfl_sync(0xFFFFFFFFu, warp_fold(lane_sum), 0);
        if (lane < gridDim.x) dsm_st(cl_mapa(part_sm + 8u * (which * CL_PARTIALS + e), lane), t);
    };
    auto total = [&](uint32_t which) { return cl_reduce(s_part[which], active, s_sum[which & 1u]); };
    double rr_l = 0.0, bb_l = 0.0;
    uint32_t ns[6] = {0u, 0u, 0u, 0u, 0u, 0u};
    W.base = 0u;
    W.o = (((lane >> 1) & 7u) + (lane >> 4)) & 1u;
#pragma unroll
    for (int k = 0; k < 16; ++k) W.q[k >> 3][(k >> 1) & 3][k & 1] = 0.0f;
    W.bc = make_int3(0, 0, 0);
#pragma unroll
    for (int n = 0; n < 6; ++n) W.nb[n] = 0u;
    if (W.mine) {
        const uint4 s0 = *reinterpret_cast<const uint4*>(m.nbr_slots + 8u * e);
        const uint4 s1 = *reinterpret_cast<const uint4*>(m.nbr_slots + 8u * e + 4u);
        ns[0] = s0.x; ns[1] = s0.y; ns[2] = s0.z; ns[3] = s0.w; ns[4] = s1.x; ns[5] = s1.y;
        W.base = s1.z * BRICK_CELLS;
        W.bc = brick_coord_of(d, s1.w);
        // the neighbours' places: their entries in the (ascending) active list
#pragma unroll
        for (int n = 0; n < 6; ++n) {
            const int3 b = add3(W.bc, nbr_off(n));
            if (b.x < 0 || b.y < 0 || b.z < 0 || b.x >= d.brick_dim.x || b.y >= d.brick_dim.y || b.z >= d.brick_dim.z) continue;
            const uint32_t key = brick_index_of(d, b);
            uint32_t lo = 0u, hi = active;
            while (lo < hi) {
                const uint32_t mid = (lo + hi) >> 1;
                if (s_active[mid] < key) lo = mid + 1u;
                else hi = mid;
            }
            if (lo < active && s_active[lo] == key)
                W.nb[n] = cl_mapa(blocks_sm + (lo % per) * uint32_t(sizeof(ResBrick)), 1u + lo / per);
        }
        auto words = [&](int l, uint16_t* w, uint32_t S) {  // the level's words of the brick's cells
            const MGLevel L = m.lv[l];
            for (uint32_t i = lane; i < S * S * S; i += 32u) {
                const int3 c = make_int3(W.bc.x * int(S) + int(i % S), W.bc.y * int(S) + int((i / S) % S), W.bc.z * int(S) + int(i / (S * S)));
                w[i] = inside3(c, L.dim) ? L.word[lin3(c, L.dim)] : uint16_t(0);
            }
        };
        words(1, W.B->w1, 4u);
        if (tail >= 2) words(2, W.B->w2, 2u);
        if (tail >= 3) words(3, W.B->w3, 1u);
        // PCGInit
#pragma unroll 1
        for (uint32_t k = 0; k < 4u; ++k) {
            const Geo g = geo_of(W.base, lane, k);
            const Q6 p = load_q6(a.p, g, ns);
            const float4 dv = ld4(a.div + g.i), dgv = ld4(d.cell_diag + g.i);
            const uint32_t w4 = quad_words(m, g);
            const X2 x = partner(p);
            double v0[2][2], v1[2][2];
            float zq[4], rq[4];
            double tq0[4], tq1[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t w = word_of(w4, j);
                const float diag = comp(dgv, j) + DIAG_EPSILON;
                rq[j] = zq[j] = 0.0f;
                tq0[j] = tq1[j] = 0.0;
                if (w & W_FLUID) {
                    float n[6];
                    nbrs6(p, x, g.h, j, n);
                    const float b = -comp(dv, j);
                    rq[j] = b - (diag * comp(p.c, j) - nb_sum(n, w));
                    zq[j] = (w & W_RED) ? red_init0(m, rq[j] / diag) : 0.0f;
                    tq0[j] = double(rq[j] * rq[j]);
                    tq1[j] = double(b * b);
                }
            }
            float zc[2][2], rs[2][2], dg[2][2];
            uint32_t wc[2] = {0u, 0u};
#pragma unroll
            for (uint32_t c = 0; c < 2u; ++c)
#pragma unroll
                for (uint32_t jj = 0; jj < 2u; ++jj) {
                    const bool odd = res_off(W, c) != 0u;
                    const uint32_t w = (w4 >> (8u * (2u * jj + (odd ? 1u : 0u)))) & 0xFFu;
                    wc[c] |= w << (8u * jj);
                    rs[c][jj] = odd ? rq[2 * jj + 1] : rq[2 * jj];
                    dg[c][jj] = (odd ? comp(dgv, int(2 * jj + 1)) : comp(dgv, int(2 * jj))) + DIAG_EPSILON;
                    zc[c][jj] = odd ? zq[2 * jj + 1] : zq[2 * jj];
                    v0[c][jj] = odd ? tq0[2 * jj + 1] : tq0[2 * jj];
                    v1[c][jj] = odd ? tq1[2 * jj + 1] : tq1[2 * jj];
                }
            rr_l = res_add(W, rr_l, v0[0], v0[1]);
            bb_l = res_add(W, bb_l, v1[0], v1[1]);
            const uint32_t i = res_entry(g);
            st2(W.B->z[0] + i, zc[0][0], zc[0][1]);
            st2(W.B->z[1] + i, zc[1][0], zc[1][1]);
#pragma unroll
            for (uint32_t c = 0; c < 2u; ++c) {
                *reinterpret_cast<uint16_t*>(W.B->word[c] + i) = uint16_t(wc[c]);
                st2(W.B->r[c] + i, rs[c][0], rs[c][1]);
                st2(W.B->dg[c] + i, dg[c][0], dg[c][1]);
                st2(W.B->rc[c] + i, 1.0f / dg[c][0], 1.0f / dg[c][1]);
            }
        }
    }
    if (rank == 0u) {
        tail_levels(m, tail, s_tail, s_levels, s_dt);
        // the tail's static part: words and colour lists behind level tail's x and b
        const uint4* img = reinterpret_cast<const uint4*>(m.tail_image);
        const uint32_t c16 = tail_pad4(m.lv[tail].cells) / 2u;
        uint32_t bytes = 0u;
        tail_offsets(m, tail, -1, &bytes);
        for (uint32_t k = c16 + threadIdx.x; k < bytes / 16u; k += CL_THREADS) reinterpret_cast<uint4*>(s_tail)[k] = img[k];
    }
    cluster_barrier();  // every CTA runs: its shared memory may be written
    send(2u, rr_l);
    send(3u, bb_l);
    cluster_barrier();
    double rho = m.scalars[0], rho_prev = 0.0, dq = 0.0, rz = 0.0, rr = total(2u);
    const double bb = total(3u);
    uint32_t it = 0u;
    bool converged = a.tol_mode != 0u && (bb > 0.0 ? sqrt(rr / bb) : 0.0) <= a.tol;
    bool run = a.limit > 0u && !converged;
    while (run) {
        const float vs = coarse_scale(m, rr), ivs = 1.0f / vs;
        auto sweep = [&](int l, uint32_t parity) {
            const uint32_t prec = m.lv[l].prec;
#define RES_CALL(S) res_sweep<S>(W, prec, parity)
            RES_LEVEL(l, RES_CALL);
#undef RES_CALL
            cluster_barrier();
        };
        res_sweep0<1u, false>(m, W, ivs);
        cluster_barrier();
        for (int k = 1; k < sweeps; ++k) {
            res_sweep0<0u, false>(m, W, ivs);
            cluster_barrier();
            res_sweep0<1u, false>(m, W, ivs);
            cluster_barrier();
        }
        res_restrict0(m, W, tail, vs);
        cluster_barrier();
        for (int l = 1; l < tail; ++l) {
            sweep(l, 1u);
            for (int k = 1; k < sweeps; ++k) {
                sweep(l, 0u);
                sweep(l, 1u);
            }
            if (l == 1) res_restrict<4>(m, W, 1, tail);
            else res_restrict<2>(m, W, 2, tail);
            cluster_barrier();
        }
        if (rank == 0u) vcycle_tail_levels(m, tail, a.coarse, s_levels);
        cluster_barrier();
        for (int l = tail - 1; l >= 1; --l) {
            if (l == 1) res_prolong<4>(m, W, 1, tail);
            else res_prolong<2>(m, W, 2, tail);
            cluster_barrier();
            for (int k = 1; k < sweeps; ++k) {
                sweep(l, 0u);
                sweep(l, 1u);
            }
            sweep(l, 0u);
        }
        if (tail == 1) {  // level 1 is the tail's: bring its x into the bricks' blocks
            if (W.mine)
                for (uint32_t i = lane; i < 64u; i += 32u) {
                    const int3 c = make_int3(W.bc.x * 4 + int(i & 3u), W.bc.y * 4 + int((i >> 2) & 3u), W.bc.z * 4 + int(i >> 4));
                    W.B->x1[i] = (W.B->w1[i] & CW_FLUID) ? dsm_ld(W.tail_sm + 4u * lin3(c, m.lv[1].dim)) : 0.0f;
                }
            cluster_barrier();
        }
        res_prolong0(m, W, ivs);
        cluster_barrier();
        for (int k = 1; k < sweeps; ++k) {
            if (k == 1) res_sweep0<0u, true>(m, W, ivs);
            else res_sweep0<0u, false>(m, W, ivs);
            cluster_barrier();
            res_sweep0<1u, false>(m, W, ivs);
            cluster_barrier();
        }
        if (sweeps == 1) res_sweep0<0u, true>(m, W, ivs);
        else res_sweep0<0u, false>(m, W, ivs);
        send(0u, res_dot_rz(W));
        cluster_barrier();
        rho_prev = rho;
        rho = total(0u);
        // UpdateD on the own cells, then ApplyA over the neighbours' new directions
        const float beta = pcg_beta(it == 0u, FLEX, rho, rz, rho_prev);
        if (W.mine) {
#pragma unroll 1
            for (uint32_t k = 0; k < 4u; ++k) {
                const Geo g = geo_of(0u, lane, k);
#pragma unroll
                for (uint32_t c = 0; c < 2u; ++c) {
                    const uint32_t i = res_entry(g);
                    const uint32_t ws = res_words(W, c, i);
                    const float2 z = ld2(W.B->z[c] + i);
                    float dn[2] = {z.x, z.y};
                    if (it != 0u) {
                        const float2 dd = ld2(W.B->d[c] + i);
                        dn[0] = z.x + beta * dd.x;
                        dn[1] = z.y + beta * dd.y;
                    }
#pragma unroll
                    for (uint32_t jj = 0; jj < 2u; ++jj)
                        if (!((ws >> (8u * jj)) & W_FLUID)) dn[jj] = 0.0f;
                    st2(W.B->d[c] + i, dn[0], dn[1]);
                }
            }
        }
        cluster_barrier();
        double dot = 0.0;
        if (W.mine) {
#pragma unroll
            for (uint32_t c = 0; c < 2u; ++c) {
                res_pull(W, RES_OFF(d), 1u - c);
                const uint32_t off = res_off(W, c);
#pragma unroll
                for (uint32_t k = 0; k < 4u; ++k) {
                    const Geo g = geo_of(0u, lane, k);
                    const Nb2 nb = res_nbrs(W, W.B->d[1u - c], g, off);
                    const uint32_t i = res_entry(g);
                    const float2 dv = ld2(W.B->d[c] + i), dg = ld2(W.B->dg[c] + i);
                    const uint32_t ws = res_words(W, c, i);
#pragma unroll
                    for (uint32_t jj = 0; jj < 2u; ++jj) {
                        const uint32_t w = (ws >> (8u * jj)) & 0xFFu;
                        W.q[c][k][jj] = (w & W_FLUID) ? (jj ? dg.y : dg.x) * (jj ? dv.y : dv.x) - nb_sum(nb.n[jj], w) : 0.0f;
                    }
                    asm volatile("" ::: "memory");
                }
            }
#pragma unroll
            for (uint32_t k = 0; k < 4u; ++k) {
                const Geo g = geo_of(0u, lane, k);
                double v[2][2];
#pragma unroll
                for (uint32_t c = 0; c < 2u; ++c) {
                    const float2 dv = ld2(W.B->d[c] + res_entry(g));
                    const uint32_t ws = res_words(W, c, res_entry(g));
#pragma unroll
                    for (uint32_t jj = 0; jj < 2u; ++jj)
                        v[c][jj] = ((ws >> (8u * jj)) & W_FLUID) ? double((jj ? dv.y : dv.x) * W.q[c][k][jj]) : 0.0;
                }
                dot = res_add(W, dot, v[0], v[1]);
            }
        }
        send(1u, dot);
        cluster_barrier();
        dq = total(1u);
        // UpdatePR
        const float alpha = ratio_f(rho, dq);
        double rr_n = 0.0, rz_n = 0.0;
        if (W.mine) {
#pragma unroll
            for (uint32_t k = 0; k < 4u; ++k) {
                const Geo g = geo_of(W.base, lane, k);
                const uint32_t i = res_entry(g);
                double v0[2][2], v1[2][2];
                float dn[2][2];
                uint32_t wc[2];
                const float4 pv = ld4(a.p + g.i);
                const float2 rc = ld2(W.B->rc[0] + i), dg = ld2(W.B->dg[0] + i);
#pragma unroll
                for (uint32_t c = 0; c < 2u; ++c) {
                    const float2 dv = ld2(W.B->d[c] + i);
                    wc[c] = res_words(W, c, i);
                    float2 zv = make_float2(0.0f, 0.0f);
                    if (FLEX) zv = ld2(W.B->z[c] + i);
                    const float2 r = ld2(W.B->r[c] + i);
                    float zo[2], rn[2] = {r.x, r.y};
#pragma unroll
                    for (uint32_t jj = 0; jj < 2u; ++jj) {
                        dn[c][jj] = jj ? dv.y : dv.x;
                        zo[jj] = 0.0f;
                        v0[c][jj] = v1[c][jj] = 0.0;
                        if (!((wc[c] >> (8u * jj)) & W_FLUID)) continue;
                        const float ri = rn[jj] - alpha * W.q[c][k][jj];
                        rn[jj] = ri;
                        if (c == 0u) zo[jj] = red_init0(m, div_by(ri, jj ? dg.y : dg.x, jj ? rc.y : rc.x));
                        v0[c][jj] = double(ri * ri);
                        if (FLEX) v1[c][jj] = double(ri * (jj ? zv.y : zv.x));
                    }
                    st2(W.B->z[c] + i, zo[0], zo[1]);
                    st2(W.B->r[c] + i, rn[0], rn[1]);
                }
                float po[4] = {pv.x, pv.y, pv.z, pv.w};
#pragma unroll
                for (uint32_t j = 0; j < 4u; ++j) {
                    const uint32_t c = (j & 1u) ^ W.o;  // colour of cell j of the quad
                    const uint32_t w = (c ? wc[1] : wc[0]) >> (8u * (j >> 1));
                    if (w & W_FLUID) po[j] = po[j] + alpha * (c ? dn[1][j >> 1] : dn[0][j >> 1]);
                }
                st4(a.p + g.i, po);
                rr_n = res_add(W, rr_n, v0[0], v0[1]);
                if (FLEX) rz_n = res_add(W, rz_n, v1[0], v1[1]);
                asm volatile("" ::: "memory");
            }
        }
        send(2u, rr_n);
        if (FLEX) send(3u, rz_n);
        cluster_barrier();
        rr = total(2u);
        if (FLEX) rz = total(3u);
        ++it;
        converged = a.tol_mode != 0u && (bb > 0.0 ? sqrt(rr / bb) : 0.0) <= a.tol;
        run = it < a.limit && !converged;
    }
    return {rho, rho_prev, dq, rr, bb, rz, it, converged};
}
#undef RES_LEVEL
#undef RES_OFF

template <bool FLEX>
__global__ void __launch_bounds__(CL_THREADS, 1) k_solve_cluster(Dev d, MGState m, ClSolve a) {
    extern __shared__ __align__(16) unsigned char s_tail[];
    __shared__ uint32_t s_warp[33];
    __shared__ double s_sum[2][32];
    __shared__ double s_part[4][CL_PARTIALS];
    __shared__ uint32_t s_active[CL_PARTIALS];
    __shared__ SLevel s_levels[SLOSH_MAX_MG_LEVELS];
    __shared__ float s_dt[16];
    if (a.setup) cl_setup(d, m, a.tail, s_warp);
    const uint32_t active = d.active_bricks[0];
    // a level-4 tail's cells have children in several bricks
    const bool resident = active <= (gridDim.x - 1u) * uint32_t(CL_WARPS) && a.tail <= 3;
    const ClState s = resident ? cl_resident<FLEX>(d, m, a, s_tail, s_sum, s_part, s_active, s_levels, s_dt) : cl_streamed<FLEX>(d, m, a, s_tail, s_sum);
    if (blockIdx.x == 0u && threadIdx.x == 0u) {
        m.ctl[0] = s.it;
        m.ctl[1] = a.limit;
        m.ctl[2] = a.tol_mode;
        m.ctl[3] = 1u;
        if (s.it > 0u && a.tol_mode != 0u && !s.converged) m.ctl[4] = 1u;  // stopped at the limit: sticky for the frame
        m.scalars[0] = s.rho;
        m.scalars[2] = s.dq;
        m.scalars[3] = s.rho_prev;
        m.scalars[4] = s.bb;
        m.scalars[5] = s.rr;
        m.scalars[8] = a.tol;
        if (FLEX) m.scalars[9] = s.rz;
    }
    if (resident) cluster_barrier();  // no CTA's shared memory goes while another may read it
}
