// efs_sweep.cuh — E and H sweeps for grids that stay in L2.
//
// On a grid whose fields, coefficients and fluxes fit in L2 a step is bound by
// launches and by the length of dependent chains, not by DRAM, so reading
// H and E twice costs little and the plane pipeline of efs_tma.cuh, which runs
// planes in series to read them once, costs most.  Here a step is two kernels
// with one thread per pair of z-adjacent cells and every cell in flight at
// once: E of all cells, UPML cells included, then, after the E-side point
// operations, H of all cells.  No cell's H has to be computed twice
// (k_deferred_h) and the UPML passes are part of the sweeps.
//
// Same operations per cell in the same order as the fused kernel and the UPML
// passes; fields and fluxes are read from one parity and written to the other.
#pragma once
#include "efs_tma.cuh"

namespace efs {

constexpr uint32_t SW_T = 256;              // threads per block

// Blocks of a sweep: every x-plane's pairs in whole blocks.
__host__ __device__ inline uint32_t sweep_plane_blocks(uint32_t Ny, uint32_t Pz) { return (Ny * (Pz / 2) + SW_T - 1) / SW_T; }

// A field load.  Sweeps without UPML may be launched early (step_begin) and
// load plainly; the others use the non-coherent path, which orders nothing
// behind the flux stores (86x87x71 with UPML: 18.8 against 20.4 us a step).
template <bool EARLY> __device__ __forceinline__ f32x2 ldf2(const float* p) {
    return EARLY ? ld2(p) : __ldg(reinterpret_cast<const f32x2*>(p));
}
template <bool EARLY> __device__ __forceinline__ float ldf(const float* p) { return EARLY ? *p : __ldg(p); }

struct SweepCell { uint32_t x, y, z; bool live, both; };   // the pair's first cell; both: the second is inside the grid
__device__ __forceinline__ SweepCell sweep_cell(const FusedGrid& g, uint32_t blk) {
    const uint32_t half = g.Pz / 2, bpp = sweep_plane_blocks(g.Ny, g.Pz);
    const uint32_t x = blk / bpp, i = (blk - x * bpp) * SW_T + threadIdx.x;
    const uint32_t y = i / half, z = 2 * (i - y * half);
    return SweepCell{x, y, z, y < g.Ny && z < g.Nz, z + 1 < g.Nz};
}

// UPML regions that hold each cell of the pair.
__device__ __forceinline__ void sweep_regions(const PmlSet& ps, const SweepCell& c, uint32_t& m0, uint32_t& m1) {
    const uint32_t xy = __ldg(ps.xm + c.x) & __ldg(ps.ym + c.y);
    const uint2 z = __ldg(reinterpret_cast<const uint2*>(ps.zm + c.z));
    m0 = xy & z.x;
    m1 = c.both ? xy & z.y : 0u;
}

// The UPML form of one cell's update, all regions that hold it in order; up[n]
// comes in as the old field and goes out as the new one.
template <bool VOLT>
__device__ __forceinline__ void sweep_upml(const PmlSet& ps, const PmlSet& pn, uint32_t m, uint32_t x, uint32_t y, uint32_t z, bool core,
                                           const float cv[3], const float ci[3], const float curl[3], float f[3]) {
    const int r = __ffs(m) - 1;
    if (m == (1u << r)) {
        const PmlRegion& R = ps.r[r];
        float a[3], b[3], fn[3], fo[3];
        pml_fetch<VOLT>(R, x, y, z, a, b, fn, fo);
        const size_t p0 = region_p(R, 0, x, y, z), nreg = (size_t)R.n[0] * R.n[1] * R.n[2];
#pragma unroll
        for (int n = 0; n < 3; ++n)
            f[n] = pml_one<VOLT>(pn.r[r], p0 + n * nreg, f[n], core, cv[n], ci[n], curl[n], a[n], b[n], fn[n], fo[n]);
    } else {
#pragma unroll
        for (int n = 0; n < 3; ++n) f[n] = pml_chain_pp<VOLT>(ps, pn, m, x, y, z, n, f[n], core, cv[n], ci[n], curl[n], true);
    }
}

// The UPML cells of a pair: their halves of f (packed old fields in fo, packed
// core updates in f) replaced by the UPML update.
template <bool VOLT>
__device__ __forceinline__ void sweep_pair_upml(const PmlSet& ps, const PmlSet& pn, const SweepCell& c, uint32_t m0, uint32_t m1,
                                                bool core0, bool core1, const PairCoef& k, const f32x2 curl[3], const f32x2 fo[3],
                                                f32x2 f[3]) {
    if (m0) {
        const float cv[3] = {lo2(k.v[0]), lo2(k.v[1]), lo2(k.v[2])}, ci[3] = {lo2(k.i[0]), lo2(k.i[1]), lo2(k.i[2])};
        const float cu[3] = {lo2(curl[0]), lo2(curl[1]), lo2(curl[2])};
        float v[3] = {lo2(fo[0]), lo2(fo[1]), lo2(fo[2])};
        sweep_upml<VOLT>(ps, pn, m0, c.x, c.y, c.z, core0, cv, ci, cu, v);
        for (int n = 0; n < 3; ++n) f[n] = pk2(v[n], hi2(f[n]));
    }
    if (m1) {
        const float cv[3] = {hi2(k.v[0]), hi2(k.v[1]), hi2(k.v[2])}, ci[3] = {hi2(k.i[0]), hi2(k.i[1]), hi2(k.i[2])};
        const float cu[3] = {hi2(curl[0]), hi2(curl[1]), hi2(curl[2])};
        float v[3] = {hi2(fo[0]), hi2(fo[1]), hi2(fo[2])};
        sweep_upml<VOLT>(ps, pn, m1, c.x, c.y, c.z + 1, core1, cv, ci, cu, v);
        for (int n = 0; n < 3; ++n) f[n] = pk2(lo2(f[n]), v[n]);
    }
}

__device__ __forceinline__ void sweep_store(float* F, uint32_t N, uint32_t c, bool both, const f32x2 f[3]) {
#pragma unroll
    for (int n = 0; n < 3; ++n) {
        if (both) st2(F + n * N + c, f[n]);
        else F[n * N + c] = lo2(f[n]);                    // the pair's second cell is padding
    }
}

// E of every cell (reads E_old, H_old and the old flux; writes E_new and the new flux).
template <bool IDX, bool PML>
__device__ __forceinline__ void sweep_e_body(const FusedGrid& g, const PmlSet& ps, const PmlSet& pn, uint32_t blk) {
    const SweepCell q = sweep_cell(g, blk);
    if (!q.live) return;
    const uint32_t N = (uint32_t)g.N, NyNz = (uint32_t)g.NyNz, Pz = g.Pz;     // 3*N < 2^32
    const uint32_t c = q.x * NyNz + q.y * Pz + q.z;
    const uint32_t dx = q.x > 0 ? NyNz : 0u, dy = q.y > 0 ? Pz : 0u, dz = q.z > 0 ? 1u : 0u;   // self at index 0
    const float *H = g.H0, *V = g.V0;
    uint2 m = make_uint2(0u, 0u);
    if (IDX || g.mat) m = __ldg(reinterpret_cast<const uint2*>(g.mat + c));
    const f32x2 hx = ldf2<!PML>(H + c), hy = ldf2<!PML>(H + N + c), hz = ldf2<!PML>(H + 2 * N + c);
    const f32x2 hzy = ldf2<!PML>(H + 2 * N + c - dy), hxy = ldf2<!PML>(H + c - dy);
    const f32x2 hzx = ldf2<!PML>(H + 2 * N + c - dx), hyx = ldf2<!PML>(H + N + c - dx);
    const float hyz = ldf<!PML>(H + N + c - dz), hxz = ldf<!PML>(H + c - dz);
    const f32x2 eo[3] = {ldf2<!PML>(V + c), ldf2<!PML>(V + N + c), ldf2<!PML>(V + 2 * N + c)};
    PairCoef k;
    if (IDX) k = pair_rows<0>(g.table, m);
    else k = pair_dense(g.vv, g.vi, N, c, true);
    uint32_t m0 = 0, m1 = 0;
    if (PML) sweep_regions(ps, q, m0, m1);
    const f32x2 curl[3] = {curl4_2(hz, hzy, hy, pk2(hyz, lo2(hy))), curl4_2(hx, pk2(hxz, lo2(hx)), hz, hzx),
                           curl4_2(hy, hyx, hx, hxy)};
    f32x2 en[3];
#pragma unroll
    for (int n = 0; n < 3; ++n) en[n] = upd_2(eo[n], k.v[n], k.i[n], curl[n], g.nz);
    if ((m.x | m.y) >> MAT_BITS) {                        // Mur targets (UPML cells are updated here)
#pragma unroll
        for (int n = 0; n < 3; ++n) {
            const f32x2 ad = adopt_mask(m, n);
            en[n] = (en[n] & ~ad) | (eo[n] & ad);
        }
    }
    if (PML && (m0 | m1)) sweep_pair_upml<true>(ps, pn, q, m0, m1, true, true, k, curl, eo, en);
    sweep_store(g.V1, N, c, q.both, en);
}

// H of every cell, from the final E_new.
template <bool IDX, bool PML>
__device__ __forceinline__ void sweep_h_body(const FusedGrid& g, const PmlSet& ps, const PmlSet& pn, uint32_t blk) {
    const SweepCell q = sweep_cell(g, blk);
    if (!q.live) return;
    const uint32_t N = (uint32_t)g.N, NyNz = (uint32_t)g.NyNz, Pz = g.Pz;
    const uint32_t c = q.x * NyNz + q.y * Pz + q.z;
    const bool core = q.x + 1 < g.Nx && q.y + 1 < g.Ny && q.both, core1 = core && q.z + 2 < g.Nz;   // H beyond the last line: pass-through
    const float* V = g.V1;
    const f32x2 ho[3] = {ldf2<!PML>(g.H0 + c), ldf2<!PML>(g.H0 + N + c), ldf2<!PML>(g.H0 + 2 * N + c)};
    PairCoef k;
#pragma unroll
    for (int n = 0; n < 3; ++n) k.v[n] = k.i[n] = 0ull;
    f32x2 curl[3] = {0ull, 0ull, 0ull};
    f32x2 hn[3] = {ho[0], ho[1], ho[2]};
    uint32_t m0 = 0, m1 = 0;
    if (PML) sweep_regions(ps, q, m0, m1);
    if (core) {
        uint2 m = make_uint2(0u, 0u);
        if (IDX) m = __ldg(reinterpret_cast<const uint2*>(g.mat + c));
        const f32x2 ex = ldf2<!PML>(V + c), ey = ldf2<!PML>(V + N + c), ez = ldf2<!PML>(V + 2 * N + c);
        const f32x2 ezy = ldf2<!PML>(V + 2 * N + c + Pz), exy = ldf2<!PML>(V + c + Pz);
        const f32x2 ezx = ldf2<!PML>(V + 2 * N + c + NyNz), eyx = ldf2<!PML>(V + N + c + NyNz);
        const float eyz = core1 ? ldf<!PML>(V + N + c + 2) : 0.f, exz = core1 ? ldf<!PML>(V + c + 2) : 0.f;
        if (IDX) k = pair_rows<6>(g.table, m);
        else k = pair_dense(g.ii, g.iv, N, c, true);
        curl[0] = curl4_2(ez, ezy, ey, pk2(hi2(ey), eyz));
        curl[1] = curl4_2(ex, pk2(hi2(ex), exz), ez, ezx);
        curl[2] = curl4_2(ey, eyx, ex, exy);
#pragma unroll
        for (int n = 0; n < 3; ++n) {
            hn[n] = upd_2(ho[n], k.v[n], k.i[n], curl[n], g.nz);
            if (!core1) hn[n] = pk2(lo2(hn[n]), hi2(ho[n]));
        }
    }
    if (PML && (m0 | m1)) sweep_pair_upml<false>(ps, pn, q, m0, m1, core, core1, k, curl, ho, hn);
    sweep_store(g.H1, N, c, q.both, hn);
}

// What rides on the E sweep's launch instead of a launch of its own (a small
// grid's step is launches; a step of 26x11x32 fell from 5.9 to 4.7 us, 81^3 with
// Mur from 13.0 to 11.8, 86x87x71 with UPML from 19.6 to 16.7, 121x109x97 with
// dense coefficients from 26.8 to 25.8, each with a port and a probe ring):
//  * the excitation (exc.ngroups > 0), when it is the first operation on the new
//    E: the block that wrote a target's cell adds to it, after its stores;
//  * the probe ring's samples of the step before, whose fields are this step's
//    inputs: blocks behind the sweep's own (ring_k: that step; ring.G == 0: none).
struct SweepRiders {
    const StepState* st;
    uint32_t k, ring_k, nb;                               // step; step sampled; blocks of the sweep itself
    PointSources exc;
    RingDev ring;
};
constexpr uint32_t SW_EXC = SW_T;                         // most excitation targets that ride (a thread each)

template <bool IDX, bool PML>
__global__ void __launch_bounds__(SW_T, 4) k_sweep_e(const FusedGrid g, const PmlSet ps, const PmlSet pn, const SweepRiders rd) {
    if (!PML) step_begin();
    const uint32_t blk = blockIdx.x;
    if (blk >= rd.nb) {
        gather_ring_body(g.V0, g.H0, rd.st, rd.ring_k, rd.ring, (blk - rd.nb) * SW_T + threadIdx.x);
        return;
    }
    sweep_e_body<IDX, PML>(g, ps, pn, blk);
    if (rd.exc.ngroups) {
        const uint32_t bpp = sweep_plane_blocks(g.Ny, g.Pz), x = blk / bpp, first = (blk - x * bpp) * 2 * SW_T;
        bool mine = false;                                // the thread's target lies in the block's run of cells
        if (threadIdx.x < rd.exc.ngroups) {
            const uint32_t cell = rd.exc.target[threadIdx.x] % (uint32_t)g.N, off = cell - x * (uint32_t)g.NyNz;
            mine = cell >= x * (uint32_t)g.NyNz && off < (uint32_t)g.NyNz && off - first < 2 * SW_T && off >= first;
        }
        if (__syncthreads_or(mine) && mine) point_sources_body<0>(g.V1, rd.st, rd.k, rd.exc, threadIdx.x);
    }
}
template <bool IDX, bool PML>
__global__ void __launch_bounds__(SW_T, 4) k_sweep_h(const FusedGrid g, const PmlSet ps, const PmlSet pn) {
    if (!PML) step_begin();
    sweep_h_body<IDX, PML>(g, ps, pn, blockIdx.x);
}

}  // namespace efs
