// efs_resident.cuh — whole runs of timesteps of a small grid in one launch.
//
// A grid of at most RS_PAIRS pairs of cells fits into the shared memory of one
// cluster, and its step is then bound by launches alone: two kernels of the
// sweep form for a few thousand cells.  Here one cluster keeps the fields in
// shared memory and the coefficients in registers, a thread per pair of
// z-adjacent cells, and runs all steps of a batch; neighbours are read from the
// other CTAs' shared memory, and the cluster's hardware barrier stands where
// the sweeps have a kernel boundary.  The excitation and the probe ring are
// applied on the way (efs_engine.cu, resident(): nothing else may act on the
// fields).  A step with a port and a probe ring, as sweeps and here: 2x2x2 3.8
// and 1.1 us, 26x11x32 4.5 and 1.4, 16x32x32 4.6 and 1.9, 16x64x32 (the most a
// cluster holds) 4.8 and 2.6; bound by the two barriers and the neighbours'
// latency, at the larger sizes by issue (16 CTAs of half the threads of 8: 1.25
// against 1.57 us).
//
// Same operations per cell in the same order as the sweeps.
#pragma once
#include "efs_sweep.cuh"

namespace efs {

constexpr uint32_t RS_T = 1024, RS_CTAS = 16;    // most threads per CTA; CTAs of the cluster (the most there are)
constexpr uint32_t RS_PAIRS = RS_T * RS_CTAS;    // a thread per pair
// One excitation target of the CTA: its place in E, the range of its further entries, the next target of the same pair.
struct RsTarget { uint32_t at, e, end, next; };
// What the targets' first entries add in RS_AHEAD steps is fetched at once: the cluster's barrier waits for
// loads in flight, and a load from L2 every step was half of the step.
constexpr uint32_t RS_AHEAD = 8;
// E, H: 3 components of 2T cells; T targets, their addends, each thread's first target
__host__ __device__ inline uint32_t resident_smem(uint32_t T) { return T * (uint32_t)(6 * 2 * 4 + sizeof(RsTarget) + 4 * RS_AHEAD + 4); }

struct Resident {
    const StepState* st;
    uint32_t steps;
    float* V; float* H;                          // fields after the last step
    PointSources exc;                            // ngroups 0: none; at most blockDim.x groups
    RingDev ring;                                // G 0: none; at most blockDim.x probes
};

__device__ __forceinline__ uint32_t rs_map(uint32_t addr, uint32_t cta) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(cta));
    return a;
}
__device__ __forceinline__ f32x2 rs_ld2(uint32_t a) {
    f32x2 v;
    asm volatile("ld.shared::cluster.b64 %0, [%1];" : "=l"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ float rs_ld(uint32_t a) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void rs_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void rs_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }

// TMAX: most threads of the launch (512 leaves a thread the registers that 1024 spills)
template <bool IDX, uint32_t TMAX>
__global__ void __launch_bounds__(TMAX, 1) k_resident(const FusedGrid g, const Resident r) {
    extern __shared__ __align__(16) float rs_smem[];
    const uint32_t T = blockDim.x, W = 2 * T, t = threadIdx.x, rank = blockIdx.x;   // the grid is one cluster
    const uint32_t N = (uint32_t)g.N, NyNz = (uint32_t)g.NyNz, Pz = g.Pz;
    const uint32_t c = 2 * (rank * T + t), c0 = rank * W;
    float* E = rs_smem;
    float* H = rs_smem + 3 * W;
    const uint32_t row = c / Pz, z = c - row * Pz, x = row / g.Ny, y = row - x * g.Ny;
    const bool in = c < N, live = in && z < g.Nz, both = z + 1 < g.Nz;
    const bool core = live && x + 1 < g.Nx && y + 1 < g.Ny && both, core1 = core && z + 2 < g.Nz;
#pragma unroll
    for (uint32_t n = 0; n < 3; ++n) {
        st2(E + n * W + 2 * t, in ? ld2(g.V0 + n * N + c) : 0ull);
        st2(H + n * W + 2 * t, in ? ld2(g.H0 + n * N + c) : 0ull);
    }
    PairCoef ke, kh;
#pragma unroll
    for (int n = 0; n < 3; ++n) ke.v[n] = ke.i[n] = kh.v[n] = kh.i[n] = 0ull;
    if (live) {
        uint2 m = make_uint2(0u, 0u);
        if (IDX) m = __ldg(reinterpret_cast<const uint2*>(g.mat + c));
        if (IDX) ke = pair_rows<0>(g.table, m);
        else ke = pair_dense(g.vv, g.vi, N, c, true);
        if (core) {
            if (IDX) kh = pair_rows<6>(g.table, m);
            else kh = pair_dense(g.ii, g.iv, N, c, true);
        }
    }
    // shared addresses of the neighbours' first component: H below, E above (self at the ends)
    const uint32_t sE = (uint32_t)__cvta_generic_to_shared(E), HO = 3 * W * 4, CW = W * 4;
    auto at = [&](uint32_t cell) {
        const uint32_t o = cell / W;
        return rs_map(sE + (cell - o * W) * 4, o);
    };
    const uint32_t cc = live ? c : c0;                    // threads without cells read their own CTA's
    const uint32_t hx_ = at(cc - (live && x > 0 ? NyNz : 0u)) + HO, hy_ = at(cc - (live && y > 0 ? Pz : 0u)) + HO,
                   hz_ = at(cc - (live && z > 0 ? 1u : 0u)) + HO;
    const uint32_t ex_ = at(core ? c + NyNz : cc), ey_ = at(core ? c + Pz : cc), ez_ = at(core1 ? c + 2 : cc);

    // this thread's excitation target and probe, if the cell is the CTA's
    RsTarget* xt = reinterpret_cast<RsTarget*>(rs_smem + 6 * W);
    float* xadd = reinterpret_cast<float*>(xt + T);
    uint32_t* xfirst = reinterpret_cast<uint32_t*>(xadd + RS_AHEAD * T);
    const uint32_t ts0 = r.st->numTS;
    xfirst[t] = ~0u;
    __syncthreads();
    uint32_t mdelay = 0;                                  // this thread's target (mine): its first entry
    float mamp = 0.f;
    bool mine = false;
    // point_sources_body<0>'s signal sample of step k (without a period its modulus is the identity)
    auto sample = [&](uint32_t delay, uint32_t k) {
        int64_t pos = (int64_t)ts0 + k - (int64_t)delay;
        if (pos < 0) pos = 0;
        if (r.exc.period > 0) pos %= (int64_t)r.exc.period;
        if (pos >= (int64_t)r.exc.len) pos = 0;
        return __ldg(r.exc.signal + pos);
    };
    auto fetch = [&](uint32_t k) {                        // addends of steps k .. k + RS_AHEAD - 1
        float v[RS_AHEAD];
#pragma unroll
        for (uint32_t i = 0; i < RS_AHEAD; ++i) v[i] = sample(mdelay, k + i);
#pragma unroll
        for (uint32_t i = 0; i < RS_AHEAD; ++i) xadd[i * T + t] = __fmul_rn(mamp, v[i]);
    };
    if (t < r.exc.ngroups) {
        const uint32_t f = r.exc.target[t], n = f / N, off = f - n * N - c0;   // wraps below the CTA's cells
        mine = off < W;
        if (mine) {
            const uint32_t e = r.exc.off[t];
            mdelay = r.exc.delay[e];
            mamp = r.exc.amp[e];
            xt[t] = RsTarget{n * W + off, e + 1, r.exc.off[t + 1], atomicExch(&xfirst[off / 2], t)};
            fetch(0);
        }
    }
    uint32_t rat = ~0u;
    if (t < r.ring.G) {
        const uint32_t f = r.ring.idx[t], n = f / N, off = f - n * N - c0;
        if (off < W) rat = n * W + off;
    }
    __syncthreads();
    const uint32_t x0 = xfirst[t];                        // targets in this thread's pair
    // steps to the next sample and its row (gather_ring_body's rule)
    uint32_t due = 0, q = 0;
    if (r.ring.G) {
        q = ts0 / r.ring.interval;
        due = (q + 1) * r.ring.interval - ts0;
    }
    float* d = nullptr;                                   // where a sample in the making goes
    float se = 0.f;
    rs_arrive();
    rs_wait();
    for (uint32_t k = 0; k < r.steps; ++k) {
        if (live) {                                       // E from the old H
            const f32x2 hx = ld2(H + 2 * t), hy = ld2(H + W + 2 * t), hz = ld2(H + 2 * W + 2 * t);
            const f32x2 hzy = rs_ld2(hy_ + 2 * CW), hxy = rs_ld2(hy_), hzx = rs_ld2(hx_ + 2 * CW), hyx = rs_ld2(hx_ + CW);
            const float hyz = rs_ld(hz_ + CW), hxz = rs_ld(hz_);
            const f32x2 curl[3] = {curl4_2(hz, hzy, hy, pk2(hyz, lo2(hy))), curl4_2(hx, pk2(hxz, lo2(hx)), hz, hzx),
                                   curl4_2(hy, hyx, hx, hxy)};
#pragma unroll
            for (int n = 0; n < 3; ++n) st2(E + n * W + 2 * t, upd_2(ld2(E + n * W + 2 * t), ke.v[n], ke.i[n], curl[n], g.nz));
        }
        for (uint32_t gi = x0; gi != ~0u; gi = xt[gi].next) {
            const RsTarget u = xt[gi];
            float v = __fadd_rn(E[u.at], xadd[k % RS_AHEAD * T + gi]);
            for (uint32_t e = u.e; e < u.end; ++e) v = __fadd_rn(v, __fmul_rn(r.exc.amp[e], sample(r.exc.delay[e], k)));
            E[u.at] = v;
        }
        const float sh = d ? H[rat] : 0.f;                // H is at rest until the barrier
        rs_arrive();
        if (d) {                                          // not before: the arrival would wait for the stores
            d[0] = se;
            d[1] = sh;
            d = nullptr;
        }
        rs_wait();
        if (core) {                                       // H from the new E
            const f32x2 ex = ld2(E + 2 * t), ey = ld2(E + W + 2 * t), ez = ld2(E + 2 * W + 2 * t);
            const f32x2 ezy = rs_ld2(ey_ + 2 * CW), exy = rs_ld2(ey_), ezx = rs_ld2(ex_ + 2 * CW), eyx = rs_ld2(ex_ + CW);
            const float eyz = core1 ? rs_ld(ez_ + CW) : 0.f, exz = core1 ? rs_ld(ez_) : 0.f;
            const f32x2 curl[3] = {curl4_2(ez, ezy, ey, pk2(hi2(ey), eyz)), curl4_2(ex, pk2(hi2(ex), exz), ez, ezx),
                                   curl4_2(ey, eyx, ex, exy)};
#pragma unroll
            for (int n = 0; n < 3; ++n) {
                const f32x2 ho = ld2(H + n * W + 2 * t);
                f32x2 hn = upd_2(ho, kh.v[n], kh.i[n], curl[n], g.nz);
                if (!core1) hn = pk2(lo2(hn), hi2(ho));
                st2(H + n * W + 2 * t, hn);
            }
        }
        if (r.ring.G && --due == 0) {
            due = r.ring.interval;
            ++q;
            if (rat != ~0u && q > r.ring.q0 && q - 1 - r.ring.q0 < r.ring.maxS) {
                d = r.ring.ring + (size_t)(q - 1 - r.ring.q0) * r.ring.G * 2 + 2 * t;
                se = E[rat];                              // E is at rest until the barrier
            }
        }
        if (mine && (k + 1) % RS_AHEAD == 0) fetch(k + 1);
        rs_arrive();
        rs_wait();
    }
    if (d) {
        d[0] = se;
        d[1] = H[rat];
    }
#pragma unroll
    for (uint32_t n = 0; n < 3; ++n) {
        if (!live) break;
        const f32x2 e = ld2(E + n * W + 2 * t), h = ld2(H + n * W + 2 * t);
        if (both) {
            st2(r.V + n * N + c, e);
            st2(r.H + n * N + c, h);
        } else {                                          // the pair's second cell is padding
            r.V[n * N + c] = lo2(e);
            r.H[n * N + c] = lo2(h);
        }
    }
}

}  // namespace efs
