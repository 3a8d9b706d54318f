// efs_fused.cuh — definitions shared by the single-pass E+H update
// (efs_tma.cuh), the UPML passes around it and the deferred H update.
//
// One timestep moves each field value through HBM once (read old, write
// new): 48 B of fields + 4 B of material index per cell.  Old and new fields
// live in separate buffers (as do the UPML flux arrays), so recomputed halo
// cells and neighbouring tiles never race.
//
// Device layout: the reference's NIJK order with the z rows padded to a
// pitch Pz (Nz rounded up to a multiple of 4 floats), so that every row and
// plane starts on a 16-byte boundary as the TMA tensor maps require.  The
// field index of (n, x, y, z) is n*N + (x*Ny + y)*Pz + z with N = Nx*Ny*Pz;
// the host translates every index a caller passes (NIJK with pitch Nz) once,
// at configure time.  Pad cells (z >= Nz) are never read as field values.
//
// H cells whose curl reads an E value that a sparse post-update operation
// rewrites (TFSF, Mur apply, excitation, PBC, series RLC, the ADE apply step)
// get a provisional H from the fused kernel and are recomputed by
// k_deferred_h, which runs after those operations (UPML cells among them are
// left to k_pml_h, which runs after them as well).  The result is the
// reference's phase order exactly, bit for bit.
#pragma once
#include "efs_kernels.cuh"

namespace efs {

constexpr int PML_MAX_OVERLAP = 4;

// The material index of a cell carries, in its top three bits, the E components
// (bit 29 + n) whose E_new is known before the core update and stands in place
// of E_old in the step's old-E buffer: the core update adopts it as is.  These
// are all components of UPML cells (k_pml_e), the Mur targets that k_mur_adopt
// computes and the applied ADE values that k_ade_adopt computes.  With dense coefficients the array holds these bits alone.
constexpr uint32_t MAT_BITS = 29, MAT_MASK = (1u << MAT_BITS) - 1u;

struct FusedGrid {
    uint32_t Nx, Ny, Nz, xchunk;
    uint32_t Pz;                        // z pitch of the device layout (Nz rounded up to a multiple of 4)
    size_t N, NyNz;                     // device component stride Nx*Ny*Pz and plane stride Ny*Pz
    const float* V0; const float* H0;   // fields at the start of the step
    float* V1; float* H1;               // fields after the step
    const uint32_t* mat; const float* table;   // mat: null with dense coefficients and no adopted cell
    const float* rowsE; const float* rowsH;    // the table's E and H halves in rows of 8 floats (varied materials, else null)
    const float* vv; const float* vi; const float* ii; const float* iv;
    uint32_t* status;                   // device status word (bit 0: a bounded wait ran out)
    uint64_t wait_ns;                   // limit of every bounded mbarrier wait (about 1 s)
    uint32_t skip_plane;                // diagnostics: loads of this x-plane are never issued (~0u: none)
    unsigned long long nz;              // two packed -0.0f (the packed products of efs_tma.cuh)
    TfsfFace tf;                        // TFSF z faces corrected in the core update (tf.n == 0: none)
};

// Face of z plane z among the TFSF faces the core update corrects, or -1.
__device__ __forceinline__ int tf_face(const TfsfFace& tf, uint32_t z) {
    return tf.n > 0 && z == tf.z[0] ? 0 : (tf.n > 1 && z == tf.z[1]) ? 1 : -1;
}

// UPML chain with separate old/new flux buffers; up to PML_MAX_OVERLAP regions per cell.
template <bool VOLT>
__device__ __forceinline__ float pml_chain_pp(const PmlSet& ps, const PmlSet& pn, uint32_t mask, uint32_t x, uint32_t y,
                                              uint32_t z, uint32_t n, float vold, bool core, float cv, float ci, float curl,
                                              bool write) {
    int reg[PML_MAX_OVERLAP];
    size_t pp[PML_MAX_OVERLAP];
    int cnt = 0;
    for (uint32_t m = mask; m; m &= m - 1) {
        const int r = __ffs(m) - 1;
        if (in_region(ps.r[r], x, y, z) && cnt < PML_MAX_OVERLAP) { reg[cnt] = r; pp[cnt] = region_p(ps.r[r], n, x, y, z); ++cnt; }
    }
    if (cnt == 0) return core ? upd(vold, cv, ci, curl) : vold;
    float fh[PML_MAX_OVERLAP];
    float v = vold;
    for (int k = 0; k < cnt; ++k) {
        const PmlRegion& R = ps.r[reg[k]];
        const float a = VOLT ? R.vv[pp[k]] : R.ii[pp[k]];
        const float b = VOLT ? R.vvfo[pp[k]] : R.iifo[pp[k]];
        const float fo = VOLT ? R.vflux[pp[k]] : R.cflux[pp[k]];
        fh[k] = __fsub_rn(__fmul_rn(a, v), __fmul_rn(b, fo));
        v = fo;
    }
    if (core) v = upd(v, cv, ci, curl);
    for (int k = 0; k < cnt; ++k) {
        const PmlRegion& R = ps.r[reg[k]];
        const float fn = VOLT ? R.vvfn[pp[k]] : R.iifn[pp[k]];
        if (write) {
            float* fl = VOLT ? pn.r[reg[k]].vflux : pn.r[reg[k]].cflux;
            fl[pp[k]] = v;
        }
        v = __fadd_rn(fh[k], __fmul_rn(fn, v));
    }
    return v;
}

// Regions that hold the cell.
__device__ __forceinline__ uint32_t cell_mask(const PmlSet& ps, uint32_t x, uint32_t y, uint32_t z) {
    return __ldg(ps.xm + x) & __ldg(ps.ym + y) & __ldg(ps.zm + z);
}

template <bool IDX>
__device__ __forceinline__ void coeffs_f(const FusedGrid& g, size_t c, uint32_t m, int base, float out[6]) {
    if (IDX) {
        // a 48-byte row is three float4: [vv0 vv1 vv2 vi0][vi1 vi2 ii0 ii1][ii2 iv0 iv1 iv2]
        const float4* t = reinterpret_cast<const float4*>(g.table) + (size_t)(m & MAT_MASK) * 3;
        if (base == 0) {
            const float4 a = __ldg(t), b = __ldg(t + 1);
            out[0] = a.x; out[1] = a.y; out[2] = a.z; out[3] = a.w; out[4] = b.x; out[5] = b.y;
        } else {
            const float4 b = __ldg(t + 1), d = __ldg(t + 2);
            out[0] = b.z; out[1] = b.w; out[2] = d.x; out[3] = d.y; out[4] = d.z; out[5] = d.w;
        }
    } else {
        const float* a = base == 0 ? g.vv : g.ii;
        const float* b = base == 0 ? g.vi : g.iv;
        out[0] = __ldg(a + c); out[1] = __ldg(a + g.N + c); out[2] = __ldg(a + 2 * g.N + c);
        out[3] = __ldg(b + c); out[4] = __ldg(b + g.N + c); out[5] = __ldg(b + 2 * g.N + c);
    }
}

// E_new of one field value from the old fields: the core update of component n
// at a cell (v: its old value), with the neighbours at index 0 the cell itself.
template <bool IDX>
__device__ __forceinline__ float core_e(const FusedGrid& g, uint32_t f, float v) {
    const uint32_t N = (uint32_t)g.N, NyNz = (uint32_t)g.NyNz, Pz = g.Pz;
    const uint32_t n = f / N, cell = f - n * N, x = cell / NyNz, r = cell - x * NyNz, y = r / Pz, z = r - y * Pz;
    const uint32_t p = n == 2 ? 0u : n + 1u, q = p == 2 ? 0u : p + 1u;       // E_n: H_q along p, H_p along q
    const uint32_t dp = p == 0 ? (x ? NyNz : 0u) : p == 1 ? (y ? Pz : 0u) : (z ? 1u : 0u);
    const uint32_t dq = q == 0 ? (x ? NyNz : 0u) : q == 1 ? (y ? Pz : 0u) : (z ? 1u : 0u);
    const float *Hq = g.H0 + q * N + cell, *Hp = g.H0 + p * N + cell;
    const float curl = curl4(Hq[0], *(Hq - dp), Hp[0], *(Hp - dq));
    float cv, ci;
    if (IDX) {
        const float* row = g.table + (size_t)(g.mat[cell] & MAT_MASK) * 12;
        cv = __ldg(row + n);
        ci = __ldg(row + 3 + n);
    } else {
        cv = __ldg(g.vv + f);
        ci = __ldg(g.vi + f);
    }
    return upd(v, cv, ci, curl);
}

// Varied materials (tma_tile_body's VARIED): how many cells have another material
// than their x-1 neighbour (out[0]), and how many of these lie more than two
// table rows from their y-1 and their z-1 neighbour's too (out[1]).
__global__ void __launch_bounds__(256) k_varied(const uint32_t* __restrict__ mat, uint32_t Nx, uint32_t Ny, uint32_t Nz, uint32_t Pz,
                                                unsigned long long* out) {
    const uint32_t plane = Ny * Pz, n = Nx * plane;
    auto far = [](uint32_t a, uint32_t b) { return a > b ? a - b > 2u : b - a > 2u; };
    uint32_t chg = 0, scat = 0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const uint32_t c = (uint32_t)i, x = c / plane, r = c - x * plane, y = r / Pz, z = r - y * Pz;
        if (x == 0 || z >= Nz) continue;
        const uint32_t m = mat[c] & MAT_MASK;
        if (m == (mat[c - plane] & MAT_MASK)) continue;
        ++chg;
        scat += y > 0 && z > 0 && far(m, mat[c - Pz] & MAT_MASK) && far(m, mat[c - 1] & MAT_MASK);
    }
    for (int o = 16; o; o >>= 1) {
        chg += __shfl_xor_sync(0xffffffffu, chg, o);
        scat += __shfl_xor_sync(0xffffffffu, scat, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(out, (unsigned long long)chg);
        atomicAdd(out + 1, (unsigned long long)scat);
    }
}
// The halves of the table as rows of 8 floats (vv0 vv1 vv2 vi0 vi1 vi2 0 0, and ii, iv).
__global__ void k_table_rows(const float* __restrict__ table, uint32_t n, float* __restrict__ E, float* __restrict__ H) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < (size_t)n * 16; i += (size_t)gridDim.x * blockDim.x) {
        const size_t r = i / 16, q = i % 16, k = q % 8;
        (q < 8 ? E : H)[r * 8 + k] = k < 6 ? table[r * 12 + (q < 8 ? 0 : 6) + k] : 0.f;
    }
}

// Adopt bits of the material index (one launch per UPML region; Mur targets; ADE cells).
__global__ void k_mat_clear(uint32_t* mat, size_t n) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) mat[i] &= MAT_MASK;
}
__global__ void k_mat_box(uint32_t* mat, uint32_t Ny, uint32_t Pz, uint32_t sx, uint32_t sy, uint32_t sz, uint32_t ny, uint32_t nz,
                          uint32_t cells) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= cells) return;
    const uint32_t z = i % nz, r = i / nz, y = r % ny, x = r / ny;
    atomicOr(mat + ((size_t)(sx + x) * Ny + sy + y) * Pz + sz + z, 7u << MAT_BITS);
}

// Mur ABC ahead of the core update (src/webgpu-fdtd.mjs:992-1023).  An entry's
// pre, post and apply steps need E_old at its two cells and E_new at the
// shifted one, which follows from the old fields, so one kernel before the core
// update computes the entry's value, writes it over E_old at the target (dead
// after the step) and the core update adopts it there: one pass over the
// entries instead of three, and no H next to a Mur face is computed twice.
//
// Entries whose target no other entry reads or writes run one per thread; the
// others in groups of lanes of one warp, which all read before any writes.
// The plan keeps entries out that anything else comes between (UPML cells,
// TFSF, periodic copies, an excitation on the target): k_mur_pre/post/apply.
//
// Bound by the sectors and latency of scattered points.  32 stub filters
// batched (4.7 M entries): 104 us a step, where the three passes took 161 us
// and the H cells next to the faces, updated again, another 122 us; 81^3 with
// six faces: 17.1 -> 13.6 us a step.
constexpr uint32_t MUR_SINGLE = 1u, MUR_LAST = 2u;   // one per thread; writes its target (the last entry that does)
constexpr uint32_t MUR_GROUP = 8u;                   // most entries of a group
struct MurAdoptDev {
    uint32_t n, first, nslots;                       // entries; first group slot (n rounded up to a warp); group slots
    const uint32_t* target; const uint32_t* shifted; const float* coeff;   // per entry, by target
    const uint8_t* kind;                             // MUR_SINGLE, MUR_LAST
    const uint32_t* slot;                            // entry of a group slot (~0: none); a group's slots lie in one warp
    float* saved;
};
template <bool IDX>
__device__ __forceinline__ float mur_value(const FusedGrid& g, const float* V, const MurAdoptDev& d, uint32_t i) {
    const uint32_t t = d.target[i], s = d.shifted[i];
    const float c = d.coeff[i], vt = V[t], vs = V[s];
    return __fadd_rn(__fsub_rn(vs, __fmul_rn(c, vt)), __fmul_rn(c, core_e<IDX>(g, s, vs)));
}
template <bool IDX>
__device__ __forceinline__ void mur_adopt_body(const FusedGrid& g, float* V, const MurAdoptDev& d, uint32_t i) {
    const bool grouped = i >= d.first;               // uniform in a warp
    uint32_t e = i;
    if (grouped) e = i - d.first < d.nslots ? d.slot[i - d.first] : ~0u;
    const bool live = e < d.n;
    const uint32_t kind = live ? d.kind[e] : 0u;
    float v = 0.f;
    if (live) v = mur_value<IDX>(g, V, d, e);        // also of entries left to the three passes: their loads are in flight with `kind`
    if (grouped) __syncwarp();
    if (!live || !(grouped || kind & MUR_SINGLE)) return;
    d.saved[e] = v;
    if (kind & MUR_LAST) V[d.target[e]] = v;
}
template <bool IDX, bool EARLY>
__global__ void __launch_bounds__(256) k_mur_adopt(const FusedGrid g, float* V, const MurAdoptDev d) {
    if (EARLY) step_begin();
    mur_adopt_body<IDX>(g, V, d, blockIdx.x * blockDim.x + threadIdx.x);
}
__global__ void k_mat_mur(uint32_t* mat, uint32_t N, const MurAdoptDev d) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < d.n && d.kind[i] & MUR_LAST) atomicOr(mat + d.target[i] % N, 1u << (MAT_BITS + d.target[i] / N));
}

// ADE state update and apply step of the voltage side ahead of the core update:
// an entry's new state follows from E_old, and what the apply step leaves at
// its cell, E_new - state, from that and the old fields, so one kernel computes
// both, writes the value over E_old and the core update adopts it.  It replaces
// the state pass, the apply pass and the second H update of every cell next to
// an entry (in a medium, of the whole medium).  Used when every entry has its
// own cell and nothing else acts on those cells (plan_ade_adopt).
//
// One entry per thread: an entry's loads are coalesced along its run.
// Bound by DRAM and its loads' latency.  200x200x100 with 1.6 M entries: the
// state and apply passes and their deferred H, 21 + 16 + 9 us a step, became 26;
// the step 159 -> 143 us.
template <bool IDX>
__device__ __forceinline__ void ade_adopt_body(const FusedGrid& g, float* V, const AdeDev& a, uint32_t i) {
    if (i >= a.n) return;
    const float st = a.state[i];
    uint32_t r = __ldg(a.grp_run + i / ADE_V) & 0x7fffffffu;
    AdeRun run = a.runs[r];
    for (uint32_t next = a.runs[r + 1].entry; i >= next; next = a.runs[r + 1].entry) run = a.runs[++r];
    const uint32_t f = run.idx + (i - run.entry);
    const float v = V[f];
    float l = run.coef >> 31 ? a.lor[i] : 0.f;
    const float en = core_e<IDX>(g, f, v);
    const float s = ade_one(v, st, l, run.coef, a.coef[run.coef & 0x7fffffffu]);
    a.state[i] = s;
    if (run.coef >> 31) a.lor[i] = l;
    V[f] = __fsub_rn(en, s);
}
template <bool IDX>
__global__ void __launch_bounds__(256) k_ade_adopt(const FusedGrid g, float* V, const AdeDev a) {
    ade_adopt_body<IDX>(g, V, a, blockIdx.x * blockDim.x + threadIdx.x);
}
__global__ void k_mat_ade(uint32_t* mat, uint32_t N, const AdeRun* runs, uint32_t nruns) {
    const uint32_t r = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;      // a warp per run
    if (r >= nruns) return;
    const uint32_t cnt = runs[r + 1].entry - runs[r].entry, f = runs[r].idx, n = f / N;
    for (uint32_t k = threadIdx.x % 32; k < cnt; k += 32) atomicOr(mat + (f + k - n * N), 1u << (MAT_BITS + n));
}

// H update of the deferred cells, after the E-side sparse operations: reads
// the final E_new and H_old, writes H_new, one thread per cell.  No deferred
// cell is a UPML cell (k_pml_h, which runs after the E-side operations too,
// updates those).
template <bool IDX>
__device__ __forceinline__ void deferred_h_body(const FusedGrid& g, const uint32_t* cells, uint32_t n, uint32_t i) {
    if (i >= n) return;
    const uint32_t c = cells[i];
    const uint32_t N = (uint32_t)g.N, NyNz = (uint32_t)g.NyNz, Pz = g.Pz;   // 3*N < 2^32
    const uint32_t x = c / NyNz, rem = c - x * NyNz, y = rem / Pz, z = rem - y * Pz;
    const bool core = (x + 1 < g.Nx) && (y + 1 < g.Ny) && (z + 1 < g.Nz);
    const float* V = g.V1;
    float ho[3], ev[9];
    ho[0] = g.H0[c]; ho[1] = g.H0[N + c]; ho[2] = g.H0[2 * N + c];
    uint32_t m = 0;
    if (core) {
        ev[0] = V[c]; ev[1] = V[N + c]; ev[2] = V[2 * N + c];
        ev[3] = V[2 * N + c + Pz]; ev[4] = V[N + c + 1]; ev[5] = V[c + 1];
        ev[6] = V[2 * N + c + NyNz]; ev[7] = V[N + c + NyNz]; ev[8] = V[c + Pz];
        m = IDX ? __ldg(g.mat + c) : 0u;
    }
    float cv[3] = {0.f, 0.f, 0.f};
    float kk[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (core) {
        cv[0] = curl4(ev[2], ev[3], ev[1], ev[4]);
        cv[1] = curl4(ev[0], ev[5], ev[2], ev[6]);
        cv[2] = curl4(ev[1], ev[7], ev[0], ev[8]);
        coeffs_f<IDX>(g, c, m, 6, kk);
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) g.H1[q * N + c] = core ? upd(ho[q], kk[q], kk[3 + q], cv[q]) : ho[q];
}
template <bool IDX>
__global__ void __launch_bounds__(256) k_deferred_h(const FusedGrid g, const uint32_t* cells, uint32_t n) {
    deferred_h_body<IDX>(g, cells, n, blockIdx.x * blockDim.x + threadIdx.x);
}

}  // namespace efs
