// efs_tma.cuh — TMA-fed single-pass E+H update (the engine's core path).
//
// A CTA owns a tile of TT_Y rows (y) x TT_Z columns (z) and streams the
// x-planes of one x-chunk through a TT_S-stage shared-memory pipeline: one
// thread issues, per plane, three cp.async.bulk.tensor loads (H with its
// low halos, E_old and the material rows, each a box of the tile plus halos)
// completing on the stage's mbarrier, about TT_S-1 planes ahead of the plane
// being computed; another stores E_new and H_new of the tile with
// cp.async.bulk.tensor from shared memory.  The copies run on the copy engine,
// so the bytes in flight per SM do not depend on how many warps are resident,
// and the warps spend no instructions on global addresses or ragged edges:
// the tensor maps span the grid's Nz x Ny x Nx cells over the padded device
// layout (row pitch Pz, a multiple of 4 floats, so every global stride is a
// multiple of 16 bytes), box columns at z >= Nz lie outside the map, are
// zero-filled on loads and clipped on stores, so pad cells are never touched.
//
// Per plane x, between two barriers, a CTA computes E_new(x) on the tile plus
// its high halo row and column from the staged H and E_old (H_old(x-1) of a
// thread's cells stays in registers), then H_new(x-1) of the owned cells from
// E_new(x-1), which the interval before left in the other of two plane
// buffers, and the thread's own E_new(x).
//
// E values known before this kernel (UPML cells by k_pml_e, Mur targets by
// k_mur_adopt, applied media by k_ade_adopt) are staged in place of E_old and
// adopted as is where the material index says so.  H of UPML cells is
// provisional here and rewritten by k_pml_h.
//
// Boundaries follow the reference's index-0 self reference: the x-1, y-1 and
// z-1 neighbours of index 0 are the cell itself (the TMA zero fill outside
// the grid is never read as a field value).  H cells whose curl reads E values
// rewritten by sparse post-update operations are written here provisionally
// and rewritten afterwards by k_deferred_h, which recomputes them from H_old.
//
// Every mbarrier wait is bounded (g.wait_ns of %globaltimer, about one
// second); a wait that runs out sets bit 0 of *g.status, the CTA drains its
// loads in flight (bounded again) and returns, and the host reports
// EFS_ERR_TIMEOUT.  A diagnostic knob (g.skip_plane) leaves one plane's loads
// unissued so that tests can make a wait run out without any fault.
#pragma once
#include "efs_fused.cuh"
#include <cuda.h>
#include <cstddef>

namespace efs {

constexpr int TT_Z = 64;                 // owned z per tile
constexpr int TT_Y = 8;                  // owned y per tile (one warp per row)
constexpr int TT_S = 4;                  // pipeline stages
constexpr int TT_HZ = TT_Z + 8;          // H box: z0-4 .. z0+TT_Z+3 (x coordinate kept 16-byte aligned)
constexpr int TT_HY = TT_Y + 2;          // H box: y0-1 .. y0+TT_Y
constexpr int TT_EZ = TT_Z + 4;          // E_old / material box: z0 .. z0+TT_Z+3
constexpr int TT_EY = TT_Y + 1;          // E_old / material box: y0 .. y0+TT_Y
constexpr uint32_t TT_DEPTH = 24;        // deepest x-chunk chosen without efs_set_plane_depth / efs_batch_set_shape
constexpr int TT_THREADS = 32 * (TT_Y + 2);   // warps 0..TT_Y-1: owned rows; TT_Y: halo row, loads; TT_Y+1: halo column, stores
constexpr uint32_t TT_H_BYTES = 3u * TT_HY * TT_HZ * 4u;
constexpr uint32_t TT_E_BYTES = 3u * TT_EY * TT_EZ * 4u;
constexpr uint32_t TT_M_BYTES = 1u * TT_EY * TT_EZ * 4u;
static_assert(TT_H_BYTES + TT_E_BYTES + TT_M_BYTES < (1u << 20), "mbarrier transaction count");

// E_new of one plane: the owned cells [component][row][z] as the store box has
// them, then the halo row and the halo column at the same component stride, so
// every neighbour of a cell is one index plus a constant per component.
constexpr int TT_EC = TT_Y * TT_Z;               // component stride
constexpr int TT_EROW = 3 * TT_EC;               // halo row (Ex, Ez used)
constexpr int TT_ECOL = TT_EROW + TT_Z;          // halo column, one cell per row (Ex, Ey)
constexpr int TT_ENEW = TT_EROW + 2 * TT_EC + TT_Z;   // floats of one E_new plane
static_assert(TT_Z + TT_Y <= TT_EC, "halo row and column fit one component stride");

struct TmaStage {
    alignas(128) float H[3][TT_HY][TT_HZ];
    alignas(128) float E[3][TT_EY][TT_EZ];
    alignas(128) uint32_t M[TT_EY][TT_EZ];
    alignas(128) float D[2][2][TF_DY];   // TFSF face corrections of the plane: [face][Ex, Ey][row]
};
struct TmaSmem {
    TmaStage st[TT_S];
    alignas(128) float En[2][TT_ENEW];   // E_new of planes x and x-1
    alignas(8) unsigned long long full[TT_S];
    alignas(128) float Hn[2][3 * TT_EC]; // H_new of planes x-1 and x-2, as the store box has them (not with varied materials)
};
constexpr size_t TT_SMEM_BYTES = sizeof(TmaSmem) + 128;   // + slack to align the base to 128 B
constexpr size_t TT_SMEM_VARIED = offsetof(TmaSmem, Hn) + 128;
static_assert(2 * (TT_SMEM_BYTES + 1024) <= 228 * 1024, "two CTAs per SM");
static_assert(2 * (TT_SMEM_VARIED + 1024) <= 196 * 1024, "two CTAs per SM and 60 KB of L1");

// What a CTA keeps across the tiles it runs back to back: the stage and its
// mbarrier phase of the next plane, and the E_new / H_new buffer it writes.
struct TmaRing {
    uint32_t s = 0, ph = 0, b = 0;
    __device__ uint32_t next() const { return s + 1 == TT_S ? 0u : s + 1; }                  // of the plane after it
    __device__ uint32_t next_ph() const { return s + 1 == TT_S ? ph ^ 1u : ph; }
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done != 0;
}

// Wait for completion of the phase with the given parity; false after ~limit_ns.
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity, uint64_t limit_ns) {
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = global_ns();
    while (!mbar_try_wait(bar, parity))
        if (global_ns() - t0 > limit_ns) return false;
    return true;
}

__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, int c3, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
        ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
        : "memory");
}

// Store one plane of the tile (its owned cells, [component][row][z]) from
// shared memory; cells beyond the grid are clipped by the tensor map.
__device__ __forceinline__ void tma_store_4d(const CUtensorMap* map, const void* src, int c0, int c1, int c2, int c3) {
    asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3, %4}], [%5];" ::"l"(
                     reinterpret_cast<uint64_t>(map)),
                 "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_u32(src))
                 : "memory");
}
__device__ __forceinline__ void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// Every store issued by this thread has read its shared memory.
__device__ __forceinline__ void tma_store_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }

// The tensor maps of one parity: loads (H_old, E_old, material, TFSF faces) and stores (E_new, H_new).
struct TmaMaps { const CUtensorMap *H, *E, *M, *D, *E1, *H1; };

// Issue the loads of plane x into stage s (one thread); dbytes > 0: also the
// plane's TFSF face corrections (rows y0 .. y0+TF_DY-1 of every face).
__device__ __forceinline__ void tt_issue(TmaSmem& S, uint32_t s, const TmaMaps& tm, bool mats, uint32_t dbytes, int x, int y0, int z0) {
    const uint32_t bar = smem_u32(&S.full[s]);
    const uint32_t bytes = TT_H_BYTES + TT_E_BYTES + (mats ? TT_M_BYTES : 0u) + dbytes;
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // earlier generic reads of the stage before the refill
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    tma_load_4d(&S.st[s].H[0][0][0], tm.H, z0 - 4, y0 - 1, x, 0, bar);
    tma_load_4d(&S.st[s].E[0][0][0], tm.E, z0, y0, x, 0, bar);
    if (mats) tma_load_3d(&S.st[s].M[0][0], tm.M, z0, y0, x, bar);
    if (dbytes) tma_load_4d(&S.st[s].D[0][0][0], tm.D, y0, x, 0, 0, bar);
}

// The CTA's shared working area: 128-byte aligned, addressed from the shared
// array itself so that every access compiles to a shared-space load or store.
__device__ __forceinline__ TmaSmem& tt_smem() {
    extern __shared__ __align__(128) unsigned char tt_smem_raw[];
    return *reinterpret_cast<TmaSmem*>(tt_smem_raw + ((128u - (smem_u32(tt_smem_raw) & 127u)) & 127u));
}

// mbarrier set-up, once per CTA (all threads call it).
__device__ __forceinline__ void tt_init(TmaSmem& S) {
    if (threadIdx.x == 0) {
#pragma unroll
        for (int s = 0; s < TT_S; ++s) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&S.full[s])));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
}

// ---------------------------------------------------------------------------
// Two z-adjacent cells per thread, as one packed f32x2 value: shared-memory
// accesses are 64 bits wide and adds, subtractions and products one
// instruction for both (each half rounded like the scalar instruction, and
// products and sums stay separate), so a warp covers the 64 cells of a row.
// ---------------------------------------------------------------------------
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pk2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float lo2(f32x2 v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float hi2(f32x2 v) { return __uint_as_float((uint32_t)(v >> 32)); }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// a * b as a*b + nz with nz = (-0, -0), which is a*b for every product, signed
// zeros included.  The compiler contracts a packed multiply followed by a
// packed add into one rounding (also when nz is a constant it can see), so nz
// comes from the launch's arguments (FusedGrid).
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b, f32x2 nz) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(nz));
    return r;
}
// curl4 and upd of both cells
__device__ __forceinline__ f32x2 curl4_2(f32x2 a, f32x2 b, f32x2 c, f32x2 d) { return add2(sub2(sub2(a, b), c), d); }
__device__ __forceinline__ f32x2 upd_2(f32x2 vold, f32x2 cv, f32x2 ci, f32x2 curl, f32x2 nz) {
    return add2(mul2(vold, cv, nz), mul2(ci, curl, nz));
}
__device__ __forceinline__ f32x2 ld2(const float* p) { return *reinterpret_cast<const f32x2*>(p); }
__device__ __forceinline__ f32x2 ldg2_once(const float* p) {   // read once: no L1 line
    f32x2 r;
    asm("ld.global.nc.L1::no_allocate.b64 %0, [%1];" : "=l"(r) : "l"(p));
    return r;
}
__device__ __forceinline__ void st2(float* p, f32x2 v) { *reinterpret_cast<f32x2*>(p) = v; }
// The halves of b that m selects (bit 0: low, bit 1: high) in place of a's.
__device__ __forceinline__ f32x2 pick2(f32x2 a, f32x2 b, uint32_t m) {
    return pk2(m & 1u ? lo2(b) : lo2(a), m & 2u ? hi2(b) : hi2(a));
}
// Coefficients of a pair: E side (BASE 0) or H side (BASE 6) of two table rows
// (a 48-byte row is three float4: [vv0 vv1 vv2 vi0][vi1 vi2 ii0 ii1][ii2 iv0 iv1 iv2]).
struct PairCoef { f32x2 v[3], i[3]; };
template <int BASE>
__device__ __forceinline__ PairCoef pair_rows(const float* table, uint2 m) {
    const float4* t0 = reinterpret_cast<const float4*>(table) + (size_t)(m.x & MAT_MASK) * 3 + (BASE ? 1 : 0);
    const float4* t1 = reinterpret_cast<const float4*>(table) + (size_t)(m.y & MAT_MASK) * 3 + (BASE ? 1 : 0);
    const float4 a0 = __ldg(t0), b0 = __ldg(t0 + 1), a1 = __ldg(t1), b1 = __ldg(t1 + 1);
    PairCoef k;
    if (BASE == 0) {
        k.v[0] = pk2(a0.x, a1.x); k.v[1] = pk2(a0.y, a1.y); k.v[2] = pk2(a0.z, a1.z);
        k.i[0] = pk2(a0.w, a1.w); k.i[1] = pk2(b0.x, b1.x); k.i[2] = pk2(b0.y, b1.y);
    } else {
        k.v[0] = pk2(a0.z, a1.z); k.v[1] = pk2(a0.w, a1.w); k.v[2] = pk2(b0.x, b1.x);
        k.i[0] = pk2(b0.y, b1.y); k.i[1] = pk2(b0.z, b1.z); k.i[2] = pk2(b0.w, b1.w);
    }
    return k;
}
// The rows of a pair's cells in one half of the table (rows of 8 floats, one
// 32-byte load each), and the pair's coefficients from them.
struct PairRows { float a[6], b[6]; };
__device__ __forceinline__ void ldg_row8(const float* rows, uint32_t m, float v[6]) {
    float pad0, pad1;
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(pad0), "=f"(pad1)
        : "l"(rows + (size_t)(m & MAT_MASK) * 8));
}
__device__ __forceinline__ PairRows pair_rows8(const float* rows, uint2 m) {
    PairRows r;
    ldg_row8(rows, m.x, r.a);
    ldg_row8(rows, m.y, r.b);
    return r;
}
__device__ __forceinline__ PairCoef pair_pack(const PairRows& r) {
    PairCoef k;
#pragma unroll
    for (int n = 0; n < 3; ++n) { k.v[n] = pk2(r.a[n], r.b[n]); k.i[n] = pk2(r.a[3 + n], r.b[3 + n]); }
    return k;
}
// All ones in the halves of a pair (material indices m) whose component n is adopted.
__device__ __forceinline__ f32x2 adopt_mask(uint2 m, int n) {
    const uint32_t lo = 0u - (m.x >> (MAT_BITS + n) & 1u), hi = 0u - (m.y >> (MAT_BITS + n) & 1u);
    return (f32x2)hi << 32 | lo;
}
// Dense coefficients of the pair at cell c (component stride N); zero for a
// pair outside the grid.  Pad cells of a padded row hold zeros.
__device__ __forceinline__ PairCoef pair_dense(const float* v, const float* i, size_t N, size_t c, bool in) {
    PairCoef k;
#pragma unroll
    for (int n = 0; n < 3; ++n) {
        k.v[n] = in ? ldg2_once(v + n * N + c) : 0ull;
        k.i[n] = in ? ldg2_once(i + n * N + c) : 0ull;
    }
    return k;
}

// One tile of the streaming update: the x-chunk starting at xs of the tile at
// (y0, z0), called by every thread of the CTA; `rg` carries the pipeline state
// from one tile of a CTA to its next.  Every load the tile issues is consumed
// before it returns; its last stores may still be reading shared memory (the
// next plane's barrier, or tt_done, waits for them).  Returns false after a
// wait ran out.
// TF: the tile may meet a TFSF face corrected here (the single engine tests it
// per tile, tma_tile; the batch sorts its tiles).
//
// Warp r < TT_Y owns tile row r, lane l the cells z0+2l and z0+2l+1.  Two more
// warps compute the E_new that their H needs beyond the tile and run the
// copies: warp TT_Y the halo row (Ex, Ez) and the loads, warp TT_Y+1 the halo
// column (Ex, Ey; one cell per lane 0..TT_Y-1) and the stores.  Per plane x,
// between two barriers:
//   E(x) of the pair from the stage; its E_new to the plane buffer;
//   H(x-1) of the pair, from the neighbours' E_new(x-1) of the interval before
//   and the thread's own E(x); its H_new to the plane buffer;
//   the refill of the stage of plane x-1 and the stores of E_new(x-1), H_new(x-2).
// A pair's coefficients stay in registers while its material does not change
// along x.
// VARIED (materials of a large table that change at most planes; the rule is
// efs_engine::plan_varied): the rows of plane x+1 are fetched at the end of plane
// x, once that plane has arrived, so their latency is not on the chain from a
// plane's arrival to its barrier, as one 32-byte load per row and side instead of
// two 16-byte loads; and H leaves straight from registers, which gives up the H
// planes in shared memory for an L1 of 60 KB instead of 28 (L1 lines bound the
// row misses in flight).  256^3, us a launch, VARIED / not: 1024 random materials
// 242 / 451, 64 K 286 / 509, 1 M 493 / 922, 64 K graded in x and z 194 / 218, a
// row per 1x2x2 cells 205 / 216; 512 random 209 / 238, 384 random 204 / 192, one
// material 153 / 141.
template <bool IDX, bool TF, bool VARIED>
__device__ __forceinline__ bool tma_tile_body(TmaSmem& S, const TmaMaps& tm, const FusedGrid& g, uint32_t xs,
                                              uint32_t y0, uint32_t z0, TmaRing& rg) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t xe = min(xs + g.xchunk, g.Nx);
    const uint32_t xl = xe < g.Nx ? xe : g.Nx - 1;           // last plane whose E this CTA computes
    const int nk = (int)(xl - xs) + 1;                       // planes streamed
    const uint32_t Ny = g.Ny, Nz = g.Nz, Pz = g.Pz;
    const size_t N = g.N, NyNz = g.NyNz;
    constexpr int HPL = TT_HY * TT_HZ;                       // one component of a staged H box
    constexpr int EPL = TT_EY * TT_EZ;                       // one component of a staged E box

    // TFSF faces meeting the tile's columns (halo column included)
    bool tf_tile = false;
    if (TF)
        for (uint32_t f = 0; f < g.tf.n; ++f) tf_tile |= g.tf.z[f] >= z0 && g.tf.z[f] <= z0 + TT_Z;
    const bool mats = IDX || g.mat;                          // the material index is staged

    if (warp == TT_Y + 1) {
        // ---- halo column: Ex and Ey of the cell (y0 + lane, z0 + TT_Z); stores
        const uint32_t y = y0 + lane, z = z0 + TT_Z;         // z >= TT_Z: never index 0
        const bool has = lane < TT_Y, in = has && y < Ny && z < Nz;
        const int hi = (lane + 1) * TT_HZ + TT_Z + 4, ei = lane * TT_EZ + TT_Z, hy_ = hi - (y == 0 ? 0 : TT_HZ);
        const size_t off = (size_t)y * Pz + z;
        const int tf = tf_tile && has ? tf_face(g.tf, z) : -1;
        float hp = in ? g.H0[(size_t)(xs > 0 ? xs - 1 : 0) * NyNz + 2 * N + off] : 0.f;   // Hz(x-1)
        float kc[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};        // dense coefficients, loaded a plane ahead
        if (!IDX && in) coeffs_f<false>(g, (size_t)xs * NyNz + off, 0u, 0, kc);
        uint32_t m = 0;                                      // the cell's material (VARIED: fetched a plane ahead)
        if (VARIED && mbar_wait_bounded(smem_u32(&S.full[rg.s]), rg.ph, g.wait_ns) && has) {
            m = (&S.st[rg.s].M[0][0])[ei];
            ldg_row8(g.rowsE, m, kc);
        }
        bool out = false;
        for (int k = 0; k < nk; ++k) {
            if (k > 0 && lane == 0) {                        // planes of the interval before: E(x-1), H(x-2)
                tma_store_4d(tm.E1, S.En[rg.b ^ 1u], (int)z0, (int)y0, (int)(xs + k) - 1, 0);
                if (!VARIED && k > 1) tma_store_4d(tm.H1, S.Hn[rg.b ^ 1u], (int)z0, (int)y0, (int)(xs + k) - 2, 0);
                tma_store_commit();
            }
            __syncwarp();
            bool ok = mbar_wait_bounded(smem_u32(&S.full[rg.s]), rg.ph, g.wait_ns);
            if (ok && has) {
                const TmaStage& st = S.st[rg.s];
                const float* Hs = &st.H[0][0][0];
                const float* Es = &st.E[0][0][0];
                if (!VARIED) m = mats ? (&st.M[0][0])[ei] : 0u;
                if (IDX && !VARIED) coeffs_f<true>(g, 0, m, 0, kc);
                const float hz = Hs[2 * HPL + hi], ex0 = Es[ei], ey0 = Es[EPL + ei];
                float ex = upd(ex0, kc[0], kc[3], curl4(hz, Hs[2 * HPL + hy_], Hs[HPL + hi], Hs[HPL + hi - 1]));
                float ey = upd(ey0, kc[1], kc[4], curl4(Hs[hi], Hs[hi - 1], hz, hp));
                if (m >> MAT_BITS & 1u) ex = ex0;            // adopted
                if (m >> MAT_BITS & 2u) ey = ey0;
                if (tf >= 0) { ex = __fadd_rn(ex, st.D[tf][0][lane]); ey = __fadd_rn(ey, st.D[tf][1][lane]); }
                S.En[rg.b][TT_ECOL + lane] = ex;
                S.En[rg.b][TT_ECOL + TT_EC + lane] = ey;
                hp = hz;
                if (!IDX && in && k + 1 < nk) coeffs_f<false>(g, (size_t)(xs + k + 1) * NyNz + off, 0u, 0, kc);
            }
            if (VARIED && ok && k + 1 < nk) {
                ok = mbar_wait_bounded(smem_u32(&S.full[rg.next()]), rg.next_ph(), g.wait_ns);
                if (ok && has) {
                    m = (&S.st[rg.next()].M[0][0])[ei];
                    ldg_row8(g.rowsE, m, kc);
                }
            }
            if (lane == 0) tma_store_wait_read();            // the buffers written in the next interval are free
            __syncwarp();
            out = __syncthreads_or(!ok) != 0;
            if (out) break;
            if (++rg.s == TT_S) { rg.s = 0; rg.ph ^= 1u; }
            rg.b ^= 1u;
        }
        if (!out && lane == 0) {                             // the last plane (E only if owned) and H before it
            if (xl < xe) tma_store_4d(tm.E1, S.En[rg.b ^ 1u], (int)z0, (int)y0, (int)xl, 0);
            if (!VARIED && nk > 1) tma_store_4d(tm.H1, S.Hn[rg.b ^ 1u], (int)z0, (int)y0, (int)xl - 1, 0);
            tma_store_commit();
        }
        __syncwarp();
        return !out;
    }

    // ---- this thread's pair (row `warp`; the halo row for warp TT_Y)
    const bool own = warp < TT_Y;
    const uint32_t y = y0 + warp, z = z0 + 2 * lane;
    const bool in = y < Ny && z < Nz;                        // the pair's first cell is inside the grid
    const bool edge = y + 1 >= Ny || z + 2 >= Nz;            // some H of the pair has no update
    const int hi = (warp + 1) * TT_HZ + 2 * lane + 4;        // index in a staged H component
    const int ei = warp * TT_EZ + 2 * lane;                  // index in a staged E component
    const int hy_ = hi - (y == 0 ? 0 : TT_HZ);               // y-1 neighbour (self at y = 0)
    const int hz_ = hi - (z == 0 ? 0 : 1);                   // z-1 neighbour of the first cell (self at z = 0)
    const int si = own ? warp * TT_Z + 2 * lane : TT_EROW + 2 * lane;   // index in an E_new / H_new plane
    const int sy_ = warp == TT_Y - 1 ? TT_EROW + 2 * lane : si + TT_Z;  // its y+1 neighbour
    const int sz_ = lane == 31 ? TT_ECOL + warp : si + 2;    // z+1 neighbour of the second cell
    int tf0 = -1, tf1 = -1;
    if (tf_tile) {
        tf0 = tf_face(g.tf, z);
        tf1 = tf_face(g.tf, z + 1);
    }

    // ---- first planes into the pipeline
    const uint32_t dbytes = tf_tile ? g.tf.n * 2u * TF_DY * 4u : 0u;
    const bool loader = threadIdx.x == 32 * TT_Y;
    int issued = 0;                                          // planes issued (the loader's count)
    if (loader)
        for (; issued < TT_S && issued < nk; ++issued)
            if (xs + issued != g.skip_plane)
                tt_issue(S, (rg.s + issued) % TT_S, tm, mats, dbytes, (int)(xs + issued), (int)y0, (int)z0);

    // H_old(xs-1) of the pair; at xs = 0 the x-1 neighbour is plane 0 itself
    const size_t off = (size_t)y * Pz + z;                   // offset inside a plane
    size_t cell = (size_t)xs * NyNz + off;
    f32x2 hp[3] = {0ull, 0ull, 0ull}, ep[3] = {0ull, 0ull, 0ull};   // H_old(x-1), E_new(x-1) of the pair
    if (in) {
        const float* H = g.H0 + (size_t)(xs > 0 ? xs - 1 : 0) * NyNz + off;
        hp[1] = ld2(H + N);
        hp[2] = ld2(H + 2 * N);
    }
    const f32x2 nz = g.nz;
    PairCoef ke, kh;                                         // E coefficients of plane x, H coefficients of plane x-1
    uint2 mp = make_uint2(0u, 0u);                           // material of the pair at x-1
    bool chg = false;                                        // it changed from plane x-2 to x-1
    f32x2 ad[3] = {0ull, 0ull, 0ull};                        // the pair's adopted components, as bit masks
    if (!IDX) ke = pair_dense(g.vv, g.vi, N, cell, in);
    PairRows re, rh;                                         // VARIED: rows of E(x) and H(x-1), and the pair's material at x
    uint2 mv = make_uint2(0u, 0u);
    if (VARIED && mbar_wait_bounded(smem_u32(&S.full[rg.s]), rg.ph, g.wait_ns)) {
        mv = *reinterpret_cast<const uint2*>(&S.st[rg.s].M[0][0] + ei);
        re = pair_rows8(g.rowsE, mv);
    }
    bool timed_out = false;
    int k = 0;

    for (; k < nk; ++k) {
        if (IDX && !VARIED && chg) kh = pair_rows<6>(g.table, mp);      // H(x-1): known before the plane arrives
        bool ok = mbar_wait_bounded(smem_u32(&S.full[rg.s]), rg.ph, g.wait_ns);
        if (ok) {
            const TmaStage& st = S.st[rg.s];
            const float* Hs = &st.H[0][0][0];
            const float* Es = &st.E[0][0][0];
            float* En = S.En[rg.b];
            const float* Ep = S.En[rg.b ^ 1u];
            f32x2 hc[3], en[3];
            // ---- E_new(x) of the pair
            if (VARIED) {
                ke = pair_pack(re);
                if (own && k > 0) kh = pair_pack(rh);
#pragma unroll
                for (int n = 0; n < 3; ++n) ad[n] = adopt_mask(mv, n);
            } else if (mats) {
                const uint2 mc = *reinterpret_cast<const uint2*>(&st.M[0][0] + ei);
                chg = k == 0 || mc.x != mp.x || mc.y != mp.y;
                if (chg) {
                    if (IDX) ke = pair_rows<0>(g.table, mc);
#pragma unroll
                    for (int n = 0; n < 3; ++n) ad[n] = adopt_mask(mc, n);
                    mp = mc;
                }
            }
            hc[0] = ld2(Hs + hi); hc[1] = ld2(Hs + HPL + hi); hc[2] = ld2(Hs + 2 * HPL + hi);
            const f32x2 hzy = ld2(Hs + 2 * HPL + hy_), hxy = ld2(Hs + hy_);
            const f32x2 hyz = pk2(Hs[HPL + hz_], lo2(hc[1])), hxz = pk2(Hs[hz_], lo2(hc[0]));
            const f32x2 eo[3] = {ld2(Es + ei), ld2(Es + EPL + ei), ld2(Es + 2 * EPL + ei)};
            en[0] = upd_2(eo[0], ke.v[0], ke.i[0], curl4_2(hc[2], hzy, hc[1], hyz), nz);
            en[1] = upd_2(eo[1], ke.v[1], ke.i[1], curl4_2(hc[0], hxz, hc[2], hp[2]), nz);
            en[2] = upd_2(eo[2], ke.v[2], ke.i[2], curl4_2(hc[1], hp[1], hc[0], hxy), nz);
#pragma unroll
            for (int n = 0; n < 3; ++n) en[n] = (en[n] & ~ad[n]) | (eo[n] & ad[n]);
            if (tf_tile) {               // the TFSF point pass's add, here
                if (tf0 >= 0) {
                    en[0] = pk2(__fadd_rn(lo2(en[0]), st.D[tf0][0][warp]), hi2(en[0]));
                    en[1] = pk2(__fadd_rn(lo2(en[1]), st.D[tf0][1][warp]), hi2(en[1]));
                }
                if (tf1 >= 0) {
                    en[0] = pk2(lo2(en[0]), __fadd_rn(hi2(en[0]), st.D[tf1][0][warp]));
                    en[1] = pk2(lo2(en[1]), __fadd_rn(hi2(en[1]), st.D[tf1][1][warp]));
                }
            }
            st2(En + si, en[0]); st2(En + TT_EC + si, en[1]); st2(En + 2 * TT_EC + si, en[2]);
            if (own) {
                // ---- H_new(x-1) of the pair
                if (k > 0) {
                    const f32x2 ezy = ld2(Ep + 2 * TT_EC + sy_), exy = ld2(Ep + sy_);
                    const f32x2 eyz = pk2(hi2(ep[1]), Ep[TT_EC + sz_]), exz = pk2(hi2(ep[0]), Ep[sz_]);
                    f32x2 hn[3];
                    hn[0] = upd_2(hp[0], kh.v[0], kh.i[0], curl4_2(ep[2], ezy, ep[1], eyz), nz);
                    hn[1] = upd_2(hp[1], kh.v[1], kh.i[1], curl4_2(ep[0], exz, ep[2], en[2]), nz);
                    hn[2] = upd_2(hp[2], kh.v[2], kh.i[2], curl4_2(ep[1], en[1], ep[0], exy), nz);
                    if (edge) {                              // H beyond the last line: pass-through
                        const uint32_t m = y + 1 >= Ny ? 3u : (z + 1 >= Nz ? 1u : 0u) | (z + 2 >= Nz ? 2u : 0u);
                        hn[0] = pick2(hn[0], hp[0], m); hn[1] = pick2(hn[1], hp[1], m); hn[2] = pick2(hn[2], hp[2], m);
                    }
                    if (!VARIED) {                           // UPML cells among them are rewritten by k_pml_h
                        float* Hn = S.Hn[rg.b];
                        st2(Hn + si, hn[0]); st2(Hn + TT_EC + si, hn[1]); st2(Hn + 2 * TT_EC + si, hn[2]);
                    } else if (in) {
                        float* H1 = g.H1 + (cell - NyNz);
                        if (z + 1 < Nz) {
                            st2(H1, hn[0]); st2(H1 + N, hn[1]); st2(H1 + 2 * N, hn[2]);
                        } else {                             // the pair's second cell is padding
                            H1[0] = lo2(hn[0]); H1[N] = lo2(hn[1]); H1[2 * N] = lo2(hn[2]);
                        }
                    }
                }
            } else if (loader && k > 0 && issued < nk) {
                if (xs + issued != g.skip_plane)             // plane k-1+TT_S into the stage of plane k-1
                    tt_issue(S, (rg.s + TT_S - 1) % TT_S, tm, mats, dbytes, (int)(xs + issued), (int)y0, (int)z0);
                ++issued;
            }
            if (!IDX) {                  // the next plane's E coefficients and this plane's H coefficients
                if (k + 1 < nk) ke = pair_dense(g.vv, g.vi, N, cell + NyNz, in);
                if (own) kh = pair_dense(g.ii, g.iv, N, cell, in);
                cell += NyNz;
            }
#pragma unroll
            for (int n = 0; n < 3; ++n) { hp[n] = hc[n]; ep[n] = en[n]; }
            if (VARIED) {                // rows of H(x) and, once its material has arrived, of E(x+1)
                cell += NyNz;
                if (own) rh = pair_rows8(g.rowsH, mv);
                if (k + 1 < nk) {
                    ok = mbar_wait_bounded(smem_u32(&S.full[rg.next()]), rg.next_ph(), g.wait_ns);
                    if (ok) {
                        mv = *reinterpret_cast<const uint2*>(&S.st[rg.next()].M[0][0] + ei);
                        re = pair_rows8(g.rowsE, mv);
                    }
                }
            }
        }
        // every read of the stage and of E_new(x-1) and every write of the plane buffers done; agree on a timeout
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the plane buffers' writes before their TMA stores
        timed_out = __syncthreads_or(!ok) != 0;
        if (timed_out) break;
        if (++rg.s == TT_S) { rg.s = 0; rg.ph ^= 1u; }
        rg.b ^= 1u;
    }
    if (timed_out) {
        if (loader) {
            atomicOr(g.status, 1u);
            for (int j = k; j < issued; ++j) {                       // drain the loads still in flight
                const uint32_t q = rg.s + (uint32_t)(j - k);         // plane k is in stage rg.s
                if (xs + j != g.skip_plane)
                    (void)mbar_wait_bounded(smem_u32(&S.full[q % TT_S]), rg.ph ^ (q / TT_S), g.wait_ns);
            }
        }
        return false;
    }
    // ---- H of the last plane x = Nx-1: no core update (pass-through; UPML cells: k_pml_h)
    if (xe == g.Nx && own && in) {
        float* H1 = g.H1 + (size_t)(g.Nx - 1) * NyNz + off;
#pragma unroll
        for (int n = 0; n < 3; ++n) {
            H1[n * N] = lo2(hp[n]);
            if (z + 1 < Nz) H1[n * N + 1] = hi2(hp[n]);
        }
    }
    return true;
}
// The CTA's last stores have left shared memory (called once, after its last tile).
__device__ __forceinline__ void tt_done() {
    if (threadIdx.x == 32 * (TT_Y + 1)) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}
// A TFSF face corrected in the core update meets the tile's columns (halo column included).
template <bool IDX, bool VARIED>
__device__ __forceinline__ bool tma_tile(TmaSmem& S, const TmaMaps& tm, const FusedGrid& g, uint32_t xs, uint32_t y0, uint32_t z0,
                                         TmaRing& rg) {
    bool tf = false;
    for (uint32_t f = 0; f < g.tf.n; ++f) tf |= g.tf.z[f] >= z0 && g.tf.z[f] <= z0 + TT_Z;
    return tf ? tma_tile_body<IDX, true, VARIED>(S, tm, g, xs, y0, z0, rg) : tma_tile_body<IDX, false, VARIED>(S, tm, g, xs, y0, z0, rg);
}

// Bound by DRAM on large grids (512^3: 1.114 ms a launch at 24 planes per CTA
// for 7.0 GB, 0.96 of the measured copy rate; 1.29 ms with one cell per lane,
// scalar accesses and stores from registers, which issued 225 warp
// instructions per 32 cells).  Small or ragged grids are bound by a plane's
// chain of wait, update and barrier, about 1.2 us with two CTAs per SM
// (64 stub filters' sizes, 32 of them: 533 us a batched step at 0.83 of the
// copy rate, 726 us before).  Tried and not kept: 7 owned rows in 8 warps (fewer warps, 128
// registers: same time at 512^3, 4% slower at 256^3), loops unrolled 2 or 4
// planes deep (slower: instruction fetch), TMA boxes without halo columns
// (no change).
template <bool IDX, bool VARIED>
__global__ void __launch_bounds__(TT_THREADS, 2)
k_fused_tma(const __grid_constant__ CUtensorMap tmH, const __grid_constant__ CUtensorMap tmE,
            const __grid_constant__ CUtensorMap tmM, const __grid_constant__ CUtensorMap tmD,
            const __grid_constant__ CUtensorMap tmE1, const __grid_constant__ CUtensorMap tmH1, const FusedGrid g) {
    const uint32_t xs = blockIdx.z * g.xchunk;
    if (xs >= g.Nx) return;                                  // uniform per CTA
    TmaSmem& S = tt_smem();
    tt_init(S);
    TmaRing rg;
    (void)tma_tile<IDX, VARIED>(S, TmaMaps{&tmH, &tmE, &tmM, &tmD, &tmE1, &tmH1}, g, xs, blockIdx.y * TT_Y, blockIdx.x * TT_Z, rg);
    tt_done();
}

// ---------------------------------------------------------------------------
// UPML cells of the TMA path, outside the streaming kernel.  Their update
// reads per-cell region coefficients and fluxes with dependent loads; run
// inside the plane pipeline those loads stalled every CTA whose tile touches a
// region.  k_pml_e runs before k_fused_tma and k_pml_h after it.  A cell that
// several regions contain is handled once, by the first of them, with the
// chain over all of them in region order.
//
// Both passes are latency-bound (a z-slab region row is 8 cells, 32 bytes,
// long).  A thread takes PML_ZC consecutive z cells of one region row and
// issues every load of them (fields, material index and, for the usual
// single-region cell, the region's flux and compact coefficient row) before
// any arithmetic.  Measured on B200 over PML_ZC in {1, 2, 4} x {2, 3, 4, 6}
// blocks per SM, one cell per thread at 4 blocks per SM (64 registers, no
// spills) is fastest: occupancy hides more latency than per-thread batching.
// ---------------------------------------------------------------------------
#ifndef EFS_PML_ZC
#define EFS_PML_ZC 1
#endif
#ifndef EFS_PML_MINB
#define EFS_PML_MINB 4
#endif
constexpr uint32_t PML_ZC = EFS_PML_ZC;     // z cells per thread
constexpr int PML_MINB = EFS_PML_MINB;      // resident 256-thread blocks per SM the register budget is set for

// Work item i -> region r, row (x, y), first z and cell count (PML_ZC cells
// per item along z, items in region order, mated regions row by row: the high
// slab's end of a row and the low slab's start of the next lie in one 64-byte
// DRAM access, see FIELD_SHIFT).
__device__ __forceinline__ bool pml_item(const PmlSet& ps, uint32_t i, int& r, uint32_t& x, uint32_t& y, uint32_t& z,
                                         uint32_t& cnt) {
    for (r = 0; r < ps.count; ++r) {
        const PmlRegion& R = ps.r[r];
        if (R.mate == -2) continue;
        const uint32_t zc = (R.n[2] + PML_ZC - 1) / PML_ZC, rc = R.mate >= 0 ? 2 * zc : zc;   // items of a row
        const uint32_t items = R.n[0] * R.n[1] * rc;
        if (i < items) {
            const uint32_t row = i / rc;
            uint32_t zi = i - row * rc, s2 = R.s[2];
            x = R.s[0] + row / R.n[1];
            y = R.s[1] + row % R.n[1];
            if (zi >= zc) {                              // the mate's half of the row
                zi -= zc;
                r = R.mate;
                s2 = ps.r[r].s[2];
            }
            z = s2 + zi * PML_ZC;
            cnt = min(PML_ZC, R.n[2] - zi * PML_ZC);
            return true;
        }
        i -= items;
    }
    return false;
}

// Every region containing (x, y, z) when region r is the first that does, else 0.
__device__ __forceinline__ uint32_t pml_owner_mask(const PmlSet& ps, int r, uint32_t x, uint32_t y, uint32_t z) {
    const uint32_t m = cell_mask(ps, x, y, z);
    return m & ((1u << r) - 1u) ? 0u : m;
}

// Region coefficients and old flux of one single-region cell (3 components).
// With the compact form the three coefficients come from one table row
// (three float4 loads that hit L1/L2) instead of nine per-cell loads.
template <bool VOLT>
__device__ __forceinline__ void pml_fetch(const PmlRegion& R, uint32_t x, uint32_t y, uint32_t z, float a[3], float b[3],
                                          float fn[3], float fo[3]) {
    const size_t p0 = region_p(R, 0, x, y, z), nreg = (size_t)R.n[0] * R.n[1] * R.n[2];
#pragma unroll
    for (int n = 0; n < 3; ++n) fo[n] = __ldg((VOLT ? R.vflux : R.cflux) + p0 + n * nreg);
    if (R.cidx) {
        const float4* row = R.ctab + 6 * (uint32_t)__ldg(R.cidx + p0) + (VOLT ? 0 : 3);
        const float4 ka = __ldg(row), kb = __ldg(row + 1), kf = __ldg(row + 2);
        a[0] = ka.x; a[1] = ka.y; a[2] = ka.z;
        b[0] = kb.x; b[1] = kb.y; b[2] = kb.z;
        fn[0] = kf.x; fn[1] = kf.y; fn[2] = kf.z;
        return;
    }
#pragma unroll
    for (int n = 0; n < 3; ++n) {
        const size_t p = p0 + n * nreg;
        a[n] = __ldg((VOLT ? R.vv : R.ii) + p);
        b[n] = __ldg((VOLT ? R.vvfo : R.iifo) + p);
        fn[n] = __ldg((VOLT ? R.vvfn : R.iifn) + p);
    }
}

// The single-region chain of pml_cell on prefetched values; writes the new flux.
template <bool VOLT>
__device__ __forceinline__ float pml_one(const PmlRegion& Rn, size_t p, float vold, bool core, float cv, float ci, float curl,
                                         float a, float b, float fn, float fo) {
    const float fh = __fsub_rn(__fmul_rn(a, vold), __fmul_rn(b, fo));
    const float v = core ? upd(fo, cv, ci, curl) : fo;
    (VOLT ? Rn.vflux : Rn.cflux)[p] = v;
    return __fadd_rn(fh, __fmul_rn(fn, v));
}

// E_new of the UPML cells (reads H_old and E_old, the old flux; writes the new
// flux).  E_new is written over E_old in `V0w` (the step's old-E buffer, dead
// after this step's core update), where k_fused_tma stages it.
template <bool IDX>
__device__ __forceinline__ void pml_e_body(const FusedGrid& g, const PmlSet& ps, const PmlSet& pn, float* V0w, uint32_t items,
                                           uint32_t i) {
    if (i >= items) return;
    int r;
    uint32_t x, y, z0, cnt;
    if (!pml_item(ps, i, r, x, y, z0, cnt)) return;
    const uint32_t N = (uint32_t)g.N, NyNz = (uint32_t)g.NyNz, Pz = g.Pz;
    const uint32_t c0 = x * NyNz + y * Pz + z0;
    const uint32_t dx = x > 0 ? NyNz : 0u, dy = y > 0 ? Pz : 0u;      // x-1 / y-1 neighbour (self at index 0)
    const float* H = g.H0;
    const PmlRegion& R = ps.r[r];
    uint32_t mask[PML_ZC], m[PML_ZC];
    float hv[PML_ZC][9], eo[PML_ZC][3], a[PML_ZC][3], b[PML_ZC][3], fn[PML_ZC][3], fo[PML_ZC][3];
    // ---- every load of the item's cells
#pragma unroll
    for (uint32_t j = 0; j < PML_ZC; ++j) {
        mask[j] = j < cnt ? pml_owner_mask(ps, r, x, y, z0 + j) : 0u;
        if (!mask[j]) continue;
        const uint32_t c = c0 + j, dz = (z0 + j) > 0 ? 1u : 0u;
        hv[j][0] = H[c]; hv[j][1] = H[N + c]; hv[j][2] = H[2 * N + c];
        hv[j][3] = H[2 * N + c - dy];      // hz(y-1)
        hv[j][4] = H[N + c - dz];          // hy(z-1)
        hv[j][5] = H[c - dz];              // hx(z-1)
        hv[j][6] = H[2 * N + c - dx];      // hz(x-1)
        hv[j][7] = H[N + c - dx];          // hy(x-1)
        hv[j][8] = H[c - dy];              // hx(y-1)
        eo[j][0] = V0w[c]; eo[j][1] = V0w[N + c]; eo[j][2] = V0w[2 * N + c];
        m[j] = IDX ? __ldg(g.mat + c) : 0u;
        if (mask[j] == (1u << r)) pml_fetch<true>(R, x, y, z0 + j, a[j], b[j], fn[j], fo[j]);
    }
    // ---- update and store
#pragma unroll
    for (uint32_t j = 0; j < PML_ZC; ++j) {
        if (!mask[j]) continue;
        const uint32_t c = c0 + j, z = z0 + j;
        const float cv[3] = {curl4(hv[j][2], hv[j][3], hv[j][1], hv[j][4]),     // backward curl, reference order
                             curl4(hv[j][0], hv[j][5], hv[j][2], hv[j][6]),
                             curl4(hv[j][1], hv[j][7], hv[j][0], hv[j][8])};
        float kk[6];
        coeffs_f<IDX>(g, c, m[j], 0, kk);
        float en[3];
        if (mask[j] == (1u << r)) {
            const size_t p0 = region_p(R, 0, x, y, z), nreg = (size_t)R.n[0] * R.n[1] * R.n[2];
#pragma unroll
            for (int n = 0; n < 3; ++n)
                en[n] = pml_one<true>(pn.r[r], p0 + n * nreg, eo[j][n], true, kk[n], kk[3 + n], cv[n], a[j][n], b[j][n],
                                      fn[j][n], fo[j][n]);
        } else {
#pragma unroll
            for (int n = 0; n < 3; ++n)
                en[n] = pml_chain_pp<true>(ps, pn, mask[j], x, y, z, n, eo[j][n], true, kk[n], kk[3 + n], cv[n], true);
        }
        V0w[c] = en[0]; V0w[N + c] = en[1]; V0w[2 * N + c] = en[2];
    }
}
template <bool IDX>
__global__ void __launch_bounds__(256, PML_MINB) k_pml_e(const FusedGrid g, const PmlSet ps, const PmlSet pn, float* V0w, uint32_t items) {
    pml_e_body<IDX>(g, ps, pn, V0w, items, blockIdx.x * blockDim.x + threadIdx.x);
}

// H_new of the UPML cells from the final E_new: runs after the E-side point
// operations (beside k_deferred_h, which leaves UPML cells to this pass).
template <bool IDX>
__device__ __forceinline__ void pml_h_body(const FusedGrid& g, const PmlSet& ps, const PmlSet& pn, uint32_t items, uint32_t i) {
    if (i >= items) return;
    int r;
    uint32_t x, y, z0, cnt;
    if (!pml_item(ps, i, r, x, y, z0, cnt)) return;
    const uint32_t N = (uint32_t)g.N, NyNz = (uint32_t)g.NyNz, Pz = g.Pz;
    const uint32_t c0 = x * NyNz + y * Pz + z0;
    const float* V = g.V1;
    const PmlRegion& R = ps.r[r];
    uint32_t mask[PML_ZC], m[PML_ZC];
    bool core[PML_ZC];
    float ev[PML_ZC][9], ho[PML_ZC][3], a[PML_ZC][3], b[PML_ZC][3], fn[PML_ZC][3], fo[PML_ZC][3];
    const bool core_xy = (x + 1 < g.Nx) && (y + 1 < g.Ny);
#pragma unroll
    for (uint32_t j = 0; j < PML_ZC; ++j) {
        mask[j] = j < cnt ? pml_owner_mask(ps, r, x, y, z0 + j) : 0u;
        if (!mask[j]) continue;
        const uint32_t c = c0 + j;
        core[j] = core_xy && (z0 + j + 1 < g.Nz);
        if (core[j]) {
            ev[j][0] = V[c]; ev[j][1] = V[N + c]; ev[j][2] = V[2 * N + c];
            ev[j][3] = V[2 * N + c + Pz];      // ez(y+1)
            ev[j][4] = V[N + c + 1];           // ey(z+1)
            ev[j][5] = V[c + 1];               // ex(z+1)
            ev[j][6] = V[2 * N + c + NyNz];    // ez(x+1)
            ev[j][7] = V[N + c + NyNz];        // ey(x+1)
            ev[j][8] = V[c + Pz];              // ex(y+1)
            m[j] = IDX ? __ldg(g.mat + c) : 0u;
        }
        ho[j][0] = g.H0[c]; ho[j][1] = g.H0[N + c]; ho[j][2] = g.H0[2 * N + c];
        if (mask[j] == (1u << r)) pml_fetch<false>(R, x, y, z0 + j, a[j], b[j], fn[j], fo[j]);
    }
#pragma unroll
    for (uint32_t j = 0; j < PML_ZC; ++j) {
        if (!mask[j]) continue;
        const uint32_t c = c0 + j, z = z0 + j;
        float cv[3] = {0.f, 0.f, 0.f};
        float kk[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        if (core[j]) {                        // forward curl, reference order
            cv[0] = curl4(ev[j][2], ev[j][3], ev[j][1], ev[j][4]);
            cv[1] = curl4(ev[j][0], ev[j][5], ev[j][2], ev[j][6]);
            cv[2] = curl4(ev[j][1], ev[j][7], ev[j][0], ev[j][8]);
            coeffs_f<IDX>(g, c, m[j], 6, kk);
        }
        float hn[3];
        if (mask[j] == (1u << r)) {
            const size_t p0 = region_p(R, 0, x, y, z), nreg = (size_t)R.n[0] * R.n[1] * R.n[2];
#pragma unroll
            for (int n = 0; n < 3; ++n)
                hn[n] = pml_one<false>(pn.r[r], p0 + n * nreg, ho[j][n], core[j], kk[n], kk[3 + n], cv[n], a[j][n], b[j][n],
                                       fn[j][n], fo[j][n]);
        } else {
#pragma unroll
            for (int n = 0; n < 3; ++n)
                hn[n] = pml_chain_pp<false>(ps, pn, mask[j], x, y, z, n, ho[j][n], core[j], kk[n], kk[3 + n], cv[n], true);
        }
        g.H1[c] = hn[0]; g.H1[N + c] = hn[1]; g.H1[2 * N + c] = hn[2];
    }
}
template <bool IDX>
__global__ void __launch_bounds__(256, PML_MINB) k_pml_h(const FusedGrid g, const PmlSet ps, const PmlSet pn, uint32_t items) {
    pml_h_body<IDX>(g, ps, pn, items, blockIdx.x * blockDim.x + threadIdx.x);
}

// ---------------------------------------------------------------------------
// Two independent passes in one launch.  The UPML passes, the deferred H and
// the NF2FF samples are latency-bound (40-56% of DRAM bandwidth alone: their
// items sit one or two per z row); launched as one grid with their blocks
// interleaved, each pass's loads overlap the other's.  Block i: while both
// passes have blocks left, even blocks run A and odd blocks run B; the rest
// run the longer pass.  Every pass uses 256-thread blocks.
// ---------------------------------------------------------------------------
template <bool IDX>
struct PassPmlE {
    FusedGrid g; PmlSet ps, pn; float* V0w; uint32_t items;
    __device__ void run(uint32_t blk) const { pml_e_body<IDX>(g, ps, pn, V0w, items, blk * 256u + threadIdx.x); }
};
template <bool IDX>
struct PassPmlH {
    FusedGrid g; PmlSet ps, pn; uint32_t items;
    __device__ void run(uint32_t blk) const { pml_h_body<IDX>(g, ps, pn, items, blk * 256u + threadIdx.x); }
};
template <bool IDX>
struct PassDeferred {
    FusedGrid g; const uint32_t* cells; uint32_t n;
    __device__ void run(uint32_t blk) const { deferred_h_body<IDX>(g, cells, n, blk * 256u + threadIdx.x); }
};
// The last operations of the step before (TFSF current points, probe ring; k1:
// that step, whose fields V, C are this step's inputs) and the TFSF face values
// of step k, each in whole blocks behind the UPML E pass; apart they are
// launches of 4 to 8 us each (a step of 200x200x100 dispersive took 142 us with
// them apart and takes 136, 256^3 240 and 237, 320x320x160 384 and 381).
struct PassTails {
    float* C; const float* V; const StepState* st;
    uint32_t k, k1, nb_tc, nb_ring, nb_face;
    PointSources tc; RingDev ring; TfsfFaceDev face;
    __device__ void run(uint32_t blk) const {
        if (blk < nb_tc) return point_sources_body<1>(C, st, k1, tc, blk * 256u + threadIdx.x);
        blk -= nb_tc;
        if (blk < nb_ring) return gather_ring_body(V, C, st, k1, ring, blk * 256u + threadIdx.x);
        tfsf_face_body(st, k, face, (blk - nb_ring) * 256u + threadIdx.x);
    }
    uint32_t blocks() const { return nb_tc + nb_ring + nb_face; }
};
struct PassNfSample {
    const float* V; const float* C; uint32_t slot; Nf2ffDev d;
    __device__ void run(uint32_t blk) const { nf2ff_sample_body(V, C, slot, d, blk * 256u + threadIdx.x); }
};
template <class A, class B>
struct PassThen {                       // na blocks of A, then B's
    A a; uint32_t na; B b;
    __device__ void run(uint32_t blk) const {
        if (blk < na) a.run(blk);
        else b.run(blk - na);
    }
};
template <class A, class B>
__global__ void __launch_bounds__(256, PML_MINB) k_pair(const A a, uint32_t na, const B b, uint32_t nb) {
    const uint32_t i = blockIdx.x, m = min(na, nb);
    if (i < 2 * m) {
        if (i & 1u) b.run(i >> 1);
        else a.run(i >> 1);
    } else if (na > nb) {
        a.run(i - m);
    } else {
        b.run(i - m);
    }
}

}  // namespace efs
