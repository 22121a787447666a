// lyd_kernels.cu -- the hot kernels of the Lyman-alpha M1 step on sm_100a.
//
//  k_advect   AdvectJandH_Cylindrical! (src/AdvectJandH.jl:526-1390) as ONE kernel. A CTA owns a
//             tile of columns (r) x rows (Z) x active bins of one cloud, its threads dealt out over
//             (column, bin) pairs (k innermost, so a warp's loads are runs of neighbouring bins),
//             and marches up the tile row by row. Face fluxes never touch HBM: the six face-flux
//             arrays and the two K_phiphi arrays of the reference are replaced by shared memory and
//             registers. Ghost cells of the four boundaries are produced on the fly from the
//             boundary conditions. k_advect_tma is the form with bulk tensor copies.
//  k_freq     LyaEmissionAbsorptionUpdate! + UpdateFreqFactors! + the per-cell tridiagonal solve
//             + the flux correction of FrequencyUpdateJLya_AllCells!, fused per cell: a warp or half
//             a warp owns one cell's whole spectrum (M contiguous bins per lane), the k +- 1 couplings
//             travel by shuffles, and the tridiagonal system is solved in FP64, by parallel
//             cyclic reduction across the lanes or by a lane-serial elimination. The epilogue
//             accumulates the next step's FindActiveBins energies and the step diagnostics into
//             per-CTA partials (fixed order, so results are run-to-run deterministic).
//  k_reduce   one CTA per cloud sums that cloud's partials and derives kmin/kmax, M_F, L, f_esc.
#include <cuda_runtime.h>

#include "lyd_internal.h"
#include "lyd_physics.cuh"

namespace lyd {

constexpr int FREQ_THREADS = 256;

// The step's kernels follow one another with programmatic dependent launches: each lets the next one's
// CTAs in as soon as all of its own have started (they fill the slots its last wave leaves empty and do
// what needs nothing from it), and every CTA waits for the kernels before it to have finished, and
// their writes to be visible, before it reads or writes anything of theirs. Every CTA of every kernel
// of the chain waits, so a kernel that has finished vouches for all before it. Launched without the
// attribute the two do nothing. What a kernel of the chain writes (J, H_r, H_Z, Delta rho u, the window, the
// partials) is read by plain loads or asynchronous copies: a kernel may be resident while its
// predecessors still write, and __ldg asks for data that nobody writes as long as the kernel lives.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename K, typename A>
static void launch_chained(bool chained, K kern, int grid, int block, size_t sm, cudaStream_t st, const A &a) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = sm;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = chained ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kern, a);
}

// Per-CTA view of one cloud of a batch.
struct View {
    long long o3, oc, orf, ozf;
    int ocol, orow, orint, ozint;
    int nr, nz, bcl, bcr, bzb, bzt;
    int jend;            // end of the rows the tiles update
    double ctdt;
};

__device__ __forceinline__ void load_view(const CloudDesc &d, View &v) {
    v.o3 = d.o3; v.oc = d.oc; v.orf = d.orf; v.ozf = d.ozf;
    v.ocol = d.ocol; v.orow = d.orow; v.orint = d.orint; v.ozint = d.ozint;
    v.nr = d.nr; v.nz = d.nz; v.bcl = d.bc_r_left; v.bcr = d.bc_r_right; v.bzb = d.bc_z_bot; v.bzt = d.bc_z_top;
    v.jend = d.j_own1;
    v.ctdt = d.ctdt;
}

template <typename S, typename R>
__device__ __forceinline__ Cell<R> ld_cell(const AdvArgs<S> &a, const View &v, int i, int j, int k) {
    long long x = v.o3 + (long long)k + (long long)a.nnu * ((long long)i + (long long)v.nr * j);
    Cell<R> c;
    c.J = R(a.J[x]);
    c.Hr = R(a.Hr[x]);
    c.HZ = R(a.HZ[x]);
    return c;
}

// Radial stencil cell with the ghost cells of src/AdvectJandH.jl:662-673 (axis, always
// reflecting) and 853-871 (outer boundary, reflecting or outflow); on a Cartesian grid the
// first X interface reflects or lets flow out (src/AdvectJandH.jl:1528-1545: both ghosts take
// cell 1 with H_X = min(H_X, 0)).
template <typename S, typename R>
__device__ __forceinline__ Cell<R> r_cell(const AdvArgs<S> &a, const View &v, int idx, int j, int k) {
    if (idx < 0) {
        if (v.bcl == 0) {
            Cell<R> c = ld_cell<S, R>(a, v, -1 - idx, j, k);
            c.Hr = -c.Hr;
            return c;
        }
        Cell<R> c = ld_cell<S, R>(a, v, 0, j, k);
        c.Hr = c.Hr < R(0) ? c.Hr : R(0);
        return c;
    }
    if (idx >= v.nr) {
        if (v.bcr == 0) {
            Cell<R> c = ld_cell<S, R>(a, v, 2 * v.nr - 1 - idx, j, k);
            c.Hr = -c.Hr;
            return c;
        }
        Cell<R> c = ld_cell<S, R>(a, v, v.nr - 1, j, k);
        c.Hr = c.Hr > R(0) ? c.Hr : R(0);
        return c;
    }
    return ld_cell<S, R>(a, v, idx, j, k);
}

// Vertical stencil cell with the ghost cells of src/AdvectJandH.jl:1000-1018 (bottom) and
// 1185-1203 (top).
template <typename S, typename R>
__device__ __forceinline__ Cell<R> z_cell(const AdvArgs<S> &a, const View &v, int i, int idx, int k) {
    if (idx < 0) {
        if (v.bzb == 0) {
            Cell<R> c = ld_cell<S, R>(a, v, i, -1 - idx, k);
            c.HZ = -c.HZ;
            return c;
        }
        Cell<R> c = ld_cell<S, R>(a, v, i, 0, k);
        c.HZ = c.HZ < R(0) ? c.HZ : R(0);
        return c;
    }
    if (idx >= v.nz) {
        if (v.bzt == 0) {
            Cell<R> c = ld_cell<S, R>(a, v, i, 2 * v.nz - 1 - idx, k);
            c.HZ = -c.HZ;
            return c;
        }
        Cell<R> c = ld_cell<S, R>(a, v, i, v.nz - 1, k);
        c.HZ = c.HZ > R(0) ? c.HZ : R(0);
        return c;
    }
    return ld_cell<S, R>(a, v, i, idx, k);
}

// alpha_F of an in-grid cell: explicit array, or alpha*H_voigt (+ alpha_cF) as set up by
// src/StaticCloudTest.jl:283-285 and PhotoThermoChemistry.jl:2151.
template <typename S, typename R>
__device__ __forceinline__ R alpha_F(const AdvArgs<S> &a, const View &v, int i, int j, int k) {
    long long c = v.oc + (long long)i + (long long)v.nr * j;
    long long x = v.o3 + (long long)k + (long long)a.nnu * ((long long)i + (long long)v.nr * j);
    if (a.aF) return R(__ldg(a.aF + x));
    R val = R(__ldg(a.alpha + c)) * R(__ldg(a.Hv + x));
    if (a.alpha_cF) val = val + R(__ldg(a.alpha_cF + c));
    return val;
}

// Asynchronous global -> shared copy of one 4- or 8-byte element (cp.async, L1-allocating).
template <typename T>
__device__ __forceinline__ void cp_async_el(T *dst, const T *src) {
    static_assert(sizeof(T) == 4 || sizeof(T) == 8, "element size");
    const unsigned sa = (unsigned)__cvta_generic_to_shared(dst);
    if constexpr (sizeof(T) == 8)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(src) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sa), "l"(src) : "memory");
}
// Asynchronous global -> shared copy of 16 bytes (cp.async.cg: L2 only, the rows are streamed).
__device__ __forceinline__ void cp_async_16(void *dst, const void *src) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// ---- bulk tensor copies (TMA) into shared memory, completed on an mbarrier -------------------
__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long *bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}
// One arrival that also announces `bytes` of copies that will complete on the barrier.
__device__ __forceinline__ void mbar_expect_tx(unsigned long long *bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long *bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Wait for the phase `parity` of the barrier to complete; gives up after a bounded number of
// polls (each poll itself returns after a short hardware time limit) and reports false.
constexpr int kMbarPolls = 1 << 20;
__device__ __forceinline__ bool mbar_wait_bounded(unsigned long long *bar, unsigned parity) {
    for (int it = 0; it < kMbarPolls; it++)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}
// Orders this thread's view of earlier generic-proxy shared-memory accesses (made visible to
// it by a barrier) before the bulk copies it issues next into the same memory.
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }
// A 3-D tile of a tensor in this GPU's global memory (the map's own buffer) into shared memory;
// x, y, z are the element coordinates of the tile's first element (x * element size a multiple
// of 16 bytes; y may be negative, out-of-range elements read as zero). No multicast.
__device__ __forceinline__ void tma_load_3d(void *dst, const void *map, int x, int y, int z,
                                            unsigned long long *bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n" ::
            "r"(smem_u32(dst)),
        "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
        : "memory");
}

// ---- k_advect_tma: one CTA = 8 columns (r) x `rows` rows (Z) x 32 bins, marching up in Z ----
//
// A ring of four rows holds, for the 8 own columns and the 2 + 2 halo columns of each row, the
// cell values every face needs: J, the reduced fluxes H/max(J, Jeps) and alpha_F, each formed once
// per cell; a ring of three rows holds the state of the own columns for the cell update. Warp w
// (0..7) owns column i0+w; warp 8 stages the halo columns and computes the tile's rightmost r face.
// Per row: stage row j+2 -> sync -> every warp computes the r face on its left (warp 8: the right
// edge) into shared memory and its Z face j+1/2 into registers -> sync -> the cell update of row j
// uses the two r faces from shared memory and the Z faces j-1/2 (carried from the previous row) and
// j+1/2.
constexpr int MT = 8;                  // own columns per CTA
constexpr int MWARPS = MT + 1;
constexpr int MTHREADS = 32 * MWARPS;
constexpr int MCOL = MT + 4;           // staged columns i0-2 .. i0+MT+1
constexpr int RING = 4;
// The own columns' state (J, H_r, H_Z in the storage type) is kept for the rows j .. j+2 only
// (staged at j+2, updated at j): a ring of three slots.
constexpr int HRING = 3;
__host__ __device__ constexpr int hslot(int r) { return ((r % HRING) + HRING) % HRING; }

// The staged-cell ring A of the bulk-copy tile: [RING][MCOL][4][32] (ring slot of the row, staged
// column lc).
template <typename R>
__device__ __forceinline__ R *a_cell(R *A, int slot, int lc) {
    return A + (slot * MCOL + lc) * 4 * 32;
}

template <typename S, typename R>
__device__ __forceinline__ Cell<R> raw_cell(const AdvArgs<S> &a, const View &v, int col, int row, int k) {
    if (col < 0 || col >= v.nr) return r_cell<S, R>(a, v, col, row, k);
    if (row < 0 || row >= v.nz) return z_cell<S, R>(a, v, col, row, k);
    return ld_cell<S, R>(a, v, col, row, k);
}

// alpha_F at a staged cell: a ghost cell takes that of the in-grid cell it clamps to.
template <typename S, typename R>
__device__ __forceinline__ R alpha_F_clamped(const AdvArgs<S> &a, const View &v, int col, int row, int k) {
    const int cc = col < 0 ? 0 : (col >= v.nr ? v.nr - 1 : col);
    const int rr = row < 0 ? 0 : (row >= v.nz ? v.nz - 1 : row);
    return alpha_F<S, R>(a, v, cc, rr, k);
}

// Stage cell (col, row) into ring slot `slot`, staged column lc (= col - i0 + 2): the flux
// inputs in the arithmetic type R, and for the tile's own columns the state (J, H_r, H_Z) in
// the storage type S, which the cell update accumulates into.
template <typename S, typename R>
__device__ __forceinline__ void stage_cell(const AdvArgs<S> &a, const View &v, R *A, S *Hh, int slot, int lc,
                                           int col, int row, int k, int lane, R jeps) {
    Cell<S> c = raw_cell<S, S>(a, v, col, row, k);
    // the alpha_F loads are issued together with the state's (one load latency per cell)
    const R aF = alpha_F_clamped<S, R>(a, v, col, row, k);
    CellF<R> f = cell_f<R>(R(c.J), R(c.Hr), R(c.HZ), jeps);
    R *p = a_cell<R>(A, slot, lc) + lane;
    p[0] = f.J; p[32] = f.fr; p[64] = f.fZ; p[96] = aF;
    if (lc >= 2 && lc < 2 + MT) {
        // the state in S; with S == R the ring's J is the state's J
        constexpr int HF = sizeof(S) == sizeof(R) ? 2 : 3;
        S *q = Hh + ((hslot(row) * MT + (lc - 2)) * HF) * 32 + lane;
        q[0] = c.Hr; q[32] = c.HZ;
        if (HF == 3) q[64] = c.J;
    }
}

// The raw tile a bulk tensor copy lands for one row: J, H_r, H_Z of the staged columns
// i0-2 .. i0+MT+1 and 32 bins, [field][column][bin] (the copy box is 32 bins x MCOL columns).
// Columns outside 0..n_r-1 land as zeros; for a ghost row (row >= n_z) the copy fetched the row
// it mirrors.
template <typename S>
__host__ __device__ constexpr int raw_tile_bytes() { return 3 * MCOL * 32 * (int)sizeof(S); }

// Stage cell (col, row) into ring slot `slot` from the raw tile, applying the ghost-cell rules
// of r_cell / z_cell: a ghost column takes the column it mirrors from the same tile (every such
// column lies in the tile: i0 < n_r), a ghost row's H_Z gets the rule of its boundary.
template <typename S, typename R>
__device__ __forceinline__ void stage_from_raw(const AdvArgs<S> &a, const View &v, const S *raw, R *A, S *Hh,
                                               int slot, int lc, int col, int row, int k, int lane, R jeps, int i0) {
    int sc = lc;
    int rule = 0;   // H_r: 1 negate, 2 keep the inward (<= 0) part, 3 keep the outward (>= 0) part
    if (col < 0) {
        if (v.bcl == 0) { sc = (-1 - col) - i0 + 2; rule = 1; }
        else { sc = -i0 + 2; rule = 2; }
    } else if (col >= v.nr) {
        if (v.bcr == 0) { sc = (2 * v.nr - 1 - col) - i0 + 2; rule = 1; }
        else { sc = (v.nr - 1) - i0 + 2; rule = 3; }
    }
    Cell<S> c;
    c.J = raw[(0 * MCOL + sc) * 32 + lane];
    c.Hr = raw[(1 * MCOL + sc) * 32 + lane];
    c.HZ = raw[(2 * MCOL + sc) * 32 + lane];
    if (rule == 1) c.Hr = -c.Hr;
    else if (rule == 2) c.Hr = c.Hr < S(0) ? c.Hr : S(0);
    else if (rule == 3) c.Hr = c.Hr > S(0) ? c.Hr : S(0);
    if (row >= v.nz) {
        if (v.bzt == 0) c.HZ = -c.HZ;
        else c.HZ = c.HZ > S(0) ? c.HZ : S(0);
    }
    const R aF = alpha_F_clamped<S, R>(a, v, col, row, k);
    CellF<R> f = cell_f<R>(R(c.J), R(c.Hr), R(c.HZ), jeps);
    R *p = a_cell<R>(A, slot, lc) + lane;
    p[0] = f.J; p[32] = f.fr; p[64] = f.fZ; p[96] = aF;
    if (lc >= 2 && lc < 2 + MT) {
        constexpr int HF = sizeof(S) == sizeof(R) ? 2 : 3;
        S *q = Hh + ((hslot(row) * MT + (lc - 2)) * HF) * 32 + lane;
        q[0] = c.Hr; q[32] = c.HZ;
        if (HF == 3) q[64] = c.J;
    }
}

// A staged cell and its alpha_F: four planes `ps` elements apart (J, f_r, f_Z, alpha_F).
template <typename R>
__device__ __forceinline__ CellF<R> staged(const R *p, int ps, R &aF) {
    CellF<R> c;
    c.J = p[0]; c.fr = p[ps]; c.fZ = p[2 * ps];
    aF = p[3 * ps];
    return c;
}

// The face between staged cells pi and pp (pm, p2: the stencil's outer cells) with the PLM intervals
// ivp and u* (src/AdvectJandH.jl:641-968, 978-1289).
template <typename R, int FLUX, bool ZDIR, typename I>
__device__ __forceinline__ void face_cells(const R *pm, const R *pi, const R *pp, const R *p2, int ps, R jeps,
                                           double us, const I *ivp, R *F, R &kL, R &kR, R &JR, R &HZR) {
    R d0, aFi, aFp, d3;
    const CellF<R> cm1 = staged<R>(pm, ps, d0);
    const CellF<R> ci = staged<R>(pi, ps, aFi);
    const CellF<R> cp1 = staged<R>(pp, ps, aFp);
    const CellF<R> cp2 = staged<R>(p2, ps, d3);
    R iv[5];
#pragma unroll
    for (int t = 0; t < 5; t++) iv[t] = R(ivp[t]);
    face_flux<R, FLUX, ZDIR>(cm1, ci, cp1, cp2, iv, aFi, aFp, R(us * kInvC), jeps, F, kL, kR, JR, HZR);
}
template <typename R, int FLUX>
__device__ __forceinline__ void face_z_cells(const R *pm, const R *pi, const R *pp, const R *p2, int ps, R jeps,
                                             double us, const double *ivp, R *F) {
    R kL, kR, JR, HZR;
    face_cells<R, FLUX, true>(pm, pi, pp, p2, ps, jeps, us, ivp, F, kL, kR, JR, HZR);
}
// r face: K_phiphi of both sides too; on the axis (f = 0) the right side's is that of the axis.
template <typename R, int FLUX, typename I>
__device__ __forceinline__ void face_r_cells(const R *pm, const R *pi, const R *pp, const R *p2, int ps, bool axis,
                                             R jeps, double us, const I *ivp, R *F, R &kL, R &kR) {
    R JR, HZR;
    face_cells<R, FLUX, false>(pm, pi, pp, p2, ps, jeps, us, ivp, F, kL, kR, JR, HZR);
    if (axis) kR = k_phiphi_axis<R>(JR, HZR, jeps);
}

// The scalars of one cell's update: face areas, c~dt/dV's factors, the velocity gradients.
struct UpdGeo {
    double ArL, ArR, AZL, AZR, idv, ga, gb, gc, gd, ge, irc;
};

// The cell update (src/AdvectJandH.jl:1302-1382) of the state (uJ, uHr, uHZ) from the fluxes of
// its faces (zL, zR; FL, FR: planes `ps` apart of flux J, H_r, H_Z, K left, K right), written at x.
template <typename S, typename R>
__device__ __forceinline__ void cell_update(const AdvArgs<S> &a, long long x, S uJ, S uHr, S uHZ, const R *zL,
                                            const R *zR, const R *FL, const R *FR, int ps, const UpdGeo &g,
                                            double ctdt, R jeps) {
    const double ctdt_c = ctdt * kInvC;
    const R sJ = R(uJ), sHr = R(uHr), sHZ = R(uHZ);
    const double fac = ctdt * g.idv;
    // increments in R, accumulated into the state in S
    S Jn, Hrn, HZn;
    const S ujeps = S(a.jeps);
    if (sizeof(R) == 8) {
        R fr_ = R(fac);
        Jn = uJ - S(fr_ * ((R(g.ArR) * FR[0] - R(g.ArL) * FL[0]) + (R(g.AZR) * zR[0] - R(g.AZL) * zL[0])));
        HZn = uHZ - S(fr_ * ((R(g.ArR) * FR[2 * ps] - R(g.ArL) * FL[2 * ps]) + (R(g.AZR) * zR[2] - R(g.AZL) * zL[2])));
        Hrn = uHr - S(fr_ * ((R(g.ArR) * FR[ps] - R(g.ArL) * FL[ps]) + (R(g.AZR) * zR[1] - R(g.AZL) * zL[1])));
    } else {
        R wrL = R(fac * g.ArL), wrR = R(fac * g.ArR), wzL = R(fac * g.AZL), wzR = R(fac * g.AZR);
        Jn = uJ - S((wrR * FR[0] - wrL * FL[0]) + (wzR * zR[0] - wzL * zL[0]));
        HZn = uHZ - S((wrR * FR[2 * ps] - wrL * FL[2 * ps]) + (wzR * zR[2] - wzL * zL[2]));
        Hrn = uHr - S((wrR * FR[ps] - wrL * FL[ps]) + (wzR * zR[1] - wzL * zL[1]));
    }
    const S Jn0 = Jn;
    Jn = Jn > ujeps ? Jn : ujeps;
    const R ga = R(g.ga), gb = R(g.gb), gc = R(g.gc), gd = R(g.gd), ge = R(g.ge);
    R DdU = work_rate<R>(sJ, sHr, sHZ, jeps, R(a.heps2), ga, gb + gc, gd, ga + gd + ge);
    R Kav = R(0.5) * (FL[4 * ps] + FR[3 * ps]);
    if (sizeof(R) == 8)
        Hrn += S(R(ctdt) * Kav * R(g.irc));
    else
        Hrn += S(R(ctdt * g.irc) * Kav);
    R cc = R(ctdt_c);
    R dHr = -cc * (sHr * ga + sHZ * gb);
    R dHZ = -cc * (sHr * gc + sHZ * gd);
    Hrn = Hrn + S(dHr);
    HZn = HZn + S(dHZ);
    Jn = Jn - S(cc * DdU * sJ);
    if (a.tape) {
        // the values before the floors and the causality limiter, for the adjoint
        a.tape[x] = double(Jn0);
        a.tape[x + a.tape_stride] = double(Jn);
        a.tape[x + 2 * a.tape_stride] = double(Hrn);
        a.tape[x + 3 * a.tape_stride] = double(HZn);
    }
    Jn = Jn > ujeps ? Jn : ujeps;
    S H2 = Hrn * Hrn + HZn * HZn;
    if (H2 > Jn * Jn) {
        S fsc;
        if constexpr (sizeof(S) == 4) {
            // a flushed (zero) root of a subnormal |H|^2 scales H to zero
            const S Hm = rsq(H2);
            fsc = Hm > S(0) ? Jn / Hm : S(0);
        } else {
            // |H|^2 > J^2 >= jeps^2, far inside the normal range
            fsc = Jn * rsqrt_nr(H2);
        }
        Hrn *= fsc;
        HZn *= fsc;
    }
    a.Jo[x] = S(Jn);
    a.Hro[x] = S(Hrn);
    a.HZo[x] = S(HZn);
}

// The per-row scalars a warp needs: the cell's geometry and velocity gradients (0..10), u*_r of
// the warp's r face (11), u*_Z of its Z face above the row (12), that face's PLM intervals
// (13..17). They are copied one per lane a row ahead of their use (cp.async into the other half
// of a per-warp double buffer in shared memory, so no register carries them across the row),
// and their loads overlap a whole row's work instead of stalling the faces and the cell update.
// The r faces' PLM intervals depend on the column only: the tile stages its MT + 1 faces' once.
constexpr int GEO_N = 18;
enum { G_ARL, G_ARR, G_AZL, G_AZR, G_IDV, G_DURDR, G_DURDZ, G_DUZDR, G_DUZDZ, G_UROR, G_IRC, G_UR, G_UZ, G_ZIV };

// Where lane `lane` finds its scalar of row j for warp column `col` (the r face of warp w is
// face col too): src + j * stride, or nowhere (src null). Each lane gets one address, so a row's
// scalars come in with one load instruction per warp. The ranges are those of the consumers:
// the cell update and the Z face run for own columns col < n_r, the r face for faces col <= n_r.
template <typename S>
__device__ __forceinline__ void geo_source(const AdvArgs<S> &a, const View &v, int lane, int col, bool own,
                                           const double *&src, int &stride) {
    src = nullptr;
    stride = 0;
    if (lane == G_UR) {
        if (col <= v.nr) { src = a.u_r_star + v.orf + col; stride = v.nr + 1; }
        return;
    }
    if (!own || col >= v.nr || lane >= GEO_N) return;
    const long long c = v.oc + col;
    stride = v.nr;
    switch (lane) {
        case G_ARL: src = a.A_r + v.orf + col; stride = v.nr + 1; break;
        case G_ARR: src = a.A_r + v.orf + col + 1; stride = v.nr + 1; break;
        case G_AZL: src = a.A_Z + v.ozf + col; break;
        case G_AZR: src = a.A_Z + v.ozf + col + v.nr; break;
        case G_IDV: src = a.inv_dV + c; break;
        case G_DURDR: src = a.dur_dr + c; break;
        case G_DURDZ: src = a.dur_dZ + c; break;
        case G_DUZDR: src = a.duZ_dr + c; break;
        case G_DUZDZ: src = a.duZ_dZ + c; break;
        case G_UROR: src = a.ur_over_r + c; break;
        case G_IRC: src = a.inv_r_cell + v.ocol + col; stride = 0; break;
        case G_UZ: src = a.u_Z_star + v.ozf + col + v.nr; break;                 // face j+1
        default: src = a.zint + v.ozint + 5 + (lane - G_ZIV); stride = 5; break;   // face j+1
    }
}

// Row j's scalar of this lane; rows at or beyond the tile's end j1 (<= n_z) fetch nothing.
__device__ __forceinline__ double geo_fetch(const double *src, int stride, int j, int j1) {
    return (src != nullptr && j < j1) ? __ldg(src + (long long)stride * j) : 0.0;
}

// Shared memory of the bulk-copy tile before its raw staging area, in bytes.
template <typename S, typename R>
__host__ __device__ constexpr size_t adv_smem_base() {
    return sizeof(R) * 32 * (RING * MCOL * 4 + (MT + 1) * 5) +
           sizeof(S) * 32 * HRING * MT * (sizeof(S) == sizeof(R) ? 2 : 3) +
           sizeof(double) * (MWARPS * 2 * GEO_N + (MT + 1) * 5);
}
__host__ __device__ constexpr size_t adv_tma_off(size_t base) { return (base + 127) / 128 * 128; }

// The advection with bulk tensor copies: rows j0+2 .. of the tile arrive as copies of one 32-bin x
// MCOL-column box per field, issued by one thread a row ahead of their use into one raw tile,
// completed on an mbarrier; the converting warps apply the ghost-cell rules. The first rows
// (j0-2 .. j0+1) are staged by per-lane loads while the first copy is in flight. The box is fixed
// when the tensor map is encoded, so this form keeps the fixed tile of 8 columns x 32 bins; the
// packed tile below is the default (see there).
template <typename S, typename R, int FLUX>
__device__ __forceinline__ void advect_tile_tma(const AdvArgs<S> &a, int tile, unsigned char *adv_smem) {
    constexpr int HF = sizeof(S) == sizeof(R) ? 2 : 3;
    R *A = reinterpret_cast<R *>(adv_smem);                            // [RING][MCOL][4][32]
    S *Hh = reinterpret_cast<S *>(A + RING * MCOL * 4 * 32);           // [HRING][MT][HF][32]
    R *Fr = reinterpret_cast<R *>(Hh + HRING * MT * HF * 32);          // [MT+1][5][32]
    double *geo = reinterpret_cast<double *>(Fr + (MT + 1) * 5 * 32);  // [MWARPS][2][GEO_N]: the row slots
    double *riv = geo + MWARPS * 2 * GEO_N;                            // [MT+1][5]: the r faces' intervals
    constexpr size_t toff = adv_tma_off(adv_smem_base<S, R>());
    S *raw = reinterpret_cast<S *>(adv_smem + toff);                                   // [3][MCOL][32]
    unsigned long long *bar = reinterpret_cast<unsigned long long *>(adv_smem + toff + raw_tile_bytes<S>());
    int *abort_flag = reinterpret_cast<int *>(bar + 1);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int4 t = a.tiles[tile];
    View v;
    load_view(a.cl[t.x], v);
    const int i0 = t.y, j0 = t.z, kb = t.w;
    const int j1 = (j0 + a.rows < v.jend) ? j0 + a.rows : v.jend;
    // the last row a tile stages: the Z face j1 - 1/2 reads rows up to j1 + 1 (ghosts beyond n_z + 1 unused)
    const int rlast = (j1 + 1 < v.nz + 1) ? j1 + 1 : v.nz + 1;
    // one bulk copy per field of row r (a ghost row fetches the row it mirrors)
    auto issue_row = [&](int r) {
        const int src = r < v.nz ? r : (v.bzt == 0 ? 2 * v.nz - 1 - r : v.nz - 1);
        const unsigned char *maps = a.tmaps + (size_t)t.x * 3 * kTensorMapBytes;
        fence_proxy_async_smem();
        mbar_expect_tx(bar, (unsigned)raw_tile_bytes<S>());
#pragma unroll
        for (int f = 0; f < 3; f++) tma_load_3d(raw + f * MCOL * 32, maps + f * kTensorMapBytes, kb, i0 - 2, src, bar);
    };
    const int k = kb + lane;
    const int kmin = a.kwin[2 * t.x], kmax = a.kwin[2 * t.x + 1];
    const bool kact = (k >= kmin) && (k <= kmax) && (k < a.nnu);
    const bool chunk_act = (kb <= kmax) && (kb + 31 >= kmin);
    const R jeps = R(a.jeps);
    const int col = i0 + w;                      // own column (warps 0..7)
    const bool own = (w < MT);

    if (!chunk_act) {
        if (own && col < v.nr && k < a.nnu) {
            for (int j = j0; j < j1; j++) {
                long long x = v.o3 + (long long)k + (long long)a.nnu * ((long long)col + (long long)v.nr * j);
                a.Jo[x] = a.J[x]; a.Hro[x] = a.Hr[x]; a.HZo[x] = a.HZ[x];
            }
        }
        return;
    }

    if (threadIdx.x == 0) {
        mbar_init(bar, 1);
        *abort_flag = 0;
    }
    __syncthreads();
    if (threadIdx.x == 0 && j0 + 2 <= rlast) issue_row(j0 + 2);
    const int hl[4] = {0, 1, MT + 2, MT + 3};
    // prologue: own columns, rows j0-2 .. j0+1
    if (own && kact && col <= v.nr + 1) {
        for (int r = j0 - 2; r <= j0 + 1; r++) {
            bool gcol = col >= v.nr, grow = (r < 0 || r >= v.nz);
            if (r < -2 || r > v.nz + 1 || (gcol && grow)) continue;
            stage_cell<S, R>(a, v, A, Hh, r & (RING - 1), w + 2, col, r, k, lane, jeps);
        }
    }
    // the halo columns of a row come with its copy, two rows before the r faces read them: the
    // prologue stages those of rows j0 and j0+1
    if (!own && kact) {
        for (int r = j0; r <= j0 + 1 && r < j1 && r < v.nz; r++) {
#pragma unroll
            for (int q = 0; q < 4; q++) {
                int c2 = i0 - 2 + hl[q];
                if (c2 <= v.nr + 1) stage_cell<S, R>(a, v, A, Hh, r & (RING - 1), hl[q], c2, r, k, lane, jeps);
            }
        }
    }
    // per-row scalars: row j0 now, every next row a row ahead (the buffer of row j is
    // g0 + ((j - j0) & 1) * GEO_N)
    const double *gsrc = nullptr;
    int gstr = 0;
    double *g0 = geo + w * 2 * GEO_N;
    geo_source<S>(a, v, lane, col, own, gsrc, gstr);
    if (lane < GEO_N) g0[lane] = geo_fetch(gsrc, gstr, j0, j1);
    for (int t = threadIdx.x; t < (MT + 1) * 5; t += blockDim.x) {
        const int f = i0 + t / 5;
        riv[t] = f <= v.nr ? __ldg(a.rint + v.orint + 5 * f + t % 5) : 0.0;
    }
    __syncthreads();
    // the Z face f of the own column: rows f-2 .. f+1 of the ring
    auto zface = [&](int f, const double *ivz, const double *up, R *F) {
        auto row = [&](int r) { return a_cell<R>(A, r & (RING - 1), w + 2) + lane; };
        face_z_cells<R, FLUX>(row(f + 2), row(f + 3), row(f), row(f + 1), 32, jeps, *up, ivz, F);
    };
    R zL[3] = {R(0), R(0), R(0)};
    if (own && kact && col < v.nr)
        zface(j0, a.zint + v.ozint + 5 * j0, a.u_Z_star + v.ozf + col + (long long)v.nr * j0, zL);   // face j0

    const double ctdt = v.ctdt;
    // FP32 arithmetic holds the next row's scalar in a register and keeps one buffer; FP64
    // arithmetic, at its register limit, copies it with cp.async into the other buffer
    constexpr bool GREG = sizeof(R) == 4;
    for (int j = j0; j < j1; j++) {
        double *g = GREG ? g0 : g0 + ((j - j0) & 1) * GEO_N;
        double gnext = 0.0;
        if constexpr (GREG) {
            gnext = geo_fetch(gsrc, gstr, j + 1, j1);
        } else {
            if (lane < GEO_N) {
                double *gn = g0 + ((j + 1 - j0) & 1) * GEO_N;
                if (gsrc != nullptr && j + 1 < j1) cp_async_el(gn + lane, gsrc + (long long)gstr * (j + 1));
                else gn[lane] = 0.0;
            }
            cp_async_commit();
        }
        // (A) row j+2 from its bulk copy: the own column, and (warp 8) the halo columns
        const int r = j + 2;
        if (r <= rlast) {
            if (!mbar_wait_bounded(bar, (unsigned)((r - (j0 + 2)) & 1))) {
                *abort_flag = 1;
                atomicOr(a.err, ERRB_TIMEOUT);
            } else if (kact) {
                const bool grow = r >= v.nz;
                if (own) {
                    if (col <= v.nr + 1 && !(col >= v.nr && grow))
                        stage_from_raw<S, R>(a, v, raw, A, Hh, r & (RING - 1), w + 2, col, r, k, lane, jeps, i0);
                } else if (!grow && r < j1) {
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        int c2 = i0 - 2 + hl[q];
                        if (c2 <= v.nr + 1)
                            stage_from_raw<S, R>(a, v, raw, A, Hh, r & (RING - 1), hl[q], c2, r, k, lane, jeps, i0);
                    }
                }
            }
        }
        __syncthreads();
        if (*reinterpret_cast<volatile int *>(abort_flag)) {
            // a copy never arrived: wait once more (bounded) for it, then leave the tile
            if (threadIdx.x == 0) mbar_wait_bounded(bar, (unsigned)((r - (j0 + 2)) & 1));
            return;
        }
        // the raw tile is free again: fetch row j+3 while this row's faces and update run
        if (threadIdx.x == 0 && j + 3 <= rlast) issue_row(j + 3);
        // (B) the r face left of the own column (warp 8: the tile's right face), the Z face j+1/2
        const int f = i0 + w;
        R zR[3] = {R(0), R(0), R(0)};
        if (kact && f <= v.nr) {
            R F[3], kL, kR;
            const R *p0 = a_cell<R>(A, j & (RING - 1), w) + lane;
            face_r_cells<R, FLUX>(p0, p0 + 128, p0 + 256, p0 + 384, 32, f == 0, jeps, g[G_UR], riv + 5 * w, F, kL, kR);
            R *p = Fr + (w * 5) * 32 + lane;
            p[0] = F[0]; p[32] = F[1]; p[64] = F[2]; p[96] = kL; p[128] = kR;
        }
        if (own && kact && col < v.nr) zface(j + 1, g + G_ZIV, g + G_UZ, zR);
        __syncthreads();
        // (C) cell update
        if (own && col < v.nr && k < a.nnu) {
            long long x = v.o3 + (long long)k + (long long)a.nnu * ((long long)col + (long long)v.nr * j);
            if (!kact) {
                a.Jo[x] = a.J[x]; a.Hro[x] = a.Hr[x]; a.HZo[x] = a.HZ[x];
            } else {
                const S *pH = Hh + ((hslot(j) * MT + w) * HF) * 32 + lane;
                const S uJ = HF == 3 ? pH[64] : S(a_cell<R>(A, j & (RING - 1), w + 2)[lane]);
                const R *FL = Fr + (w * 5) * 32 + lane;
                const UpdGeo ug = {g[G_ARL], g[G_ARR], g[G_AZL], g[G_AZR], g[G_IDV], g[G_DURDR], g[G_DURDZ],
                                   g[G_DUZDR], g[G_DUZDZ], g[G_UROR], g[G_IRC]};
                cell_update<S, R>(a, x, uJ, pH[0], pH[32], zL, zR, FL, FL + 5 * 32, 32, ug, ctdt, jeps);
            }
        }
        zL[0] = zR[0]; zL[1] = zR[1]; zL[2] = zR[2];
        if constexpr (GREG) {
            // the next row's scalars replace this row's once every lane of the warp has read them
            __syncwarp();
            if (lane < GEO_N) g[lane] = gnext;
        } else {
            // the next row's scalars have landed (each lane waits for its own copy; the warp
            // barrier shows them to the other lanes and keeps this row's buffer until every lane
            // has read it)
            cp_async_wait<0>();
        }
        __syncwarp();
    }
}

template <typename S, typename R, int FLUX, int MINB>
__global__ void __launch_bounds__(MTHREADS, MINB) k_advect_tma(AdvArgs<S> a) {
    extern __shared__ __align__(128) unsigned char adv_smem[];
    pdl_trigger();
    pdl_wait();
    advect_tile_tma<S, R, FLUX>(a, blockIdx.x, adv_smem);
}

// ---- k_advect: the packed tile ---------------------------------------------------------------
//
// A CTA of 256 threads owns `ncol` columns (r) x `rows` rows (Z) x `nbk` bins of one cloud and
// marches up its rows. The active window holds nact = kmax - kmin + 1 of the n_nu bins (24 of 48
// in the ragged batches, 50 of 64 in the benchmark's cloud), so lanes fixed to bins stand idle for
// a quarter to two thirds of the work: here the window is cut into nb chunks of nbk = ceil(nact /
// nb) bins and the threads are dealt out over (column, bin) pairs, thread t to column t / nbk and
// bin t % nbk of the chunk; a row's cells are runs of nbk consecutive bins, so a warp's loads stay
// a few contiguous runs. The window is known on the device only, so the CTA works out its own
// nb, nbk and ncol (pack_bins) from its place in the cloud's work list, which is as long as the
// widest need; CTAs beyond the window's share leave at once. Bins outside the window are copied
// through, the rows of a tile shared out over its chunks.
// A ring of four rows in shared memory holds, for the ncol + 1 columns that have an r face, what
// every face needs: J, the reduced fluxes H / max(J, Jeps) (so the reciprocal of J is taken once per
// cell) and alpha_F; the three columns beyond (two left, one right) keep the current row alone. Per
// row: stage row j+2 -> barrier -> each thread computes the r face on its left into shared memory
// and its Z face j+1/2 into registers -> barrier -> the cell update of row j from the two r faces in
// shared memory and the Z faces j-1/2 (carried) and j+1/2. Faces never touch HBM. Every staged
// input comes a row ahead by cp.async, but for the halo of the mixed form, which is loaded where it is
// staged: with four CTAs per SM, which a caller may set, there is no room for its landing row (at the default
// three there would be: not tried). Its own columns' rows loaded so too: 256^2 x 64 171 us, with
// those a row ahead 167.
// Bound by dependent FP64 latency and instruction issue (24 warps per SM, 80 registers: FP64 pipe 36 %,
// issue 59 %). Per launch, against tiles of 8 columns x 32 fixed bins with one warp per column and
// branches in the faces: 256^2 x 64 with 53 active bins 262 -> 195 us (FP64), 187 -> 158 us (mixed),
// 171 -> 132 us (FP32 storage); 512^2 x 128 with 85 active 1877 -> 1088 us; 24 clouds of 17..96
// cells a side x 48 bins 254 -> 125 us; 131 x 203 x 50 with the HLL flux 155 -> 95 us. Executed warp
// instructions at 256^2 x 64 early in a run, 16 rows: 153 -> 92 million. A ninth warp for the
// halo columns and the right face (288 threads, 72 registers) was slower (210 us): it stages four
// cells to the others' one and holds up the row's barrier.
constexpr int PT = 256;                // threads
constexpr int PNC = 18;                // most columns with an r face (own columns + 1)
constexpr int PHALO = 96;              // 3 halo columns x 32 bins
// Per-row scalars of each column: areas of its left r face and of its two Z faces, 1/dV, the
// velocity gradients, u*_r of the left r face, u*_Z of the Z face above, and, for the row staged
// three rows later, alpha and alpha_cF; then the PLM intervals of the Z face above the row.
enum { P_AR, P_UR, P_AZL, P_AZR, P_IDV, P_DURDR, P_DURDZ, P_DUZDR, P_DUZDZ, P_UROR, P_UZ, P_AL, P_ACF, P_N };
constexpr int PGEO = P_N * PNC + 5;
static_assert(PGEO <= PT, "one copy per thread");
static_assert(PT == FREQ_THREADS, "the persistent step's CTAs run tiles and items alike");

// How a window of nact bins of a cloud of nr columns is cut: nb chunks of nbk <= 32 bins, tiles of
// ncol columns (ncol + 1 columns of nbk bins fit the CTA's threads), the fewest tiles of four
// candidates; then the columns are shared out evenly over the tiles.
struct Pack { int nb, nbk, ncol, nct; };
__host__ __device__ __forceinline__ int up_div(int a, int b) { return (int)((unsigned)(a + b - 1) / (unsigned)b); }
__host__ __device__ __forceinline__ Pack pack_of(int nact, int nr, int nb) {
    Pack p;
    p.nb = nb;
    p.nbk = up_div(nact, nb);
    const int nc = (int)((unsigned)PT / (unsigned)p.nbk) - 1;
    p.nct = up_div(nr, nc < PNC - 1 ? nc : PNC - 1);
    p.ncol = up_div(nr, p.nct);
    return p;
}
// device: lane q of every warp weighs candidate nb0 + q, and every lane takes the best one's quotients. Every tile
// waits for this arithmetic: with thirteen divisions in series, the height's loop and its late load of
// `share` instead of eight and none, 256^2 x 64 took 197.4 us against 195.1 (FP32 storage 135 against 132).
__device__ __forceinline__ Pack pack_bins(int nact, int nr) {
    const int q = threadIdx.x & 3, nb0 = (nact + 31) / 32;
    Pack p = pack_of(nact, nr, nb0 + q);
    const int best = (int)(__reduce_min_sync(0xffffffffu, (unsigned)(p.nb * p.nct) * 4u + (unsigned)q) & 3u);
    p.nb = nb0 + best;
    p.nbk = __shfl_sync(0xffffffffu, p.nbk, best);
    p.ncol = __shfl_sync(0xffffffffu, p.ncol, best);
    p.nct = __shfl_sync(0xffffffffu, p.nct, best);
    return p;
}
// Rows per tile when the caller leaves them open: nz rows, tpb tiles to a band of rows, for a
// cloud whose share of the GPU's resident CTAs is `share`. A field that one wave of tiles of up to 12
// rows covers is cut until its tiles just fill the wave, down to two rows: its time is a tile's
// latency (64^2 x 64: 25 us with 2 rows, 28 / 36 / 58 us with 4 / 8 / 16; 131 x 203 x 50: 95 us with 10,
// 105 / 112 with 8 / 16). Beyond, a tile's prologue (about 1.3 rows of work) pulls towards tall tiles
// and the last wave, which runs partly empty, towards short ones: rows^2 = 4 x the rows of a single
// wave balances the two (256^2 x 64: 194 us with 12 rows, 195 / 199 with 9 / 16, mixed 158 / 162 / 171;
// the 24 clouds 134 us with 8, 156 / 145 with 16 / 4; 512^2 x 128: 1084 us with 16, 1097 / 1158 with 12 / 8).
constexpr int kPackRows = 16;
__host__ __device__ __forceinline__ int pack_rows(int tpb, int nz, int share) {
    const int wave = up_div(tpb * nz, share);                 // rows per tile of a single wave
    int rows = wave < 2 ? 2 : wave;
    if (wave > 12) rows = wave > kPackRows * kPackRows / 4 ? kPackRows : (int)ceilf(sqrtf(4.0f * wave));
    return up_div(nz, up_div(nz, rows));
}
// host: the most tiles any window of 1..nnu bins makes of `nz` rows
int adv_tiles(int nnu, int nr, int nz, int rows, int share) {
    int most = 1;
    for (int n = 1; n <= nnu; n++) {
        int tpb = 1 << 30;
        for (int q = 0; q < 4; q++) {
            const Pack p = pack_of(n, nr, (n + 31) / 32 + q);
            tpb = p.nb * p.nct < tpb ? p.nb * p.nct : tpb;
        }
        const int r = rows > 0 ? rows : pack_rows(tpb, nz, share);
        const int m = tpb * ((nz + r - 1) / r);
        most = m > most ? m : most;
    }
    return most;
}

// The column a staged stencil column copies, and the boundary rule that r_cell applies to the copy's H_r
// (1: negate; 2: keep the part <= 0; 3: keep the part >= 0). A ghost row's source and rule change from
// row to row and are found where it is copied; a corner cell (ghost in both directions) is never staged.
struct ColSrc { int i, rule; };
__device__ __forceinline__ ColSrc col_src(const View &v, int col) {
    if (col < 0) return v.bcl == 0 ? ColSrc{-1 - col, 1} : ColSrc{0, 2};
    if (col >= v.nr) return v.bcr == 0 ? ColSrc{2 * v.nr - 1 - col, 1} : ColSrc{v.nr - 1, 3};
    return ColSrc{col, 0};
}
template <typename S>
__device__ __forceinline__ S bc_rule(S h, int rule) {
    if (rule == 0) return h;                  // (all but the ghosts: one branch past the rules)
    if (rule == 1) return -h;
    if (rule == 2) return h < S(0) ? h : S(0);
    return h > S(0) ? h : S(0);
}

// The own columns' rows land a row ahead in every form; the halo columns' when their landing row fits
// beside it, i.e. when S and R agree.
template <typename S, typename R> __host__ __device__ constexpr bool adv_ahead() { return sizeof(S) == sizeof(R); }
// The halo's landing row fills the gaps of its staged row's planes (96 of 256 values) in FP64;
// with FP32 it has its own space.
template <typename S, typename R> __host__ __device__ constexpr bool adv_overlay() { return sizeof(S) == 8 && sizeof(R) == 8; }
template <typename S, typename R>
__host__ __device__ constexpr size_t adv_pack_smem() {
    size_t b = sizeof(R) * ((RING + 1) * 4 * PT + 5 * PT);           // ring, halo row, r faces
    b += sizeof(S) * RING * (adv_ahead<S, R>() ? 2 : 3) * PT;        // the state's rows
    b += sizeof(S) * (adv_ahead<S, R>() ? 2 : 1) * PT;               // landing row: J (mixed: lands in the state's), H_voigt
    if (adv_ahead<S, R>() && !adv_overlay<S, R>()) b += sizeof(S) * 4 * PHALO + sizeof(double) * 2 * PHALO;
    return b + sizeof(double) * (2 * PGEO + PNC * 5 + PNC);
}

// One tile of the work list by the calling CTA of PT threads, in dynamic shared memory `sm`: the
// body of k_advect, also run by the persistent batch kernel.
template <typename S, typename R, int FLUX>
__device__ __forceinline__ void advect_tile(const AdvArgs<S> &a, int tile, unsigned char *sm) {
    constexpr bool AHEAD = adv_ahead<S, R>(), OVER = adv_overlay<S, R>();
    constexpr int HF = AHEAD ? 2 : 3;
    R *A = reinterpret_cast<R *>(sm);                       // [RING][4][PT]
    R *HB = A + RING * 4 * PT;                              // [4][PT]: the halo columns' current row
    R *Fr = HB + 4 * PT;                                    // [5][PT]
    S *Hs = reinterpret_cast<S *>(Fr + 5 * PT);             // [RING][HF][PT]: H_r, H_Z (, J) as stored
    S *raw = Hs + RING * HF * PT;                           // [HF == 3 ? 1 : 2][PT]: (J,) H_voigt (or alpha_F) landing
    constexpr int RJ = HF == 3 ? 0 : PT;                    // where H_voigt lands in it
    double *geo = reinterpret_cast<double *>(raw + RJ + PT);                // [2][PGEO]
    double *irc = geo + 2 * PGEO;                           // [PNC]: <1/r>
    R *riv = reinterpret_cast<R *>(irc + PNC);              // [PNC][5] of a double's room: the r faces' intervals
    double *hal = irc + PNC + PNC * 5;                      // AHEAD, not OVER: [2][PHALO], then [4][PHALO] of S
    const int t = threadIdx.x;
    const int4 it = a.tiles[tile];                          // cloud, rows [y, w), place z in their list
    View v;
    load_view(a.cl[it.x], v);
    const int share = a.cl[it.x].adv_share;                 // (asked for with the rest, not when it is needed)
    int kmin = a.kwin[2 * it.x], kmax = a.kwin[2 * it.x + 1];
    kmin = kmin > 0 ? kmin : 0;
    kmax = kmax < a.nnu - 1 ? kmax : a.nnu - 1;
    const int nact = kmax >= kmin ? kmax - kmin + 1 : 0;
    const Pack pk = pack_bins(nact > 0 ? nact : 1, v.nr);
    const int tpb = pk.nb * pk.nct, band = (int)((unsigned)it.z / (unsigned)tpb), e0 = it.z - band * tpb;
    const int kb = (int)((unsigned)e0 / (unsigned)pk.nct), ct = e0 - kb * pk.nct;
    const int rows = a.rows > 0 ? a.rows : pack_rows(tpb, it.w - it.y, share);
    const int j0 = it.y + band * rows;
    if (j0 >= it.w) return;
    const int j1 = j0 + rows < it.w ? j0 + rows : it.w;
    const int nbk = pk.nbk, i0 = ct * pk.ncol;
    int ncol = pk.ncol;
    if (i0 >= v.nr) return;                                 // (shares rounded up can leave a last one empty)
    ncol = i0 + ncol <= v.nr ? ncol : v.nr - i0;
    const int kbeg = kmin + kb * nbk;
    const R jeps = R(a.jeps);

    // Bins outside the window pass through, the rows of the tile in turn over its chunks. A thread's first
    // two are loaded here and stored once the prologue's own loads have gone out.
    const int nin = a.nnu - nact, prow = ncol * nin;
    const int npass = prow * ((j1 - j0 - kb + pk.nb - 1) / pk.nb);
    auto pass_at = [&](int e) {
        const int q = e / prow, f = e - q * prow, cc = f / nin, m = f - cc * nin;
        return v.o3 + (long long)a.nnu * (i0 + cc + (long long)v.nr * (j0 + kb + q * pk.nb)) + (m < kmin ? m : m + nact);
    };
    Cell<S> pv[2];
    long long px[2] = {-1, -1};
#pragma unroll
    for (int q = 0; q < 2; q++)
        if (t + q * PT < npass) {
            px[q] = pass_at(t + q * PT);
            pv[q].J = a.J[px[q]]; pv[q].Hr = a.Hr[px[q]]; pv[q].HZ = a.HZ[px[q]];
        }
    auto pass_rest = [&]() {
#pragma unroll
        for (int q = 0; q < 2; q++)
            if (px[q] >= 0) { a.Jo[px[q]] = pv[q].J; a.Hro[px[q]] = pv[q].Hr; a.HZo[px[q]] = pv[q].HZ; }
        for (int e = t + 2 * PT; e < npass; e += PT) {
            const long long x = pass_at(e);
            a.Jo[x] = a.J[x]; a.Hro[x] = a.Hr[x]; a.HZo[x] = a.HZ[x];
        }
    };
    if (nact == 0 || kbeg > kmax) {
        pass_rest();
        return;
    }

    // this thread's item: column i0 + c (c = ncol: the column right of the tile, for its r face)
    const int c = t / nbk, k = kbeg + (t - c * nbk), col = i0 + c;
    const bool item = c <= ncol && k <= kmax && col <= v.nr + 1;
    const bool own = item && c < ncol;
    const bool busy = __any_sync(0xffffffffu, item);
    const int cg = c < ncol ? c : ncol;
    // and its halo cell, counted from the top so that the threads without an own cell come first:
    // columns i0-2, i0-1 and i0+ncol+1
    const int hq = PT - 1 - t, hc = hq / nbk, hk = kbeg + (hq - hc * nbk);
    const int hcol = hc < 2 ? i0 - 2 + hc : i0 + ncol + 1;
    const bool halo = hc < 3 && hk <= kmax && hcol <= v.nr + 1;
    R *hp = HB + hq;
    S *hraw = nullptr;
    int hps = 0;                                            // plane stride of the halo's landing row
    double *hal0 = nullptr, *hal1 = nullptr;                // its alpha, alpha_cF
    if constexpr (OVER) {
        hraw = reinterpret_cast<S *>(HB) + PHALO + hq;
        hps = PT;
        hal0 = reinterpret_cast<double *>(HB) + (hq >> 6) * PT + 2 * PHALO + (hq & 63);
        hal1 = hal0 + 2 * PT;
    } else if constexpr (AHEAD) {
        hraw = reinterpret_cast<S *>(hal + 2 * PHALO) + hq;
        hps = PHALO;
        hal0 = hal + hq;
        hal1 = hal0 + PHALO;
    }

    // ---- copies a row ahead ----
    // a cell's column and bin are the thread's own: what changes from row to row is the source row
    const unsigned rstr = (unsigned)a.nnu * (unsigned)v.nr;
    auto copy_cell = [&](long long xc, long long xac, int row, S *dJ, S *dHr, S *dHZ, S *dHv) {
        int sj = row, rj = row;
        if (row >= v.nz) {
            sj = v.bzt == 0 ? 2 * v.nz - 1 - row : v.nz - 1;
            rj = v.nz - 1;
        }
        const long long x = xc + (long long)((unsigned long long)rstr * (unsigned)sj);
        const long long xa = xac + (long long)((unsigned long long)rstr * (unsigned)rj);
        cp_async_el(dJ, a.J + x);
        cp_async_el(dHr, a.Hr + x);
        cp_async_el(dHZ, a.HZ + x);
        cp_async_el(dHv, (a.aF ? a.aF : a.Hv) + xa);
    };
    // where a (possibly ghost) column's cells and opacities come from, and the rule of its H_r
    auto col_base = [&](int cc, int kk, long long &xc, long long &xac, int &rule) {
        const ColSrc s = col_src(v, cc);
        const int ci = cc < 0 ? 0 : (cc >= v.nr ? v.nr - 1 : cc);
        xc = v.o3 + kk + (long long)a.nnu * s.i;
        xac = v.o3 + kk + (long long)a.nnu * ci;
        rule = s.rule;
    };
    long long xo = 0, xoa = 0, xh = 0, xha = 0;
    int orule = 0, hrule = 0;
    if (item) col_base(col, k, xo, xoa, orule);
    if (AHEAD && halo) col_base(hcol, hk, xh, xha, hrule);
    // rows the own columns stage: up to j1 + 1 and the second ghost row; no corner ghosts
    auto stages = [&](int r) { return item && r <= j1 + 1 && r <= v.nz + 1 && !(col >= v.nr && r >= v.nz); };
    auto issue_own = [&](int r) {
        if (stages(r)) {
            S *h = Hs + (r & (RING - 1)) * HF * PT + t;
            copy_cell(xo, xoa, r, HF == 3 ? h + 2 * PT : raw + t, h, h + PT, raw + RJ + t);
        }
    };
    auto issue_halo = [&](int r) {
        if (halo && r < j1) {
            copy_cell(xh, xha, r, hraw, hraw + hps, hraw + 2 * hps, hraw + 3 * hps);
            if (!a.aF) {
                const int ci = hcol < 0 ? 0 : (hcol >= v.nr ? v.nr - 1 : hcol);
                const long long cl = v.oc + ci + (long long)v.nr * r;
                cp_async_el(hal0, a.alpha + cl);
                if (a.alpha_cF) cp_async_el(hal1, a.alpha_cF + cl);
            }
        }
    };
    auto put = [&](R *p, S J, S Hr, S HZ, R aF) {
        const CellF<R> f = cell_f<R>(R(J), R(Hr), R(HZ), jeps);
        p[0] = f.J; p[PT] = f.fr; p[2 * PT] = f.fZ; p[3 * PT] = aF;
    };
    auto aF_of = [&](S hv, double al, double acF) {
        if (a.aF) return R(hv);
        R x = R(al) * R(hv);
        if (a.alpha_cF) x = x + R(acF);
        return x;
    };
    // an own cell's state as stored
    auto keep = [&](S *h, const Cell<S> &x) {
        h[0] = x.Hr; h[PT] = x.HZ;
        if (HF == 3) h[2 * PT] = x.J;
    };

    // ---- per-row scalars: entry t of a row's slot comes from gsrc + row * gstr ----
    const double *gsrc = nullptr;
    int gstr = 0;
    const int gi = t / PNC, gc = t - gi * PNC, gcol = i0 + gc;
    if (gi < P_N) {
        const bool face = gi == P_AR || gi == P_UR, al = gi >= P_AL;
        if (gc <= ncol && (face ? gcol <= v.nr : al ? gcol <= v.nr + 1 : (gc < ncol && gcol < v.nr))) {
            const int cc = gcol < v.nr ? gcol : v.nr - 1;
            gstr = face ? v.nr + 1 : v.nr;
            switch (gi) {
                case P_AR: gsrc = a.A_r + v.orf + gcol; break;
                case P_UR: gsrc = a.u_r_star + v.orf + gcol; break;
                case P_AZL: gsrc = a.A_Z + v.ozf + gcol; break;
                case P_AZR: gsrc = a.A_Z + v.ozf + gcol + v.nr; break;
                case P_IDV: gsrc = a.inv_dV + v.oc + gcol; break;
                case P_DURDR: gsrc = a.dur_dr + v.oc + gcol; break;
                case P_DURDZ: gsrc = a.dur_dZ + v.oc + gcol; break;
                case P_DUZDR: gsrc = a.duZ_dr + v.oc + gcol; break;
                case P_DUZDZ: gsrc = a.duZ_dZ + v.oc + gcol; break;
                case P_UROR: gsrc = a.ur_over_r + v.oc + gcol; break;
                case P_UZ: gsrc = a.u_Z_star + v.ozf + gcol + v.nr; break;       // face j + 1
                case P_AL: gsrc = !a.aF ? a.alpha + v.oc + cc : nullptr; break;
                default: gsrc = !a.aF && a.alpha_cF ? a.alpha_cF + v.oc + cc : nullptr; break;
            }
        }
    } else if (t < PGEO) {
        gsrc = a.zint + v.ozint + 5 + (t - P_N * PNC);                           // face j + 1
        gstr = 5;
    }
    const bool g_al = gi == P_AL || gi == P_ACF;
    auto geo_copy = [&](int jb) {
        int row = jb;
        if (g_al) row = jb + 3 < v.nz ? jb + 3 : v.nz - 1;
        if (gsrc != nullptr && (g_al || jb < j1)) cp_async_el(geo + (jb & 1) * PGEO + t, gsrc + (long long)gstr * row);
    };

    // ---- prologue: the first copies, then rows j0-2 .. j0+1 by loads ----
    issue_own(j0 + 2);
    if constexpr (AHEAD) issue_halo(j0);
    geo_copy(j0);
    if (g_al) geo_copy(j0 - 1);
    cp_async_commit();
    if (item) {
        // (the loads of all four rows first, then their conversions)
        Cell<S> x[4];
        R aF[4];
        auto skip = [&](int r) { return r < -2 || r > v.nz + 1 || (col >= v.nr && (r < 0 || r >= v.nz)); };
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int r = j0 - 2 + q;
            if (skip(r)) continue;
            x[q] = raw_cell<S, S>(a, v, col, r, k);
            aF[q] = alpha_F_clamped<S, R>(a, v, col, r, k);
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int r = j0 - 2 + q, sl = r & (RING - 1);
            if (skip(r)) continue;
            put(A + sl * 4 * PT + t, x[q].J, x[q].Hr, x[q].HZ, aF[q]);
            // (the state of rows below j0 is not needed, and row j0-2's slot is row j0+2's)
            if (q >= 2) keep(Hs + sl * HF * PT + t, x[q]);
        }
    }
    for (int e = t; e < PNC * 5; e += PT) {
        const int f = i0 + e / 5;
        if (f <= v.nr) riv[e] = R(__ldg(a.rint + v.orint + 5 * f + e % 5));
    }
    if (t < PNC && i0 + t < v.nr) irc[t] = __ldg(a.inv_r_cell + v.ocol + i0 + t);
    pass_rest();
    cp_async_wait<0>();
    __syncthreads();
    auto zface = [&](int f, const double *ivz, double us, R *F) {
        auto row = [&](int r) { return A + (r & (RING - 1)) * 4 * PT + t; };
        face_z_cells<R, FLUX>(row(f + 2), row(f + 3), row(f), row(f + 1), PT, jeps, us, ivz, F);
    };
    R zL[3] = {R(0), R(0), R(0)};
    if (own) zface(j0, a.zint + v.ozint + 5 * j0, __ldg(a.u_Z_star + v.ozf + col + (long long)v.nr * j0), zL);
    long long x = v.o3 + (long long)k + (long long)a.nnu * ((long long)col + (long long)v.nr * j0);

    for (int j = j0; j < j1; j++) {
        const double *g = geo + (j & 1) * PGEO;
        // (A) row j+2 of the own columns and row j of the halo columns
        const int r = j + 2;
        if constexpr (!AHEAD) {
            if (halo) {
                const Cell<S> x = raw_cell<S, S>(a, v, hcol, j, hk);
                put(hp, x.J, x.Hr, x.HZ, alpha_F_clamped<S, R>(a, v, hcol, j, hk));
            }
        }
        if (stages(r)) {
            const int zrule = r < v.nz ? 0 : (v.bzt == 0 ? 1 : 3);
            const S *h = Hs + (r & (RING - 1)) * HF * PT + t;
            const double *gp = geo + ((j - 1) & 1) * PGEO + c;
            put(A + (r & (RING - 1)) * 4 * PT + t, HF == 3 ? h[2 * PT] : raw[t], bc_rule(h[0], orule),
                bc_rule(h[PT], zrule), aF_of(raw[RJ + t], gp[P_AL * PNC], gp[P_ACF * PNC]));
        }
        issue_own(r + 1);
        if constexpr (AHEAD) {
            if (halo) {
                put(hp, hraw[0], bc_rule(hraw[hps], hrule), hraw[2 * hps],
                    aF_of(hraw[3 * hps], *hal0, *hal1));
                issue_halo(j + 1);
            }
        }
        __syncthreads();
        geo_copy(j + 1);
        cp_async_commit();
        // (B) the r face left of the column, the Z face j+1/2: computed by every thread of a warp that
        // has an item (a thread without one reads what lies in its places and keeps nothing), so that
        // the two faces are one straight run of code
        R zR[3] = {R(0), R(0), R(0)};
        if (busy) {
            const R *p = A + (j & (RING - 1)) * 4 * PT + t;
            const R *hb = HB + (k - kbeg);
            R F[3], kL, kR;
            face_r_cells<R, FLUX>(c >= 2 ? p - 2 * nbk : hb + c * nbk, c >= 1 ? p - nbk : hb + nbk, p,
                                  c < ncol ? p + nbk : hb + 2 * nbk, PT, col == 0, jeps, g[P_UR * PNC + cg],
                                  riv + 5 * cg, F, kL, kR);
            zface(j + 1, g + P_N * PNC, g[P_UZ * PNC + cg], zR);
            R *o = Fr + t;
            o[0] = F[0]; o[PT] = F[1]; o[2 * PT] = F[2]; o[3 * PT] = kL; o[4 * PT] = kR;
        }
        __syncthreads();
        // (C) cell update
        if (own) {
            const S *h = Hs + (j & (RING - 1)) * HF * PT + t;
            const S uJ = HF == 3 ? h[2 * PT] : S(A[(j & (RING - 1)) * 4 * PT + t]);
            const double *q = g + c;
            const UpdGeo ug = {q[P_AR * PNC],    q[P_AR * PNC + 1], q[P_AZL * PNC],   q[P_AZR * PNC],
                               q[P_IDV * PNC],   q[P_DURDR * PNC],  q[P_DURDZ * PNC], q[P_DUZDR * PNC],
                               q[P_DUZDZ * PNC], q[P_UROR * PNC],   irc[c]};
            cell_update<S, R>(a, x, uJ, h[0], h[PT], zL, zR, Fr + t, Fr + t + nbk, PT, ug, v.ctdt, jeps);
        }
        x += (long long)a.nnu * v.nr;
        zL[0] = zR[0]; zL[1] = zR[1]; zL[2] = zR[2];
        cp_async_wait<0>();
    }
}

template <typename S, typename R, int FLUX, int MINB>
__global__ void __launch_bounds__(PT, MINB) k_advect(AdvArgs<S> a) {
    extern __shared__ __align__(128) unsigned char adv_smem[];
    pdl_trigger();
    pdl_wait();                                             // (the tile's very shape is the last step's decision)
    advect_tile<S, R, FLUX>(a, blockIdx.x, adv_smem);
}

// ------------------------------------------------------------------------------------------
// Frequency kernel helpers
// ------------------------------------------------------------------------------------------
template <int M>
struct Row {
    double a[M], b[M], c[M], d[M];
};

// (A cell's bins lie across a group of G lanes, M contiguous bins to a lane; `ln` is the lane's place in
// its group, and every shuffle stays inside the group.)
// Fetch, for every owned row r = lane*M + m, the quantity v of row r - s (dir = -1) or r + s
// (dir = +1). Rows outside [0, 32M) read the identity-row value `idv`.
template <int M>
__device__ __forceinline__ void nbr(const double (&v)[M], double (&out)[M], int s, int dir, int lane, double idv) {
    if (s < M) {
#pragma unroll
        for (int m = 0; m < M; m++) {
            int mm = m + dir * s;
            if (mm >= 0 && mm < M) {
                out[m] = v[mm];
            } else {
                int src = mm < 0 ? mm + M : mm - M;
                double w = 0.0;
#pragma unroll
                for (int q = 0; q < M; q++)
                    if (q == src) w = v[q];
                double got = dir < 0 ? __shfl_up_sync(0xffffffffu, w, 1) : __shfl_down_sync(0xffffffffu, w, 1);
                bool oob = dir < 0 ? (lane == 0) : (lane == 31);
                out[m] = oob ? idv : got;
            }
        }
    } else {
        int t = s / M;
#pragma unroll
        for (int m = 0; m < M; m++) {
            double got = dir < 0 ? __shfl_up_sync(0xffffffffu, v[m], t) : __shfl_down_sync(0xffffffffu, v[m], t);
            bool oob = dir < 0 ? (lane < t) : (lane + t > 31);
            out[m] = oob ? idv : got;
        }
    }
}

// Parallel cyclic reduction of the 32*M-row tridiagonal system held by the warp (8 bins per lane; fewer
// take cr_pcr_solve below) (row r = lane*M + m; a = sub-, b = main-, c = super-diagonal, d = right-hand side).
// Decoupled rows are identity rows. Returns x in d.
template <int M>
__device__ __forceinline__ void pcr_solve(Row<M> &R_, int lane) {
#pragma unroll
    for (int s = 1; s < 32 * M; s <<= 1) {
        double ib[M];
#pragma unroll
        for (int m = 0; m < M; m++) ib[m] = rcp<double>(R_.b[m]);
        double am[M], cm[M], dm[M], ibm[M], ap[M], cp[M], dp[M], ibp[M];
        nbr<M>(R_.a, am, s, -1, lane, 0.0);
        nbr<M>(R_.c, cm, s, -1, lane, 0.0);
        nbr<M>(R_.d, dm, s, -1, lane, 0.0);
        nbr<M>(ib, ibm, s, -1, lane, 1.0);
        nbr<M>(R_.a, ap, s, +1, lane, 0.0);
        nbr<M>(R_.c, cp, s, +1, lane, 0.0);
        nbr<M>(R_.d, dp, s, +1, lane, 0.0);
        nbr<M>(ib, ibp, s, +1, lane, 1.0);
#pragma unroll
        for (int m = 0; m < M; m++) {
            double al = -R_.a[m] * ibm[m];
            double ga = -R_.c[m] * ibp[m];
            double nb = R_.b[m] + al * cm[m] + ga * ap[m];
            double nd = R_.d[m] + al * dm[m] + ga * dp[m];
            R_.a[m] = al * am[m];
            R_.c[m] = ga * cp[m];
            R_.b[m] = nb;
            R_.d[m] = nd;
        }
    }
#pragma unroll
    for (int m = 0; m < M; m++) R_.d[m] = R_.d[m] * rcp<double>(R_.b[m]);
}

// Lane-serial elimination of the same system: the group writes its rows to shared memory and its
// first lane runs the forward elimination and back substitution of dgtsv's no-interchange branch
// (the Thomas algorithm), then the rows are read back. `sm` holds 4*G*M doubles of the group.
template <int M, int G>
__device__ __forceinline__ void thomas_solve(Row<M> &R_, int ln, double *sm) {
    constexpr int N = G * M;
    double *a = sm, *b = sm + N, *c = sm + 2 * N, *d = sm + 3 * N;
#pragma unroll
    for (int m = 0; m < M; m++) {
        int r = ln * M + m;
        a[r] = R_.a[m]; b[r] = R_.b[m]; c[r] = R_.c[m]; d[r] = R_.d[m];
    }
    __syncwarp();
    if (ln == 0) {
        for (int r = 1; r < N; r++) {
            double fact = a[r] / b[r - 1];
            b[r] = b[r] - fact * c[r - 1];
            d[r] = d[r] - fact * d[r - 1];
        }
        d[N - 1] = d[N - 1] / b[N - 1];
        for (int r = N - 2; r >= 0; r--) d[r] = (d[r] - c[r] * d[r + 1]) / b[r];
    }
    __syncwarp();
#pragma unroll
    for (int m = 0; m < M; m++) {
        int r = ln * M + m;
        R_.d[m] = d[r];
        R_.b[m] = b[r];
    }
    __syncwarp();
}

template <int G>
__device__ __forceinline__ double up1(double v, int s = 1) { return __shfl_up_sync(0xffffffffu, v, s, G); }
template <int G>
__device__ __forceinline__ double dn1(double v, int s = 1) { return __shfl_down_sync(0xffffffffu, v, s, G); }

// PCR over one row per lane (lane ln of a group holds row ln of a G-row system coupled to ln +- s),
// every row scaled to a unit diagonal so that a level fetches three values from each neighbour;
// returns the last level's diagonal (the pivot, before scaling) in eb and x in ed. A lane with no
// neighbour at distance s gets its own values back from the shuffle, and its coupling that way is zero
// (the first row's a and the last row's c are, and a level carries the zeros on to lanes ln < 2 s and
// from the far end), so nothing is selected (256^2 x 64 FP64 139 -> 137 us, 512^2 x 128 1025 -> 1006).
template <int G>
__device__ __forceinline__ void pcr_lanes(double ea, double &eb, double ec, double &ed) {
    double ib = rcp<double>(eb);
    double na = ea * ib, nc = ec * ib, nd = ed * ib;
#pragma unroll
    for (int s = 1; s < G; s <<= 1) {
        double am = up1<G>(na, s), cm = up1<G>(nc, s), dm = up1<G>(nd, s);
        double ap = dn1<G>(na, s), cp = dn1<G>(nc, s), dp = dn1<G>(nd, s);
        eb = fma(-na, cm, fma(-nc, ap, 1.0));
        const double a2 = -na * am, c2 = -nc * cp;
        const double d2 = fma(-na, dm, fma(-nc, dp, nd));
        ib = rcp<double>(eb);
        na = a2 * ib;
        nc = c2 * ib;
        nd = d2 * ib;
    }
    ed = nd;
}

template <int G>
__device__ __forceinline__ void cr_pcr_solve(Row<1> &R_) {
    pcr_lanes<G>(R_.a[0], R_.b[0], R_.c[0], R_.d[0]);
}

// Two rows per lane (rows 2l and 2l+1): one cyclic-reduction step eliminates the odd rows, leaving
// one row per lane, which PCR across the group solves; the odd rows then follow by
// back-substitution. Half the divisions and shuffles of PCR on all rows, the same arithmetic per
// eliminated row. Returns x in d; b holds the pivots for the zero-pivot check.
template <int G>
__device__ __forceinline__ void cr_pcr_solve(Row<2> &R_) {
    // odd row o = 2l+1 of this lane; o- = 2l-1 is the previous lane's odd row
    const double ibo = rcp<double>(R_.b[1]);
    double a_om = up1<G>(R_.a[1]), c_om = up1<G>(R_.c[1]), d_om = up1<G>(R_.d[1]), ib_om = up1<G>(ibo);
    // even row e = 2l: eliminate x_{e-1} (row o-) and x_{e+1} (row o)
    const double al = -R_.a[0] * ib_om, ga = -R_.c[0] * ibo;
    const double ea = al * a_om, ec = ga * R_.c[1];
    double eb = R_.b[0] + al * c_om + ga * R_.a[1];
    double ed = R_.d[0] + al * d_om + ga * R_.d[1];
    pcr_lanes<G>(ea, eb, ec, ed);
    // odd rows: x_o = (d_o - a_o x_e - c_o x_{e+2}) / b_o
    const double xe2 = dn1<G>(ed);
    R_.d[0] = ed;
    R_.d[1] = (R_.d[1] - R_.a[1] * ed - R_.c[1] * xe2) * ibo;
    R_.b[0] = eb;
}

// Three rows per lane (rows 3l .. 3l+2): rows 3l+1 and 3l+2 eliminated down the lane, which leaves
// row 3l coupled to the neighbouring lanes' rows 3l -+ 3 for the PCR; then back-substitution.
template <int G>
__device__ __forceinline__ void cr_pcr_solve(Row<3> &R_) {
    const double ib1 = rcp<double>(R_.b[1]);
    const double f = -R_.a[2] * ib1;
    const double a2 = f * R_.a[1], b2 = fma(f, R_.c[1], R_.b[2]), d2 = fma(f, R_.d[1], R_.d[2]);
    const double ib2 = rcp<double>(b2);
    // x2 = A2 + B2 x0 + C2 x3, x1 = A1 + B1 x0 + C1 x3
    const double A2 = d2 * ib2, B2 = -a2 * ib2, C2 = -R_.c[2] * ib2;
    const double g = -R_.c[1] * ib1;
    const double A1 = fma(g, A2, R_.d[1] * ib1), B1 = fma(g, B2, -R_.a[1] * ib1), C1 = g * C2;
    const double A2m = up1<G>(A2), B2m = up1<G>(B2), C2m = up1<G>(C2);
    const double ea = R_.a[0] * B2m, ec = R_.c[0] * C1;
    double eb = fma(R_.a[0], C2m, fma(R_.c[0], B1, R_.b[0]));
    double ed = fma(-R_.a[0], A2m, fma(-R_.c[0], A1, R_.d[0]));
    pcr_lanes<G>(ea, eb, ec, ed);
    const double x3 = dn1<G>(ed);
    R_.d[0] = ed;
    R_.d[1] = fma(C1, x3, fma(B1, ed, A1));
    R_.d[2] = fma(C2, x3, fma(B2, ed, A2));
    R_.b[0] = eb;
    R_.b[2] = b2;
}

// Four rows per lane (rows 4l .. 4l+3): two cyclic-reduction steps (the odd rows, then rows
// 4l+2) leave row 4l, solved by PCR across the group; rows 4l+2, then the odd rows follow by
// back-substitution.
template <int G>
__device__ __forceinline__ void cr_pcr_solve(Row<4> &R_) {
    const double ib1 = rcp<double>(R_.b[1]), ib3 = rcp<double>(R_.b[3]);
    double a3p = up1<G>(R_.a[3]), c3p = up1<G>(R_.c[3]), d3p = up1<G>(R_.d[3]), ib3p = up1<G>(ib3);
    // level 1: rows 4l (eliminate 4l-1, 4l+1) and 4l+2 (eliminate 4l+1, 4l+3)
    double al = -R_.a[0] * ib3p, ga = -R_.c[0] * ib1;
    double a0 = al * a3p, b0 = R_.b[0] + al * c3p + ga * R_.a[1], c0 = ga * R_.c[1];
    double d0 = R_.d[0] + al * d3p + ga * R_.d[1];
    al = -R_.a[2] * ib1;
    ga = -R_.c[2] * ib3;
    double a2 = al * R_.a[1], b2 = R_.b[2] + al * R_.c[1] + ga * R_.a[3], c2 = ga * R_.c[3];
    double d2 = R_.d[2] + al * R_.d[1] + ga * R_.d[3];
    // level 2: row 4l eliminates 4l-2 (previous lane's row 2) and 4l+2
    const double ib2 = rcp<double>(b2);
    double a2p = up1<G>(a2), c2p = up1<G>(c2), d2p = up1<G>(d2), ib2p = up1<G>(ib2);
    al = -a0 * ib2p;
    ga = -c0 * ib2;
    double eb = b0 + al * c2p + ga * a2, ed = d0 + al * d2p + ga * d2;
    pcr_lanes<G>(al * a2p, eb, ga * c2, ed);
    const double x0 = ed;
    const double x4 = dn1<G>(x0);
    const double x2 = (d2 - a2 * x0 - c2 * x4) * ib2;
    R_.d[1] = (R_.d[1] - R_.a[1] * x0 - R_.c[1] * x2) * ib1;
    R_.d[3] = (R_.d[3] - R_.a[3] * x2 - R_.c[3] * x4) * ib3;
    R_.d[0] = x0;
    R_.d[2] = x2;
    R_.b[0] = eb;
    R_.b[2] = b2;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
// over a group of G lanes
template <int G>
__device__ __forceinline__ double group_sum(double v) {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Per-bin constants of UpdateFreqFactors! staged in shared memory once per CTA. With the half-widths
// dl = nuC - nu (left) and dr = nu_{k+1} - nuC (right) of a bin, the Peclet number at one of the three
// places a row needs is P = C r, r = d / K, C = vel nuC + K (h/kT - 2 / nuC) (src/FreqFactors.jl:205-250),
// i.e. P = vel (nuC d) / K + (h/kT) d - 2 d / nuC: KC_A* = nuC d, KC_D* = d, KC_B* = -2 d / nuC (zero without
// recoil). *P: the left half of bin k+1, stored at k; *R: the right half of bin k (and, read at k-1,
// of bin k-1). KC_EXP2: the 32 entries of exp_tab's table.
enum { KC_AP, KC_DP, KC_BP, KC_AR, KC_DR, KC_BR, KC_IDNU, KC_DNU, KC_EXP2 };

// Per-cell inputs staged in shared memory, 32 cells at a time per warp, one cell per lane, already in
// the combinations the cell loop uses: opacities times c~ dt, the source, the prefactor of K, h/kT, the
// velocity gradients over c (g0 = du_r/dr, g12 = du_r/dZ + du_Z/dr, g3 = du_Z/dZ, tr = the trace with
// u_r/r), dV, the emitted power. CS_SUM_R / CS_SUM_Z receive each cell's sum over bins of
// dnu (H_old - H), which the warp's lanes turn into the cell's momentum, force and diagnostics once per
// 32 cells, one cell per lane.
enum { CS_AL, CS_AC, CS_APD, CS_ACF, CS_SRC, CS_PREF, CS_REC0, CS_G0, CS_G12, CS_G3, CS_TR, CS_DV, CS_POW,
       CS_DRU_R, CS_DRU_Z, CS_SUM_R, CS_SUM_Z, CS_N };

// A lane's M contiguous doubles of a shared-memory row, as 16-byte loads where M allows.
template <int M>
__device__ __forceinline__ void lds_row(const double *p, double (&v)[M]) {
    if constexpr (M % 2 == 0) {
#pragma unroll
        for (int m = 0; m < M; m += 2) {
            const double2 t = *reinterpret_cast<const double2 *>(p + m);
            v[m] = t.x;
            v[m + 1] = t.y;
        }
    } else {
#pragma unroll
        for (int m = 0; m < M; m++) v[m] = p[m];
    }
}

// Shared memory of the frequency kernel, in doubles: the FP64 per-bin constants (NP = G M padded bins);
// per warp the staged cell inputs; up to 64 bins, per warp two slots (the cells at hand and the next
// ones, whose rows are copied in meanwhile) of `ns` rows: J, H_r, H_Z, H_voigt, and with G = 32 J_old when
// it is not J's own buffer; and the lane-serial solver's rows when it runs. A warp's reduction row
// overlays its slots, which are free once its cells are done. 71 KB per CTA at 64 bins, 87 KB at 48:
// two CTAs per SM. A third CTA per SM would fit at 64 bins, but its 80-register bound spills in the cell
// loop (FP64 at 256^2 x 64: 0.258 ms against 0.184 ms at two CTAs).
template <int M, int G> __host__ __device__ constexpr bool freq_prefetch() { return G * M <= 64; }
template <int M, int G>
__host__ __device__ constexpr int freq_rows_warp(int ns) {      // doubles per warp
    return freq_prefetch<M, G>() ? 2 * ns * 32 * M : 32 * M + 8;
}
template <int M, int G>
__host__ __device__ constexpr int freq_smem_off_cs() { return KC_EXP2 * G * M + 32; }
template <int M, int G>
__host__ __device__ constexpr int freq_smem_off_rows(int nwarps) { return freq_smem_off_cs<M, G>() + nwarps * CS_N * 32; }
template <int M, int G>
__host__ __device__ constexpr int freq_smem_off_tsm(int nwarps, int ns) {
    return freq_smem_off_rows<M, G>(nwarps) + nwarps * freq_rows_warp<M, G>(ns);
}
template <int M, int G>
__host__ __device__ constexpr int freq_smem_doubles(int nwarps, bool thomas, int ns) {
    return freq_smem_off_tsm<M, G>(nwarps, ns) + (thomas ? nwarps * 4 * 32 * M : 0);
}
// rows of a slot
template <int G> __host__ __device__ constexpr int freq_ns(bool jo_alias) { return G == 32 && !jo_alias ? 5 : 4; }

// A lane's M contiguous bins of one row as whole 16-byte words, when the row layout allows it
// (k_freq's `vec` path): loads from shared memory and stores to global memory.
template <typename S, int M>
struct LaneRow {
    static constexpr bool ok = (M * sizeof(S)) % 16 == 0;
    static constexpr int words = (M * (int)sizeof(S)) / 16;
    __device__ __forceinline__ static void load(const S *src, S (&v)[M]) {
        if constexpr (ok) {
#pragma unroll
            for (int w = 0; w < words; w++) {
                const float4 t = reinterpret_cast<const float4 *>(src)[w];
                memcpy(&v[w * (16 / sizeof(S))], &t, 16);
            }
        }
    }
    __device__ __forceinline__ static void store(S *dst, const S (&v)[M]) {
        if constexpr (ok) {
#pragma unroll
            for (int w = 0; w < words; w++) {
                float4 t;
                memcpy(&t, &v[w * (16 / sizeof(S))], 16);
                reinterpret_cast<float4 *>(dst)[w] = t;
            }
        }
    }
};

// The cells [wbeg, wend) of a work item that warp `warp` of `nw` handles: one contiguous run
// per warp, of a multiple of `cpw` cells.
__device__ __forceinline__ void warp_cell_run(int4 it, int warp, int nw, int cpw, int &wbeg, int &wend) {
    const int per = ((it.z - it.y + nw - 1) / nw + cpw - 1) / cpw * cpw;
    wbeg = it.y + warp * per;
    wend = min(it.z, wbeg + per);
}

// Up to four bins per lane the kernel is held to 2 CTAs per SM (128 registers).
// A cell's bins lie across a group of G lanes, M contiguous bins to a lane: up to 48 bins half a warp
// (two cells per warp, 1, 2 or 3 bins per lane), beyond a whole warp. With whole warps 48 bins left 8 of
// 32 lanes idle and the solve took five levels across 32 lanes for each cell; by halves every lane has
// work, a level serves two cells and there are four: 24 clouds x 48 bins 123 -> 86 us per launch. At 64
// bins half warps (4 bins per lane) spill: 149 us against 140 at 256^2 in FP64, so they keep the
// whole warp.
// RC is the arithmetic of the cell-centre closure D(J, H) and of D:grad u that enter the Doppler
// term of the frequency factors: R in the FP64 and FP32-storage forms, FP32 in the mixed form.
// The closure only sets the velocity of the Peclet numbers; every factor is then formed in FP64
// from that one velocity, so its rounding moves the step like a velocity field off by 1e-7
// relative, not like the rounding of F against F+ + F- that the factors themselves cannot take
// (mixed frequency kernel at 256^2 x 64: 0.259 -> 0.246 ms; the mixed form's M_F after 2000
// steps 5.93e-7 -> 5.95e-7 from FP64).
//
// Bound by instruction issue and dependent FP64 latency (16 warps per SM). What a cell's 32 lanes
// share (opacities times c~ dt, the prefactor of K, h/kT, the gradients' combinations, column and row) is
// formed once per 32 cells, one cell per lane; the Peclet numbers come from per-bin constants by
// three multiply-adds; and the factors of a lane's bins are straight-line code (no branch per bin,
// padding bins computed and dropped). Warp instructions per launch at 256^2 x 64: 114 -> 91 million;
// per launch 178 -> 141 us (FP64), 174 -> 138 (mixed), 163 -> 129 (FP32 storage); 512^2 x 128 1474 ->
// 1026 us, 24 clouds x 48 bins 158 -> 123 us, 64^2 x 64 27 -> 24 us.
//
// freq_item is one work item (`item` of `nitems`) by the calling CTA of FREQ_THREADS threads, in dynamic
// shared memory `fsm`: the body of k_freq, also run by the persistent batch kernel.
template <typename S, typename R, int M, int G, typename RC>
__device__ __forceinline__ void freq_item(const FreqArgs<S> &a, int item, int nitems, double *fsm) {
    constexpr int nw = FREQ_THREADS / 32;
    constexpr int NP = G * M, WN = 32 * M, CPW = 32 / G;   // a cell's padded bins, a warp's, a warp's cells
    constexpr bool PF = freq_prefetch<M, G>(), PARK = M == 3;
    static_assert(freq_rows_warp<M, G>(4) >= NP + 8, "a warp's reduction row fits its rows");
    const bool jo_alias = a.Jold == a.Jin;
    const int ns = freq_ns<G>(jo_alias);                  // rows of a slot
    double *kc = fsm;                                     // [KC_EXP2][NP], then the exponentials' table
    double *tsm = fsm + freq_smem_off_tsm<M, G>(nw, ns);  // [nwarps][CPW][4][NP] (lane-serial solver)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ln = lane & (G - 1), sub = lane / G;        // place in the cell's group, the group's cell
    const int nnu = a.nnu;
    for (int t = threadIdx.x; t < NP; t += blockDim.x) {
        const bool up = t + 1 < nnu, in = t < nnu;
        const double dp = up ? a.nuC[t + 1] - a.nu[t + 1] : 0.0, dr = in ? a.nu[t + 1] - a.nuC[t] : 0.0;
        kc[KC_AP * NP + t] = up ? a.nuC[t + 1] * dp : 0.0;
        kc[KC_DP * NP + t] = dp;
        kc[KC_BP * NP + t] = up && a.recoil ? -2.0 * dp * a.inv_nuC[t + 1] : 0.0;
        kc[KC_AR * NP + t] = in ? a.nuC[t] * dr : 0.0;
        kc[KC_DR * NP + t] = dr;
        kc[KC_BR * NP + t] = in && a.recoil ? -2.0 * dr * a.inv_nuC[t] : 0.0;
        kc[KC_IDNU * NP + t] = in ? a.inv_dnu[t] : 0.0;
        kc[KC_DNU * NP + t] = in ? a.dnu[t] : 0.0;
    }
    if (threadIdx.x < 32) kc[KC_EXP2 * NP + threadIdx.x] = kExp2Tab[threadIdx.x];
    pdl_wait();                               // (the constants above are none of the step's own)
    __syncthreads();

    const int4 it = a.items[item];
    const CloudDesc &cd = a.cl[it.x];
    const long long o3 = cd.o3, oc = cd.oc;
    const int nr = cd.nr, nz = cd.nz, bzb = cd.bc_z_bot;
    const double c_tilde = cd.c_tilde, dt = cd.dt, ctdt = cd.ctdt, z_center = cd.z_center;
    const double jeps = a.jeps;
    const double dw = 1.0 / ctdt;
    double acc_e[M];
#pragma unroll
    for (int m = 0; m < M; m++) acc_e[m] = 0.0;
    double acc_tot = 0.0, acc_mf = 0.0, acc_net = 0.0, acc_out = 0.0, acc_L = 0.0, acc_esc = 0.0;
    int bad = 0;

    int wbeg, wend;
    warp_cell_run(it, warp, nw, CPW, wbeg, wend);
    double *cs = fsm + freq_smem_off_cs<M, G>() + warp * CS_N * 32;      // [CS_N][32]
    S *rows = reinterpret_cast<S *>(fsm + freq_smem_off_rows<M, G>(nw) + warp * freq_rows_warp<M, G>(ns));
    const bool need_ff = a.do_freq && a.update_ff, need_js = a.do_emission || (a.parts & PART_DIAG);
    // With `vec`, every lane's M bins of a row are whole 16-byte words in global and shared memory
    // (row starts 16-byte aligned, n_nu a multiple of M). A group of a whole warp (G = 32) then moves its
    // rows lane by lane, bin m of lane l at l*M + m, else element by element, bin m of lane l at
    // m*32 + l; groups of 16 copy their two cells' rows as the one run they are in memory.
    using LR = LaneRow<S, M>;
    const bool vec = LR::ok && a.vec16 && nnu % M == 0;
    // copies of the rows of cells cl .. into slot b
    auto issue = [&](int cl, int b) {
        const long long base = o3 + (long long)cl * nnu;
        S *d = rows + b * ns * WN;
        constexpr int per = 16 / sizeof(S);
        if constexpr (G == 32) {
            if constexpr (LR::ok) {
                if (vec) {
                    if (lane * M < nnu) {
                        const long long g = base + lane * M;
                        const int q = lane * M;
#pragma unroll
                        for (int w = 0; w < LR::words; w++) {
                            cp_async_16(d + q + w * per, a.Jin + g + w * per);
                            cp_async_16(d + WN + q + w * per, a.Hrin + g + w * per);
                            cp_async_16(d + 2 * WN + q + w * per, a.HZin + g + w * per);
                            cp_async_16(d + 3 * WN + q + w * per, a.Hv + g + w * per);
                            if (!jo_alias) cp_async_16(d + 4 * WN + q + w * per, a.Jold + g + w * per);
                        }
                    }
                    return;
                }
            }
#pragma unroll
            for (int m = 0; m < M; m++) {
                const int k = lane * M + m, q = m * 32 + lane;
                if (k < nnu) {
                    cp_async_el(d + q, a.Jin + base + k);
                    cp_async_el(d + WN + q, a.Hrin + base + k);
                    cp_async_el(d + 2 * WN + q, a.HZin + base + k);
                    cp_async_el(d + 3 * WN + q, a.Hv + base + k);
                    if (!jo_alias) cp_async_el(d + 4 * WN + q, a.Jold + base + k);
                }
            }
        } else {
            const int n = min(CPW, wend - cl) * nnu;
            if (a.vec16) {
                for (int e = lane * per; e < n; e += 32 * per) {
                    cp_async_16(d + e, a.Jin + base + e);
                    cp_async_16(d + WN + e, a.Hrin + base + e);
                    cp_async_16(d + 2 * WN + e, a.HZin + base + e);
                    cp_async_16(d + 3 * WN + e, a.Hv + base + e);
                }
            } else {
                for (int e = lane; e < n; e += 32) {
                    cp_async_el(d + e, a.Jin + base + e);
                    cp_async_el(d + WN + e, a.Hrin + base + e);
                    cp_async_el(d + 2 * WN + e, a.HZin + base + e);
                    cp_async_el(d + 3 * WN + e, a.Hv + base + e);
                }
            }
        }
    };
    // a lane's bins of a row that starts at p (in shared or global memory), zeros beyond n_nu
    auto row_get = [&](const S *p, bool ok, S (&v)[M]) {
        if (vec) {
            if (ok && ln * M < nnu) {
                LR::load(p + ln * M, v);
            } else {
#pragma unroll
                for (int m = 0; m < M; m++) v[m] = S(0);
            }
        } else {
#pragma unroll
            for (int m = 0; m < M; m++) v[m] = (ok && ln * M + m < nnu) ? p[ln * M + m] : S(0);
        }
    };
    auto row_put = [&](S *p, bool ok, const S (&v)[M]) {
        if (vec) {
            if (ok && ln * M < nnu) LR::store(p + ln * M, v);
        } else {
#pragma unroll
            for (int m = 0; m < M; m++)
                if (ok && ln * M + m < nnu) p[ln * M + m] = v[m];
        }
    };
    const double k4 = kFourPiOverC * (1.0 / c_tilde) * a.j_scale;
    const double inv_dt = 1.0 / dt;
    // emission/absorption steps over c~ dt; its source in storage units
    const double ctdt_e = c_tilde * dt, src_w = c_tilde * dt / a.j_scale;
    // the per-cell part of the epilogue for cells [gb, ge) of the run (ge - gb <= 32), one
    // cell per lane: the momentum Delta rho u, this step's force, and the M_F, L and radial
    // partials (Update_f_Lya_MF_L_Lya!, src/ConstantsAndFunctions.jl:588-674)
    auto flush = [&](int gb, int ge) {
        __syncwarp();
        const int cl = gb + lane;
        if (cl >= ge) return;
        const long long c = oc + cl;
        const double drs = cs[CS_SUM_R * 32 + lane], dzs = cs[CS_SUM_Z * 32 + lane];
        if (a.do_emission && a.dru_r) {
            a.dru_r[c] = cs[CS_DRU_R * 32 + lane] + k4 * drs;
            a.dru_Z[c] = cs[CS_DRU_Z * 32 + lane] + k4 * dzs;
        }
        if (a.parts & PART_DIAG) {
            const int i = cl % nr, j = cl / nr;
            const double dV = cs[CS_DV * 32 + lane];
            double fr = (k4 * drs) * inv_dt, fz = (k4 * dzs) * inv_dt;
            if (a.f_r) { a.f_r[c] = fr; a.f_Z[c] = fz; }
            acc_mf += dV * sqrt(fr * fr + fz * fz);
            acc_L += cs[CS_POW * 32 + lane];
            double drr = __ldg(a.rCoM + cd.ocol + i), dzz = __ldg(a.ZCoM + cd.orow + j) - z_center;
            double dist = sqrt(drr * drr + dzz * dzz);
            double frad = 0.0;
            if (dist > 0.0) {
                double id = 1.0 / dist;
                frad = fr * (drr * id) + fz * (dzz * id);
            }
            acc_net += dV * frad;
            acc_out += dV * (frad > 0.0 ? frad : 0.0);
        }
    };
    if constexpr (PF) {
        if (wbeg < wend) issue(wbeg, 0);
        cp_async_commit();
    }
    int g0 = wbeg;
    int i = (wbeg + sub) % nr, j = (wbeg + sub) / nr;     // the cell's column and row, advanced with it
    S nonfin = S(0);                           // 0 x everything written: NaN once something is not finite
    for (int c0 = wbeg; c0 < wend; c0 += CPW) {
        const int cl = c0 + sub;               // this group's cell (a last odd one leaves groups idle)
        const bool ok = G == 32 || cl < wend;
        const long long base = o3 + (long long)cl * nnu;
        if (((c0 - wbeg) & 31) == 0) {
            if (c0 > wbeg) flush(g0, c0);
            // stage the per-cell inputs of the next 32 cells of the run (one coalesced load per
            // field instead of a dependent load per cell)
            g0 = c0;
            __syncwarp();
            const bool v = c0 + lane < wend;
            const long long cc = oc + c0 + lane;
            auto ld = [&](const double *p, bool need) { return (v && need && p) ? __ldg(p + cc) : 0.0; };
            const double alv = ld(a.alpha, a.do_emission || need_ff), js = ld(a.js, need_js);
            const double dV = ld(a.dV, a.parts != 0);
            cs[CS_AL * 32 + lane] = alv * ctdt_e;
            cs[CS_AC * 32 + lane] = ld(a.alpha_c, a.do_emission) * ctdt_e;
            cs[CS_APD * 32 + lane] = alv * ld(a.pd, a.do_emission) * ctdt_e;
            cs[CS_ACF * 32 + lane] = ld(a.alpha_cF, a.do_emission) * ctdt_e;
            cs[CS_SRC * 32 + lane] = js * src_w * (a.phi ? 1.0 : ld(a.phi_inv, a.do_emission));
            if (need_ff) {
                // (the padding lanes get a temperature and no opacity)
                const double T = v ? ld(a.T, true) : 1.0, dnuD = compute_dnuD(T);
                cs[CS_PREF * 32 + lane] = 0.5 * (alv > a.alpha_floor ? alv : a.alpha_floor) * (dnuD * dnuD);
                cs[CS_REC0 * 32 + lane] = a.recoil ? kHOverKB / T : 0.0;
                const double g0 = ld(a.dur_dr, true), g3 = ld(a.duZ_dZ, true);
                cs[CS_G0 * 32 + lane] = g0 * kInvC;
                cs[CS_G12 * 32 + lane] = (ld(a.dur_dZ, true) + ld(a.duZ_dr, true)) * kInvC;
                cs[CS_G3 * 32 + lane] = g3 * kInvC;
                cs[CS_TR * 32 + lane] = (g0 + g3 + ld(a.ur_over_r, true)) * kInvC;
            }
            cs[CS_DV * 32 + lane] = dV;
            cs[CS_POW * 32 + lane] = kFourPi * dV * js;
            const bool du = v && a.do_emission && a.dru_r;       // (flush writes them: no __ldg)
            cs[CS_DRU_R * 32 + lane] = du ? a.dru_r[cc] : 0.0;
            cs[CS_DRU_Z * 32 + lane] = du ? a.dru_Z[cc] : 0.0;
            __syncwarp();
        }
        const double *cv = cs + (cl - g0);        // cv[f * 32]: field f of this cell
        S J[M], Hr[M], HZ[M];
        R Hv[M];
        double Jo[M];
        S *rH = rows;                             // where H_r, H_Z wait: rows WN apart
        if constexpr (G == 32 && PF) {
            const int b = (c0 - wbeg) & 1;
            if (c0 + 1 < wend) issue(c0 + 1, b ^ 1);
            cp_async_commit();
            cp_async_wait<1>();                   // this cell's copies (each lane reads its own)
            const S *d = rows + b * ns * WN;
            bool done = false;
            if constexpr (LR::ok) {
                if (vec) {
                    if (lane * M < nnu) {
                        const int q = lane * M;
                        S hv[M], jo[M];
                        LR::load(d + q, J);
                        LR::load(d + WN + q, Hr);
                        LR::load(d + 2 * WN + q, HZ);
                        LR::load(d + 3 * WN + q, hv);
                        LR::load(d + (jo_alias ? 0 : 4 * WN) + q, jo);
#pragma unroll
                        for (int m = 0; m < M; m++) { Hv[m] = R(hv[m]); Jo[m] = double(jo[m]); }
                    } else {
#pragma unroll
                        for (int m = 0; m < M; m++) { J[m] = Hr[m] = HZ[m] = S(0); Hv[m] = R(0); Jo[m] = 0.0; }
                    }
                    done = true;
                }
            }
            if (!done) {
#pragma unroll
                for (int m = 0; m < M; m++) {
                    const int k = lane * M + m, q = m * 32 + lane;
                    const bool vld = k < nnu;
                    J[m] = vld ? d[q] : S(0);
                    Hr[m] = vld ? d[WN + q] : S(0);
                    HZ[m] = vld ? d[2 * WN + q] : S(0);
                    Hv[m] = vld ? R(d[3 * WN + q]) : R(0);
                    Jo[m] = vld ? double(jo_alias ? d[q] : d[4 * WN + q]) : 0.0;
                }
            }
        } else if constexpr (G == 32) {
#pragma unroll
            for (int m = 0; m < M; m++) {
                int k = lane * M + m;
                bool vld = k < nnu;
                J[m] = vld ? a.Jin[base + k] : S(0);
                Hr[m] = vld ? a.Hrin[base + k] : S(0);
                HZ[m] = vld ? a.HZin[base + k] : S(0);
                Hv[m] = vld ? R(__ldg(a.Hv + base + k)) : R(0);
                Jo[m] = vld ? double(a.Jold[base + k]) : 0.0;
            }
        } else {
            S hv[M], jo[M];
            if (!jo_alias) row_get(a.Jold + base, ok, jo);
            const int b = ((c0 - wbeg) / CPW) & 1;
            __syncwarp();                         // every lane is done with the other slot
            if (c0 + CPW < wend) issue(c0 + CPW, b ^ 1);
            cp_async_commit();
            cp_async_wait<1>();                   // these cells' copies
            __syncwarp();
            S *d = rows + b * ns * WN + sub * nnu;
            row_get(d, ok, J);
            row_get(d + WN, ok, Hr);
            row_get(d + 2 * WN, ok, HZ);
            row_get(d + 3 * WN, ok, hv);
            rH = d + WN;
#pragma unroll
            for (int m = 0; m < M; m++) {
                Hv[m] = R(hv[m]);
                Jo[m] = double(jo_alias ? J[m] : jo[m]);
            }
        }
        double dr_sum = 0.0, dz_sum = 0.0;
        // ---- LyaEmissionAbsorptionUpdate! (src/ConstantsAndFunctions.jl:526-567) ----
        if (a.do_emission) {
            const R al = R(cv[CS_AL * 32]), ac = R(cv[CS_AC * 32]), apd = R(cv[CS_APD * 32]);
            const R acF = R(cv[CS_ACF * 32]), src = R(cv[CS_SRC * 32]);
            double dn[M];
            lds_row<M>(kc + KC_DNU * NP + ln * M, dn);
#pragma unroll
            for (int m = 0; m < M; m++) {
                const int k = ln * M + m;
                R phi = (k >= a.phi_kmin && k <= a.phi_kmax) ? Hv[m] : R(0);
                R aH = al * Hv[m] + acF;
                if (a.phi) phi = ok && k < nnu ? R(__ldg(a.phi + base + k)) : R(0);
                if (a.aF) aH = ok && k < nnu ? R(__ldg(a.aF + base + k)) * R(ctdt_e) : R(0);
                // (bins beyond n_nu hold zeros and have no width)
                const R Jn = (R(Jo[m]) + src * phi) * rcp<R>(R(1) + (ac + apd * Hv[m]));
                const R iden = rcp<R>(R(1) + aH);
                const R hr = R(Hr[m]) * iden, hz = R(HZ[m]) * iden;
                dr_sum += dn[m] * (double(Hr[m]) - double(hr));
                dz_sum += dn[m] * (double(HZ[m]) - double(hz));
                Hr[m] = S(hr);
                HZ[m] = S(hz);
                J[m] = S(Jn);
                Jo[m] = double(J[m]);
            }
            dr_sum = group_sum<G>(dr_sum);
            dz_sum = group_sum<G>(dz_sum);
        }
        if (ln == 0) {       // turned into the cell's momentum and diagnostics by flush()
            cs[CS_SUM_R * 32 + (cl - g0)] = dr_sum;
            cs[CS_SUM_Z * 32 + (cl - g0)] = dz_sum;
        }
        // ---- FrequencyUpdateJLya_AllCells! (src/UpdateLyaJandH.jl:231-391) ----
        if (a.do_freq) {
            Row<M> sys;
            double Fp[M], F0[M], Fm[M];
            if (a.update_ff) {
                // UpdateFreqFactors!, src/FreqFactors.jl:181-275, for every bin the lane holds (rows 0 and
                // n_nu - 1, and padding bins, form values nobody keeps), so the lane's bins are one
                // straight run of code.
                // The frequency factors stay FP64 in every precision variant: with F/dw up to
                // ~1e9 at tau0 = 1e8, an FP32 rounding of F0 against Fm + Fp acts as a spurious
                // source or sink tens of times larger than the step's own change.
                const double pref = cv[CS_PREF * 32], rec0 = cv[CS_REC0 * 32];
                const RC g0 = RC(cv[CS_G0 * 32]), g12 = RC(cv[CS_G12 * 32]), g3 = RC(cv[CS_G3 * 32]);
                const RC tr = RC(cv[CS_TR * 32]);
                // 1/K_k = 1 / (pref H_voigt[k]) once per bin; the k+-1 neighbours come by shuffle
                double iK[M];
#pragma unroll
                for (int m = 0; m < M; m++) iK[m] = rcp<double>(pref * double(Hv[m]));
                const double iK_up = up1<G>(iK[M - 1]), iK_dn = dn1<G>(iK[0]);
                const double *kl = kc + ln * M, *etab = kc + KC_EXP2 * NP;
                // the right half of the bin below the lane's first
                const int kb = ln > 0 ? -1 : 0;
                double ar = kl[KC_AR * NP + kb], drr = kl[KC_DR * NP + kb], br = kl[KC_BR * NP + kb];
                // three bins per lane: H_r and H_Z wait in their rows while the factors and the solve use the
                // registers (24 clouds x 48 bins 94 -> 86 us)
                double vel[M];
                auto vel_of = [&](int m) {
                    return double(work_rate<RC>(RC(J[m]), RC(Hr[m]), RC(HZ[m]), RC(jeps), RC(a.heps2), g0, g12, g3, tr));
                };
                if constexpr (PARK) {
#pragma unroll
                    for (int m = 0; m < M; m++) vel[m] = vel_of(m);
                    row_put(rH, ok, Hr);
                    row_put(rH + WN, ok, HZ);
                }
                constexpr int W = M % 2 == 0 ? 2 : 1;   // bins whose constants are held at a time
#pragma unroll
                for (int mb = 0; mb < M; mb += W) {
                    double AP[W], DP[W], BP[W], AR[W], DR[W], BR[W], idn[W];
                    lds_row<W>(kl + KC_AP * NP + mb, AP);
                    lds_row<W>(kl + KC_DP * NP + mb, DP);
                    lds_row<W>(kl + KC_BP * NP + mb, BP);
                    lds_row<W>(kl + KC_AR * NP + mb, AR);
                    lds_row<W>(kl + KC_DR * NP + mb, DR);
                    lds_row<W>(kl + KC_BR * NP + mb, BR);
                    lds_row<W>(kl + KC_IDNU * NP + mb, idn);
#pragma unroll
                    for (int w = 0; w < W; w++) {
                        const int m = mb + w;
                        if constexpr (!PARK) vel[m] = vel_of(m);
                        const double iKm = (m > 0) ? iK[m > 0 ? m - 1 : 0] : iK_up;
                        const double iKp = (m < M - 1) ? iK[m < M - 1 ? m + 1 : 0] : iK_dn;
                        const double rkp = DP[w] * iKp, rk = DR[w] * iK[m], rkm = drr * iKm;
                        const double Pkp = clamp_P(fma(vel[m] * AP[w], iKp, fma(rec0, DP[w], BP[w])));
                        const double Pk = clamp_P(fma(vel[m] * AR[w], iK[m], fma(rec0, DR[w], BR[w])));
                        const double Pkm = clamp_P(fma(vel[m] * ar, iKm, fma(rec0, drr, br)));
                        double oRkp, xRkp, oLk, xLk, oRk, xRk, oLkm, xLkm;
                        omphi_R(Pkp, oRkp, xRkp, etab);
                        omphi_LR(Pk, oLk, xLk, oRk, xRk, etab);
                        omphi_L(Pkm, oLkm, xLkm, etab);
                        const double dkp = idn[w] * rcp<double>(xLk * rk - xRkp * rkp);
                        const double dkm = idn[w] * rcp<double>(xLkm * rkm - xRk * rk);
                        Fp[m] = oRkp * dkp;
                        Fm[m] = oLkm * dkm;
                        F0[m] = oLk * dkp + oRk * dkm;
                        ar = AR[w]; drr = DR[w]; br = BR[w];
                    }
                }
                if (a.Fkp) {
#pragma unroll
                    for (int m = 0; m < M; m++) {
                        int k = ln * M + m;
                        const bool in = k >= 1 && k <= nnu - 2;
                        if (ok && k < nnu) {
                            a.Fkp[base + k] = in ? Fp[m] : 0.0;
                            a.Fk[base + k] = in ? F0[m] : 0.0;
                            a.Fkm[base + k] = in ? Fm[m] : 0.0;
                        }
                    }
                }
            } else {
#pragma unroll
                for (int m = 0; m < M; m++) {
                    int k = ln * M + m;
                    bool in = (ok && k >= 1 && k <= nnu - 2);
                    Fp[m] = in ? a.Fkp[base + k] : 0.0;
                    F0[m] = in ? a.Fk[base + k] : 0.0;
                    Fm[m] = in ? a.Fkm[base + k] : 0.0;
                }
            }
            // rows k = 1 .. nnu-2 of src/UpdateLyaJandH.jl:200-214; the couplings of the
            // first and last rows to k = 0 and k = nnu-1 are dropped (TridiagonalSolver.jl:45-46)
#pragma unroll
            for (int m = 0; m < M; m++) {
                int k = ln * M + m;
                bool in = (ok && k >= 1 && k <= nnu - 2);
                sys.a[m] = (in && k >= 2) ? Fm[m] : 0.0;
                sys.b[m] = in ? -(F0[m] + dw) : 1.0;
                sys.c[m] = (in && k <= nnu - 3) ? Fp[m] : 0.0;
                sys.d[m] = in ? -dw * Jo[m] : 0.0;
            }
            if (a.solver == SOLVER_THOMAS)
                thomas_solve<M, G>(sys, ln, tsm + (warp * CPW + sub) * 4 * NP);
            else
                if constexpr (M <= 4) cr_pcr_solve<G>(sys);
                else pcr_solve<M>(sys, lane);
            if constexpr (PARK) {
                if (a.update_ff) {
                    row_get(rH, ok, Hr);
                    row_get(rH + WN, ok, HZ);
                }
            }
            // flux correction, src/UpdateLyaJandH.jl:341-377
#pragma unroll
            for (int m = 0; m < M; m++) {
                int k = ln * M + m;
                bool in = (k >= 1 && k <= nnu - 2);
                double Jn = in ? sys.d[m] : double(J[m]);
                if (!(sys.b[m] != 0.0)) bad |= ERRB_SOLVE;
                double Jf = Jn > jeps ? Jn : jeps;
                double ratio = Jf * rcp<double>(Jo[m] > jeps ? Jo[m] : jeps);
                double hr = double(Hr[m]) * ratio, hz = double(HZ[m]) * ratio;
                double H2 = hr * hr + hz * hz;
                if (H2 > Jf * Jf) {
                    double fsc = Jf * rsqrt_nr(H2);   // |H|^2 > J^2 >= jeps^2: normal
                    hr *= fsc;
                    hz *= fsc;
                }
                J[m] = S(Jf);
                Hr[m] = S(hr);
                HZ[m] = S(hz);
            }
        }
        // ---- store (bins beyond n_nu hold the floor and zeros) ----
#pragma unroll
        for (int m = 0; m < M; m++) nonfin += J[m] * S(0) + Hr[m] * S(0) + HZ[m] * S(0);
        row_put(a.Jout + base, ok, J);
        row_put(a.Hrout + base, ok, Hr);
        row_put(a.HZout + base, ok, HZ);
        // ---- epilogue partials ----
        if (a.parts & PART_ACTIVE) {
            // (bins beyond n_nu have no width)
            const double dV = cv[CS_DV * 32];
            double dn[M];
            lds_row<M>(kc + KC_DNU * NP + ln * M, dn);
#pragma unroll
            for (int m = 0; m < M; m++) {
                const double Jv = double(J[m]), w = dn[m] * dV;
                const double e1 = Jv - 10.0 * jeps, e0 = Jv - jeps;
                acc_e[m] += w * (e1 > 0.0 ? e1 : 0.0);
                acc_tot += w * (e0 > 0.0 ? e0 : 0.0);
            }
        }
        if (a.parts & PART_DIAG) {
            // escaping flux through the outer r face, the top face and (outflow) the bottom face
            double esc = 0.0;
            const bool rb = ok && i == nr - 1, zt = ok && j == nz - 1, zb = ok && j == 0 && bzb == 1;
            if (rb || zt || zb) {
                const double Arr = rb ? __ldg(a.A_r + cd.orf + nr + (long long)(nr + 1) * j) * kFourPi : 0.0;
                const double AZt = zt ? __ldg(a.A_Z + cd.ozf + i + (long long)nr * nz) * kFourPi : 0.0;
                const double AZb = zb ? __ldg(a.A_Z + cd.ozf + i) * kFourPi : 0.0;
#pragma unroll
                for (int m = 0; m < M; m++) {
                    int k = ln * M + m;
                    if (k >= nnu) continue;
                    double dn = kc[KC_DNU * NP + k];
                    double hr = double(S(Hr[m])) * a.j_scale, hz = double(S(HZ[m])) * a.j_scale;
                    if (rb) esc += dn * (Arr * (hr > 0.0 ? hr : 0.0));
                    if (zt) esc += dn * (AZt * (hz > 0.0 ? hz : 0.0));
                    if (zb) esc += dn * (AZb * (-hz > 0.0 ? -hz : 0.0));
                }
            }
            acc_esc += esc;
        }
        for (i += CPW; i >= nr; i -= nr) j++;
    }
    if (wbeg < wend) flush(g0, wend);
    if (nonfin != S(0)) bad |= ERRB_NONFINITE;
    if constexpr (PF) cp_async_wait<0>();
    if (bad) atomicOr(a.err, bad);
    if (!a.parts) return;
    // ---- CTA reduction of the partials, fixed order ----
    // (the warp's reduction row overlays its rows, whose last copies landed above)
    auto red_row = [&](int w) { return fsm + freq_smem_off_rows<M, G>(nw) + w * freq_rows_warp<M, G>(ns); };
    double *red = red_row(warp);
    __syncwarp();
#pragma unroll
    for (int m = 0; m < M; m++)
#pragma unroll
        for (int o = G; o < 32; o <<= 1) acc_e[m] += __shfl_xor_sync(0xffffffffu, acc_e[m], o);
    if (lane < G) {
#pragma unroll
        for (int m = 0; m < M; m++) red[lane * M + m] = acc_e[m];
    }
    acc_tot = warp_sum(acc_tot);
    acc_esc = warp_sum(acc_esc);
    acc_mf = warp_sum(acc_mf);
    acc_net = warp_sum(acc_net);
    acc_out = warp_sum(acc_out);
    acc_L = warp_sum(acc_L);
    if (lane == 0) {
        red[NP + 0] = acc_tot;
        red[NP + 1] = acc_mf;
        red[NP + 2] = acc_net;
        red[NP + 3] = acc_out;
        red[NP + 4] = acc_L;
        red[NP + 5] = acc_esc;
    }
    __syncthreads();
    const int ncols = nnu + kExtraCols;
    for (int col = threadIdx.x; col < ncols; col += blockDim.x) {
        int src = col < nnu ? col : NP + (col - nnu);
        double s = 0.0;
        for (int w2 = 0; w2 < nw; w2++) s += red_row(w2)[src];
        a.partials[(size_t)col * nitems + item] = s;
    }
}

template <typename S, typename R, int M, int G, typename RC = R>
__global__ void __launch_bounds__(FREQ_THREADS, M <= 4 ? 2 : 1) k_freq(FreqArgs<S> a) {
    extern __shared__ __align__(16) double fsm[];
    pdl_trigger();
    freq_item<S, R, M, G, RC>(a, a.item0 + (int)blockIdx.x, a.nitems_all ? a.nitems_all : (int)gridDim.x, fsm);
}

// FindActiveBins partials of the current J (src/UpdateLyaJandH.jl:47-97): one warp per cell, over
// the work items of k_freq.
template <typename S, int M>
__global__ void __launch_bounds__(FREQ_THREADS) k_find_active(const S *J, int nnu, const double *dnu,
                                                              const double *dV, const CloudDesc *cl, const int4 *items,
                                                              double jeps, double *partials) {
    extern __shared__ __align__(16) double fsm[];
    constexpr int NP = 32 * M;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int4 it = items[blockIdx.x];
    const long long o3 = cl[it.x].o3, oc = cl[it.x].oc;
    double acc_e[M];
#pragma unroll
    for (int m = 0; m < M; m++) acc_e[m] = 0.0;
    double acc_tot = 0.0;
    int wbeg, wend;
    warp_cell_run(it, warp, nw, 1, wbeg, wend);
    for (int c = wbeg; c < wend; c++) {
        const double v = __ldg(dV + oc + c);
#pragma unroll
        for (int m = 0; m < M; m++) {
            int k = lane * M + m;
            if (k >= nnu) continue;
            double Jv = double(__ldg(J + o3 + (long long)c * nnu + k));
            double dn = __ldg(dnu + k);
            const double e1 = Jv - 10.0 * jeps, e0 = Jv - jeps, w = dn * v;
            acc_e[m] += w * (e1 > 0.0 ? e1 : 0.0);
            acc_tot += w * (e0 > 0.0 ? e0 : 0.0);
        }
    }
    const int stride = NP + 8;
#pragma unroll
    for (int m = 0; m < M; m++) fsm[warp * stride + lane * M + m] = acc_e[m];
    acc_tot = warp_sum(acc_tot);
    if (lane == 0) fsm[warp * stride + NP] = acc_tot;
    __syncthreads();
    for (int col = threadIdx.x; col <= nnu; col += blockDim.x) {
        int src = col < nnu ? col : NP;
        double s = 0.0;
        for (int w = 0; w < nw; w++) s += fsm[w * stride + src];
        partials[(size_t)col * gridDim.x + blockIdx.x] = s;
    }
}

// Column sums of each cloud's partials (one warp per column, a fixed order), then, by one thread
// per cloud, FindActiveBins' decision and the diagnostics of Update_f_Lya_MF_L_Lya! /
// Compute_f_esc_Lya_Cylindrical. With a.cnt set, each cloud's columns are spread over CTAs of
// 8 warps, one column per warp, whose sums go through a.colsum; the last CTA of the cloud to
// finish takes the decision. Without, one CTA per cloud sums every column. The last decision
// of the launch advances the record index.
// reduce_block is block `vb` of that launch by the calling CTA (all its warps): the body of
// k_reduce, also run by the persistent batch kernel.
__device__ __forceinline__ void reduce_block(const RedArgs &a, int vb) {
    __shared__ double col[256 + kExtraCols];
    __shared__ int is_last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int ncols = a.nnu + kExtraCols;
    const bool split = a.cnt != nullptr;
    const int nchunks = split ? (ncols + nw - 1) / nw : 1;
    const int cloud = vb / nchunks, chunk = vb % nchunks;
    const CloudDesc &cd = a.cl[cloud];
    const int npb = cd.npb;
    const double *pbase = a.partials + cd.pb0;
    const int c0 = split ? chunk * nw : 0, c1 = split ? min(ncols, c0 + nw) : ncols;
    for (int cc = c0 + warp; cc < c1; cc += nw) {
        bool need = (cc < a.nnu + 1) ? (a.parts & PART_ACTIVE) : (a.parts & PART_DIAG);
        double s = 0.0;
        if (need) {
            const double *p = pbase + (size_t)cc * a.nblocks;
            // (eight loads in flight, added in order)
            for (int b0 = lane; b0 < npb; b0 += 256) {
                double v[8];
#pragma unroll
                for (int q = 0; q < 8; q++) v[q] = b0 + 32 * q < npb ? __ldcg(p + b0 + 32 * q) : 0.0;
#pragma unroll
                for (int q = 0; q < 8; q++) s += v[q];
            }
        }
        s = warp_sum(s);
        if (lane == 0) {
            col[cc] = s;
            if (split) a.colsum[(size_t)cloud * ncols + cc] = s;
        }
    }
    if (split) {
        // the last CTA of this cloud gathers the other CTAs' sums (threadfence reduction)
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) is_last = atomicAdd(a.cnt + cloud, 1) == nchunks - 1;
        __syncthreads();
        if (!is_last) return;
        __threadfence();
        for (int cc = threadIdx.x; cc < ncols; cc += blockDim.x) col[cc] = __ldcg(a.colsum + (size_t)cloud * ncols + cc);
        if (threadIdx.x == 0) a.cnt[cloud] = 0;
    }
    __syncthreads();
    // the decisions: one warp looks the bins over, its first lane writes
    if (warp != 0) return;
    int *kw = a.kwin + 2 * cloud;
    const int used_kmin = kw[0], used_kmax = kw[1];
    __syncwarp();
    if (a.parts & PART_ACTIVE) {
        double Etot = col[a.nnu];
        int kmin = a.nnu - 1, kmax = 0;
        for (int k = lane; k < a.nnu; k += 32) {
            if (col[k] > kEpsActive * Etot) {
                kmin = k < kmin ? k : kmin;
                kmax = k > kmax ? k : kmax;
            }
        }
        kmin = __reduce_min_sync(0xffffffffu, kmin);
        kmax = __reduce_max_sync(0xffffffffu, kmax);
        kmax = kmax > a.kcore_max ? kmax : a.kcore_max;
        kmin = kmin < a.kcore_min ? kmin : a.kcore_min;
        if (lane == 0) {
            kw[0] = kmin;
            kw[1] = kmax;
            if (a.kwin_copy) {
                a.kwin_copy[2 * cloud] = kmin;
                a.kwin_copy[2 * cloud + 1] = kmax;
            }
        }
    }
    if (lane == 0 && (a.parts & PART_DIAG)) {
        double MF = col[a.nnu + 1], net = col[a.nnu + 2], outw = col[a.nnu + 3];
        double L = col[a.nnu + 4];
        if (L > 0.0) {
            double kk = 1.0 / (L / kC);
            MF *= kk; net *= kk; outw *= kk;
        } else {
            MF = 0.0; net = 0.0; outw = 0.0;
        }
        double Ltot = (cd.bc_z_bot == 0) ? 2.0 * L : L;
        double Lsim = (cd.bc_z_bot == 0) ? 0.5 * Ltot : Ltot;
        double fesc = (Ltot > 0.0 && Lsim > 0.0) ? col[a.nnu + 5] / Lsim : 0.0;
        double rec[7] = {MF, net, outw, Ltot, fesc, (double)used_kmin, (double)used_kmax};
        if (a.last)
            for (int q = 0; q < 7; q++) a.last[(size_t)cloud * 7 + q] = rec[q];
        if (a.diag && a.step_counter) {
            int idx = *a.step_counter;
            if (idx < a.hist_capacity)
                for (int q = 0; q < 7; q++) a.diag[((size_t)idx * a.nclouds + cloud) * 7 + q] = rec[q];
            __threadfence();
            int done = atomicAdd(a.done, 1);
            if (done == a.nclouds - 1) {
                *a.step_counter = idx + 1;
                *a.done = 0;
            }
        }
    }
}

__global__ void __launch_bounds__(1024) k_reduce(RedArgs a) {
    pdl_trigger();
    pdl_wait();
    reduce_block(a, blockIdx.x);
}

// ---- the persistent step: one cooperative launch runs the three phases -----------------------
//
// A grid barrier with a bounded wait: the CTAs of the launch arrive on a counter; the last to
// arrive resets it and advances the generation the others wait on. A wait that outlasts `polls`
// polls sets ERRB_TIMEOUT and the CTA leaves the launch (the others then time out at this or
// the next barrier), so a launch never hangs. Fences order each CTA's writes of one phase before
// the other CTAs' reads of the next.
__device__ __forceinline__ bool grid_barrier(unsigned *bar, unsigned nblocks, long long polls, int *err) {
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        volatile unsigned *gen = bar + 1;
        const unsigned g = *gen;
        __threadfence();
        int good = 1;
        if (atomicAdd(bar, 1u) + 1u == nblocks) {
            bar[0] = 0u;
            __threadfence();
            atomicAdd(bar + 1, 1u);
        } else {
            long long it = 0;
            while (*gen == g) {
                if (++it > polls) {
                    good = 0;
                    atomicOr(err, ERRB_TIMEOUT);
                    break;
                }
                __nanosleep(64);
            }
        }
        __threadfence();
        ok = good;
    }
    __syncthreads();
    return ok != 0;
}

// One fused static step of every cloud of a batch in one launch: the packed advection tiles, a grid
// barrier, the frequency-kernel items, a grid barrier, the reduction blocks, each as its own kernel's
// CTAs of 8 warps run them; each CTA walks the work lists with a grid stride. Within a launch every buffer one phase reads was written by an
// earlier launch or after a barrier, so no read meets a stale copy: the advection reads the set
// the previous launch's frequency phase wrote.
template <typename S>
struct PersistArgs {
    AdvArgs<S> adv;
    FreqArgs<S> freq;
    RedArgs red;
    int ntiles, nitems, nred;
    unsigned *bar;          // [0] arrivals, [1] generation; [0] zero before the launch
    long long polls;
    int *err;
};

// RA: arithmetic of the advection; RF, RC: of the frequency step and its closure (as k_freq).
template <typename S, typename RA, typename RF, typename RC, int FLUX, int M, int G>
__global__ void __launch_bounds__(PT, 2) k_step_persistent(PersistArgs<S> p) {
    extern __shared__ __align__(128) unsigned char psm[];
    for (int t = blockIdx.x; t < p.ntiles; t += gridDim.x) {
        advect_tile<S, RA, FLUX>(p.adv, t, psm);
        __syncthreads();
    }
    if (!grid_barrier(p.bar, gridDim.x, p.polls, p.err)) return;
    for (int it = blockIdx.x; it < p.nitems; it += gridDim.x) {
        freq_item<S, RF, M, G, RC>(p.freq, it, p.nitems, reinterpret_cast<double *>(psm));
        __syncthreads();
    }
    if (!grid_barrier(p.bar, gridDim.x, p.polls, p.err)) return;
    for (int vb = blockIdx.x; vb < p.nred; vb += gridDim.x) {
        reduce_block(p.red, vb);
        __syncthreads();
    }
}

// ---- launch wrappers ----------------------------------------------------------------------
template <typename S, typename R, int FLUX, int MINB>
static void adv_launch(const void *args, cudaStream_t st) {
    static bool attr = false;
    const AdvArgs<S> &a = *static_cast<const AdvArgs<S> *>(args);
    // the bulk-copy form runs when the caller encoded tensor maps for this launch's input state
    if (a.tmaps) {
        constexpr size_t sm = adv_tma_off(adv_smem_base<S, R>()) + raw_tile_bytes<S>() + 16;   // + mbarrier, abort flag
        static bool attr_t = false;
        if (!attr_t) {
            cudaFuncSetAttribute(k_advect_tma<S, R, FLUX, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
            attr_t = true;
        }
        launch_chained(a.chained, k_advect_tma<S, R, FLUX, MINB>, a.ntiles, MTHREADS, sm, st, a);
        return;
    }
    constexpr size_t sm = adv_pack_smem<S, R>();
    if (!attr) {
        cudaFuncSetAttribute(k_advect<S, R, FLUX, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
        attr = true;
    }
    launch_chained(a.chained, k_advect<S, R, FLUX, MINB>, a.ntiles, PT, sm, st, a);
}

template <typename S, typename R, int FLUX>
static void adv_occ(const void *args, cudaStream_t st, int ctas) {
    if (ctas >= 4) adv_launch<S, R, FLUX, 4>(args, st);
    else if (ctas == 2) adv_launch<S, R, FLUX, 2>(args, st);
    else adv_launch<S, R, FLUX, 3>(args, st);
}

int adv_ctas_per_sm(int prec, int want) {
    if (prec == PREC_K_FP64) return (want == 2) ? 2 : 3;   // FP64: 75 KB of shared memory, 80 registers
    // FP32 arithmetic: three CTAs of 80 registers against four of 64: mixed 158 against 161 us at 256^2 x 64,
    // 533 / 541 at 512^2 x 64, level on small fields; FP32 storage 133 against 130
    return (want >= 2 && want <= 4) ? want : prec == PREC_K_FP32 ? 4 : 3;
}

void launch_advect(int prec, int flux, const void *args, int ctas, cudaStream_t st) {
    ctas = adv_ctas_per_sm(prec, ctas);
    if (prec == PREC_K_FP64) {
        if (static_cast<const AdvArgs<double> *>(args)->ntiles <= 0) return;
        if (ctas == 3) {
            if (flux == 0) adv_launch<double, double, 0, 3>(args, st);
            else adv_launch<double, double, 1, 3>(args, st);
        } else {
            if (flux == 0) adv_launch<double, double, 0, 2>(args, st);
            else adv_launch<double, double, 1, 2>(args, st);
        }
    } else if (prec == PREC_K_MIXED) {
        if (static_cast<const AdvArgs<double> *>(args)->ntiles <= 0) return;
        if (flux == 0) adv_occ<double, float, 0>(args, st, ctas);
        else adv_occ<double, float, 1>(args, st, ctas);
    } else {
        if (static_cast<const AdvArgs<float> *>(args)->ntiles <= 0) return;
        if (flux == 0) adv_occ<float, float, 0>(args, st, ctas);
        else adv_occ<float, float, 1>(args, st, ctas);
    }
}

int bins_per_lane(int nnu) { return nnu <= 32 ? 1 : nnu <= 64 ? 2 : nnu <= 128 ? 4 : 8; }

int freq_blocks(int ncell, int dev) {
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    int want = (ncell + (FREQ_THREADS / 32) - 1) / (FREQ_THREADS / 32);
    int cap = sms * 4;
    return want < cap ? (want > 0 ? want : 1) : cap;
}

static bool al16(const void *p) { return p == nullptr || (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Every row of every cloud starts on a 16-byte boundary when the buffers do and a row (n_nu elements) is
// a multiple of 16 bytes: cloud offsets are sums of whole rows.
template <typename S>
static int rows_vec16(const FreqArgs<S> &f) {
    return (f.nnu * sizeof(S)) % 16 == 0 && al16(f.Jin) && al16(f.Hrin) && al16(f.HZin) && al16(f.Jold) && al16(f.Hv) &&
           al16(f.Jout) && al16(f.Hrout) && al16(f.HZout);
}

template <typename S, typename R, int M, int G, typename RC>
static void freq_launch(const void *args, int nitems, cudaStream_t st) {
    FreqArgs<S> fa = *static_cast<const FreqArgs<S> *>(args);
    fa.vec16 = rows_vec16(fa);
    const size_t sm = sizeof(double) * freq_smem_doubles<M, G>(FREQ_THREADS / 32, fa.solver == SOLVER_THOMAS,
                                                               freq_ns<G>(fa.Jold == fa.Jin));
    static bool attr = false;
    if (!attr) {
        const size_t smax = sizeof(double) * freq_smem_doubles<M, G>(FREQ_THREADS / 32, true, 5);
        cudaFuncSetAttribute(k_freq<S, R, M, G, RC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smax);
        attr = true;
    }
    launch_chained(fa.chained, k_freq<S, R, M, G, RC>, nitems, FREQ_THREADS, sm, st, fa);
}

// How a cell's bins lie across lanes: groups of G lanes, M bins to a lane (see freq_item).
static int freq_shape(int nnu) {
    return nnu <= 16 ? 0 : nnu <= 32 ? 1 : nnu <= 48 ? 2 : nnu <= 64 ? 3 : nnu <= 128 ? 4 : 5;
}
int freq_cells_per_warp(int nnu) { return nnu <= 48 ? 2 : 1; }

void launch_freq(int prec, const void *args, int nnu, int nitems, cudaStream_t st) {
    if (nitems <= 0) return;
#define LYD_FQ(S_, R_, RC_)                                                  \
    switch (freq_shape(nnu)) {                                               \
    case 0: freq_launch<S_, R_, 1, 16, RC_>(args, nitems, st); break;        \
    case 1: freq_launch<S_, R_, 2, 16, RC_>(args, nitems, st); break;        \
    case 2: freq_launch<S_, R_, 3, 16, RC_>(args, nitems, st); break;        \
    case 3: freq_launch<S_, R_, 2, 32, RC_>(args, nitems, st); break;        \
    case 4: freq_launch<S_, R_, 4, 32, RC_>(args, nitems, st); break;        \
    default: freq_launch<S_, R_, 8, 32, RC_>(args, nitems, st); break;       \
    }
    // the mixed variant keeps the frequency step in FP64 (its state, factors and solve need
    // it) except the closure that sets the Doppler velocity (see k_freq)
    if (prec == PREC_K_FP32) {
        LYD_FQ(float, float, float)
    } else if (prec == PREC_K_MIXED) {
        LYD_FQ(double, double, float)
    } else {
        LYD_FQ(double, double, double)
    }
#undef LYD_FQ
}

template <typename S, int M>
static void active_launch(const S *J, int nnu, const double *dnu, const double *dV, const CloudDesc *cl,
                          const int4 *items, int nitems, double jeps, double *partials, cudaStream_t st) {
    size_t sm = sizeof(double) * (FREQ_THREADS / 32) * (32 * M + 8);
    k_find_active<S, M><<<nitems, FREQ_THREADS, sm, st>>>(J, nnu, dnu, dV, cl, items, jeps, partials);
}

void launch_find_active(int sprec, const void *J, int nnu, const double *dnu, const double *dV, const CloudDesc *cl,
                        const int4 *items, int nitems, double jeps, double *partials, cudaStream_t st) {
    if (nitems <= 0) return;
    int M = bins_per_lane(nnu);
#define LYD_ACT(T, MM) \
    active_launch<T, MM>(static_cast<const T *>(J), nnu, dnu, dV, cl, items, nitems, jeps, partials, st)
    if (sprec == 0) {
        switch (M) { case 1: LYD_ACT(double, 1); break; case 2: LYD_ACT(double, 2); break;
                     case 4: LYD_ACT(double, 4); break; default: LYD_ACT(double, 8); break; }
    } else {
        switch (M) { case 1: LYD_ACT(float, 1); break; case 2: LYD_ACT(float, 2); break;
                     case 4: LYD_ACT(float, 4); break; default: LYD_ACT(float, 8); break; }
    }
#undef LYD_ACT
}

template <typename S, typename RA, typename RF, typename RC, int FLUX, int M, int G>
static cudaError_t persist_launch(const void *adv, const void *freq, const RedArgs &red, int nitems,
                                  unsigned *bar, long long polls, int *err, cudaStream_t st) {
    PersistArgs<S> p;
    p.adv = *static_cast<const AdvArgs<S> *>(adv);
    p.freq = *static_cast<const FreqArgs<S> *>(freq);
    p.freq.vec16 = rows_vec16(p.freq);
    p.red = red;
    if (!red.colsum) p.red.cnt = nullptr;
    const int ncols = red.nnu + kExtraCols, rw = PT / 32;
    p.ntiles = p.adv.ntiles;
    p.nitems = nitems;
    p.nred = p.red.cnt ? red.nclouds * ((ncols + rw - 1) / rw) : red.nclouds;
    p.bar = bar;
    p.polls = polls;
    p.err = err;
    auto kern = k_step_persistent<S, RA, RF, RC, FLUX, M, G>;
    const size_t sa = adv_pack_smem<S, RA>();
    const size_t sf = sizeof(double) * freq_smem_doubles<M, G>(FREQ_THREADS / 32, p.freq.solver == SOLVER_THOMAS,
                                                               freq_ns<G>(p.freq.Jold == p.freq.Jin));
    const size_t sm = sa > sf ? sa : sf;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    int dev = 0, sms = 0, per = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, PT, sm);
    if (e != cudaSuccess) return e;
    if (per < 1) return cudaErrorInvalidConfiguration;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(per * sms));
    cfg.blockDim = dim3(PT);
    cfg.dynamicSmemBytes = sm;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    e = cudaMemsetAsync(bar, 0, 2 * sizeof(unsigned), st);
    if (e != cudaSuccess) return e;
    return cudaLaunchKernelEx(&cfg, kern, p);
}

cudaError_t launch_persistent(int prec, int flux, const void *adv, const void *freq, const RedArgs &red, int nnu,
                              int nitems, unsigned *bar, long long polls, int *err, cudaStream_t st) {
#define LYD_PS1(S_, RA_, RF_, RC_, M_, G_)                                                                 \
    return flux == 0 ? persist_launch<S_, RA_, RF_, RC_, 0, M_, G_>(adv, freq, red, nitems, bar, polls, err, st) \
                     : persist_launch<S_, RA_, RF_, RC_, 1, M_, G_>(adv, freq, red, nitems, bar, polls, err, st);
#define LYD_PS(S_, RA_, RF_, RC_)                                                                         \
    switch (freq_shape(nnu)) {                                                                            \
    case 0: LYD_PS1(S_, RA_, RF_, RC_, 1, 16)                                                             \
    case 1: LYD_PS1(S_, RA_, RF_, RC_, 2, 16)                                                             \
    case 2: LYD_PS1(S_, RA_, RF_, RC_, 3, 16)                                                             \
    case 3: LYD_PS1(S_, RA_, RF_, RC_, 2, 32)                                                             \
    case 4: LYD_PS1(S_, RA_, RF_, RC_, 4, 32)                                                             \
    default: LYD_PS1(S_, RA_, RF_, RC_, 8, 32)                                                            \
    }
    // the arithmetic of each phase as in launch_advect and launch_freq
    if (prec == PREC_K_FP32) {
        LYD_PS(float, float, float, float)
    } else if (prec == PREC_K_MIXED) {
        LYD_PS(double, float, double, float)
    } else {
        LYD_PS(double, double, double, double)
    }
#undef LYD_PS
#undef LYD_PS1
}

void launch_reduce(const RedArgs &a, cudaStream_t st) {
    if (a.nclouds <= 0) return;
    if (a.cnt && a.colsum) {
        const int nchunks = (a.nnu + kExtraCols + 7) / 8;
        launch_chained(a.chained, k_reduce, a.nclouds * nchunks, 256, 0, st, a);
    } else {
        RedArgs b = a;
        b.cnt = nullptr;
        launch_chained(a.chained, k_reduce, a.nclouds, 1024, 0, st, b);
    }
}

}  // namespace lyd
