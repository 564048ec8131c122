// Fused Yee time step: E update + E-CPML + soft sources + H update + H-CPML
// in ONE pass over HBM per time step (sm_103a, TMA + mbarrier pipeline).
//
// Semantics are exactly those of the in-place sequence
//   update_e -> cpml_e -> sources -> update_h -> cpml_h
// (2nd_order-Yee/CUDA/fdtd3d_201_250x250x320cell_15npml_100000tstep.cu:718-742,
//  operation grouping of 2nd_order-Yee/Numpy/fdtd3d.py:4-13), computed with
// the same round-to-nearest operations, so the result is bit-identical to
// the unfused kernels and to the FP32 oracle.
//
// Design
//  * The state lives in two buffers (ping-pong): a step reads buffer `cur`
//    and writes buffer `1-cur`.  E-psi slabs are ping-ponged too; H-psi is
//    updated in place (only its owner touches it).
//  * A CTA owns a tile of TZ=64 (z) x TY (y) cells for a chunk of x planes
//    and marches along x.  A thread owns a group of 4 z cells of one row, so
//    every shared and global access of the plain path is 16 bytes wide: about
//    50 instructions a cell and step, where a thread with two cells and
//    64-bit plane indices took 300 and kept the schedulers 58 % busy.
//  * For plane i the tile needs H(i), H(i+1), E(i), CE(i) with a one-cell
//    halo at j0-1 / k0-1 (and j0+TY / k0+TZ for H).  3-D TMA box loads
//    (cp.async.bulk.tensor) bring stage q = {E(q), CE(q), H(q+1)} into rings
//    of NS (E, CE) and NS+1 (H) shared-memory slots; one mbarrier a stage.
//  * E_new is computed on the tile plus the j0-1 row and k0-1 column
//    (halo cells are recomputed from the untouched input buffer, never read
//    from a neighbour), then H_new(i) for the tile uses E_new(i) from shared
//    memory (two buffers) and E_new(i-1) kept in registers.  One CTA barrier
//    a plane: after it E_new is visible and the plane's slots are free, and
//    the spare lane of the halo warp refills them.
//  * A chunk starting at x0 > 0 recomputes E_new(x0-1) without storing it.
//  * What bounds it: DRAM on plain grids (512^3 1.25 ms a step, 6.4 TB/s on 60
//    bytes a cell, 0.95 of the measured copy; the kernel before this one 1.8 ms),
//    on absorbing grids the instruction stream of the slab planes (a plane of
//    a z-edge tile executes twice a plain one's) and halos read twice where
//    tiles of different speed drift apart.  Measured and dropped: 2 cells a
//    thread (1024x1024x512 with CPML 7.2 against 6.1 ms), the E and the H phase
//    on warps of their own (8.4 ms: 96 registers a thread, spills), the z-slab
//    terms on two extra warps (7.1 ms: warps on different code miss the
//    instruction cache), psi prefetched into registers a plane ahead (no gain
//    over the L2 prefetch), two stages with 3 CTAs per SM (6.6 ms).
//  * Every mbarrier wait is bounded; on expiry the kernel records
//    FDTD_ERR_TIMEOUT in a device status word and the CTA leaves its loop.
#pragma once
#include <cuda.h>

#include <type_traits>

#include "common.cuh"

namespace fdtd {
namespace fused {

// Tile: TZ cells along z (4 per thread) x TY rows.
constexpr int TZ = 64;
constexpr int GZ = TZ / 4;   // groups of 4 z cells in a tile row
constexpr int HC = TZ + 8;   // H box:    k0-4 .. k0+TZ+3 (needs k0-1 .. k0+TZ)
constexpr int EC = TZ + 4;   // E/CE box: k0-4 .. k0+TZ-1 (needs k0-1 .. k0+TZ-1); E_new rows too
constexpr int MAX_LOCAL_SRC = 128;
constexpr int MAX_ORDERED = 32;     // x chunks whose order a plan holds
constexpr int MAX_BAND_SRC = 32;
constexpr uint64_t WAIT_NS = 1000000000ull;  // a wait gives up after 1 s

constexpr int al128(int b) { return (b + 127) / 128 * 128; }

// Shared-memory layout of one CTA for tile height TY and NS pipeline stages.
// Threads 0 .. OWN-1 own the tile's groups (E and H); the next HALO threads
// recompute E_new on the halo row j0-1 (GZ groups) and on the halo column
// k0-1 (one group a row, of which the last cell counts); the last thread
// issues the TMA copies.
template <int TY, int NS>
struct Layout {
    static constexpr int HR = TY + 2, ER = TY + 1, NH = NS + 1;
    static constexpr int HBOX = HR * HC, EBOX = ER * EC;  // floats per component box
    static constexpr int HBOXB = al128(HBOX * 4), EBOXB = al128(EBOX * 4);
    static constexpr int HSLOT = 3 * HBOXB, ESLOT = 6 * EBOXB;  // H(3); E(3), CE(3)
    static constexpr uint32_t TX_H = 3 * HBOX * 4, TX_E = 6 * EBOX * 4;
    static constexpr int OWN = TY * GZ, HALO = GZ + TY;
    static constexpr int THREADS = (OWN + HALO + 1 + 31) / 32 * 32;
    static constexpr int PRODUCER = THREADS - 1;
    static constexpr int OFF_E = NH * HSLOT;
    static constexpr int OFF_N = OFF_E + NS * ESLOT;  // E_new: two buffers of three boxes
    static constexpr int OFF_BAR = OFF_N + 2 * 3 * EBOXB;
    static constexpr int OFF_TAB = OFF_BAR + 128 + 16;  // z groups read up to 4 floats before a table
    static constexpr int SMEM = OFF_TAB + 16 + 128 /*align slack*/;  // plus the CPML tables
    // CTAs per SM that shared memory allows: what the register budget is sized for
    static constexpr int FIT = 232448 / (SMEM + 2048);
    static constexpr int MINB = FIT < 1 ? 1 : (FIT > 4 ? 4 : FIT);
};

struct TMaps {
    CUtensorMap h[3];   // hx, hy, hz of the input buffer, box (HC, TY+2, 1)
    CUtensorMap e[3];   // ex, ey, ez of the input buffer, box (EC, TY+1, 1)
    CUtensorMap ce[3];  // cex, cey, cez,                  box (EC, TY+1, 1)
};

struct Params {
    int64_t nx, ny, nz, sx, sy;
    int32_t ntz, nty, nxc, x_chunk;
    // tile rows at either end that hold y slab cells (item order)
    int32_t yf, yb;
    uint8_t xorder[MAX_ORDERED];  // the x chunks in item order, when there are no more than that
    float *out[6];  // ex, ey, ez, hx, hy, hz of the output buffer
    const float *psi_e_in[6];
    float *psi_e_out[6];
    float *psi_h[6];
    int32_t P[3];
    int32_t faces;
    const float *tb_e[3], *ta_e[3], *tk_e[3];
    const float *tb_h[3], *ta_h[3], *tk_h[3];
    int32_t nsrc;
    const int32_t *src_ijk;
    const int32_t *src_comp;
    const float *src_amp;
    int64_t namp;
    int64_t t;
    int32_t *status;
    int32_t vpsi;         // 1: rows of the x/y psi slabs are 16-byte multiples (float4 accesses)
    // 1: the z-slab CPML is finished by the band kernels.  The fused kernel
    // leaves them the E z-psi correction, the sources on E z-slab nodes and
    // every H cell of the band (k in [1, P+1] and [n-P-1, n-1]).  0: the fused
    // kernel applies the z terms itself, like the x and y ones.
    int32_t zfix;
    const float *in[6];   // input buffer fields (read by the band kernels)
    const float *in_ce[3];
    // sources on E z-slab nodes, applied by the E band kernel in list order;
    // nbsrc < 0: more than MAX_BAND_SRC of them, the band kernel scans the list
    int32_t nbsrc;
    int32_t bsrc[MAX_BAND_SRC];
    // Drude box (drude = 1): cells [i0, i0+ni) x [j0, j0+nj) x [k0, k0+nk); dense J, CJA, CJB;
    // J is read from dj_in and written to dj_out (ping-pong like E-psi)
    int32_t drude, dvec;  // dvec: the box's rows are 16-byte multiples on the grid's groups of 4 cells
    int64_t dbox[6];  // i0, j0, k0, ni, nj, nk
    const float *dj_in[3];
    float *dj_out[3];
    const float *dcja[3], *dcjb[3];
    // TFSF plane wave (tfsf = 1): box corners tp1, tp2 (p2 = pt2 + 1), face bits, axis;
    // incident table per half (0: E faces read th1d, 1: H faces read te1d), face, slot:
    // coefficient and 1-D index (tix >= 0: fixed; < 0: coordinate along the axis + tvo)
    int32_t tfsf, tfaces, taxis, tvo;
    int32_t tp1[3], tp2[3];
    float tcoef[2][6][2];
    int32_t tix[2][6][2];
    const float *te1d, *th1d;
    // test hook of single-grid plans (plan creation sets 0 and -1): wait_ns > 0
    // replaces the 1 s wait limit; test_withhold >= 0 makes CTA 0 skip the
    // copies of that plane of its first work item, so its wait runs out with
    // no copy in flight.
    uint64_t wait_ns;
    int32_t test_withhold;
};

// extents (elements) of a field array and of psi array q (0, 1: x slab;
// 2, 3: y slab; 4, 5: z slab), for the bounds-checked build
__host__ __device__ __forceinline__ int64_t fext_y(const Params &p) { return p.nx * p.sx; }
__host__ __device__ __forceinline__ int64_t pext_y(const Params &p, int q) {
    const int ax = q / 2;
    const int64_t P2 = 2 * (int64_t)p.P[ax];
    return ax == 0 ? P2 * p.ny * p.nz : (ax == 1 ? p.nx * P2 * p.nz : p.nx * p.ny * P2);
}


// Many independent grids advanced by one launch: work items of all grids are
// numbered consecutively; item_off[s] is the first item of grid s.
struct BatchDesc {
    int32_t nsims;
    int32_t cur;             // buffer holding the current state (same for every grid)
    int64_t t;               // step number (source amplitude index)
    const Params *params;    // [2*nsims]: grid s reading buffer b at params[2*s + b]
    const TMaps *maps;       // [2*nsims]: tensor maps of grid s, input buffer b
    const int64_t *item_off; // [nsims + 1]
    // work queue: [0] next item, [1] CTAs finished; zero between launches (the
    // last CTA to finish clears both)
    int32_t *queue;
};

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ uint64_t globaltimer_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// Bounded wait: true on completion; false after limit_ns, or early when
// another CTA has already recorded a timeout in the status word (status may
// be null: then only the deadline applies).
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, uint32_t parity, const int32_t *status,
                                                  uint64_t limit_ns = WAIT_NS) {
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = globaltimer_ns();
    for (uint32_t n = 1;; n++) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((n & 255) == 0) {
            if (globaltimer_ns() - t0 > limit_ns) return false;
            if (status && *(volatile const int32_t *)status == FDTD_ERR_TIMEOUT) return false;
        }
    }
}

__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *map, uint64_t *bar, int c0, int c1,
                                            int c2) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ void prefetch_tmap(const CUtensorMap *map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

// CPML slab index of an E node / H node along one axis, or -1.
__device__ __forceinline__ int slab_e(int idx, int P, int n, int front, int back) {
    if (P <= 0) return -1;
    if (front && idx >= 1 && idx <= P) return idx - 1;
    if (back && idx >= n - P - 1 && idx <= n - 2) return P + idx - (n - P - 1);
    return -1;
}
__device__ __forceinline__ int slab_h(int idx, int P, int n, int front, int back) {
    if (P <= 0) return -1;
    if (front && idx >= 1 && idx <= P) return idx - 1;
    if (back && idx >= n - P && idx <= n - 1) return P + idx - (n - P);
    return -1;
}

// H cells whose update reads an E z-slab node or that carry a z psi:
// k in [1, P+1] (front) or [n-P-1, n-1] (back)
__device__ __forceinline__ bool in_zband_h(int k, int P, int n, int front, int back) {
    if (P <= 0) return false;
    return (front && k >= 1 && k <= P + 1) || (back && k >= n - P - 1 && k <= n - 1);
}

// CPML table entry of one slab node (b, a, 1/kappa - 1).
struct Coef {
    float b, a, km;
};

// psi <- b psi + a d; returns km1 d + psi (the CPML correction term)
__device__ __forceinline__ float corr(float &psi, const Coef &c, float d) {
    psi = fadd(fmul(c.b, psi), fmul(c.a, d));
    return fadd(fmul(c.km, d), psi);
}

// Coefficients of slab node s from the shared-memory tables of one axis
// (base = first of the six tables, n2 = 2P entries each; eh = 0 E, 1 H).
__device__ __forceinline__ Coef tab_coef(const float *tabs, int base, int n2, int eh, int s) {
    const float *t = tabs + base + eh * 3 * n2;
    return Coef{t[s], t[n2 + s], t[2 * n2 + s]};
}

// Four consecutive z cells.
struct V4 {
    float v[4];
};
__device__ __forceinline__ V4 lds4(const float *s) {
    const float4 t = *reinterpret_cast<const float4 *>(s);
    return V4{{t.x, t.y, t.z, t.w}};
}
__device__ __forceinline__ void sts4(float *s, const V4 &a) {
    *reinterpret_cast<float4 *>(s) = make_float4(a.v[0], a.v[1], a.v[2], a.v[3]);
}
__device__ __forceinline__ bool bit(uint32_t m, int e) { return (m >> e) & 1; }

// Elements q .. q+3 of a global array of n elements: the cells of mask m, as
// one 16-byte access where vec says that the group is aligned (it then lies
// in the array whole) and, for a store, m has all four.
__device__ __forceinline__ V4 ldg4(const float *a, int64_t q, uint32_t m, bool vec, [[maybe_unused]] int64_t n) {
    V4 r{};
    if (vec) {
        if (m && FDTD_IN(q, n) && FDTD_IN(q + 3, n)) r = lds4(a + q);
    } else {
#pragma unroll
        for (int e = 0; e < 4; e++)
            if (bit(m, e) && FDTD_IN(q + e, n)) r.v[e] = a[q + e];
    }
    return r;
}
__device__ __forceinline__ void stg4(float *a, int64_t q, uint32_t m, bool vec, const V4 &r,
                                     [[maybe_unused]] int64_t n) {
    if (vec && m == 0xFu) {
        if (FDTD_IN(q, n) && FDTD_IN(q + 3, n)) sts4(a + q, r);
    } else {
#pragma unroll
        for (int e = 0; e < 4; e++)
            if (bit(m, e) && FDTD_IN(q + e, n)) a[q + e] = r.v[e];
    }
}

// The z-slab nodes of a group: m its cells (bits) on front or back nodes, s(e)
// the slab index of cell e.  A group on nodes of both sides (grids of at most
// 2P+5 cells along z) has two bases, else one (add = 0).
struct ZSlab {
    uint32_t m;
    int base, add;  // slab index of cell 0; what the back nodes add to it
    uint32_t bm;    // cells on back nodes, where the group has both
    __device__ __forceinline__ int s(int e) const { return base + e + (bit(bm, e) ? add : 0); }
};
__device__ __forceinline__ ZSlab zslab(int kk, int P, int n, int front, int back, bool e, uint32_t in) {
    const int s0 = kk - 1, s1 = kk + P - (e ? n - P - 1 : n - P);
    uint32_t fm = 0, bm = 0;
#pragma unroll
    for (int c = 0; c < 4; c++) {
        const int k = kk + c;
        fm |= (uint32_t)(P > 0 && front && k >= 1 && k <= P) << c;
        bm |= (uint32_t)(P > 0 && back && (e ? k >= n - P - 1 && k <= n - 2 : k >= n - P && k <= n - 1)) << c;
    }
    fm &= in;
    bm &= in;
    return fm ? ZSlab{fm | bm, s0, s1 - s0, bm} : ZSlab{bm, s1, 0, 0u};
}
// psi of the group's z-slab cells (row: first element of the dense z-psi row):
// one address and constant offsets but for groups with two bases
__device__ __forceinline__ V4 ldz4(const float *a, int64_t row, uint32_t m, const ZSlab &z, [[maybe_unused]] int64_t n) {
    V4 r{};
    if (z.bm == 0) {
        const float *b = a + (row + z.base);
#pragma unroll
        for (int e = 0; e < 4; e++)
            if (bit(m, e) && FDTD_IN(row + z.base + e, n)) r.v[e] = b[e];
    } else {
#pragma unroll 1
        for (int e = 0; e < 4; e++)
            if (bit(m, e) && FDTD_IN(row + z.s(e), n)) {
                const float t = a[row + z.s(e)];
#pragma unroll
                for (int u = 0; u < 4; u++) r.v[u] = u == e ? t : r.v[u];
            }
    }
    return r;
}
__device__ __forceinline__ void stz4(float *a, int64_t row, uint32_t m, const ZSlab &z, const V4 &r,
                                     [[maybe_unused]] int64_t n) {
    if (z.bm == 0) {
        float *b = a + (row + z.base);
#pragma unroll
        for (int e = 0; e < 4; e++)
            if (bit(m, e) && FDTD_IN(row + z.base + e, n)) b[e] = r.v[e];
    } else {
#pragma unroll 1
        for (int e = 0; e < 4; e++)
            if (bit(m, e) && FDTD_IN(row + z.s(e), n)) {
                float t = r.v[0];
#pragma unroll
                for (int u = 1; u < 4; u++) t = u == e ? r.v[u] : t;
                a[row + z.s(e)] = t;
            }
    }
}
__device__ __forceinline__ void prefetch_l2(const float *a) {
    asm volatile("prefetch.global.L2 [%0];" ::"l"(a));
}

// One CPML term of a group: f += S * cf * (km1 d + psi'), psi' = b psi + a d,
// d = hi - lo, on the cells of m; without a branch a cell (values of the
// other cells are computed and dropped).
template <int S>
__device__ __forceinline__ void term_cell(float &f, float cf, float &psi, const Coef &c, float d, bool in) {
    float ps = psi;
    const float t = fmul(cf, corr(ps, c, d));
    const float v = S > 0 ? fadd(f, t) : fsub(f, t);
    f = in ? v : f;
    psi = ps;
}
template <int S>
__device__ __forceinline__ void slab_term(V4 &f, const V4 &cf, V4 &psi, const Coef &c, const V4 &hi, const V4 &lo,
                                          uint32_t m) {
#pragma unroll
    for (int e = 0; e < 4; e++) term_cell<S>(f.v[e], cf.v[e], psi.v[e], c, fsub(hi.v[e], lo.v[e]), bit(m, e));
}
// the z slab's: coefficients by cell (tab: b of the family's tables, n2 entries
// each; cells off the slab read a neighbouring table's entry, at most 3 floats past)
template <int S>
__device__ __forceinline__ void z_term(V4 &f, const V4 &cf, V4 &psi, const float *tab, int n2, const ZSlab &z,
                                       const V4 &hi, const V4 &lo, uint32_t m) {
#pragma unroll
    for (int e = 0; e < 4; e++) {
        const float *t = tab + (z.bm == 0 ? z.base + e : (bit(z.m, e) ? z.s(e) : 0));
        const Coef c{t[0], t[n2], t[2 * n2]};
        term_cell<S>(f.v[e], cf.v[e], psi.v[e], c, fsub(hi.v[e], lo.v[e]), bit(m, e));
    }
}
// tile and x chunk of work item u: the tile rows that hold y slab cells first
// (their planes take up to twice as long: started last, they would be the
// launch's tail; 256^3 with y faces alone 213 -> 180 us), z tile fastest, and
// of either kind the x chunks with most slab, Drude and TFSF planes first (the
// first and the last one, where there are too many for the table).  Not so
// the z-edge tiles, which are as slow: apart from their neighbours in time,
// they would share no halo reads through L2 (1024x1024x512: 6.1 -> 7.0 ms).
__device__ __forceinline__ void item_tile(const Params &p, int u, int &tz, int &ty, int &xc) {
    const int ye = p.yf + p.yb, nm = p.nty - ye, edge = p.ntz * ye * p.nxc;
    const bool first = u < edge;
    if (!first) u -= edge;
    const int tiles = p.ntz * (first ? ye : nm), c = u / tiles, t = u % tiles, r = t / p.ntz;
    tz = t % p.ntz;
    ty = first ? (r < p.yf ? r : p.nty - ye + r) : p.yf + r;
    xc = p.nxc <= MAX_ORDERED ? p.xorder[c] : c == 0 ? 0 : (c == 1 ? p.nxc - 1 : c - 1);
}

__device__ __forceinline__ bool tin(int64_t x, int32_t lo, int32_t hi) { return x >= lo && x <= hi; }

// TFSF corrections (kuFDTD/v0.2.0/dim3/tfsf.py:79-89, e1/e2 slices :154-186).  Two face
// families can correct a component, in this order: ex, hx the y then the z face; ey, hy
// x, z; ez, hz x, y: families 0 .. 5.  E faces lie at p1-1 and p2, H faces at p1 and p2.
//
// Cells of the group (row j, cells k .. k+3) that each family corrects on the planes it
// acts on: 4 bits a family, from bit 0.
__device__ __forceinline__ uint32_t tfsf_masks(const Params &p, int eh, int64_t j, int64_t k, uint32_t inm) {
    const int32_t j1 = p.tp1[1], k1 = p.tp1[2], j2 = p.tp2[1], k2 = p.tp2[2], f = p.tfaces;
    // components that run along an axis end one cell before p2: E in the face's slot, H in the other
    const bool ja = tin(j, j1, eh ? j2 : j2 - 1), jb = tin(j, j1, eh ? j2 - 1 : j2);
    const bool yon = (j == (eh ? j1 : j1 - 1) && ((f >> 2) & 1)) || (j == j2 && ((f >> 3) & 1));
    uint32_t m = 0;
#pragma unroll
    for (int e = 0; e < 4; e++) {
        if (!((inm >> e) & 1)) continue;
        const int64_t kc = k + e;
        const bool ka = tin(kc, k1, eh ? k2 : k2 - 1), kb = tin(kc, k1, eh ? k2 - 1 : k2);
        const bool zon = (kc == (eh ? k1 : k1 - 1) && ((f >> 4) & 1)) || (kc == k2 && ((f >> 5) & 1));
        m |= ((uint32_t)(yon && ka) | (uint32_t)(zon && ja) << 4 | (uint32_t)(jb && ka) << 8 |
              (uint32_t)(zon && jb) << 12 | (uint32_t)(ja && kb) << 16 | (uint32_t)(yon && kb) << 20)
             << e;
    }
    return m;
}

// v += 0.5 (c * F1d[idx]) on the cells m of the group: one face, slot 0 or 1 of it.
// The 1-D arrays go through the read-only path (plain loads: 200^3 194 -> 214 us a step).
// Nothing writes them while this kernel is resident, as the 1-D step before it calls no
// grid_release(); and no load can move above the wait, after which zero is known.
__device__ __forceinline__ void tfsf_term(const Params &p, int zero, int eh, int face, int slot, int ax, uint32_t m,
                                          V4 &v) {
    const float *f1d = eh == 0 ? p.th1d : p.te1d;
    const float c = p.tcoef[eh][face][slot];
    const int ix = p.tix[eh][face][slot];
    const int at = (ix >= 0 ? ix : ax + p.tvo) + zero, step = ix < 0 && p.taxis == 2 ? 1 : 0;
#pragma unroll
    for (int e = 0; e < 4; e++)
        if ((m >> e) & 1) v.v[e] = fadd(v.v[e], fmul(0.5f, fmul(c, __ldg(f1d + at + e * step))));
}

// The terms of one group (m: its masks) on plane i, E (eh = 0) or H (eh = 1).  A family
// at a time, 4 cells each: one cell at a time, with the family's face and table looked up
// for each, a plane of a tile with a y face row took 3 times as long (256^3, 12-cell
// CPML, all faces of a 128^3 box: 404 us a step, 340 with this form; without a wave 247).
__device__ __forceinline__ void tfsf_group(const Params &p, int zero, int eh, uint32_t m, int i, int j, int k, V4 &vx,
                                           V4 &vy, V4 &vz) {
    const int32_t i1 = p.tp1[0], i2 = p.tp2[0];
    const bool xb = i == i2, xface = (i == (eh ? i1 : i1 - 1) && (p.tfaces & 1)) || (xb && ((p.tfaces >> 1) & 1));
    if (!tin(i, i1, eh ? i2 - 1 : i2)) m &= ~0x0000ffu;  // y, z faces of the x component
    if (!xface) m &= ~0x0f0f00u;
    if (!tin(i, i1, eh ? i2 : i2 - 1)) m &= ~0xf0f000u;  // y, z faces of the z, y component
    if (!m) return;
    const int ax = p.taxis == 0 ? i : (p.taxis == 1 ? j : k);
    const int fx = xb ? 1 : 0, fy = j == p.tp2[1] ? 3 : 2;
    const uint32_t back = k <= p.tp2[2] && p.tp2[2] < k + 4 ? 1u << (p.tp2[2] - k) : 0u;
    auto zfaces = [&](uint32_t z, int slot, V4 &v) {
        if (z & ~back) tfsf_term(p, zero, eh, 4, slot, ax, z & ~back, v);
        if (z & back) tfsf_term(p, zero, eh, 5, slot, ax, z & back, v);
    };
    if (m & 15u) tfsf_term(p, zero, eh, fy, 1, ax, m & 15u, vx);
    if ((m >> 4) & 15u) zfaces((m >> 4) & 15u, 0, vx);
    if ((m >> 8) & 15u) tfsf_term(p, zero, eh, fx, 0, ax, (m >> 8) & 15u, vy);
    if ((m >> 12) & 15u) zfaces((m >> 12) & 15u, 1, vy);
    if ((m >> 16) & 15u) tfsf_term(p, zero, eh, fx, 1, ax, (m >> 16) & 15u, vz);
    if (m >> 20) tfsf_term(p, zero, eh, fy, 0, ax, m >> 20, vz);
}

// EXT: bit 0: the Drude box is compiled in, bit 1: the TFSF faces, bit 2: the
// z-slab terms (else they are the band kernels').  A plan
// launches the variant its grid needs: code a step does not use still costs it
// registers and instruction-cache space.
template <int TY, int NS, bool BATCH, int EXT>
__global__ void __launch_bounds__(Layout<TY, NS>::THREADS, Layout<TY, NS>::MINB)
k_yee_fused(const __grid_constant__ TMaps mk, const __grid_constant__ Params pk, const __grid_constant__ BatchDesc bd) {
    using L = Layout<TY, NS>;
    constexpr bool DRUDE = EXT & 1, TFSF = EXT & 2, ZIN = EXT & 4;
    static_assert(NS * 8 <= 128, "the mbarriers live in 128 bytes");
    extern __shared__ unsigned char smem_raw[];
    // 128-byte aligned base, computed from the shared-window offset so the
    // pointer stays in the shared address space (shared loads, not generic ones)
    unsigned char *smem =
        smem_raw + ((128u - (static_cast<uint32_t>(__cvta_generic_to_shared(smem_raw)) & 127u)) & 127u);
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + L::OFF_BAR);
    // CPML tables: tab[(axis*2 + eh)*3 + {b,a,km}] has 2P[axis] entries
    float *tabs = reinterpret_cast<float *>(smem + L::OFF_TAB);
    // batched launches: parameters of the grid the current item belongs to
    __shared__ __align__(16) Params s_p;
    __shared__ int s_nls, s_smin, s_smax;
    // sources of the current work item, list order: (i << 16 | j), (k << 2 | comp), list index
    __shared__ uint32_t s_ls_ij[MAX_LOCAL_SRC];
    __shared__ int s_ls_kc[MAX_LOCAL_SRC], s_ls_s[MAX_LOCAL_SRC];

    // the next step's CTAs may set up while this launch drains (not the band kernels,
    // which wait for its end)
    if (BATCH || !pk.zfix) grid_release();

    const int tid = threadIdx.x, lane = tid & 31;
    const bool own_t = tid < L::OWN, e_t = tid < L::OWN + L::HALO, producer = tid == L::PRODUCER;
    // box row (row j0-1+er) and box column (first of the group) of this thread
    int er = 0, col = 0;
    if (own_t) {
        er = 1 + tid / GZ;
        col = 4 + 4 * (tid % GZ);
    } else if (tid < L::OWN + GZ) {
        col = 4 + 4 * (tid - L::OWN);
    } else if (e_t) {
        er = 1 + tid - L::OWN - GZ;
    }
    const float *const h_t = reinterpret_cast<const float *>(smem) + er * HC + col;
    const float *const e_t0 = reinterpret_cast<const float *>(smem + L::OFF_E) + er * EC + col;
    float *const n_t = reinterpret_cast<float *>(smem + L::OFF_N) + er * EC + col;
    constexpr int HB = L::HBOXB / 4, EB = L::EBOXB / 4;  // component strides (floats)
    const Params &p = BATCH ? s_p : pk;

    // stage the CPML coefficient tables of the current grid: the loads of all
    // 18 tables are in flight together (in turn they cost 18 memory latencies)
    auto stage_tables = [&]() {
        for (int x0 = 0; x0 < 2 * max(p.P[0], max(p.P[1], p.P[2])); x0 += L::THREADS) {
            const int x = x0 + tid;
            float v[18];
#pragma unroll
            for (int a = 0; a < 3; a++) {
                const bool in = x < 2 * p.P[a];
                const float *src[6] = {p.tb_e[a], p.ta_e[a], p.tk_e[a], p.tb_h[a], p.ta_h[a], p.tk_h[a]};
#pragma unroll
                for (int q = 0; q < 6; q++) v[6 * a + q] = in ? src[q][x] : 0.f;
            }
            int off = 0;
#pragma unroll
            for (int a = 0; a < 3; a++) {
                const int n2 = 2 * p.P[a];
#pragma unroll
                for (int q = 0; q < 6; q++)
                    if (x < n2) tabs[off + q * n2 + x] = v[6 * a + q];
                off += 6 * n2;
            }
        }
    };

    if (tid == 0) {
        for (int s = 0; s < NS; s++) mbar_init(&bars[s], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    [[maybe_unused]] int zero = 0;  // of a value that the compiler knows only after the wait (tfsf_term)
    if (!BATCH) {
        if (producer)
            for (int c = 0; c < 3; c++) {
                prefetch_tmap(&mk.h[c]);
                prefetch_tmap(&mk.e[c]);
                prefetch_tmap(&mk.ce[c]);
            }
        grid_wait();
        if (TFSF) asm volatile("" : "+r"(zero) : : "memory");
        stage_tables();
    } else {
        grid_wait();
    }

    // ring positions: stage slot and H slot of the current plane, parity of the stage
    int es = 0, hs = 0;
    uint32_t par = 0;
    int q_abort = 0, q_issued = -1;
    bool aborted = false;
    const uint64_t wlim = (!BATCH && pk.wait_ns) ? pk.wait_ns : WAIT_NS;
    bool first_item = true;
    const int64_t nitems = BATCH ? bd.item_off[bd.nsims] : (int64_t)pk.ntz * pk.nty * pk.nxc;
    int cur_sim = -1;

    // Batched launches take items from a queue (grids ordered with the longest
    // items first, so the short ones fill the tail); a single grid has one CTA
    // an item (the hardware hands them out as CTAs end), or walks them in a
    // fixed stride when the caller limits the CTAs per SM.
    __shared__ int s_item;
    int64_t gitem = blockIdx.x;
    if (BATCH) {
        if (tid == 0) s_item = atomicAdd(&bd.queue[0], 1);
        __syncthreads();
        gitem = s_item;
    }
    while (gitem < nitems && !aborted) {
        int64_t item = gitem;
        const TMaps *mp = &mk;
        if (BATCH) {
            // grid of this item: largest s with item_off[s] <= gitem
            int lo = 0, hi = bd.nsims - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (bd.item_off[mid] <= gitem) lo = mid;
                else hi = mid - 1;
            }
            item = gitem - bd.item_off[lo];
            mp = &bd.maps[2 * lo + bd.cur];
            if (lo != cur_sim) {
                __syncthreads();  // every thread is done with the previous grid's parameters
                for (int w = tid; w < (int)(sizeof(Params) / 4); w += L::THREADS)
                    reinterpret_cast<int32_t *>(&s_p)[w] =
                        reinterpret_cast<const int32_t *>(&bd.params[2 * lo + bd.cur])[w];
                __syncthreads();
                if (tid == 0) s_p.t = bd.t;
                if (producer)
                    for (int c = 0; c < 3; c++) {
                        prefetch_tmap(&mp->h[c]);
                        prefetch_tmap(&mp->e[c]);
                        prefetch_tmap(&mp->ce[c]);
                    }
                stage_tables();
                cur_sim = lo;
            }
        }
        const TMaps &maps = *mp;
        const int nx = (int)p.nx, ny = (int)p.ny, nz = (int)p.nz;
        const int P0 = p.P[0], P1 = p.P[1], P2 = p.P[2], faces = p.faces;
        int tzi, tyi, xci;
        item_tile(p, (int)item, tzi, tyi, xci);
        const int k0 = tzi * TZ, j0 = tyi * TY;
        const int x0 = xci * p.x_chunk, x1 = min(x0 + p.x_chunk, nx);
        const int i_start = x0 > 0 ? x0 - 1 : 0;
        const int nit = x1 - i_start;  // planes i_start .. x1-1; H(x1) feeds E(x1-1)

        __syncthreads();  // previous item finished by every thread
        // stage q into E slot se and H slot sh: E(q), CE(q), H(q+1) (and H(0) with
        // stage 0).  Past the last plane the copies read zeros: H(nx) only feeds
        // E components that are never updated at i = nx-1.
        auto issue = [&](int q, int se, int sh) {
            if (!BATCH && first_item && blockIdx.x == 0 && q == pk.test_withhold) return;  // test hook
            q_issued = q;
            uint64_t *bar = &bars[se];
            mbar_arrive_expect_tx(bar, L::TX_E + (q == 0 ? 2 : 1) * L::TX_H);
            const int xc = i_start + q;
            unsigned char *hd = smem + sh * L::HSLOT, *ed = smem + L::OFF_E + se * L::ESLOT;
            if (q == 0) {
                unsigned char *h0 = smem + (sh == 0 ? L::NH - 1 : sh - 1) * L::HSLOT;
                for (int c = 0; c < 3; c++) tma_load_3d(h0 + c * L::HBOXB, &maps.h[c], bar, k0 - 4, j0 - 1, xc);
            }
            for (int c = 0; c < 3; c++) tma_load_3d(hd + c * L::HBOXB, &maps.h[c], bar, k0 - 4, j0 - 1, xc + 1);
            for (int c = 0; c < 3; c++) tma_load_3d(ed + c * L::EBOXB, &maps.e[c], bar, k0 - 4, j0 - 1, xc);
            for (int c = 0; c < 3; c++)
                tma_load_3d(ed + (3 + c) * L::EBOXB, &maps.ce[c], bar, k0 - 4, j0 - 1, xc);
        };
        if (producer) {
            q_issued = -1;
            for (int q = 0; q < NS && q < nit; q++) {
                int se = es + q, sh = hs + q + 1;
                if (se >= NS) se -= NS;
                if (sh >= L::NH) sh -= L::NH;
                issue(q, se, sh);
            }
        }

        // sources inside the extended region of this work item, in list order,
        // found by one warp (32 a round: one memory latency for each round)
        if (tid < 32) {
            int n = 0, smin = 0x7fffffff, smax = -1;
            if (p.t >= 0 && p.t < p.namp) {
                for (int s0 = 0; s0 < p.nsrc; s0 += 32) {
                    const int s = s0 + lane;
                    bool in = false;
                    int si = 0, sj = 0, sk = 0;
                    if (s < p.nsrc) {
                        si = p.src_ijk[3 * s];
                        sj = p.src_ijk[3 * s + 1];
                        sk = p.src_ijk[3 * s + 2];
                        in = si >= i_start && si < x1 && sj >= j0 - 1 && sj < j0 + TY && sk >= k0 - 1 && sk < k0 + TZ &&
                             !(p.zfix && slab_e(sk, P2, nz, (faces >> 4) & 1, (faces >> 5) & 1) >= 0);
                    }
                    const uint32_t m = __ballot_sync(0xffffffffu, in);
                    const int at = n + __popc(m & ((1u << lane) - 1));
                    if (in && at < MAX_LOCAL_SRC) {
                        // packing: si, sj < 65536 (grid extents) and sk < 2^28 (checked at
                        // plan creation), so neither field overflows
                        s_ls_ij[at] = ((uint32_t)si << 16) | (uint32_t)sj;
                        s_ls_kc[at] = (sk << 2) | p.src_comp[s];
                        s_ls_s[at] = s;
                    }
                    if (in) {
                        smin = min(smin, si);
                        smax = max(smax, si);
                    }
                    n += __popc(m);
                }
                smin = __reduce_min_sync(0xffffffffu, smin);
                smax = __reduce_max_sync(0xffffffffu, smax);
            }
            if (lane == 0) {
                s_nls = n > MAX_LOCAL_SRC ? -1 : n;  // -1: more than the list holds, the planes scan all sources
                s_smin = smin;
                s_smax = smax;
            }
        }
        __syncthreads();  // source list and tables ready
        const int nls = s_nls, smin = s_smin, smax = s_smax;

        // ---- per-item, per-thread description of the group (row jj, cells kk .. kk+3) ----
        const int jj = j0 - 1 + er, kk = k0 - 4 + col;
        const bool row_in = e_t && jj >= 0 && jj < ny;
        const bool j_lt = jj < ny - 1, j_gt = jj > 0;
        uint32_t inm = 0, ltm = 0, gtm = 0, hbm = 0;  // cells in the grid, with k < nz-1, with k > 0, in the H band
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int k = kk + e;
            inm |= (uint32_t)(row_in && k >= 0 && k < nz) << e;
            ltm |= (uint32_t)(k < nz - 1) << e;
            gtm |= (uint32_t)(k > 0) << e;
            hbm |= (uint32_t)(p.zfix && in_zband_h(k, P2, nz, (faces >> 4) & 1, (faces >> 5) & 1)) << e;
        }
        const bool emask = !(j_lt && ltm == 0xFu), hmask = !(j_gt && gtm == 0xFu);
        const int sye = row_in ? slab_e(jj, P1, ny, (faces >> 2) & 1, (faces >> 3) & 1) : -1;
        const int syh = own_t && row_in ? slab_h(jj, P1, ny, (faces >> 2) & 1, (faces >> 3) & 1) : -1;
        const bool zin = ZIN && P2 > 0 && !p.zfix;
        const ZSlab ze = zslab(kk, zin ? P2 : 0, nz, (faces >> 4) & 1, (faces >> 5) & 1, true, inm);
        const ZSlab zh = zslab(kk, zin ? P2 : 0, nz, (faces >> 4) & 1, (faces >> 5) & 1, false, own_t ? inm : 0u);
        const bool vpsi = p.vpsi != 0;
        // the item's E region (planes i_start..x1-1, rows j0-1.., columns k0-1..) meets the Drude box
        const bool dtile = DRUDE && p.drude && i_start < p.dbox[0] + p.dbox[3] && x1 > p.dbox[0] &&
                           j0 - 1 < p.dbox[1] + p.dbox[4] && j0 + TY > p.dbox[1] &&
                           k0 - 1 < p.dbox[2] + p.dbox[5] && k0 + TZ > p.dbox[2];
        uint32_t dmask = 0;  // cells of the group in the box's columns, when its row is in the box
        if (DRUDE && dtile && jj >= p.dbox[1] && jj < p.dbox[1] + p.dbox[4])
#pragma unroll
            for (int e = 0; e < 4; e++)
                dmask |= (uint32_t)(bit(inm, e) && kk + e >= p.dbox[2] && kk + e < p.dbox[2] + p.dbox[5]) << e;
        // TFSF faces in this item (E faces at p1-1 and p2, H faces at p1 and p2): the tile's
        // rows and columns meet the box's y/z extent [p1-1, p2], and then either hold a y or
        // z face row/column (all planes of the box's x extent) or, per plane, an x face plane
        const bool t_rows = TFSF && p.tfsf && j0 - 1 <= p.tp2[1] && j0 + TY - 1 >= p.tp1[1] - 1 &&
                            k0 - 1 <= p.tp2[2] && k0 + TZ - 1 >= p.tp1[2] - 1;
        auto holds = [](int lo, int hi, int v) { return v >= lo && v <= hi; };
        const bool t_yz = t_rows && i_start <= p.tp2[0] && x1 - 1 >= p.tp1[0] - 1 &&
                          (holds(j0 - 1, j0 + TY - 1, p.tp1[1] - 1) || holds(j0 - 1, j0 + TY - 1, p.tp1[1]) ||
                           holds(j0 - 1, j0 + TY - 1, p.tp2[1]) || holds(k0 - 1, k0 + TZ - 1, p.tp1[2] - 1) ||
                           holds(k0 - 1, k0 + TZ - 1, p.tp1[2]) || holds(k0 - 1, k0 + TZ - 1, p.tp2[2]));
        // plane-uniform: an x face plane; any TFSF correction on this plane
        auto tfsf_x = [&](int i) { return i == p.tp1[0] - 1 || i == p.tp1[0] || i == p.tp2[0]; };
        auto tfsf_plane = [&](int i) {
            return TFSF && t_rows && (tfsf_x(i) || (t_yz && i >= p.tp1[0] - 1 && i <= p.tp2[0]));
        };
        uint32_t te = 0, th = 0;  // TFSF cells of the group, zero outside the box's faces
        if (TFSF && t_rows) {
            te = tfsf_masks(p, 0, jj, kk, inm);
            if (own_t) th = tfsf_masks(p, 1, jj, kk, inm);
        }

        V4 hyc{}, hzc{};                // own hy, hz of the current plane
        V4 prev_ey{}, prev_ez{};        // E_new of the plane before
        int nb = 0;                     // E_new buffer
        // planes that need more than the curl updates: all of them in tiles of a y or z
        // slab, else the x-slab, Drude, TFSF and source planes
        const bool tile_gen = __syncthreads_or(sye >= 0 || syh >= 0 || (ZIN && (ze.m || zh.m)));
        // One plane: E phase, barrier, H phase.  Copies of the code (gen: with the Drude, TFSF
        // and source terms; slab: with the CPML terms too): most planes run the shortest one,
        // which fits the instruction cache.  Returns false when a wait ran out.
        auto plane = [&](auto gen_c, auto slab_c, int q, bool late) -> bool {
            constexpr bool gen = decltype(gen_c)::value, slab = decltype(slab_c)::value;
            const int i = i_start + q;
            const bool i_lt = i < nx - 1, i_gt = i > 0, own = own_t && i >= x0;
            // plane-uniform: x slab nodes
            const int sxe = slab ? slab_e(i, P0, nx, faces & 1, (faces >> 1) & 1) : -1,
                      sxh = slab ? slab_h(i, P0, nx, faces & 1, (faces >> 1) & 1) : -1;
            // psi of this plane's slab cells: E psi now, H psi before the barrier below
            // (px, py, pz: the two arrays of the x, y and z slab)
            V4 px0{}, px1{}, py0{}, py1{}, pz0{}, pz1{};
            const int64_t qx = ((int64_t)(sxe >= 0 ? sxe : 0) * ny + jj) * nz + kk;
            const int64_t qy = ((int64_t)i * 2 * P1 + (sye >= 0 ? sye : 0)) * nz + kk;
            const int64_t qz = ((int64_t)i * ny + jj) * 2 * P2;
            if (sxe >= 0) {
                px0 = ldg4(p.psi_e_in[0], qx, inm, vpsi, pext_y(p, 0));
                px1 = ldg4(p.psi_e_in[1], qx, inm, vpsi, pext_y(p, 1));
            }
            if (slab && sye >= 0) {
                py0 = ldg4(p.psi_e_in[2], qy, inm, vpsi, pext_y(p, 2));
                py1 = ldg4(p.psi_e_in[3], qy, inm, vpsi, pext_y(p, 3));
            }
            if (ZIN && slab && ze.m) {
                pz0 = ldz4(p.psi_e_in[4], qz, ze.m, ze, pext_y(p, 4));
                pz1 = ldz4(p.psi_e_in[5], qz, ze.m, ze, pext_y(p, 5));
            }
            if (slab && q + 1 < nit) {
                // the next plane's psi into L2: one plane is long enough for DRAM, and the
                // loads above and before the barrier then wait for L2 only
                const int64_t dx = (int64_t)ny * nz, dy = (int64_t)2 * P1 * nz, dz = (int64_t)ny * 2 * P2;
                if (inm) {
                    if (sxe >= 0 && sxe + 1 < 2 * P0) {
                        prefetch_l2(p.psi_e_in[0] + qx + dx);
                        prefetch_l2(p.psi_e_in[1] + qx + dx);
                    }
                    if (sye >= 0) {
                        prefetch_l2(p.psi_e_in[2] + qy + dy);
                        prefetch_l2(p.psi_e_in[3] + qy + dy);
                    }
                    if (ZIN && ze.m) {
                        prefetch_l2(p.psi_e_in[4] + qz + dz + ze.s(__ffs(ze.m) - 1));
                        prefetch_l2(p.psi_e_in[5] + qz + dz + ze.s(__ffs(ze.m) - 1));
                    }
                    if (own_t) {
                        if (sxh >= 0 && sxh + 1 < 2 * P0) {
                            const int64_t u = ((int64_t)(sxh + 1) * ny + jj) * nz + kk;
                            prefetch_l2(p.psi_h[0] + u);
                            prefetch_l2(p.psi_h[1] + u);
                        }
                        if (syh >= 0) {
                            const int64_t u = ((int64_t)(i + 1) * 2 * P1 + syh) * nz + kk;
                            prefetch_l2(p.psi_h[2] + u);
                            prefetch_l2(p.psi_h[3] + u);
                        }
                        if (ZIN && zh.m) {
                            prefetch_l2(p.psi_h[4] + qz + dz + zh.s(__ffs(zh.m) - 1));
                            prefetch_l2(p.psi_h[5] + qz + dz + zh.s(__ffs(zh.m) - 1));
                        }
                    }
                }
            }
            const bool dplane = gen && DRUDE && dmask && i >= p.dbox[0] && i < p.dbox[0] + p.dbox[3];
            int64_t jb = 0;
            if (gen && DRUDE && dplane) {
                jb = ((i - p.dbox[0]) * p.dbox[4] + (jj - p.dbox[1])) * p.dbox[5] - p.dbox[2] + kk;
                if (q + 1 < nit && i + 1 < p.dbox[0] + p.dbox[3]) {  // the next plane's box arrays into L2
                    const int64_t u = jb + p.dbox[4] * p.dbox[5] + __ffs(dmask) - 1;
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        prefetch_l2(p.dj_in[c] + u);
                        prefetch_l2(p.dcja[c] + u);
                        prefetch_l2(p.dcjb[c] + u);
                    }
                }
            }

            const float *H0 = h_t + hs * (L::HSLOT / 4);
            const float *H1 = h_t + (hs + 1 == L::NH ? 0 : hs + 1) * (L::HSLOT / 4);
            const float *E0 = e_t0 + es * (L::ESLOT / 4);
            float *N0 = n_t + nb * (3 * EB);
            const bool tplane = gen && TFSF && tfsf_plane(i);  // TFSF corrections on this plane
            // ---- E phase ----
            V4 hx{}, hy1{}, hz1{}, ex{}, ey{}, ez{};
            if (e_t) {
                if (q == 0) {
                    hyc = lds4(H0 + HB);
                    hzc = lds4(H0 + 2 * HB);
                }
                hx = lds4(H0);
                hy1 = lds4(H1 + HB);
                hz1 = lds4(H1 + 2 * HB);
                const V4 hxj = lds4(H0 + HC), hzj = lds4(H0 + 2 * HB + HC);
                const float hxk4 = H0[4], hyk4 = H0[HB + 4];
                const V4 ex0 = lds4(E0), ey0 = lds4(E0 + EB), ez0 = lds4(E0 + 2 * EB);
                const V4 cx = lds4(E0 + 3 * EB), cy = lds4(E0 + 4 * EB), cz = lds4(E0 + 5 * EB);
                auto hxk = [&](int e) { return e < 3 ? hx.v[e + 1] : hxk4; };
                auto hyk = [&](int e) { return e < 3 ? hyc.v[e + 1] : hyk4; };
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    ex.v[e] = fadd(ex0.v[e], fmul(cx.v[e], curl4(hzj.v[e], hzc.v[e], hyk(e), hyc.v[e])));
                    ey.v[e] = fadd(ey0.v[e], fmul(cy.v[e], curl4(hxk(e), hx.v[e], hz1.v[e], hzc.v[e])));
                    ez.v[e] = fadd(ez0.v[e], fmul(cz.v[e], curl4(hy1.v[e], hyc.v[e], hxj.v[e], hx.v[e])));
                }
                if (!i_lt || emask) {
                    // component masks (cells the reference does not update keep their value)
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        if (!(j_lt && bit(ltm, e))) ex.v[e] = ex0.v[e];
                        if (!(i_lt && bit(ltm, e))) ey.v[e] = ey0.v[e];
                        if (!(i_lt && j_lt)) ez.v[e] = ez0.v[e];
                    }
                }
                if (gen && DRUDE && dplane) {  // Drude ADE, before the CPML terms
                    [[maybe_unused]] const int64_t nd = p.dbox[3] * p.dbox[4] * p.dbox[5];
                    const bool dv = p.dvec != 0;
                    V4 dj[3], da[3], db[3];
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        dj[c] = ldg4(p.dj_in[c], jb, dmask, dv, nd);
                        da[c] = ldg4(p.dcja[c], jb, dmask, dv, nd);
                        db[c] = ldg4(p.dcjb[c], jb, dmask, dv, nd);
                    }
                    auto ade = [&](V4 &v, const V4 &cf, int c) {
                        V4 jn;
#pragma unroll
                        for (int e = 0; e < 4; e++) {
                            const float n = drude_cell(v.v[e], cf.v[e], dj[c].v[e], da[c].v[e], db[c].v[e], jn.v[e]);
                            v.v[e] = bit(dmask, e) ? n : v.v[e];
                        }
                        if (own) stg4(p.dj_out[c], jb, dmask, dv, jn, nd);
                    };
                    ade(ex, cx, 0);
                    ade(ey, cy, 1);
                    ade(ez, cz, 2);
                }
                if (slab && sxe >= 0) {  // x slab: ey -= cey (..dHz/dx..), ez += cez (..dHy/dx..)
                    const Coef c = tab_coef(tabs, 0, 2 * P0, 0, sxe);
                    const uint32_t m0 = inm & ltm, m1 = j_lt ? inm : 0u;
                    slab_term<-1>(ey, cy, px0, c, hz1, hzc, m0);
                    slab_term<+1>(ez, cz, px1, c, hy1, hyc, m1);
                    if (own) {
                        stg4(p.psi_e_out[0], qx, m0, vpsi, px0, pext_y(p, 0));
                        stg4(p.psi_e_out[1], qx, m1, vpsi, px1, pext_y(p, 1));
                    }
                }
                if (slab && sye >= 0) {  // y slab: ez -= cez (..dHx/dy..), ex += cex (..dHz/dy..)
                    const Coef c = tab_coef(tabs, 12 * P0, 2 * P1, 0, sye);
                    const uint32_t m0 = i_lt ? inm : 0u, m1 = inm & ltm;
                    slab_term<-1>(ez, cz, py0, c, hxj, hx, m0);
                    slab_term<+1>(ex, cx, py1, c, hzj, hzc, m1);
                    if (own) {
                        stg4(p.psi_e_out[2], qy, m0, vpsi, py0, pext_y(p, 2));
                        stg4(p.psi_e_out[3], qy, m1, vpsi, py1, pext_y(p, 3));
                    }
                }
                if (ZIN && slab && ze.m) {  // z slab: ex -= cex (..dHy/dz..), ey += cey (..dHx/dz..)
                    const uint32_t m0 = j_lt ? ze.m : 0u, m1 = i_lt ? ze.m : 0u;
                    const V4 hxs{{hx.v[1], hx.v[2], hx.v[3], hxk4}}, hys{{hyc.v[1], hyc.v[2], hyc.v[3], hyk4}};
                    z_term<-1>(ex, cx, pz0, tabs + 12 * (P0 + P1), 2 * P2, ze, hys, hyc, m0);
                    z_term<+1>(ey, cy, pz1, tabs + 12 * (P0 + P1), 2 * P2, ze, hxs, hx, m1);
                    if (own) {
                        stz4(p.psi_e_out[4], qz, m0, ze, pz0, pext_y(p, 4));
                        stz4(p.psi_e_out[5], qz, m1, ze, pz1, pext_y(p, 5));
                    }
                }
                // TFSF: E += 0.5 (c * H1d), after the CPML terms, before the sources
                if (gen && TFSF && tplane && te) tfsf_group(p, zero, 0, te, i, jj, kk, ex, ey, ez);
                if (gen && i >= smin && i <= smax) {  // soft sources, list order
                    const uint32_t ij_here = ((uint32_t)i << 16) | (uint32_t)jj;
                    const int ns = nls >= 0 ? nls : p.nsrc;
                    for (int s = 0; s < ns; s++) {
                        int kc, ls = s;
                        if (nls >= 0) {
                            if (s_ls_ij[s] != ij_here) continue;
                            kc = s_ls_kc[s];
                            ls = s_ls_s[s];
                        } else {
                            if (p.src_ijk[3 * s] != i || p.src_ijk[3 * s + 1] != jj) continue;
                            kc = (p.src_ijk[3 * s + 2] << 2) | p.src_comp[s];
                            if (p.zfix && slab_e(kc >> 2, P2, nz, (faces >> 4) & 1, (faces >> 5) & 1) >= 0) continue;
                        }
                        const int d = (kc >> 2) - kk;
                        if (d < 0 || d > 3) continue;
                        const float v = p.src_amp[(int64_t)ls * p.namp + p.t];
#pragma unroll
                        for (int e = 0; e < 4; e++) {
                            if (e != d) continue;
                            if ((kc & 3) == 0) ex.v[e] = fadd(ex.v[e], v);
                            else if ((kc & 3) == 1) ey.v[e] = fadd(ey.v[e], v);
                            else ez.v[e] = fadd(ez.v[e], v);
                        }
                    }
                }
                sts4(N0, ex);
                sts4(N0 + EB, ey);
                sts4(N0 + 2 * EB, ez);
            }
            // H psi of the slab cells (in place: only this thread touches them)
            const int64_t ux = ((int64_t)(sxh >= 0 ? sxh : 0) * ny + jj) * nz + kk;
            const int64_t uy = ((int64_t)i * 2 * P1 + (syh >= 0 ? syh : 0)) * nz + kk;
            if (own) {
                if (slab && sxh >= 0) {
                    px0 = ldg4(p.psi_h[0], ux, inm, vpsi, pext_y(p, 0));
                    px1 = ldg4(p.psi_h[1], ux, inm, vpsi, pext_y(p, 1));
                }
                if (slab && syh >= 0) {
                    py0 = ldg4(p.psi_h[2], uy, inm, vpsi, pext_y(p, 2));
                    py1 = ldg4(p.psi_h[3], uy, inm, vpsi, pext_y(p, 3));
                }
                if (ZIN && slab && zh.m) {
                    pz0 = ldz4(p.psi_h[4], qz, zh.m, zh, pext_y(p, 4));
                    pz1 = ldz4(p.psi_h[5], qz, zh.m, zh, pext_y(p, 5));
                }
            }
            // E_new of plane i visible; E(q), CE(q) and H(q) read by every thread; the
            // barrier also agrees on whether any thread's wait ran out
            if (__syncthreads_or(late)) {
                return false;
            }
            if (producer && q + NS < nit) issue(q + NS, es, hs);

            // ---- H phase ----
            if (own) {
                const V4 ez_j = lds4(N0 + 2 * EB - EC), ex_j = lds4(N0 - EC);
                const float eyk0 = N0[EB - 1], exk0 = N0[-1];
                auto ey_k = [&](int e) { return e ? ey.v[e - 1] : eyk0; };
                auto ex_k = [&](int e) { return e ? ex.v[e - 1] : exk0; };
                V4 ox, oy, oz;  // H_new
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    ox.v[e] = fsub(hx.v[e], fmul(0.5f, curl4(ez.v[e], ez_j.v[e], ey.v[e], ey_k(e))));
                    oy.v[e] = fsub(hyc.v[e], fmul(0.5f, curl4(ex.v[e], ex_k(e), ez.v[e], prev_ez.v[e])));
                    oz.v[e] = fsub(hzc.v[e], fmul(0.5f, curl4(ey.v[e], prev_ey.v[e], ex.v[e], ex_j.v[e])));
                }
                if (!i_gt || hmask) {
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        if (!(j_gt && bit(gtm, e))) ox.v[e] = hx.v[e];
                        if (!(i_gt && bit(gtm, e))) oy.v[e] = hyc.v[e];
                        if (!(i_gt && j_gt)) oz.v[e] = hzc.v[e];
                    }
                }
                const V4 half{{0.5f, 0.5f, 0.5f, 0.5f}};
                if (slab && sxh >= 0) {  // x slab: hy += (..dEz/dx..), hz -= (..dEy/dx..)
                    const Coef c = tab_coef(tabs, 0, 2 * P0, 1, sxh);
                    const uint32_t m0 = inm & gtm & ~hbm, m1 = j_gt ? inm & ~hbm : 0u;
                    slab_term<+1>(oy, half, px0, c, ez, prev_ez, m0);
                    slab_term<-1>(oz, half, px1, c, ey, prev_ey, m1);
                    stg4(p.psi_h[0], ux, m0, vpsi, px0, pext_y(p, 0));
                    stg4(p.psi_h[1], ux, m1, vpsi, px1, pext_y(p, 1));
                }
                if (slab && syh >= 0) {  // y slab: hz += (..dEx/dy..), hx -= (..dEz/dy..)
                    const Coef c = tab_coef(tabs, 12 * P0, 2 * P1, 1, syh);
                    const uint32_t m0 = i_gt ? inm & ~hbm : 0u, m1 = inm & gtm & ~hbm;
                    slab_term<+1>(oz, half, py0, c, ex, ex_j, m0);
                    slab_term<-1>(ox, half, py1, c, ez, ez_j, m1);
                    stg4(p.psi_h[2], uy, m0, vpsi, py0, pext_y(p, 2));
                    stg4(p.psi_h[3], uy, m1, vpsi, py1, pext_y(p, 3));
                }
                if (ZIN && slab && zh.m) {  // z slab: hx += (..dEy/dz..), hy -= (..dEx/dz..)
                    const uint32_t m0 = j_gt ? zh.m : 0u, m1 = i_gt ? zh.m : 0u;
                    const V4 eys{{eyk0, ey.v[0], ey.v[1], ey.v[2]}}, exs{{exk0, ex.v[0], ex.v[1], ex.v[2]}};
                    z_term<+1>(ox, half, pz0, tabs + 12 * (P0 + P1) + 6 * P2, 2 * P2, zh, ey, eys, m0);
                    z_term<-1>(oy, half, pz1, tabs + 12 * (P0 + P1) + 6 * P2, 2 * P2, zh, ex, exs, m1);
                    stz4(p.psi_h[4], qz, m0, zh, pz0, pext_y(p, 4));
                    stz4(p.psi_h[5], qz, m1, zh, pz1, pext_y(p, 5));
                }
                // TFSF: H += 0.5 (c * E1d), after the CPML terms
                if (gen && TFSF && tplane && th) tfsf_group(p, zero, 1, th, i, jj, kk, ox, oy, oz);
                const int64_t gi = (int64_t)i * p.sx + (int64_t)jj * p.sy + kk;
                stg4(p.out[0], gi, inm, true, ex, fext_y(p));
                stg4(p.out[1], gi, inm, true, ey, fext_y(p));
                stg4(p.out[2], gi, inm, true, ez, fext_y(p));
                stg4(p.out[3], gi, inm, true, ox, fext_y(p));
                stg4(p.out[4], gi, inm, true, oy, fext_y(p));
                stg4(p.out[5], gi, inm, true, oz, fext_y(p));
            }
            prev_ey = ey;
            prev_ez = ez;
            hyc = hy1;
            hzc = hz1;
            nb ^= 1;
            return true;
        };
        for (int q = 0; q < nit; q++) {
            const int i = i_start + q;
            // E(q), CE(q) and H(q+1) have arrived (H(q) with the stage before)
            const bool late = !mbar_wait_bounded(&bars[es], par, p.status, wlim);
            const bool slab = tile_gen || (P0 > 0 && (i <= P0 || i >= nx - P0 - 1));
            const bool ext = (i >= smin && i <= smax) ||
                             (DRUDE && dtile && i >= p.dbox[0] && i < p.dbox[0] + p.dbox[3]) || (TFSF && tfsf_plane(i));
            // Drude and TFSF planes off the slabs run a copy without the CPML terms (256^3 with
            // bands: 343 -> 310 us a step with a 128^3 wave box, 295 -> 287 with a 128^3 Drude
            // box).  Not where the kernel has the z terms: those grids are small, their planes
            // of all kinds alternate, and a third copy costs more (64^3, Drude: 17.1 -> 19.0).
            using std::true_type, std::false_type;
            constexpr bool own_copy = (DRUDE || TFSF) && !ZIN;
            const bool ok = slab || (!own_copy && ext) ? plane(true_type{}, true_type{}, q, late)
                            : own_copy && ext          ? plane(true_type{}, std::bool_constant<!own_copy>{}, q, late)
                                                       : plane(false_type{}, false_type{}, q, late);
            if (!ok) {
                aborted = true;
                q_abort = q;
                break;
            }
            if (++es == NS) {
                es = 0;
                par ^= 1;
            }
            if (++hs == L::NH) hs = 0;
        }
        if (aborted) break;
        first_item = false;
        if (++hs == L::NH) hs = 0;  // an item uses one H plane more than stages
        if (BATCH) {
            __syncthreads();  // every thread has read s_item
            if (tid == 0) s_item = atomicAdd(&bd.queue[0], 1);
            __syncthreads();
            gitem = s_item;
        } else {
            gitem += gridDim.x;
        }
    }

    if (BATCH && tid == 0) {
        // the last CTA to finish clears the queue for the next launch
        __threadfence();
        if (atomicAdd(&bd.queue[1], 1) == (int)gridDim.x - 1) {
            bd.queue[0] = 0;
            bd.queue[1] = 0;
            __threadfence();
        }
    }
    if (aborted) {
        if (producer) {
            atomicExch(p.status, FDTD_ERR_TIMEOUT);
            // Let the copies still in flight land before the CTA's shared
            // memory is released (each wait bounded).
            for (int q = q_abort; q <= q_issued; q++) {
                mbar_wait_bounded(&bars[es], par, nullptr, wlim);
                if (++es == NS) {
                    es = 0;
                    par ^= 1;
                }
            }
        }
        __syncthreads();
    }
}


// ---------------------------------------------------------------------------
// z band kernels (single-grid and batched plans).  The fused kernel treats z-slab tiles
// like interior tiles; these two kernels then finish the band in the same
// operation order as the in-kernel path (and the reference's cpml_e/cpml_h):
//   E: on E z-slab nodes, psi_e(z) update and E correction, then the sources
//      on those cells (list order);
//   H: on k in [1, P+1] and [n-P-1, n-1], H recomputed from the input buffer
//      and the final E with its x, y and z CPML terms (x/y psi_h were left
//      untouched there by the fused kernel).
// One thread per cell; z is the fastest index inside each band.
// ---------------------------------------------------------------------------
__device__ __forceinline__ Coef gcoef(const float *b, const float *a, const float *k, int s) {
    return Coef{b[s], a[s], k[s]};
}

// first k of the back H band
__host__ __device__ __forceinline__ int64_t zband_h_start(const Params &p) {
    const int P = p.P[2], f = (p.faces >> 4) & 1, b = (p.faces >> 5) & 1;
    const int64_t fend = f ? P + 1 : 0;
    return b ? (p.nz - P - 1 > fend + 1 ? p.nz - P - 1 : fend + 1) : p.nz;
}

// All loads come first, then the arithmetic, then the stores: a store could
// alias a later load as far as the compiler knows, so loads placed after
// stores would not be overlapped.
// E band cells per (i, j) row: the front slab's nodes, then the back slab's
__host__ __device__ __forceinline__ int zband_e_row(const Params &p) {
    return (((p.faces >> 4) & 1) ? p.P[2] : 0) + (((p.faces >> 5) & 1) ? p.P[2] : 0);
}

// E band cell kb of row (i, j)
__device__ __forceinline__ void zband_e_at(const Params &p, int64_t tstep, int64_t i, int64_t j, int kb) {
    const int P = p.P[2];
    const int nf = ((p.faces >> 4) & 1) ? P : 0;
    const int64_t k = kb < nf ? 1 + kb : p.nz - P - 1 + (kb - nf);
    const int sz = kb < nf ? kb : P + (kb - nf);
    const int64_t c = i * p.sx + j * p.sy + k, qz = (i * p.ny + j) * 2 * P + sz;
    const Coef cf = gcoef(p.tb_e[2], p.ta_e[2], p.tk_e[2], sz);
    const bool ux = j < p.ny - 1, uy = i < p.nx - 1;  // exz / eyz elements that exist
    float px = 0.f, py = 0.f, hyd = 0.f, hxd = 0.f, ex = 0.f, ey = 0.f, cx = 0.f, cy = 0.f;
    if (ux) {
        px = (FDTD_IN(qz, pext_y(p, 4)) ? p.psi_e_in[4][qz] : 0.f);
        hyd = fsub((FDTD_IN(c + 1, fext_y(p)) ? p.in[4][c + 1] : 0.f), (FDTD_IN(c, fext_y(p)) ? p.in[4][c] : 0.f));
        ex = (FDTD_IN(c, fext_y(p)) ? p.out[0][c] : 0.f);
        cx = (FDTD_IN(c, fext_y(p)) ? p.in_ce[0][c] : 0.f);
    }
    if (uy) {
        py = (FDTD_IN(qz, pext_y(p, 5)) ? p.psi_e_in[5][qz] : 0.f);
        hxd = fsub((FDTD_IN(c + 1, fext_y(p)) ? p.in[3][c + 1] : 0.f), (FDTD_IN(c, fext_y(p)) ? p.in[3][c] : 0.f));
        ey = (FDTD_IN(c, fext_y(p)) ? p.out[1][c] : 0.f);
        cy = (FDTD_IN(c, fext_y(p)) ? p.in_ce[1][c] : 0.f);
    }
    if (ux) {  // ex -= cex (..dHy/dz..)
        const float tc = corr(px, cf, hyd);
        if (FDTD_IN(qz, pext_y(p, 4))) p.psi_e_out[4][qz] = px;
        if (FDTD_IN(c, fext_y(p))) p.out[0][c] = fsub(ex, fmul(cx, tc));
    }
    if (uy) {  // ey += cey (..dHx/dz..)
        const float tc = corr(py, cf, hxd);
        if (FDTD_IN(qz, pext_y(p, 5))) p.psi_e_out[5][qz] = py;
        if (FDTD_IN(c, fext_y(p))) p.out[1][c] = fadd(ey, fmul(cy, tc));
    }
    if (tstep >= 0 && tstep < p.namp) {  // sources on this cell, list order
        const int n = p.nbsrc < 0 ? p.nsrc : p.nbsrc;
        for (int b = 0; b < n; b++) {
            const int s = p.nbsrc < 0 ? b : p.bsrc[b];
            if (p.src_ijk[3 * s] != i || p.src_ijk[3 * s + 1] != j || p.src_ijk[3 * s + 2] != k) continue;
            float *f = p.out[p.src_comp[s]] + c;
            if (FDTD_IN(c, fext_y(p))) *f = fadd(*f, p.src_amp[(int64_t)s * p.namp + tstep]);
        }
    }
}

// H band cells per (i, j) row: k = 1 .. P+1 (front), then bstart .. nz-1 (back)
__host__ __device__ __forceinline__ int zband_h_row(const Params &p) {
    const int64_t fend = ((p.faces >> 4) & 1) ? p.P[2] + 1 : 0;
    return (int)(fend + (p.nz - zband_h_start(p)));
}

// H band cell kb of row (i, j): H recomputed from the input buffer and the
// final E, with its curl, then the x, y and z CPML terms (in-kernel order)
__device__ __forceinline__ void zband_h_at(const Params &p, int64_t i, int64_t j, int kb) {
    const int P = p.P[2];
    const int front = (p.faces >> 4) & 1, back = (p.faces >> 5) & 1;
    const int64_t nz = p.nz, ny = p.ny, nx = p.nx;
    const int64_t fend = front ? P + 1 : 0;          // front band: k = 1 .. fend
    const int64_t bstart = zband_h_start(p);         // back band: k = bstart .. nz-1
    const int nf = (int)fend;
    const int64_t k = kb < nf ? 1 + kb : bstart + (kb - nf);
    const int64_t c = i * p.sx + j * p.sy + k;
    const int f0 = p.faces & 1, b0 = (p.faces >> 1) & 1, f1 = (p.faces >> 2) & 1, b1 = (p.faces >> 3) & 1;
    const int sxh = slab_h((int)i, p.P[0], (int)nx, f0, b0), syh = slab_h((int)j, p.P[1], (int)ny, f1, b1);
    const int szh = slab_h((int)k, P, (int)nz, front, back);
    const int P1 = p.P[1];
    const bool ux = j > 0 && k > 0, uy = i > 0 && k > 0, uz = i > 0 && j > 0;  // update masks
    // ---- loads
    const float *__restrict__ ex = p.out[0];
    const float *__restrict__ ey = p.out[1];
    const float *__restrict__ ez = p.out[2];
    const float hx0 = (FDTD_IN(c, fext_y(p)) ? p.in[3][c] : 0.f), hy0 = (FDTD_IN(c, fext_y(p)) ? p.in[4][c] : 0.f), hz0 = (FDTD_IN(c, fext_y(p)) ? p.in[5][c] : 0.f);
    const float ex_c = (FDTD_IN(c, fext_y(p)) ? ex[c] : 0.f), ey_c = (FDTD_IN(c, fext_y(p)) ? ey[c] : 0.f), ez_c = (FDTD_IN(c, fext_y(p)) ? ez[c] : 0.f);
    const float ez_j = j > 0 ? (FDTD_IN(c - p.sy, fext_y(p)) ? ez[c - p.sy] : 0.f) : 0.f, ex_j = j > 0 ? (FDTD_IN(c - p.sy, fext_y(p)) ? ex[c - p.sy] : 0.f) : 0.f;
    const float ey_i = i > 0 ? (FDTD_IN(c - p.sx, fext_y(p)) ? ey[c - p.sx] : 0.f) : 0.f, ez_i = i > 0 ? (FDTD_IN(c - p.sx, fext_y(p)) ? ez[c - p.sx] : 0.f) : 0.f;
    const float ey_k = (FDTD_IN(c - 1, fext_y(p)) ? ey[c - 1] : 0.f), ex_k = (FDTD_IN(c - 1, fext_y(p)) ? ex[c - 1] : 0.f);  // k >= 1 in the band
    const int64_t qy = syh >= 0 ? (i * 2 * P1 + syh) * nz + k : 0;
    const int64_t qx = sxh >= 0 ? ((int64_t)sxh * ny + j) * nz + k : 0;
    const int64_t qz = szh >= 0 ? (i * ny + j) * 2 * P + szh : 0;
    float ps_hxy = 0.f, ps_hxz = 0.f, ps_hyx = 0.f, ps_hyz = 0.f, ps_hzx = 0.f, ps_hzy = 0.f;
    if (syh >= 0) {
        if (ux) ps_hxy = (FDTD_IN(qy, pext_y(p, 3)) ? p.psi_h[3][qy] : 0.f);
        if (uz) ps_hzy = (FDTD_IN(qy, pext_y(p, 2)) ? p.psi_h[2][qy] : 0.f);
    }
    if (sxh >= 0) {
        if (uy) ps_hyx = (FDTD_IN(qx, pext_y(p, 0)) ? p.psi_h[0][qx] : 0.f);
        if (uz) ps_hzx = (FDTD_IN(qx, pext_y(p, 1)) ? p.psi_h[1][qx] : 0.f);
    }
    if (szh >= 0) {
        if (ux) ps_hxz = (FDTD_IN(qz, pext_y(p, 4)) ? p.psi_h[4][qz] : 0.f);
        if (uy) ps_hyz = (FDTD_IN(qz, pext_y(p, 5)) ? p.psi_h[5][qz] : 0.f);
    }
    // ---- arithmetic
    float hx = hx0, hy = hy0, hz = hz0;
    if (ux) {
        hx = fsub(hx, fmul(0.5f, curl4(ez_c, ez_j, ey_c, ey_k)));
        if (syh >= 0)
            hx = fsub(hx, fmul(0.5f, corr(ps_hxy, gcoef(p.tb_h[1], p.ta_h[1], p.tk_h[1], syh), fsub(ez_c, ez_j))));
        if (szh >= 0)
            hx = fadd(hx, fmul(0.5f, corr(ps_hxz, gcoef(p.tb_h[2], p.ta_h[2], p.tk_h[2], szh), fsub(ey_c, ey_k))));
    }
    if (uy) {
        hy = fsub(hy, fmul(0.5f, curl4(ex_c, ex_k, ez_c, ez_i)));
        if (sxh >= 0)
            hy = fadd(hy, fmul(0.5f, corr(ps_hyx, gcoef(p.tb_h[0], p.ta_h[0], p.tk_h[0], sxh), fsub(ez_c, ez_i))));
        if (szh >= 0)
            hy = fsub(hy, fmul(0.5f, corr(ps_hyz, gcoef(p.tb_h[2], p.ta_h[2], p.tk_h[2], szh), fsub(ex_c, ex_k))));
    }
    if (uz) {
        hz = fsub(hz, fmul(0.5f, curl4(ey_c, ey_i, ex_c, ex_j)));
        if (sxh >= 0)
            hz = fsub(hz, fmul(0.5f, corr(ps_hzx, gcoef(p.tb_h[0], p.ta_h[0], p.tk_h[0], sxh), fsub(ey_c, ey_i))));
        if (syh >= 0)
            hz = fadd(hz, fmul(0.5f, corr(ps_hzy, gcoef(p.tb_h[1], p.ta_h[1], p.tk_h[1], syh), fsub(ex_c, ex_j))));
    }
    // ---- stores
    if (FDTD_IN(c, fext_y(p))) p.out[3][c] = hx;
    if (FDTD_IN(c, fext_y(p))) p.out[4][c] = hy;
    if (FDTD_IN(c, fext_y(p))) p.out[5][c] = hz;
    if (syh >= 0) {
        if (ux) if (FDTD_IN(qy, pext_y(p, 3))) p.psi_h[3][qy] = ps_hxy;
        if (uz) if (FDTD_IN(qy, pext_y(p, 2))) p.psi_h[2][qy] = ps_hzy;
    }
    if (sxh >= 0) {
        if (uy) if (FDTD_IN(qx, pext_y(p, 0))) p.psi_h[0][qx] = ps_hyx;
        if (uz) if (FDTD_IN(qx, pext_y(p, 1))) p.psi_h[1][qx] = ps_hzx;
    }
    if (szh >= 0) {
        if (ux) if (FDTD_IN(qz, pext_y(p, 4))) p.psi_h[4][qz] = ps_hxz;
        if (uy) if (FDTD_IN(qz, pext_y(p, 5))) p.psi_h[5][qz] = ps_hyz;
    }
}

// Host stub of one fused-kernel instantiation (launched through a pointer).
typedef void (*FusedKernel)(const TMaps, const Params, const BatchDesc);

// Tile heights and pipeline depths compiled in: X(TY, NS) for each.
#define FDTD_FUSED_TILES(X) X(4, 3) X(4, 4) X(4, 6) X(8, 3) X(8, 4) X(16, 3)

// Instantiations compiled in separate translation units (the build compiles
// them in parallel): single-grid kernels without (EXT 0..3) and with (EXT 4..7)
// the z-slab terms, batched kernels without (EXT 0, 1) and with them (EXT 4, 5).
// false when (ty, ns) is not compiled in.
bool single_kernels(int ty, int ns, FusedKernel out[4]);
bool single_kernels_z(int ty, int ns, FusedKernel out[4]);
bool batch_kernels(int ty, int ns, FusedKernel out[2]);
bool batch_kernels_z(int ty, int ns, FusedKernel out[2]);

}  // namespace fused
}  // namespace fdtd
