// Fused Yee time step: host side (plans, tensor maps, launches) and the
// z-band kernels.  The fused kernel itself is in yee_fused.cuh.
#include <cuda.h>

#include <algorithm>
#include <cstring>
#include <unordered_map>
#include <vector>

#include "yee_fused.cuh"

namespace fdtd {
namespace fused {

// Band kernels: a thread per band cell, a plane's rows (blockIdx.y: i) one after
// the other, so that no lane is idle.  A warp a row left 6 to 8 of 32 lanes so with
// a 12-cell layer, and more with a thinner one; us a step without / with: 128^3 with
// 8 cells 61.8 / 59.5, 256x256x128 159.2 / 157.5, 203x331x157 206.6 / 204.4.  What
// bounds them is DRAM: 64 bytes at either end of every row (31 us for the H band of
// 256x256x128, whose 115 MB a copy would move in 17).
__global__ void __launch_bounds__(128) k_zband_e(const __grid_constant__ Params p) {
    const uint32_t nk = zband_e_row(p), u = blockIdx.x * 128 + threadIdx.x, j = u / nk;
    if (j >= p.ny) return;
    zband_e_at(p, p.t, blockIdx.y, j, (int)(u - j * nk));
}

__global__ void __launch_bounds__(128) k_zband_h(const __grid_constant__ Params p) {
    const uint32_t nk = zband_h_row(p), u = blockIdx.x * 128 + threadIdx.x, j = u / nk;
    if (j >= p.ny) return;
    zband_h_at(p, blockIdx.y, j, (int)(u - j * nk));
}

// The same over all grids of a batched plan: off[s] is the first block of grid s,
// whose planes take as many whole blocks each.  A block copies its grid's parameters
// into shared memory once.
struct BandBatch {
    int32_t nsims, cur;
    int64_t t;
    const Params *params;
    const int64_t *off;
};
constexpr int kBandBlock = 256;
__host__ __device__ __forceinline__ int64_t band_plane_blocks(const Params &p, int nk) {
    return (p.ny * nk + kBandBlock - 1) / kBandBlock;
}
template <bool E>
__global__ void __launch_bounds__(kBandBlock) k_zband_batch(const __grid_constant__ BandBatch d) {
    __shared__ __align__(16) unsigned char s_p[sizeof(Params)];
    int g = -1;  // the last grid that starts at or before this block
    for (int b = 0; b < d.nsims; b += kBandBlock) {
        const int s = b + (int)threadIdx.x;
        g += __syncthreads_count(s < d.nsims && d.off[s] <= (int64_t)blockIdx.x);
    }
    static_assert(sizeof(Params) % 8 == 0, "copied as 8-byte words");
    const uint64_t *src = reinterpret_cast<const uint64_t *>(d.params + 2 * g + d.cur);
    for (int w = threadIdx.x; w < (int)(sizeof(Params) / 8); w += kBandBlock) reinterpret_cast<uint64_t *>(s_p)[w] = src[w];
    __syncthreads();
    const Params &p = *reinterpret_cast<const Params *>(s_p);
    const uint32_t nk = E ? zband_e_row(p) : zband_h_row(p), nb = (uint32_t)band_plane_blocks(p, nk);
    const uint32_t local = (uint32_t)(blockIdx.x - d.off[g]), i = local / nb;
    const uint32_t u = (local - i * nb) * kBandBlock + threadIdx.x, j = u / nk;
    if (j >= p.ny) return;
    if (E) zband_e_at(p, d.t, i, j, (int)(u - j * nk));
    else zband_h_at(p, i, j, (int)(u - j * nk));
}

}  // namespace fused
}  // namespace fdtd

// ---------------------------------------------------------------------------
// Host side: plan = encoded tensor maps + launch configuration.
// ---------------------------------------------------------------------------
using namespace fdtd;
using namespace fdtd::fused;

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void *ptr = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &ptr, 12000, cudaEnableDefault, &q) !=
                cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            return nullptr;
        fn = reinterpret_cast<EncodeTiledFn>(ptr);
    }
    return fn;
}

struct KernelEntry {
    int ty, ns, threads, smem;  // smem: without the CPML tables
    FusedKernel fn[2][4];       // single grid: without / with the z-slab terms; bit 0: Drude, bit 1: TFSF
    FusedKernel fn_batch[2][2]; // batched: without / with the z-slab terms, Drude (no plane wave)
};

template <int TY, int NS>
static KernelEntry entry() {
    KernelEntry e{TY, NS, Layout<TY, NS>::THREADS, Layout<TY, NS>::SMEM, {}, {}};
    single_kernels(TY, NS, e.fn[0]);
    single_kernels_z(TY, NS, e.fn[1]);
    batch_kernels(TY, NS, e.fn_batch[0]);
    batch_kernels_z(TY, NS, e.fn_batch[1]);
    return e;
}

// Tile heights and pipeline depths compiled in (the autotuner picks among them).
static const KernelEntry *find_kernel(int ty, int ns) {
#define FDTD_ENTRY(TY, NS) entry<TY, NS>(),
    static const KernelEntry table[] = {FDTD_FUSED_TILES(FDTD_ENTRY)};
#undef FDTD_ENTRY
    for (const KernelEntry &e : table)
        if (e.ty == ty && e.ns == ns) return &e;
    return nullptr;
}

struct fdtd_yee_plan {
    Grid g;
    const KernelEntry *k;
    FusedKernel fn;  // the kernel variant launched (with or without the Drude / TFSF code)
    int smem;
    int x_chunk;
    int64_t nitems;
    int nblocks;
    int cluster;  // CTAs of a cluster (consecutive work items)
    int cur;
    TMaps maps[2];
    Params base;
    float *f[2][6];
    float *psi_e[2][6];
    float *dj[2][3];  // Drude J buffers
    bool has_tfsf;
    fdtd_tfsf tfsf;   // plane-wave source (1-D grid arrays owned by the caller)
};

// 3-D FP32 tensor map: dims (n0 fastest, n1, n2), element strides s1, s2,
// box (b0, b1, 1); out-of-range elements read as zero.
static int encode_map3(EncodeTiledFn enc, CUtensorMap *m, const float *ptr, int64_t n0, int64_t n1, int64_t n2,
                       int64_t s1, int64_t s2, int b0, int b1, CUtensorMapL2promotion promo) {
    cuuint64_t dims[3] = {(cuuint64_t)n0, (cuuint64_t)n1, (cuuint64_t)n2};
    cuuint64_t strides[2] = {(cuuint64_t)s1 * 4, (cuuint64_t)s2 * 4};
    cuuint32_t box[3] = {(cuuint32_t)b0, (cuuint32_t)b1, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float *>(ptr), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, promo,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? FDTD_OK : FDTD_ERR_CUDA;
}

static int encode_map(EncodeTiledFn enc, CUtensorMap *m, const float *ptr, const Grid &g, int box_z, int box_y,
                      CUtensorMapL2promotion promo) {
    return encode_map3(enc, m, ptr, g.nz, g.ny, g.nx, g.sy, g.sx, box_z, box_y, promo);
}

// Default launch shape: tile rows and pipeline stages.
constexpr int kTileY = 8, kStages = 3;
constexpr int kCluster = 8;

// Whether a single grid's z slab (slab nodes a row) is left to the band kernels.
// In the fused kernel a z-edge tile takes twice the time of a plain one a plane
// (its row warps run the z code for a quarter of their lanes), and its neighbours
// then share no halo reads with it; the band kernels cost two launches and a second
// pass over the row ends.  Measured, fused / bands, us a step with an 8-cell CPML on
// all faces: 48^3 16 / 21, 64^3 16 / 21, 80^3 34 / 33, 100x100x64 28 / 29, 100^3
// 51 / 46, 52x162x171 65 / 54, 125x125x130 89 / 73, with a Drude box 104 / 77; with 12
// cells 256x256x128 186 / 160, 512^3 1739 / 1545.  Rows that are mostly slab lose
// earlier: 200x200x20 with a Drude box 112 / 70, 1000x60x20 157 / 101 (the kernels before
// these 104 and 132).  So do launch shapes of the caller's with a Drude box or a wave,
// fused / bands (the kernels before): 80^3, 4 cells, both, tiles of 4 rows 92 / 67 (69),
// 60x200x40 92 / 64 (72); a wave and a chunk of 8 planes, 48^3 53 / 46 (49); and so do
// long chunks on their own, whose items march many planes at a plane's latency: 64^3 with
// 8 cells, chunks of 31 109 / 77 (86), 57x100x124 84 / 46 (60).  Grids of few (i, j) rows
// keep the bands' three launches, which plan_info reports and the tests of it expect, and
// so does one chunk on grids below 393 kcells keep its one launch.
static bool use_bands(const Grid &g, int slab, const fdtd_tile *tile, bool drude, bool tfsf) {
    const int64_t rows = g.nx * g.ny, cells = rows * g.nz;
    const bool own = tile && tile->tile_y != 16 &&  // (tiles of 16 rows: 60x70x90, a Drude box, 26 / 27)
                     (tile->tile_y || tile->x_chunk || tile->ctas_per_sm > 0 || tile->stages);
    if (own && tile->x_chunk && (tfsf || tile->x_chunk >= 8))
        return tfsf || drude || rows < 2048 || tile->x_chunk < g.nx || cells >= 3 << 17;
    const int line = own && (drude || tfsf) ? 5 << 16 : own && !tile->x_chunk ? 3 << 17 : 2 * slab > g.nz ? 3 << 18 : 13 << 16;
    return rows < 2048 || cells >= line;
}

static bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

extern "C" {

// Shared memory, resident CTAs and SM count of a kernel variant.
static int fused_residency(FusedKernel fn, int threads, int smem, int *nsm, int *occ) {
    int dev = 0, optin = 0;
    cudaFuncAttributes fa;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, (const void *)fn);
    if (e != cudaSuccess) { set_cuda_error(e); return FDTD_ERR_CUDA; }
    const int max_dyn = optin - (int)fa.sharedSizeBytes;
    if (smem > max_dyn) return FDTD_ERR_UNSUPPORTED;
    // the attribute is an upper bound; every plan of this kernel fits under it
    e = cudaFuncSetAttribute((const void *)fn, cudaFuncAttributeMaxDynamicSharedMemorySize, max_dyn);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(nsm, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ, (const void *)fn, threads, smem);
    if (e != cudaSuccess) { set_cuda_error(e); return FDTD_ERR_CUDA; }
    return *occ < 1 ? FDTD_ERR_UNSUPPORTED : FDTD_OK;
}

// Default x chunk of a single grid: of the splits of nx into 1 .. nx chunks,
// the one whose launch is shortest when `slots` resident CTAs work through
// tiles * chunks items of chunk + kItemPlanes plane steps (an item's pipeline
// fill and its recomputed halo plane); the longer chunk on a tie.
constexpr int kItemPlanes = 4;
static int single_chunk(int64_t nx, int64_t tiles, int64_t slots) {
    int64_t best = nx, best_t = -1;
    for (int64_t n = 1; n <= nx; n++) {
        const int64_t c = (nx + n - 1) / n, items = tiles * ((nx + c - 1) / c);
        const int64_t t = (items + slots - 1) / slots * (c + kItemPlanes);
        if (c > 128 && n < nx) continue;
        if (c < 2) break;  // one-plane items would compute every E plane twice
        if (best_t < 0 || t < best_t) {
            best_t = t;
            best = c;
        }
    }
    return (int)best;
}

// The chunk for which the number of sources an item may hold is counted when the
// caller gives none: 128 planes, halved down to 8 until there are 3 items an SM.
// It fixes which source layouts are refused, whatever chunk the step then takes;
// a longer chunk's items may hold more than their list does, and scan all sources.
static int capacity_chunk(int64_t nx, int64_t tiles, int nsm) {
    int xc = 128;
    while (xc > 8 && tiles * ((nx + xc - 1) / xc) < 3 * (int64_t)nsm) xc /= 2;
    return xc;
}

// batch_chunk > 0: a grid of a batched plan, which pools every grid's items over
// one launch (with that chunk unless the caller gives one); batch_bands: the
// batched plan's band kernels finish the z slab
static int yee_plan_create(fdtd_yee_plan **out, const fdtd_grid *gp, const fdtd_yee_state *s, const fdtd_cpml *c,
                           const fdtd_sources *src, const fdtd_tile *tile, int32_t *status_dev, int32_t cur,
                           void *stream, int batch_chunk, bool batch_bands) {
    if (!out || !s || !status_dev) return FDTD_ERR_ARG;
    *out = nullptr;
    Grid g;
    FDTD_TRY(validate_grid(gp, &g));
    if (g.nx < 2 || g.ny < 2 || g.nz < 2) return FDTD_ERR_SHAPE;
    if (g.nx > (1 << 30) || g.ny > (1 << 30) || g.nz > (1 << 30)) return FDTD_ERR_SHAPE;
    if ((g.sx & 3) || (g.sy & 3)) return FDTD_ERR_ALIGN;
    if (cur != 0 && cur != 1) return FDTD_ERR_ARG;
    for (int b = 0; b < 2; b++)
        for (int q = 0; q < 6; q++) {
            if (!s->f[b][q]) return FDTD_ERR_ARG;
            if (!aligned16(s->f[b][q])) return FDTD_ERR_ALIGN;
        }
    for (int q = 0; q < 3; q++) {
        if (!s->ce[q]) return FDTD_ERR_ARG;
        if (!aligned16(s->ce[q])) return FDTD_ERR_ALIGN;
    }
    const int ty = tile && tile->tile_y ? tile->tile_y : kTileY;
    const int ns = tile && tile->stages ? tile->stages : kStages;
    const KernelEntry *ke = find_kernel(ty, ns);
    if (!ke) return FDTD_ERR_UNSUPPORTED;
    int xch = tile && tile->x_chunk ? tile->x_chunk : 0;  // 0: chosen below
    if (xch < 0) return FDTD_ERR_ARG;

    fdtd_yee_plan *pl = new fdtd_yee_plan();
    pl->g = g;
    pl->k = ke;
    pl->cur = cur;
    Params &p = pl->base;
    p = Params{};
    p.nx = g.nx; p.ny = g.ny; p.nz = g.nz; p.sx = g.sx; p.sy = g.sy;
    p.ntz = (int)((g.nz + TZ - 1) / TZ);
    p.nty = (int)((g.ny + ty - 1) / ty);
    p.status = status_dev;
    p.wait_ns = 0;         // the 1 s limit
    p.test_withhold = -1;  // every copy issued

    const bool pml = c && (c->npml[0] > 0 || c->npml[1] > 0 || c->npml[2] > 0);
    if (pml) {
        const int64_t n[3] = {g.nx, g.ny, g.nz};
        p.faces = c->faces;
        for (int a = 0; a < 3; a++) {
            p.P[a] = c->npml[a];
            if (c->npml[a] < 0) { delete pl; return FDTD_ERR_ARG; }
            if (c->npml[a] == 0) continue;
            if (n[a] < 2 * (int64_t)c->npml[a] + 2) { delete pl; return FDTD_ERR_SHAPE; }
            if (!all_nonnull(c->b_e[a], c->a_e[a], c->km1_e[a], c->b_h[a], c->a_h[a], c->km1_h[a])) {
                delete pl; return FDTD_ERR_ARG;
            }
            for (int b = 0; b < 2; b++)
                if (!s->psi_e[b][2 * a] || !s->psi_e[b][2 * a + 1]) { delete pl; return FDTD_ERR_ARG; }
            if (!s->psi_h[2 * a] || !s->psi_h[2 * a + 1]) { delete pl; return FDTD_ERR_ARG; }
            p.tb_e[a] = c->b_e[a]; p.ta_e[a] = c->a_e[a]; p.tk_e[a] = c->km1_e[a];
            p.tb_h[a] = c->b_h[a]; p.ta_h[a] = c->a_h[a]; p.tk_h[a] = c->km1_h[a];
        }
        for (int q = 0; q < 6; q++) p.psi_h[q] = s->psi_h[q];
    }
    for (int q = 0; q < 3; q++) p.in_ce[q] = s->ce[q];
    if (s->drude) {
        const int st = validate_drude(g, s->drude);
        if (st != FDTD_OK) { delete pl; return st; }
        const fdtd_drude &d = *s->drude;
        p.drude = 1;
        const int64_t box[6] = {d.i0, d.j0, d.k0, d.ni, d.nj, d.nk};
        for (int q = 0; q < 6; q++) p.dbox[q] = box[q];
        for (int q = 0; q < 3; q++) {
            if (!d.j2[q]) { delete pl; return FDTD_ERR_ARG; }
            pl->dj[0][q] = d.j[q];
            pl->dj[1][q] = d.j2[q];
            p.dcja[q] = d.cja[q];
            p.dcjb[q] = d.cjb[q];
        }
    }
    if (s->tfsf) {
        const int st = validate_tfsf(g, s->tfsf);
        if (st != FDTD_OK) { delete pl; return st; }
        const fdtd_tfsf &t = *s->tfsf;
        // the box's face cells (p1-1 .. p2) stay clear of the CPML slabs and of the
        // z band, which the band kernels finish after the fused kernel
        const int64_t n3[3] = {g.nx, g.ny, g.nz};
        for (int a = 0; a < 3; a++) {
            const int64_t P = c ? c->npml[a] : 0;
            if (P > 0 && (t.p1[a] - 1 < P + 2 || t.p2[a] + 1 > n3[a] - P - 2)) { delete pl; return FDTD_ERR_UNSUPPORTED; }
        }
        pl->has_tfsf = true;
        pl->tfsf = t;
        p.tfsf = 1;
        p.tfaces = t.faces;
        p.taxis = t.axis;
        for (int a = 0; a < 3; a++) {
            p.tp1[a] = (int32_t)t.p1[a];
            p.tp2[a] = (int32_t)t.p2[a];
        }
        tfsf_table(&t, p.tcoef, p.tix, &p.tvo);
        p.te1d = t.e1d;
        p.th1d = t.h1d;
    }
    // the z slab (when a z face has CPML): inside the fused kernel or by the band kernels
    p.zfix = 0;
    if (p.P[2] > 0 && ((p.faces >> 4) & 3))
        p.zfix = batch_chunk ? batch_bands : use_bands(g, zband_e_row(p), tile, p.drude, p.tfsf);
    // tile rows with y slab cells (rows j0-1 .. j0+ty-1), counted from either end
    if (p.P[1] > 0)
        for (int t = 0; t < p.nty; t++) {
            if (((p.faces >> 2) & 1) && t * ty - 1 <= p.P[1]) p.yf = t + 1;
            if (((p.faces >> 3) & 1) && (int64_t)(t + 1) * ty - 1 >= g.ny - p.P[1] - 1) {
                p.yb = p.nty - std::max(t, p.yf);
                break;
            }
        }
    // launch configuration: shared memory, resident CTAs, x chunk
    pl->smem = ke->smem + 6 * 2 * (p.P[0] + p.P[1] + p.P[2]) * 4;
    pl->fn = ke->fn[p.P[2] > 0 && ((p.faces >> 4) & 3) && !p.zfix][(p.drude ? 1 : 0) | (p.tfsf ? 2 : 0)];
    int nsm = 0, occ = 0;
    {
        const int st = fused_residency(pl->fn, ke->threads, pl->smem, &nsm, &occ);
        if (st != FDTD_OK) { delete pl; return st; }
    }
    const int max_ctas = tile ? (int)tile->ctas_per_sm : 0;
    if (max_ctas > 0) occ = std::min(occ, max_ctas);
    const int cap_chunk = xch ? xch : capacity_chunk(g.nx, (int64_t)p.ntz * p.nty, nsm);
    if (!xch) {
        xch = batch_chunk ? batch_chunk : single_chunk(g.nx, (int64_t)p.ntz * p.nty, (int64_t)nsm * occ);
        // With a wave and CPML a tile's planes take up to three times as long where they hold
        // faces and slabs, and a launch of one round lasts as long as its slowest item: no
        // longer chunks than give 3 items an SM.  us a step, one round / this, a box 5 cells
        // off the layer: 180^3 with 4 cells 249 / 170, 150^3 with 8 211 / 152, 300x120x120
        // 198 / 154, with a Drude box 211 / 182 (the kernels before these: 223, 191, 184, 217);
        // 256^3 takes several rounds and keeps its chunk.  Not on other launch shapes: one CTA an
        // SM (100x100x64 with 4 cells 63 / 87) and tiles of 4 rows (80^3, 6 stages, 72 / 84) lose.
        if (p.tfsf && pml && ty == kTileY && ns == kStages && max_ctas <= 0) xch = std::min(xch, cap_chunk);
    }
    pl->x_chunk = p.x_chunk = (int)std::min<int64_t>(xch, g.nx);
    p.nxc = (int)((g.nx + pl->x_chunk - 1) / pl->x_chunk);
    pl->nitems = (int64_t)p.ntz * p.nty * p.nxc;
    if (p.nxc <= MAX_ORDERED) {
        // item order of the x chunks: those with the slowest planes first, counting a plane
        // of an x slab, of the Drude box or of the wave's box as two, so that no slow items are
        // left for the launch's tail.  Against the x slab chunks alone first, us a step, 12-cell
        // CPML and a box of half of each extent: 400x300x200 TFSF 567 -> 479, Drude 570 -> 478;
        // 512^3 1831 -> 1731, 1862 -> 1840; 256^3 310 -> 305, 286 -> 281 (both boxes 347 -> 358).
        int cost[MAX_ORDERED];
        for (int q = 0; q < p.nxc; q++) {
            const int64_t x0 = (int64_t)q * p.x_chunk, x1 = std::min<int64_t>(x0 + p.x_chunk, g.nx);
            cost[q] = 0;
            for (int64_t i = x0; i < x1; i++)
                cost[q] += 1 + (p.P[0] > 0 && (((p.faces & 1) && i <= p.P[0]) || ((p.faces & 2) && i >= g.nx - p.P[0] - 1))) +
                           (p.drude && i >= p.dbox[0] && i < p.dbox[0] + p.dbox[3]) +
                           (p.tfsf && i >= p.tp1[0] - 1 && i <= p.tp2[0]);
            p.xorder[q] = (uint8_t)q;
        }
        std::stable_sort(p.xorder, p.xorder + p.nxc, [&](uint8_t a, uint8_t b) { return cost[a] > cost[b]; });
    }
    if (pl->nitems >= ((int64_t)1 << 31)) { delete pl; return FDTD_ERR_UNSUPPORTED; }
    // one CTA an item, or a persistent grid where the caller limits the CTAs per SM
    pl->nblocks = (int)(max_ctas > 0 ? std::min<int64_t>(pl->nitems, (int64_t)nsm * occ) : pl->nitems);
    // Launches of several rounds: clusters of 8 consecutive items.  A cluster's CTAs
    // start together, so neighbouring tiles stay on nearby planes and share their halo
    // reads through L2, which items that start one by one do not after the first
    // rounds.  Measured without / with, us a step (27 rounds: 1024x1024x512, 6.7:
    // 512^3): 5098 / 4837 plain and 6563 / 6015 with CPML; 1241 / 1223 and 1652 / 1587.
    // With 3 rounds (256^3) the slots that wait for 8 to be free cost more: 164 / 172.
    pl->cluster = 1;
    if (max_ctas <= 0 && pl->nitems >= 4 * (int64_t)nsm * occ) {
        pl->cluster = kCluster;
        pl->nblocks = (pl->nblocks + kCluster - 1) / kCluster * kCluster;  // the excess CTAs find no item
    }
    if (src && src->nsrc > 0) {
        if (!all_nonnull(src->ijk, src->comp, src->amp) || src->namp < 0) { delete pl; return FDTD_ERR_ARG; }
        p.nsrc = src->nsrc; p.src_ijk = src->ijk; p.src_comp = src->comp; p.src_amp = src->amp; p.namp = src->namp;
        // capacity: sources per work item's extended region, in chunks of cap_chunk planes
        // read on the caller's stream (after any pending write of the list), then wait for it
        int32_t *hijk = new int32_t[3 * (size_t)src->nsrc];
        cudaError_t ce = cudaMemcpyAsync(hijk, src->ijk, sizeof(int32_t) * 3 * src->nsrc, cudaMemcpyDeviceToHost,
                                         as_stream(stream));
        if (ce == cudaSuccess) ce = cudaStreamSynchronize(as_stream(stream));
        if (ce != cudaSuccess) {
            set_cuda_error(ce);
            delete[] hijk; delete pl; return FDTD_ERR_CUDA;
        }
        // sources on E z-slab nodes: applied by the E band kernel
        if (p.zfix) {
            const int64_t P2 = p.P[2];
            const int f2 = (p.faces >> 4) & 1, b2 = (p.faces >> 5) & 1;
            for (int a = 0; a < src->nsrc; a++) {
                const int64_t sk = hijk[3 * a + 2];
                const bool node = (f2 && sk >= 1 && sk <= P2) || (b2 && sk >= g.nz - P2 - 1 && sk <= g.nz - 2);
                if (!node) continue;
                if (p.nbsrc == MAX_BAND_SRC) {  // too many for the list: the band kernel scans all sources
                    p.nbsrc = -1;
                    break;
                }
                p.bsrc[p.nbsrc++] = a;
            }
        }
        // sources per work item, counted with the kernel's own membership test
        // (x in [i_start, x1), y in [j0-1, j0+TY), z in [k0-1, k0+TZ)); a source
        // lies in at most two chunks/tiles per axis
        std::unordered_map<int64_t, int> per_item;
        const int64_t xc = std::min<int64_t>(cap_chunk, g.nx);
        const int64_t ntz = (g.nz + TZ - 1) / TZ, nty = (g.ny + ty - 1) / ty;
        for (int a = 0; a < src->nsrc; a++) {
            const int64_t si = hijk[3 * a], sj = hijk[3 * a + 1], sk = hijk[3 * a + 2];
            if (si < 0 || si >= g.nx || sj < 0 || sj >= g.ny || sk < 0 || sk >= g.nz || sk >= (int64_t(1) << 28)) {
                delete[] hijk; delete pl; return FDTD_ERR_ARG;
            }
            for (int64_t xi = si / xc; xi <= (si + 1) / xc; xi++) {
                const int64_t x0 = xi * xc, x1 = std::min(x0 + xc, (int64_t)g.nx);
                const int64_t is = x0 > 0 ? x0 - 1 : 0;
                if (x0 >= g.nx || si < is || si >= x1) continue;
                for (int64_t yi = sj / ty; yi <= (sj + 1) / ty && yi < nty; yi++) {
                    const int64_t j0 = yi * ty;
                    if (sj < j0 - 1 || sj >= j0 + ty) continue;
                    for (int64_t zi = sk / TZ; zi <= (sk + 1) / TZ && zi < ntz; zi++) {
                        const int64_t k0 = zi * TZ;
                        if (sk < k0 - 1 || sk >= k0 + TZ) continue;
                        if (++per_item[(xi * nty + yi) * ntz + zi] > MAX_LOCAL_SRC) {
                            delete[] hijk; delete pl; return FDTD_ERR_CAPACITY;
                        }
                    }
                }
            }
        }
        delete[] hijk;
    }

    EncodeTiledFn enc = get_encode_fn();
    if (!enc) { delete pl; return FDTD_ERR_CUDA; }
    for (int b = 0; b < 2; b++) {
        for (int q = 0; q < 6; q++) {
            pl->f[b][q] = s->f[b][q];
            pl->psi_e[b][q] = s->psi_e[b][q];
        }
        const int pm = tile ? tile->l2_promotion : 0;
        const CUtensorMapL2promotion promo = pm == 1   ? CU_TENSOR_MAP_L2_PROMOTION_NONE
                                             : pm == 2 ? CU_TENSOR_MAP_L2_PROMOTION_L2_64B
                                             : pm == 3 ? CU_TENSOR_MAP_L2_PROMOTION_L2_128B
                                                       : CU_TENSOR_MAP_L2_PROMOTION_L2_256B;
        int st = FDTD_OK;
        for (int q = 0; q < 3 && st == FDTD_OK; q++) {
            st = encode_map(enc, &pl->maps[b].h[q], s->f[b][3 + q], g, HC, ty + 2, promo);
            if (st == FDTD_OK) st = encode_map(enc, &pl->maps[b].e[q], s->f[b][q], g, EC, ty + 1, promo);
            if (st == FDTD_OK) st = encode_map(enc, &pl->maps[b].ce[q], s->ce[q], g, EC, ty + 1, promo);
        }
        if (st != FDTD_OK) { delete pl; return st; }
    }
    // 16-byte accesses of the x/y psi slabs: rows of nz floats must be 16-byte
    // multiples
    p.vpsi = g.nz % 4 == 0;
    for (int q = 0; q < 4 && pml; q++)
        if (p.P[q / 2] > 0)
            p.vpsi = p.vpsi && aligned16(s->psi_e[0][q]) && aligned16(s->psi_e[1][q]) && aligned16(s->psi_h[q]);
    if (p.drude) {
        p.dvec = p.dbox[2] % 4 == 0 && p.dbox[5] % 4 == 0;
        for (int q = 0; q < 3; q++)
            p.dvec = p.dvec && aligned16(pl->dj[0][q]) && aligned16(pl->dj[1][q]) && aligned16(p.dcja[q]) &&
                     aligned16(p.dcjb[q]);
    }
    *out = pl;
    return FDTD_OK;
}

int fdtd_yee_plan_create(fdtd_yee_plan **out, const fdtd_grid *gp, const fdtd_yee_state *s, const fdtd_cpml *c,
                         const fdtd_sources *src, const fdtd_tile *tile, int32_t *status_dev, int32_t cur,
                         void *stream) {
    return yee_plan_create(out, gp, s, c, src, tile, status_dev, cur, stream, 0, false);
}

int fdtd_yee_plan_run(fdtd_yee_plan *pl, int64_t t0, int64_t nsteps, void *stream) {
    if (!pl || nsteps < 0) return FDTD_ERR_ARG;
    cudaStream_t st = as_stream(stream);
    // TFSF: the 1-D E step of each step runs before its fused kernel (whose E
    // faces read the 1-D H of the previous step, H faces the new 1-D E), the
    // 1-D H step after it
    if (pl->has_tfsf && nsteps > 0) {
        if (t0 + nsteps - 1 >= pl->tfsf.namp || t0 < 0) return FDTD_ERR_ARG;
        FDTD_TRY(tfsf_launch_1d(&pl->tfsf, 0, t0, st));
    }
    for (int64_t n = 0; n < nsteps; n++) {
        NvtxRange nvtx_range("fdtd_yee_step");
        const int in = pl->cur, outb = 1 - pl->cur;
        Params p = pl->base;
        for (int q = 0; q < 6; q++) {
            p.out[q] = pl->f[outb][q];
            p.psi_e_in[q] = pl->psi_e[in][q];
            p.psi_e_out[q] = pl->psi_e[outb][q];
        }
        for (int q = 0; q < 3; q++) {
            p.dj_in[q] = pl->dj[in][q];
            p.dj_out[q] = pl->dj[outb][q];
        }
        p.t = t0 + n;
        BatchDesc bd{};
        launch_chained(pl->fn, dim3((unsigned)pl->nblocks), dim3((unsigned)pl->k->threads), (size_t)pl->smem, st,
                       (unsigned)pl->cluster, pl->maps[in], p, bd);
        if (p.zfix) {
            for (int q = 0; q < 6; q++) p.in[q] = pl->f[in][q];
            // (a plane's band cells number less than 2^32: the arrays would not fit otherwise)
            auto plane = [&](int nk) { return dim3((unsigned)((p.ny * nk + 127) / 128), (unsigned)p.nx); };
            // launched the plain way: started early, their waiting blocks hold back the
            // kernel before them (256^3 253 -> 261 us a step)
            k_zband_e<<<plane(zband_e_row(p)), 128, 0, st>>>(p);
            k_zband_h<<<plane(zband_h_row(p)), 128, 0, st>>>(p);
        }
        FDTD_TRY(check_launch());
        if (pl->has_tfsf) FDTD_TRY(tfsf_launch_1d(&pl->tfsf, n + 1 < nsteps ? 2 : 1, t0 + n + 1, st));
        pl->cur = outb;
    }
    return FDTD_OK;
}

int fdtd_yee_plan_current(const fdtd_yee_plan *pl) { return pl ? pl->cur : -1; }

int fdtd_yee_plan_test_timeout(fdtd_yee_plan *pl, int64_t wait_ns, int32_t withhold_plane) {
    if (!pl || wait_ns < 0 || withhold_plane < -1) return FDTD_ERR_ARG;
    pl->base.wait_ns = (uint64_t)wait_ns;
    pl->base.test_withhold = withhold_plane;
    return FDTD_OK;
}

int fdtd_yee_plan_set_current(fdtd_yee_plan *pl, int32_t cur) {
    if (!pl || (cur != 0 && cur != 1)) return FDTD_ERR_ARG;
    pl->cur = cur;
    return FDTD_OK;
}

int fdtd_yee_plan_info(const fdtd_yee_plan *pl, int32_t *info, int32_t n) {
    if (!pl || !info || n < 6) return FDTD_ERR_ARG;
    info[0] = pl->k->ty;
    info[1] = pl->k->ns;
    info[2] = pl->x_chunk;
    info[3] = pl->nblocks;
    info[4] = pl->k->threads;
    info[5] = pl->smem;
    if (n >= 8) {
        info[6] = pl->base.zfix;                  // 1: z slab on the band kernels
        info[7] = (pl->base.zfix ? 3 : 1) + (pl->has_tfsf ? 1 : 0);  // kernel launches per step
    }
    return FDTD_OK;
}

int fdtd_yee_plan_destroy(fdtd_yee_plan *pl) {
    delete pl;
    return FDTD_OK;
}

int fdtd_yee_step_f32(const fdtd_grid *g, const fdtd_yee_state *st, const fdtd_cpml *c, const fdtd_sources *src,
                      int32_t *status_dev, int32_t cur, int64_t t0, int64_t nsteps, int32_t *cur_out,
                      void *stream) {
    if (nsteps < 0) return FDTD_ERR_ARG;
    fdtd_yee_plan *pl = nullptr;
    FDTD_TRY(fdtd_yee_plan_create(&pl, g, st, c, src, nullptr, status_dev, cur, stream));
    const int r = fdtd_yee_plan_run(pl, t0, nsteps, stream);
    if (cur_out) *cur_out = pl->cur;
    fdtd_yee_plan_destroy(pl);  // host-side only: the launches hold copies of everything they use
    return r;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Batched plan: many grids, one launch per step.  Every grid gets an ordinary
// plan (validation, tensor maps, parameters); their Params/TMaps and the item
// offsets live in a caller-provided device workspace.
// ---------------------------------------------------------------------------
struct fdtd_batch_plan {
    int32_t nsims;
    const KernelEntry *k;
    FusedKernel fn;  // batched variant launched (with the Drude code when a grid has a Drude box)
    int smem;
    int nblocks;
    int cur;
    int64_t nitems;
    TMaps *d_maps;
    Params *d_params;
    int64_t *d_off;        // work-item offsets of the fused kernel, then the band kernels' block offsets (E, H)
    int64_t band_e, band_h;  // blocks of the band kernels
    int32_t *d_queue;        // work queue of the fused kernel (2 counters)
};

static size_t batch_ws_layout(int32_t nsims, size_t *off_params, size_t *off_items) {
    size_t o = 0;
    o += (size_t)2 * nsims * sizeof(TMaps);
    o = (o + 63) / 64 * 64;
    *off_params = o;
    o += (size_t)2 * nsims * sizeof(Params);
    o = (o + 63) / 64 * 64;
    *off_items = o;  // work-item offsets, band block offsets (E, H), then the queue
    o += (size_t)3 * (nsims + 1) * sizeof(int64_t);
    o += 64;
    return o;
}

extern "C" {

size_t fdtd_batch_workspace_bytes(int32_t nsims) {
    size_t a, b;
    return nsims > 0 ? batch_ws_layout(nsims, &a, &b) : 0;
}

int fdtd_batch_plan_create(fdtd_batch_plan **out, int32_t nsims, const fdtd_grid *grids, const fdtd_yee_state *states,
                           const fdtd_cpml *cpmls, const fdtd_sources *srcs, const fdtd_tile *tile,
                           int32_t *status_dev, void *workspace, size_t workspace_bytes, int32_t cur,
                           void *stream) {
    if (!out || nsims <= 0 || !grids || !states || !status_dev || !workspace) return FDTD_ERR_ARG;
    *out = nullptr;
    if ((reinterpret_cast<uintptr_t>(workspace) & 63) != 0) return FDTD_ERR_ALIGN;
    size_t off_p, off_i;
    const size_t need = batch_ws_layout(nsims, &off_p, &off_i);
    if (workspace_bytes < need) return FDTD_ERR_CAPACITY;
    std::vector<TMaps> maps((size_t)2 * nsims);
    std::vector<Params> params((size_t)2 * nsims);
    std::vector<int64_t> off((size_t)3 * (nsims + 1), 0);
    int64_t *off_e = off.data() + (nsims + 1), *off_h = off_e + (nsims + 1);
    const KernelEntry *ke = nullptr;
    int tab_bytes = 0;
    bool any_drude = false, any_zin = false;  // z terms in the kernel
    const int ty = tile && tile->tile_y ? tile->tile_y : kTileY;
    int chunk = tile ? tile->x_chunk : 0;
    if (ty > 0 && !chunk) {
        // default chunk for all grids: of 8 .. 128 planes, the one for which the
        // items (planes + kItemPlanes each) of all grids, spread evenly over
        // the CTAs, plus one last item end first
        int dev = 0, nsm = 0;
        if (cudaGetDevice(&dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || nsm < 1)
            nsm = 1;
        double best_t = -1;
        for (int c : {128, 96, 64, 48, 32, 24, 16, 12, 8}) {
            double work = 0;
            int64_t longest = 0;
            for (int32_t s = 0; s < nsims; s++) {
                const int64_t tiles = ((grids[s].nz + TZ - 1) / TZ) * ((grids[s].ny + ty - 1) / ty);
                work += (double)tiles * (double)(grids[s].nx + kItemPlanes * ((grids[s].nx + c - 1) / c));
                longest = std::max(longest, std::min<int64_t>(c, grids[s].nx) + kItemPlanes);
            }
            const double t = work / (2.0 * nsm) + (double)longest;
            if (best_t < 0 || t < best_t) {
                best_t = t;
                chunk = c;
            }
        }
    }
    int64_t cells = 0;
    for (int32_t s = 0; s < nsims; s++) cells += grids[s].nx * grids[s].ny * grids[s].nz;
    // The z slab on band kernels (three launches a step) or in the kernel, where the tiles of a
    // z slab, half of all on grids of up to 192 cells, execute twice a plain one's instructions.
    // us a step in the kernel / on bands: 8 grids of 24..96 cells an axis, 1.6 Mcells in all,
    // 97 / 84; 24 of 24..64 (2.1 M) 110 / 105; 64 of 32..192 (80 M) 2022 / 1617; but 8 of 24..64
    // (0.8 M) 45 / 50 and 4 of 64^3 (1.0 M) 45 / 51, where the launches count.  Tiles of 4 rows,
    // a third of whose warps are halo, are faster on bands at any size: 64 of 14..24 (0.4 M) 93 / 71,
    // with Drude boxes 115 / 92 (the kernels before these 92 and 99)
    const bool bands = cells >= 3 << 19 || ty == 4;
    // grids with the longest items (x planes per chunk, then tile rows) come first
    std::vector<int32_t> order((size_t)nsims);
    for (int32_t s = 0; s < nsims; s++) order[s] = s;
    auto item_len = [&](int32_t s) {
        return std::min<int64_t>(chunk, grids[s].nx) * 65536 + std::min<int64_t>(grids[s].ny, 65535);
    };
    std::stable_sort(order.begin(), order.end(), [&](int32_t a, int32_t b) { return item_len(a) > item_len(b); });
    for (int32_t s = 0; s < nsims; s++)
        if (states[s].tfsf) return FDTD_ERR_UNSUPPORTED;  // plane waves: single-grid plans only
    for (int32_t s = 0; s < nsims; s++) {
        const int32_t u = order[s];
        fdtd_yee_plan *pl = nullptr;
        const int st = yee_plan_create(&pl, &grids[u], &states[u], cpmls ? &cpmls[u] : nullptr,
                                       srcs ? &srcs[u] : nullptr, tile, status_dev, cur, stream, std::max(chunk, 1),
                                       bands);
        if (st != FDTD_OK) return st;
        ke = pl->k;
        any_drude = any_drude || pl->base.drude;
        any_zin = any_zin || (pl->base.P[2] > 0 && ((pl->base.faces >> 4) & 3) && !pl->base.zfix);
        tab_bytes = std::max(tab_bytes, 6 * 2 * (pl->base.P[0] + pl->base.P[1] + pl->base.P[2]) * 4);
        for (int b = 0; b < 2; b++) {
            Params p = pl->base;
            for (int q = 0; q < 6; q++) {
                p.out[q] = pl->f[1 - b][q];
                p.psi_e_in[q] = pl->psi_e[b][q];
                p.psi_e_out[q] = pl->psi_e[1 - b][q];
                p.in[q] = pl->f[b][q];
            }
            for (int q = 0; q < 3; q++) {
                p.dj_in[q] = pl->dj[b][q];
                p.dj_out[q] = pl->dj[1 - b][q];
            }
            params[2 * s + b] = p;
            maps[2 * s + b] = pl->maps[b];
        }
        off[s + 1] = off[s] + pl->nitems;
        const Params &p = pl->base;
        off_e[s + 1] = off_e[s] + (p.zfix ? p.nx * band_plane_blocks(p, zband_e_row(p)) : 0);
        off_h[s + 1] = off_h[s] + (p.zfix ? p.nx * band_plane_blocks(p, zband_h_row(p)) : 0);
        fdtd_yee_plan_destroy(pl);
    }
    // fill the workspace on the caller's stream (ordered after that stream's
    // earlier launches that may still read it), then wait for the copies: the
    // host-side tables are freed on return
    unsigned char *ws = static_cast<unsigned char *>(workspace);
    cudaStream_t cs = as_stream(stream);
    cudaError_t e = cudaMemcpyAsync(ws, maps.data(), maps.size() * sizeof(TMaps), cudaMemcpyHostToDevice, cs);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(ws + off_p, params.data(), params.size() * sizeof(Params), cudaMemcpyHostToDevice, cs);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(ws + off_i, off.data(), off.size() * sizeof(int64_t), cudaMemcpyHostToDevice, cs);
    if (e == cudaSuccess) e = cudaMemsetAsync(ws + off_i + off.size() * sizeof(int64_t), 0, 64, cs);
    if (e == cudaSuccess) e = cudaStreamSynchronize(cs);
    if (e != cudaSuccess) { set_cuda_error(e); return FDTD_ERR_CUDA; }

    fdtd_batch_plan *bp = new fdtd_batch_plan();
    bp->nsims = nsims;
    bp->k = ke;
    bp->smem = ke->smem + tab_bytes;
    bp->cur = cur;
    bp->nitems = off[nsims];
    bp->d_maps = reinterpret_cast<TMaps *>(ws);
    bp->d_params = reinterpret_cast<Params *>(ws + off_p);
    bp->d_off = reinterpret_cast<int64_t *>(ws + off_i);
    bp->d_queue = reinterpret_cast<int32_t *>(ws + off_i + off.size() * sizeof(int64_t));
    bp->band_e = off_e[nsims];
    bp->band_h = off_h[nsims];
    bp->fn = ke->fn_batch[any_zin ? 1 : 0][any_drude ? 1 : 0];
    int nsm = 0, occ = 0;
    const int rs = fused_residency(bp->fn, ke->threads, bp->smem, &nsm, &occ);
    if (rs != FDTD_OK) { delete bp; return rs; }
    if (tile && tile->ctas_per_sm > 0) occ = std::min(occ, (int)tile->ctas_per_sm);
    bp->nblocks = (int)std::min<int64_t>(bp->nitems, (int64_t)nsm * occ);
    *out = bp;
    return FDTD_OK;
}

int fdtd_batch_plan_run(fdtd_batch_plan *bp, int64_t t0, int64_t nsteps, void *stream) {
    if (!bp || nsteps < 0) return FDTD_ERR_ARG;
    cudaStream_t st = as_stream(stream);
    TMaps dummy_maps;
    memset(&dummy_maps, 0, sizeof(dummy_maps));
    Params dummy{};
    for (int64_t n = 0; n < nsteps; n++) {
        NvtxRange nvtx_range("fdtd_batch_step");
        BatchDesc bd{};
        bd.nsims = bp->nsims;
        bd.cur = bp->cur;
        bd.t = t0 + n;
        bd.params = bp->d_params;
        bd.maps = bp->d_maps;
        bd.item_off = bp->d_off;
        bd.queue = bp->d_queue;
        launch_chained(bp->fn, dim3((unsigned)bp->nblocks), dim3((unsigned)bp->k->threads), (size_t)bp->smem, st, 1,
                       dummy_maps, dummy, bd);
        if (bp->band_h > 0) {
            BandBatch d{bp->nsims, bp->cur, t0 + n, bp->d_params, bp->d_off + (bp->nsims + 1)};
            k_zband_batch<true><<<(unsigned)bp->band_e, kBandBlock, 0, st>>>(d);
            d.off += bp->nsims + 1;
            k_zband_batch<false><<<(unsigned)bp->band_h, kBandBlock, 0, st>>>(d);
        }
        FDTD_TRY(check_launch());
        bp->cur = 1 - bp->cur;
    }
    return FDTD_OK;
}

int fdtd_batch_plan_current(const fdtd_batch_plan *bp) { return bp ? bp->cur : -1; }

int fdtd_batch_plan_set_current(fdtd_batch_plan *bp, int32_t cur) {
    if (!bp || (cur != 0 && cur != 1)) return FDTD_ERR_ARG;
    bp->cur = cur;
    return FDTD_OK;
}

int fdtd_batch_plan_info(const fdtd_batch_plan *bp, int32_t *info, int32_t n) {
    if (!bp || !info || n < 6) return FDTD_ERR_ARG;
    info[0] = bp->k->ty;
    info[1] = bp->k->ns;
    info[2] = (int32_t)std::min<int64_t>(bp->nitems, 0x7fffffff);
    info[3] = bp->nblocks;
    info[4] = bp->k->threads;
    info[5] = bp->smem;
    if (n >= 8) {
        info[6] = bp->band_h > 0;
        info[7] = bp->band_h > 0 ? 3 : 1;
    }
    return FDTD_OK;
}

int fdtd_batch_plan_destroy(fdtd_batch_plan *bp) {
    delete bp;
    return FDTD_OK;
}

int fdtd_batched_run_f32(int32_t nsims, const fdtd_grid *grids, const fdtd_yee_state *states,
                         const fdtd_cpml *cpmls, const fdtd_sources *srcs, int32_t *status_dev, void *workspace,
                         size_t workspace_bytes, int32_t cur, int64_t t0, int64_t nsteps, int32_t *cur_out,
                         void *stream) {
    if (nsteps < 0) return FDTD_ERR_ARG;
    fdtd_batch_plan *bp = nullptr;
    FDTD_TRY(fdtd_batch_plan_create(&bp, nsims, grids, states, cpmls, srcs, nullptr, status_dev, workspace,
                                    workspace_bytes, cur, stream));
    const int r = fdtd_batch_plan_run(bp, t0, nsteps, stream);
    if (cur_out) *cur_out = fdtd_batch_plan_current(bp);
    fdtd_batch_plan_destroy(bp);  // the launches read the caller's workspace, not the plan
    return r;
}

}  // extern "C"
