// In-place, reference-shaped kernels: one thread per cell, z-coalesced.
//
// Semantics (index ranges, operation grouping) follow
//   2nd_order-Yee/Numpy/fdtd3d.py:4-37                   (E, H, periodic planes)
//   kuFDTD/v0.2.0/dim3/cpu/core/cpml_non_kappa.c:14-429  (psi recursion, slab ranges)
//   kuFDTD/before_CUDA/v0.3.0/boundary/core/cpml_core.c:238-263 (kappa term)
// Arithmetic uses explicit round-to-nearest intrinsics so results equal the
// FP32 NumPy/C evaluation bit for bit.
#include <initializer_list>

#include "common.cuh"

namespace fdtd {

constexpr int kBlockZ = 128;

// one cell (i, j, k) at offset c
__device__ __forceinline__ void cell_e(const Grid &g, int64_t i, int64_t j, int64_t k, int64_t c, float *ex, float *ey,
                                       float *ez, const float *hx, const float *hy, const float *hz, const float *cex,
                                       const float *cey, const float *cez) {
    if (j < g.ny - 1 && k < g.nz - 1)
        ex[c] = fadd(ex[c], fmul(cex[c], curl4(hz[c + g.sy], hz[c], hy[c + 1], hy[c])));
    if (i < g.nx - 1 && k < g.nz - 1)
        ey[c] = fadd(ey[c], fmul(cey[c], curl4(hx[c + 1], hx[c], hz[c + g.sx], hz[c])));
    if (i < g.nx - 1 && j < g.ny - 1)
        ez[c] = fadd(ez[c], fmul(cez[c], curl4(hy[c + g.sx], hy[c], hx[c + g.sy], hx[c])));
}
__device__ __forceinline__ void cell_h(const Grid &g, int64_t i, int64_t j, int64_t k, int64_t c, const float *ex,
                                       const float *ey, const float *ez, float *hx, float *hy, float *hz,
                                       const float *chx, const float *chy, const float *chz) {
    if (j > 0 && k > 0)
        hx[c] = fsub(hx[c], fmul(chx ? chx[c] : 0.5f, curl4(ez[c], ez[c - g.sy], ey[c], ey[c - 1])));
    if (i > 0 && k > 0)
        hy[c] = fsub(hy[c], fmul(chy ? chy[c] : 0.5f, curl4(ex[c], ex[c - 1], ez[c], ez[c - g.sx])));
    if (i > 0 && j > 0)
        hz[c] = fsub(hz[c], fmul(chz ? chz[c] : 0.5f, curl4(ey[c], ey[c - g.sx], ex[c], ex[c - g.sy])));
}

__global__ void __launch_bounds__(kBlockZ)
k_update_e(Grid g, float *__restrict__ ex, float *__restrict__ ey, float *__restrict__ ez,
           const float *__restrict__ hx, const float *__restrict__ hy, const float *__restrict__ hz,
           const float *__restrict__ cex, const float *__restrict__ cey, const float *__restrict__ cez) {
    const int64_t k = (int64_t)blockIdx.x * kBlockZ + threadIdx.x;
    const int64_t j = blockIdx.y, i = blockIdx.z;
    if (k >= g.nz) return;
    cell_e(g, i, j, k, i * g.sx + j * g.sy + k, ex, ey, ez, hx, hy, hz, cex, cey, cez);
}

__global__ void __launch_bounds__(kBlockZ)
k_update_h(Grid g, const float *__restrict__ ex, const float *__restrict__ ey, const float *__restrict__ ez,
           float *__restrict__ hx, float *__restrict__ hy, float *__restrict__ hz,
           const float *__restrict__ chx, const float *__restrict__ chy, const float *__restrict__ chz) {
    const int64_t k = (int64_t)blockIdx.x * kBlockZ + threadIdx.x;
    const int64_t j = blockIdx.y, i = blockIdx.z;
    if (k >= g.nz) return;
    cell_h(g, i, j, k, i * g.sx + j * g.sy + k, ex, ey, ez, hx, hy, hz, chx, chy, chz);
}

// ---------------------------------------------------------------------------
// The same updates with 4 z cells a thread, for arrays whose rows start on
// 16-byte boundaries (strides of a multiple of 4 floats, aligned bases): every
// access but the one neighbour past the group is 16 bytes wide and all loads
// precede the stores.  One thread a cell keeps too few bytes in flight: on
// 250x250x320 (beyond L2) E 180 us (5.3 TB/s of its 48 bytes a cell) and H 161
// us (4.5 TB/s of 36); this form 131 and 98 (7.3 TB/s, part of it from L2).
// Threads run over the (j, group) pairs of an x plane, so short rows leave no
// lanes idle.
// ---------------------------------------------------------------------------
struct F4 {
    float v[4];
};
__device__ __forceinline__ F4 ld4(const float *p) {
    const float4 t = *reinterpret_cast<const float4 *>(p);
    return F4{{t.x, t.y, t.z, t.w}};
}
// cells lo .. hi-1 of r
__device__ __forceinline__ void st4(float *p, const F4 &r, int lo, int hi) {
    if (lo == 0 && hi == 4) {
        *reinterpret_cast<float4 *>(p) = make_float4(r.v[0], r.v[1], r.v[2], r.v[3]);
    } else {
#pragma unroll
        for (int e = 0; e < 4; e++)
            if (e >= lo && e < hi) p[e] = r.v[e];
    }
}
// (j, first cell) of this thread's group on its plane; false past the end
__device__ __forceinline__ bool group4(const Grid &g, uint32_t ng, uint32_t &j, uint32_t &k) {
    const uint32_t t = blockIdx.x * kBlockZ + threadIdx.x;
    j = t / ng;
    k = 4 * (t - j * ng);
    return j < (uint32_t)g.ny;
}

__global__ void __launch_bounds__(kBlockZ)
k_update_e4(Grid g, uint32_t ng, float *__restrict__ ex, float *__restrict__ ey, float *__restrict__ ez,
            const float *__restrict__ hx, const float *__restrict__ hy, const float *__restrict__ hz,
            const float *__restrict__ cex, const float *__restrict__ cey, const float *__restrict__ cez) {
    uint32_t j, k;
    if (!group4(g, ng, j, k)) return;
    const int64_t i = blockIdx.y, c = i * g.sx + (int64_t)j * g.sy + k;
    const bool jl = j < g.ny - 1, il = i < g.nx - 1;  // rows / planes with a neighbour above
    if (g.nz - k < 4) {  // the ragged end of a row: cell by cell, nothing past it is read
        for (int64_t q = k; q < g.nz; q++) cell_e(g, i, j, q, c + (q - k), ex, ey, ez, hx, hy, hz, cex, cey, cez);
        return;
    }
    const int kl = g.nz - 1 - k < 4 ? 3 : 4;  // cells with k < nz-1
    const int64_t Y = jl ? g.sy : 0, X = il ? g.sx : 0, n = kl == 4 ? 4 : 0;  // (offset 0: loaded, not used)
    const F4 ax = ld4(hx + c), ay = ld4(hy + c), az = ld4(hz + c);
    const F4 xj = ld4(hx + c + Y), zj = ld4(hz + c + Y), yi = ld4(hy + c + X), zi = ld4(hz + c + X);
    const float xk = hx[c + n], yk = hy[c + n];
    F4 rx = ld4(ex + c), ry = ld4(ey + c), rz = ld4(ez + c);
    const F4 cx = ld4(cex + c), cy = ld4(cey + c), cz = ld4(cez + c);
#pragma unroll
    for (int e = 0; e < 4; e++) {
        const float xk1 = e < 3 ? ax.v[e < 3 ? e + 1 : 3] : xk, yk1 = e < 3 ? ay.v[e < 3 ? e + 1 : 3] : yk;
        rx.v[e] = fadd(rx.v[e], fmul(cx.v[e], curl4(zj.v[e], az.v[e], yk1, ay.v[e])));
        ry.v[e] = fadd(ry.v[e], fmul(cy.v[e], curl4(xk1, ax.v[e], zi.v[e], az.v[e])));
        rz.v[e] = fadd(rz.v[e], fmul(cz.v[e], curl4(yi.v[e], ay.v[e], xj.v[e], ax.v[e])));
    }
    if (jl) st4(ex + c, rx, 0, kl);
    if (il) st4(ey + c, ry, 0, kl);
    if (il && jl) st4(ez + c, rz, 0, 4);
}

template <bool CH>
__global__ void __launch_bounds__(kBlockZ)
k_update_h4(Grid g, uint32_t ng, const float *__restrict__ ex, const float *__restrict__ ey,
            const float *__restrict__ ez, float *__restrict__ hx, float *__restrict__ hy, float *__restrict__ hz,
            const float *__restrict__ chx, const float *__restrict__ chy, const float *__restrict__ chz) {
    uint32_t j, k;
    if (!group4(g, ng, j, k)) return;
    const int64_t i = blockIdx.y, c = i * g.sx + (int64_t)j * g.sy + k;
    const bool jg = j > 0, ig = i > 0;
    if (g.nz - k < 4) {
        for (int64_t q = k; q < g.nz; q++) cell_h(g, i, j, q, c + (q - k), ex, ey, ez, hx, hy, hz, chx, chy, chz);
        return;
    }
    const int k0 = k == 0 ? 1 : 0;  // first cell with k > 0
    const int64_t Y = jg ? g.sy : 0, X = ig ? g.sx : 0, n = k0 ? 0 : 1;  // (offset 0: loaded, not used)
    const F4 ax = ld4(ex + c), ay = ld4(ey + c), az = ld4(ez + c);
    const F4 zj = ld4(ez + c - Y), xj = ld4(ex + c - Y), zi = ld4(ez + c - X), yi = ld4(ey + c - X);
    const float xk = ex[c - n], yk = ey[c - n];
    F4 rx = ld4(hx + c), ry = ld4(hy + c), rz = ld4(hz + c);
    F4 cx{{0.5f, 0.5f, 0.5f, 0.5f}}, cy = cx, cz = cx;
    if (CH) {
        cx = ld4(chx + c);
        cy = ld4(chy + c);
        cz = ld4(chz + c);
    }
#pragma unroll
    for (int e = 0; e < 4; e++) {
        const float xk1 = e ? ax.v[e ? e - 1 : 0] : xk, yk1 = e ? ay.v[e ? e - 1 : 0] : yk;
        rx.v[e] = fsub(rx.v[e], fmul(cx.v[e], curl4(az.v[e], zj.v[e], ay.v[e], yk1)));
        ry.v[e] = fsub(ry.v[e], fmul(cy.v[e], curl4(ax.v[e], xk1, az.v[e], zi.v[e])));
        rz.v[e] = fsub(rz.v[e], fmul(cz.v[e], curl4(ay.v[e], yi.v[e], ax.v[e], xj.v[e])));
    }
    if (jg) st4(hx + c, rx, k0, 4);
    if (ig) st4(hy + c, ry, k0, 4);
    if (ig && jg) st4(hz + c, rz, 0, 4);
}

// Periodic planes, fdtd3d.py:16-37.  grid: (ceil(m/128), n_other, 1)
__global__ void k_pbc_plane(Grid g, int axis, int e_or_h, float *f1, float *f2) {
    const int64_t a = (int64_t)blockIdx.x * kBlockZ + threadIdx.x;
    const int64_t b = blockIdx.y;
    int64_t lo, hi;  // offsets of the first and last plane cell
    if (axis == 0) {  // plane (j=b, k=a)
        if (a >= g.nz || b >= g.ny) return;
        lo = b * g.sy + a;
        hi = lo + (g.nx - 1) * g.sx;
    } else if (axis == 1) {  // plane (i=b, k=a)
        if (a >= g.nz || b >= g.nx) return;
        lo = b * g.sx + a;
        hi = lo + (g.ny - 1) * g.sy;
    } else {  // plane (i=b, j=a)
        if (a >= g.ny || b >= g.nx) return;
        lo = b * g.sx + a * g.sy;
        hi = lo + g.nz - 1;
    }
    if (e_or_h == 0) {  // E: last plane <- first plane
        f1[hi] = f1[lo];
        f2[hi] = f2[lo];
    } else {            // H: first plane <- last plane
        f1[lo] = f1[hi];
        f2[lo] = f2[hi];
    }
}

struct CpmlAxis {
    int64_t P;
    int front, back;
    const float *b, *a, *km1;
    float *psi1, *psi2;
};

__device__ __forceinline__ float cpml_term(float &psi, float b, float a, float km1, float d) {
    psi = fadd(fmul(b, psi), fmul(a, d));
    return fadd(fmul(km1, d), psi);
}

// E, x axis: ey -= cey*(...dHz/dx...), ez += cez*(...dHy/dx...)
__global__ void k_cpml_e_x(Grid g, CpmlAxis A, float *ey, float *ez, const float *hy, const float *hz,
                           const float *cey, const float *cez) {
    const int64_t k = (int64_t)blockIdx.x * kBlockZ + threadIdx.x;
    const int64_t j = blockIdx.y, s = blockIdx.z;
    if (k >= g.nz) return;
    if (!(s < A.P ? A.front : A.back)) return;
    const int64_t i = slab_node_e(s, A.P, g.nx);
    const int64_t c = i * g.sx + j * g.sy + k, p = (s * g.ny + j) * g.nz + k;
    const float b = A.b[s], a = A.a[s], km1 = A.km1[s];
    if (k < g.nz - 1) {
        float psi = A.psi1[p];
        float t = cpml_term(psi, b, a, km1, fsub(hz[c + g.sx], hz[c]));
        A.psi1[p] = psi;
        ey[c] = fsub(ey[c], fmul(cey[c], t));
    }
    if (j < g.ny - 1) {
        float psi = A.psi2[p];
        float t = cpml_term(psi, b, a, km1, fsub(hy[c + g.sx], hy[c]));
        A.psi2[p] = psi;
        ez[c] = fadd(ez[c], fmul(cez[c], t));
    }
}

// E, y axis: ez -= cez*(...dHx/dy...), ex += cex*(...dHz/dy...)
__global__ void k_cpml_e_y(Grid g, CpmlAxis A, float *ez, float *ex, const float *hx, const float *hz,
                           const float *cez, const float *cex) {
    const int64_t k = (int64_t)blockIdx.x * kBlockZ + threadIdx.x;
    const int64_t s = blockIdx.y, i = blockIdx.z;
    if (k >= g.nz) return;
    if (!(s < A.P ? A.front : A.back)) return;
    const int64_t j = slab_node_e(s, A.P, g.ny);
    const int64_t c = i * g.sx + j * g.sy + k, p = (i * 2 * A.P + s) * g.nz + k;
    const float b = A.b[s], a = A.a[s], km1 = A.km1[s];
    if (i < g.nx - 1) {
        float psi = A.psi1[p];
        float t = cpml_term(psi, b, a, km1, fsub(hx[c + g.sy], hx[c]));
        A.psi1[p] = psi;
        ez[c] = fsub(ez[c], fmul(cez[c], t));
    }
    if (k < g.nz - 1) {
        float psi = A.psi2[p];
        float t = cpml_term(psi, b, a, km1, fsub(hz[c + g.sy], hz[c]));
        A.psi2[p] = psi;
        ex[c] = fadd(ex[c], fmul(cex[c], t));
    }
}

// E, z axis: ex -= cex*(...dHy/dz...), ey += cey*(...dHx/dz...)
__global__ void k_cpml_e_z(Grid g, CpmlAxis A, float *ex, float *ey, const float *hx, const float *hy,
                           const float *cex, const float *cey) {
    const uint32_t t = blockIdx.x * kBlockZ + threadIdx.x, twoP = 2 * (uint32_t)A.P;  // (j, s) of plane i
    const int64_t j = t / twoP, s = t % twoP, i = blockIdx.y;
    if (j >= g.ny || !(s < A.P ? A.front : A.back)) return;
    const int64_t k = slab_node_e(s, A.P, g.nz);
    const int64_t c = i * g.sx + j * g.sy + k, p = i * g.ny * twoP + t;
    const float b = A.b[s], a = A.a[s], km1 = A.km1[s];
    // loads before stores: a store could alias a later load as far as the compiler
    // knows (with 32-bit cell decoding: E 25.7 -> 20.1, H 23.3 -> 16.8 us at 250x250x320)
    const bool u1 = j < g.ny - 1, u2 = i < g.nx - 1;
    float p1 = 0.f, p2 = 0.f, d1 = 0.f, d2 = 0.f, v1 = 0.f, v2 = 0.f, c1 = 0.f, c2 = 0.f;
    if (u1) {
        p1 = A.psi1[p];
        d1 = fsub(hy[c + 1], hy[c]);
        v1 = ex[c];
        c1 = cex[c];
    }
    if (u2) {
        p2 = A.psi2[p];
        d2 = fsub(hx[c + 1], hx[c]);
        v2 = ey[c];
        c2 = cey[c];
    }
    if (u1) {
        const float tt = cpml_term(p1, b, a, km1, d1);
        A.psi1[p] = p1;
        ex[c] = fsub(v1, fmul(c1, tt));
    }
    if (u2) {
        const float tt = cpml_term(p2, b, a, km1, d2);
        A.psi2[p] = p2;
        ey[c] = fadd(v2, fmul(c2, tt));
    }
}

// H, x axis: hy += ch*(...dEz/dx...), hz -= ch*(...dEy/dx...)
__global__ void k_cpml_h_x(Grid g, CpmlAxis A, float *hy, float *hz, const float *ey, const float *ez,
                           const float *chy, const float *chz) {
    const int64_t k = (int64_t)blockIdx.x * kBlockZ + threadIdx.x;
    const int64_t j = blockIdx.y, s = blockIdx.z;
    if (k >= g.nz) return;
    if (!(s < A.P ? A.front : A.back)) return;
    const int64_t i = slab_node_h(s, A.P, g.nx);
    const int64_t c = i * g.sx + j * g.sy + k, p = (s * g.ny + j) * g.nz + k;
    const float b = A.b[s], a = A.a[s], km1 = A.km1[s];
    if (k > 0) {
        float psi = A.psi1[p];
        float t = cpml_term(psi, b, a, km1, fsub(ez[c], ez[c - g.sx]));
        A.psi1[p] = psi;
        hy[c] = fadd(hy[c], fmul(chy ? chy[c] : 0.5f, t));
    }
    if (j > 0) {
        float psi = A.psi2[p];
        float t = cpml_term(psi, b, a, km1, fsub(ey[c], ey[c - g.sx]));
        A.psi2[p] = psi;
        hz[c] = fsub(hz[c], fmul(chz ? chz[c] : 0.5f, t));
    }
}

// H, y axis: hz += ch*(...dEx/dy...), hx -= ch*(...dEz/dy...)
__global__ void k_cpml_h_y(Grid g, CpmlAxis A, float *hz, float *hx, const float *ex, const float *ez,
                           const float *chz, const float *chx) {
    const int64_t k = (int64_t)blockIdx.x * kBlockZ + threadIdx.x;
    const int64_t s = blockIdx.y, i = blockIdx.z;
    if (k >= g.nz) return;
    if (!(s < A.P ? A.front : A.back)) return;
    const int64_t j = slab_node_h(s, A.P, g.ny);
    const int64_t c = i * g.sx + j * g.sy + k, p = (i * 2 * A.P + s) * g.nz + k;
    const float b = A.b[s], a = A.a[s], km1 = A.km1[s];
    if (i > 0) {
        float psi = A.psi1[p];
        float t = cpml_term(psi, b, a, km1, fsub(ex[c], ex[c - g.sy]));
        A.psi1[p] = psi;
        hz[c] = fadd(hz[c], fmul(chz ? chz[c] : 0.5f, t));
    }
    if (k > 0) {
        float psi = A.psi2[p];
        float t = cpml_term(psi, b, a, km1, fsub(ez[c], ez[c - g.sy]));
        A.psi2[p] = psi;
        hx[c] = fsub(hx[c], fmul(chx ? chx[c] : 0.5f, t));
    }
}

// H, z axis: hx += ch*(...dEy/dz...), hy -= ch*(...dEx/dz...)
__global__ void k_cpml_h_z(Grid g, CpmlAxis A, float *hx, float *hy, const float *ex, const float *ey,
                           const float *chx, const float *chy) {
    const uint32_t t = blockIdx.x * kBlockZ + threadIdx.x, twoP = 2 * (uint32_t)A.P;  // (j, s) of plane i
    const int64_t j = t / twoP, s = t % twoP, i = blockIdx.y;
    if (j >= g.ny || !(s < A.P ? A.front : A.back)) return;
    const int64_t k = slab_node_h(s, A.P, g.nz);
    const int64_t c = i * g.sx + j * g.sy + k, p = i * g.ny * twoP + t;
    const float b = A.b[s], a = A.a[s], km1 = A.km1[s];
    const bool u1 = j > 0, u2 = i > 0;
    float p1 = 0.f, p2 = 0.f, d1 = 0.f, d2 = 0.f, v1 = 0.f, v2 = 0.f, c1 = 0.5f, c2 = 0.5f;
    if (u1) {
        p1 = A.psi1[p];
        d1 = fsub(ey[c], ey[c - 1]);
        v1 = hx[c];
        if (chx) c1 = chx[c];
    }
    if (u2) {
        p2 = A.psi2[p];
        d2 = fsub(ex[c], ex[c - 1]);
        v2 = hy[c];
        if (chy) c2 = chy[c];
    }
    if (u1) {
        const float tt = cpml_term(p1, b, a, km1, d1);
        A.psi1[p] = p1;
        hx[c] = fadd(v1, fmul(c1, tt));
    }
    if (u2) {
        const float tt = cpml_term(p2, b, a, km1, d2);
        A.psi2[p] = p2;
        hy[c] = fsub(v2, fmul(c2, tt));
    }
}

// The x and y slabs with 4 z cells a thread (rows, psi rows and bases on 16-byte
// boundaries): as k_cpml_{e,h}_{x,y}, the pair (f1, g1, c1) first, then (f2, g2,
// c2); E: f1 -= , f2 +=; H: f1 +=, f2 -=.  One cell a thread ran at 4.5 TB/s of
// its 48 bytes (250x250x320, 15 cells: E 26 and H 24 us an axis); this form 16
// and 14 us.
template <bool E, int AX>
__global__ void __launch_bounds__(kBlockZ)
k_cpml_xy4(Grid g, uint32_t ng, CpmlAxis A, float *__restrict__ f1, float *__restrict__ f2,
           const float *__restrict__ g1, const float *__restrict__ g2, const float *__restrict__ c1,
           const float *__restrict__ c2) {
    const uint32_t t = blockIdx.x * kBlockZ + threadIdx.x, r = t / ng;  // row j (x slab) or slab index (y slab)
    const int64_t k = 4 * (int64_t)(t - r * ng);
    if (r >= (AX == 0 ? (uint32_t)g.ny : 2 * (uint32_t)A.P)) return;
    const int64_t s = AX == 0 ? (int64_t)blockIdx.y : (int64_t)r, P = A.P;
    if (!(s < P ? A.front : A.back)) return;
    const int64_t n = AX == 0 ? g.nx : g.ny, node = E ? slab_node_e(s, P, n) : slab_node_h(s, P, n);
    const int64_t i = AX == 0 ? node : (int64_t)blockIdx.y, j = AX == 0 ? (int64_t)r : node;
    const int64_t c = i * g.sx + j * g.sy + k, st = E ? (AX == 0 ? g.sx : g.sy) : -(AX == 0 ? g.sx : g.sy);
    const int64_t p = AX == 0 ? (s * g.ny + j) * g.nz + k : (i * 2 * P + s) * g.nz + k;
    const float b = A.b[s], a = A.a[s], km1 = A.km1[s];
    // cells that a component updates: all but the one at the z edge (lo .. hi-1), or all of the row or none
    const int lo = !E && k == 0 ? 1 : 0, hi = E && k + 4 == g.nz ? 3 : 4;
    const bool row = AX == 0 ? (E ? j < g.ny - 1 : j > 0) : (E ? i < g.nx - 1 : i > 0);
    const bool u1 = AX == 0 || row, u2 = AX == 1 || row;
    const int lo1 = AX == 0 ? lo : 0, hi1 = AX == 0 ? hi : 4, lo2 = AX == 0 ? 0 : lo, hi2 = AX == 0 ? 4 : hi;
    F4 d1{}, d2{}, p1{}, p2{}, v1{}, v2{}, k1{{0.5f, 0.5f, 0.5f, 0.5f}}, k2 = k1;
    auto load = [&](const float *gf, const float *cf, const float *ps, const float *f, F4 &d, F4 &q, F4 &v, F4 &kc) {
        const F4 x = ld4(gf + c), y = ld4(gf + c + st);
#pragma unroll
        for (int e = 0; e < 4; e++) d.v[e] = E ? fsub(y.v[e], x.v[e]) : fsub(x.v[e], y.v[e]);
        if (E || cf) kc = ld4(cf + c);
        q = ld4(ps + p);
        v = ld4(f + c);
    };
    if (u1) load(g1, c1, A.psi1, f1, d1, p1, v1, k1);
    if (u2) load(g2, c2, A.psi2, f2, d2, p2, v2, k2);
#pragma unroll
    for (int e = 0; e < 4; e++) {
        const float t1 = fmul(k1.v[e], cpml_term(p1.v[e], b, a, km1, d1.v[e]));
        const float t2 = fmul(k2.v[e], cpml_term(p2.v[e], b, a, km1, d2.v[e]));
        v1.v[e] = E ? fsub(v1.v[e], t1) : fadd(v1.v[e], t1);
        v2.v[e] = E ? fadd(v2.v[e], t2) : fsub(v2.v[e], t2);
    }
    if (u1) {
        st4(A.psi1 + p, p1, lo1, hi1);
        st4(f1 + c, v1, lo1, hi1);
    }
    if (u2) {
        st4(A.psi2 + p, p2, lo2, hi2);
        st4(f2 + c, v2, lo2, hi2);
    }
}

// Soft sources, sequential in list order (duplicates accumulate in order).
// Drude ADE on the box of d, one thread per box cell (z fastest).
__global__ void __launch_bounds__(kBlockZ)
k_drude_e(Grid g, fdtd_drude d, float *ex, float *ey, float *ez, const float *cex, const float *cey,
          const float *cez) {
    const int64_t t = (int64_t)blockIdx.x * kBlockZ + threadIdx.x;
    if (t >= d.ni * d.nj * d.nk) return;
    const int64_t k = t % d.nk, j = (t / d.nk) % d.nj, i = t / (d.nk * d.nj);
    const int64_t c = (d.i0 + i) * g.sx + (d.j0 + j) * g.sy + d.k0 + k;
    float *E[3] = {ex, ey, ez};
    const float *CE[3] = {cex, cey, cez};
#pragma unroll
    for (int q = 0; q < 3; q++) {
        float jn;
        E[q][c] = drude_cell(E[q][c], CE[q][c], d.j[q][t], d.cja[q][t], d.cjb[q][t], jn);
        d.j[q][t] = jn;
    }
}

__global__ void k_sources(Grid g, fdtd_sources src, int64_t t, float *ex, float *ey, float *ez) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    if (t < 0 || t >= src.namp) return;
    for (int s = 0; s < src.nsrc; s++) {
        const int64_t si = src.ijk[3 * s], sj = src.ijk[3 * s + 1], sk = src.ijk[3 * s + 2];
        if (si < 0 || si >= g.nx || sj < 0 || sj >= g.ny || sk < 0 || sk >= g.nz) continue;
        const int64_t c = si * g.sx + sj * g.sy + sk;
        float *f = src.comp[s] == 0 ? ex : (src.comp[s] == 1 ? ey : ez);
        f[c] = fadd(f[c], src.amp[(int64_t)s * src.namp + t]);
    }
}

static dim3 cell_grid(const Grid &g) {
    return dim3((unsigned)((g.nz + kBlockZ - 1) / kBlockZ), (unsigned)g.ny, (unsigned)g.nx);
}

// 4 cells a thread where rows start on 16-byte boundaries.
static bool rows16(const Grid &g, std::initializer_list<const void *> arrays) {
    if ((g.sx & 3) || (g.sy & 3) || g.ny * ((g.nz + 3) / 4) >= ((int64_t)1 << 31)) return false;
    for (const void *p : arrays)
        if (reinterpret_cast<uintptr_t>(p) & 15) return false;
    return true;
}

static void launch_update_e(const Grid &g, float *ex, float *ey, float *ez, const float *hx, const float *hy,
                            const float *hz, const float *cex, const float *cey, const float *cez, cudaStream_t st) {
    if (rows16(g, {ex, ey, ez, hx, hy, hz, cex, cey, cez})) {
        const uint32_t ng = (uint32_t)((g.nz + 3) / 4);
        const dim3 grid((unsigned)((g.ny * ng + kBlockZ - 1) / kBlockZ), (unsigned)g.nx);
        k_update_e4<<<grid, kBlockZ, 0, st>>>(g, ng, ex, ey, ez, hx, hy, hz, cex, cey, cez);
    } else {
        k_update_e<<<cell_grid(g), kBlockZ, 0, st>>>(g, ex, ey, ez, hx, hy, hz, cex, cey, cez);
    }
}

static void launch_update_h(const Grid &g, const float *ex, const float *ey, const float *ez, float *hx, float *hy,
                            float *hz, const float *chx, const float *chy, const float *chz, cudaStream_t st) {
    const int nch = (chx != nullptr) + (chy != nullptr) + (chz != nullptr);  // (one or two: a mixed call)
    if ((nch == 0 || nch == 3) && rows16(g, {ex, ey, ez, hx, hy, hz, chx, chy, chz})) {
        const uint32_t ng = (uint32_t)((g.nz + 3) / 4);
        const dim3 grid((unsigned)((g.ny * ng + kBlockZ - 1) / kBlockZ), (unsigned)g.nx);
        if (nch) k_update_h4<true><<<grid, kBlockZ, 0, st>>>(g, ng, ex, ey, ez, hx, hy, hz, chx, chy, chz);
        else k_update_h4<false><<<grid, kBlockZ, 0, st>>>(g, ng, ex, ey, ez, hx, hy, hz, chx, chy, chz);
    } else {
        k_update_h<<<cell_grid(g), kBlockZ, 0, st>>>(g, ex, ey, ez, hx, hy, hz, chx, chy, chz);
    }
}

static int validate_cpml(const Grid &g, const fdtd_cpml *c, const fdtd_psi *psi, bool e) {
    if (!c || !psi) return FDTD_ERR_ARG;
    const int64_t n[3] = {g.nx, g.ny, g.nz};
    for (int a = 0; a < 3; a++) {
        const int64_t P = c->npml[a];
        if (P < 0) return FDTD_ERR_ARG;
        if (P == 0) continue;
        if (n[a] < 2 * P + 2) return FDTD_ERR_SHAPE;
        if (a < 2 && 2 * P > 65535) return FDTD_ERR_SHAPE;
        const float *const *tb = e ? c->b_e : c->b_h;
        const float *const *ta = e ? c->a_e : c->a_h;
        const float *const *tk = e ? c->km1_e : c->km1_h;
        float *const *ps = e ? psi->e : psi->h;
        if (!all_nonnull(tb[a], ta[a], tk[a], ps[2 * a], ps[2 * a + 1])) return FDTD_ERR_ARG;
    }
    return FDTD_OK;
}

static CpmlAxis make_axis(const fdtd_cpml *c, const fdtd_psi *psi, int a, bool e) {
    CpmlAxis A;
    A.P = c->npml[a];
    A.front = (c->faces >> (2 * a)) & 1;
    A.back = (c->faces >> (2 * a + 1)) & 1;
    A.b = e ? c->b_e[a] : c->b_h[a];
    A.a = e ? c->a_e[a] : c->a_h[a];
    A.km1 = e ? c->km1_e[a] : c->km1_h[a];
    A.psi1 = e ? psi->e[2 * a] : psi->h[2 * a];
    A.psi2 = e ? psi->e[2 * a + 1] : psi->h[2 * a + 1];
    return A;
}

template <bool E, int AX>
static void launch_cpml_xy4(const Grid &g, const CpmlAxis &A, float *f1, float *f2, const float *g1, const float *g2,
                            const float *c1, const float *c2, cudaStream_t st) {
    const uint32_t ng = (uint32_t)(g.nz / 4);
    const int64_t rows = AX == 0 ? g.ny : 2 * A.P;
    const dim3 grid((unsigned)((rows * ng + kBlockZ - 1) / kBlockZ), (unsigned)(AX == 0 ? 2 * A.P : g.nx));
    k_cpml_xy4<E, AX><<<grid, kBlockZ, 0, st>>>(g, ng, A, f1, f2, g1, g2, c1, c2);
}

static int launch_cpml_e(const Grid &g, const fdtd_cpml *c, const fdtd_psi *psi, float *ex, float *ey,
                         float *ez, const float *hx, const float *hy, const float *hz, const float *cex,
                         const float *cey, const float *cez, cudaStream_t st) {
    const bool v4 = g.nz % 4 == 0 && rows16(g, {ex, ey, ez, hx, hy, hz, cex, cey, cez});
    if (c->npml[0] > 0) {
        CpmlAxis A = make_axis(c, psi, 0, true);
        if (v4 && rows16(g, {A.psi1, A.psi2})) {
            launch_cpml_xy4<true, 0>(g, A, ey, ez, hz, hy, cey, cez, st);
        } else {
            dim3 grid((unsigned)((g.nz + kBlockZ - 1) / kBlockZ), (unsigned)g.ny, (unsigned)(2 * A.P));
            k_cpml_e_x<<<grid, kBlockZ, 0, st>>>(g, A, ey, ez, hy, hz, cey, cez);
        }
    }
    if (c->npml[1] > 0) {
        CpmlAxis A = make_axis(c, psi, 1, true);
        if (v4 && rows16(g, {A.psi1, A.psi2})) {
            launch_cpml_xy4<true, 1>(g, A, ez, ex, hx, hz, cez, cex, st);
        } else {
            dim3 grid((unsigned)((g.nz + kBlockZ - 1) / kBlockZ), (unsigned)(2 * A.P), (unsigned)g.nx);
            k_cpml_e_y<<<grid, kBlockZ, 0, st>>>(g, A, ez, ex, hx, hz, cez, cex);
        }
    }
    if (c->npml[2] > 0) {
        CpmlAxis A = make_axis(c, psi, 2, true);
        const dim3 grid((unsigned)((g.ny * 2 * A.P + kBlockZ - 1) / kBlockZ), (unsigned)g.nx);
        k_cpml_e_z<<<grid, kBlockZ, 0, st>>>(g, A, ex, ey, hx, hy, cex, cey);
    }
    return check_launch();
}

static int launch_cpml_h(const Grid &g, const fdtd_cpml *c, const fdtd_psi *psi, const float *ex,
                         const float *ey, const float *ez, float *hx, float *hy, float *hz, const float *chx,
                         const float *chy, const float *chz, cudaStream_t st) {
    const bool v4 = g.nz % 4 == 0 && rows16(g, {ex, ey, ez, hx, hy, hz, chx, chy, chz});
    if (c->npml[0] > 0) {
        CpmlAxis A = make_axis(c, psi, 0, false);
        if (v4 && rows16(g, {A.psi1, A.psi2})) {
            launch_cpml_xy4<false, 0>(g, A, hy, hz, ez, ey, chy, chz, st);
        } else {
            dim3 grid((unsigned)((g.nz + kBlockZ - 1) / kBlockZ), (unsigned)g.ny, (unsigned)(2 * A.P));
            k_cpml_h_x<<<grid, kBlockZ, 0, st>>>(g, A, hy, hz, ey, ez, chy, chz);
        }
    }
    if (c->npml[1] > 0) {
        CpmlAxis A = make_axis(c, psi, 1, false);
        if (v4 && rows16(g, {A.psi1, A.psi2})) {
            launch_cpml_xy4<false, 1>(g, A, hz, hx, ex, ez, chz, chx, st);
        } else {
            dim3 grid((unsigned)((g.nz + kBlockZ - 1) / kBlockZ), (unsigned)(2 * A.P), (unsigned)g.nx);
            k_cpml_h_y<<<grid, kBlockZ, 0, st>>>(g, A, hz, hx, ex, ez, chz, chx);
        }
    }
    if (c->npml[2] > 0) {
        CpmlAxis A = make_axis(c, psi, 2, false);
        const dim3 grid((unsigned)((g.ny * 2 * A.P + kBlockZ - 1) / kBlockZ), (unsigned)g.nx);
        k_cpml_h_z<<<grid, kBlockZ, 0, st>>>(g, A, hx, hy, ex, ey, chx, chy);
    }
    return check_launch();
}

static int validate_sources(const Grid &g, const fdtd_sources *s) {
    if (!s) return FDTD_ERR_ARG;
    if (s->nsrc < 0 || s->namp < 0) return FDTD_ERR_ARG;
    if (s->nsrc > 0 && !all_nonnull(s->ijk, s->comp, s->amp)) return FDTD_ERR_ARG;
    return FDTD_OK;
}

}  // namespace fdtd

using namespace fdtd;

extern "C" {

int fdtd_update_e_f32(const fdtd_grid *gp, float *ex, float *ey, float *ez, const float *hx, const float *hy,
                      const float *hz, const float *cex, const float *cey, const float *cez, void *stream) {
    Grid g;
    FDTD_TRY(validate_grid(gp, &g));
    if (!all_nonnull(ex, ey, ez, hx, hy, hz, cex, cey, cez)) return FDTD_ERR_ARG;
    launch_update_e(g, ex, ey, ez, hx, hy, hz, cex, cey, cez, as_stream(stream));
    return check_launch();
}

int fdtd_update_h_f32(const fdtd_grid *gp, const float *ex, const float *ey, const float *ez, float *hx,
                      float *hy, float *hz, const float *chx, const float *chy, const float *chz, void *stream) {
    Grid g;
    FDTD_TRY(validate_grid(gp, &g));
    if (!all_nonnull(ex, ey, ez, hx, hy, hz)) return FDTD_ERR_ARG;
    launch_update_h(g, ex, ey, ez, hx, hy, hz, chx, chy, chz, as_stream(stream));
    return check_launch();
}

static int pbc_common(const fdtd_grid *gp, int32_t axes, float *f0, float *f1, float *f2, int e_or_h,
                      void *stream) {
    Grid g;
    FDTD_TRY(validate_grid(gp, &g));
    if (!all_nonnull(f0, f1, f2)) return FDTD_ERR_ARG;
    if (axes & ~7) return FDTD_ERR_ARG;
    cudaStream_t st = as_stream(stream);
    // E: x -> (ey, ez), y -> (ez, ex), z -> (ex, ey); H likewise with h.
    if (axes & 1)
        k_pbc_plane<<<dim3((unsigned)((g.nz + kBlockZ - 1) / kBlockZ), (unsigned)g.ny), kBlockZ, 0, st>>>(
            g, 0, e_or_h, f1, f2);
    if (axes & 2)
        k_pbc_plane<<<dim3((unsigned)((g.nz + kBlockZ - 1) / kBlockZ), (unsigned)g.nx), kBlockZ, 0, st>>>(
            g, 1, e_or_h, f2, f0);
    if (axes & 4)
        k_pbc_plane<<<dim3((unsigned)((g.ny + kBlockZ - 1) / kBlockZ), (unsigned)g.nx), kBlockZ, 0, st>>>(
            g, 2, e_or_h, f0, f1);
    return check_launch();
}

int fdtd_update_pbc_e_f32(const fdtd_grid *g, int32_t axes, float *ex, float *ey, float *ez, void *stream) {
    return pbc_common(g, axes, ex, ey, ez, 0, stream);
}

int fdtd_update_pbc_h_f32(const fdtd_grid *g, int32_t axes, float *hx, float *hy, float *hz, void *stream) {
    return pbc_common(g, axes, hx, hy, hz, 1, stream);
}

int fdtd_cpml_e_f32(const fdtd_grid *gp, const fdtd_cpml *c, float *ex, float *ey, float *ez, const float *hx,
                    const float *hy, const float *hz, const float *cex, const float *cey, const float *cez,
                    const fdtd_psi *psi, void *stream) {
    Grid g;
    FDTD_TRY(validate_grid(gp, &g));
    if (!all_nonnull(ex, ey, ez, hx, hy, hz, cex, cey, cez)) return FDTD_ERR_ARG;
    FDTD_TRY(validate_cpml(g, c, psi, true));
    return launch_cpml_e(g, c, psi, ex, ey, ez, hx, hy, hz, cex, cey, cez, as_stream(stream));
}

int fdtd_cpml_h_f32(const fdtd_grid *gp, const fdtd_cpml *c, const float *ex, const float *ey, const float *ez,
                    float *hx, float *hy, float *hz, const float *chx, const float *chy, const float *chz,
                    const fdtd_psi *psi, void *stream) {
    Grid g;
    FDTD_TRY(validate_grid(gp, &g));
    if (!all_nonnull(ex, ey, ez, hx, hy, hz)) return FDTD_ERR_ARG;
    FDTD_TRY(validate_cpml(g, c, psi, false));
    return launch_cpml_h(g, c, psi, ex, ey, ez, hx, hy, hz, chx, chy, chz, as_stream(stream));
}

int fdtd_add_sources_f32(const fdtd_grid *gp, const fdtd_sources *src, int64_t t, float *ex, float *ey,
                         float *ez, void *stream) {
    Grid g;
    FDTD_TRY(validate_grid(gp, &g));
    if (!all_nonnull(ex, ey, ez)) return FDTD_ERR_ARG;
    FDTD_TRY(validate_sources(g, src));
    if (src->nsrc == 0) return FDTD_OK;
    k_sources<<<1, 32, 0, as_stream(stream)>>>(g, *src, t, ex, ey, ez);
    return check_launch();
}

int fdtd_drude_update_e_f32(const fdtd_grid *gp, const fdtd_drude *d, float *ex, float *ey, float *ez,
                            const float *cex, const float *cey, const float *cez, void *stream) {
    Grid g;
    FDTD_TRY(validate_grid(gp, &g));
    if (!all_nonnull(ex, ey, ez, cex, cey, cez)) return FDTD_ERR_ARG;
    FDTD_TRY(validate_drude(g, d));
    const int64_t n = d->ni * d->nj * d->nk;
    k_drude_e<<<(unsigned)((n + kBlockZ - 1) / kBlockZ), kBlockZ, 0, as_stream(stream)>>>(g, *d, ex, ey, ez, cex,
                                                                                         cey, cez);
    return check_launch();
}

int fdtd_step_unfused_f32(const fdtd_grid *gp, float *const f[6], const float *const ce[3],
                          const float *const ch[3], const fdtd_cpml *c, const fdtd_psi *psi,
                          const fdtd_sources *src, int64_t t, void *stream) {
    NvtxRange nvtx_range("fdtd_step_unfused");
    Grid g;
    FDTD_TRY(validate_grid(gp, &g));
    if (!f || !ce) return FDTD_ERR_ARG;
    if (!all_nonnull(f[0], f[1], f[2], f[3], f[4], f[5], ce[0], ce[1], ce[2])) return FDTD_ERR_ARG;
    const float *chx = ch ? ch[0] : nullptr, *chy = ch ? ch[1] : nullptr, *chz = ch ? ch[2] : nullptr;
    const bool pml = c && (c->npml[0] > 0 || c->npml[1] > 0 || c->npml[2] > 0);
    if (pml) {
        FDTD_TRY(validate_cpml(g, c, psi, true));
        FDTD_TRY(validate_cpml(g, c, psi, false));
    }
    if (src) FDTD_TRY(validate_sources(g, src));
    cudaStream_t st = as_stream(stream);
    launch_update_e(g, f[0], f[1], f[2], f[3], f[4], f[5], ce[0], ce[1], ce[2], st);
    FDTD_TRY(check_launch());
    if (pml) FDTD_TRY(launch_cpml_e(g, c, psi, f[0], f[1], f[2], f[3], f[4], f[5], ce[0], ce[1], ce[2], st));
    if (src && src->nsrc > 0) {
        k_sources<<<1, 32, 0, st>>>(g, *src, t, f[0], f[1], f[2]);
        FDTD_TRY(check_launch());
    }
    launch_update_h(g, f[0], f[1], f[2], f[3], f[4], f[5], chx, chy, chz, st);
    FDTD_TRY(check_launch());
    if (pml) FDTD_TRY(launch_cpml_h(g, c, psi, f[0], f[1], f[2], f[3], f[4], f[5], chx, chy, chz, st));
    return FDTD_OK;
}

}  // extern "C"
