// 4th-order stage on a group of 4 z cells: one thread of the edge kernels
// (symp_pair.cu).
//
// A cell's stage reads 4 values along each of two axes for each component: one
// cell a thread, 24 to 36 scalar loads for 3 results.  A group loads whole
// 16-byte words and the few cells of the neighbouring groups, a third of the
// instructions, and twice to four times the bytes in flight for each thread.
// Measured, 512^3 with a 10-cell CPML, us a pass over its 14.3 Mcells: edge H
// 250 -> 204 (880 MB of DRAM traffic), edge E 256 -> 255 (1120 MB); the step 8475
// -> 8254, 256^3 1414 -> 1373, and on whole small grids (in-place, one cell a
// thread -> edge kernels) 64^3 98 -> 75.  Rows of psi that are no 16-byte
// multiple are read and written one cell at a time, 4 lines an instruction, and
// gain nothing (300x301x303: 2210 and 2213).  As the in-place stage kernel
// (k_symp_stage) the group form was slower, 1714 -> 1865 at 256^3.  With each
// component's results gathered before its stores (Out) 512^3 8142 -> 8096 and 200^3 with 8 cells
// 782 -> 768; 128^3, through plain loads, 266 where the read-only path took 267.
//
// H nodes take a backward stencil (offsets -2 .. 1), E nodes a forward one
// (-1 .. 2); with that, both have the same form.  G: the field that is read.
//   component 0: curl of G2 along y, G1 along z; CPML terms in order y, z
//   component 1: curl of G0 along z, G2 along x; x, z
//   component 2: curl of G1 along x, G0 along y; x, y
#pragma once
#include "common.cuh"

namespace fdtd {
namespace sg {

struct F4 {
    float v[4];
};
// the 4 stencil values of each cell along one axis, in the axis' direction
struct Window {
    F4 a, b, c, d;
};
// CPML tables of one stage along one axis
struct Tab {
    const float *b, *a, *km1;
};

template <bool RO, typename T>
__device__ __forceinline__ T ld1(const T *p) {
    return RO ? __ldg(p) : *p;
}

// slab index of node x of n along an axis with P cells a face, -1 outside
template <bool E>
__device__ __forceinline__ int slab(int P, bool front, bool back, int x, int n) {
    const int b0 = E ? n - P - 1 : n - P, b1 = E ? n - 2 : n - 1;
    int s = -1;
    if (P > 0 && front && x >= 1 && x <= P) s = x - 1;
    if (P > 0 && back && x >= b0 && x <= b1) s = P + x - b0;
    return s;
}

// cells k .. k+3 of row (i, j); k is a multiple of 4, and so are the row and
// plane strides Y and X; n: elements of a field array
struct Group {
    int32_t nx, ny, nz;
    uint32_t X, Y;
    int i, j, k;
    uint32_t c, in;  // offset of cell k; cells inside the grid
    int64_t n;
    __device__ __forceinline__ Group(int nx_, int ny_, int nz_, uint32_t sx, uint32_t sy, int i_, int j_, int k_)
        : nx(nx_), ny(ny_), nz(nz_), X(sx), Y(sy), i(i_), j(j_), k(k_),
          c((uint32_t)i_ * sx + (uint32_t)j_ * sy + (uint32_t)k_), in(k_ + 4 <= nz_ ? 0xFu : (1u << (nz_ - k_)) - 1),
          n((int64_t)nx_ * sx) {}
    // the group at offset at of a field, RO: through the read-only path.  A chained kernel
    // takes plain loads: the launch before may write the field while this one is resident,
    // and the read-only path is for memory that nothing writes in that time.
    template <bool RO>
    __device__ __forceinline__ F4 ldf(const float *f, uint32_t at) const {
        if (!RO) return ld(f, at, in, true, n);
        F4 r{};
        if (in == 0xFu) {
            if (FDTD_IN(at, n) && FDTD_IN(at + 3, n)) {
                const float4 t = ld1<RO>(reinterpret_cast<const float4 *>(f + at));
                r = F4{{t.x, t.y, t.z, t.w}};
            }
        } else {
#pragma unroll
            for (int e = 0; e < 4; e++)
                if (((in >> e) & 1) && FDTD_IN(at + e, n)) r.v[e] = ld1<RO>(f + at + e);
        }
        return r;
    }
    // elements at .. at+3 of a psi array or of the updated field, those of mask m
    __device__ static __forceinline__ F4 ld(const float *f, uint32_t at, uint32_t m, bool vec, int64_t ext) {
        F4 r{};
        if (m == 0xFu && vec) {
            if (FDTD_IN(at, ext) && FDTD_IN(at + 3, ext)) {
                const float4 t = *reinterpret_cast<const float4 *>(f + at);
                r = F4{{t.x, t.y, t.z, t.w}};
            }
        } else {
#pragma unroll
            for (int e = 0; e < 4; e++)
                if (((m >> e) & 1) && FDTD_IN(at + e, ext)) r.v[e] = f[at + e];
        }
        return r;
    }
    __device__ static __forceinline__ void st(float *f, uint32_t at, uint32_t m, bool vec, const F4 &a, int64_t ext) {
        if (m == 0xFu && vec) {
            if (FDTD_IN(at, ext) && FDTD_IN(at + 3, ext))
                *reinterpret_cast<float4 *>(f + at) = make_float4(a.v[0], a.v[1], a.v[2], a.v[3]);
        } else {
#pragma unroll
            for (int e = 0; e < 4; e++)
                if (((m >> e) & 1) && FDTD_IN(at + e, ext)) f[at + e] = a.v[e];
        }
    }
    // stencil along x or y (stride s); the rows must exist
    template <bool E, bool RO>
    __device__ __forceinline__ Window rows(const float *f, uint32_t s) const {
        return E ? Window{ldf<RO>(f, c - s), ldf<RO>(f, c), ldf<RO>(f, c + s), ldf<RO>(f, c + 2 * s)}
                 : Window{ldf<RO>(f, c - 2 * s), ldf<RO>(f, c - s), ldf<RO>(f, c), ldf<RO>(f, c + s)};
    }
    // stencil along z; past either end of the row the values are zeros that no updated cell uses
    template <bool E, bool RO>
    __device__ __forceinline__ Window along_z(const float *f) const {
        const F4 o = ldf<RO>(f, c);
        if (E) {
            const float l = k > 0 && FDTD_IN(c - 1, n) ? ld1<RO>(f + c - 1) : 0.f;
            float r0 = 0.f, r1 = 0.f;
            if (k + 5 < nz) {
                if (FDTD_IN(c + 5, n)) {
                    const float2 t = ld1<RO>(reinterpret_cast<const float2 *>(f + c + 4));
                    r0 = t.x;
                    r1 = t.y;
                }
            } else if (k + 4 < nz && FDTD_IN(c + 4, n)) {
                r0 = ld1<RO>(f + c + 4);
            }
            return Window{{{l, o.v[0], o.v[1], o.v[2]}}, o, {{o.v[1], o.v[2], o.v[3], r0}}, {{o.v[2], o.v[3], r0, r1}}};
        }
        float l0 = 0.f, l1 = 0.f;
        if (k > 0 && FDTD_IN(c - 2, n)) {
            const float2 t = ld1<RO>(reinterpret_cast<const float2 *>(f + c - 2));
            l0 = t.x;
            l1 = t.y;
        }
        const float r = k + 4 < nz && FDTD_IN(c + 4, n) ? ld1<RO>(f + c + 4) : 0.f;
        return Window{{{l0, l1, o.v[0], o.v[1]}}, {{l1, o.v[0], o.v[1], o.v[2]}}, o, {{o.v[1], o.v[2], o.v[3], r}}};
    }
};

// 4th-order difference of a cell: 27 (c - b) - (d - a)
__device__ __forceinline__ float diff4(const Window &w, int e) {
    return fsub(fmul(27.0f, fsub(w.c.v[e], w.b.v[e])), fsub(w.d.v[e], w.a.v[e]));
}

// NST stages in a row (they read the same G; psi is carried from one to the next).  Ctx:
//   fin(q), fout(q), g(q)   updated field (input, output), read field
//   psi_in(n), psi_out(n)   psi array n (two an axis), vpsi: its x, y rows are 16-byte multiples
//   P(ax), front(ax), back(ax), tab(st, ax), coef(st)
//   cv(q, grp)              coefficient of the cells
//   main(st, v, cv, d27)    the stage's main term
//   RO                      fields that are only read go through the read-only path
//   SPLIT                   the thread advances component `only`, else all three
template <bool E, int NST, class Ctx>
__device__ __forceinline__ void stage(const Group &g, const Ctx &x, int only) {
    auto inside = [](int v, int n) { return E ? v > 0 && v < n - 2 : v > 1 && v < n - 1; };
    const bool iin = inside(g.i, g.nx), jin = inside(g.j, g.ny);
    const int sx = slab<E>(x.P(0), x.front(0), x.back(0), g.i, g.nx);
    const int sy = slab<E>(x.P(1), x.front(1), x.back(1), g.j, g.ny);
    int sz[4];
    uint32_t km = 0, zm = 0;
#pragma unroll
    for (int e = 0; e < 4; e++) {
        km |= (uint32_t)(((g.in >> e) & 1) && inside(g.k + e, g.nz)) << e;
        sz[e] = slab<E>(x.P(2), x.front(2), x.back(2), g.k + e, g.nz);
        zm |= (uint32_t)(sz[e] >= 0) << e;
    }
    const uint32_t px = ((uint32_t)(sx >= 0 ? sx : 0) * g.ny + g.j) * g.nz + g.k;
    const uint32_t py = ((uint32_t)g.i * 2u * x.P(1) + (sy >= 0 ? sy : 0)) * g.nz + g.k;
    const uint32_t pz = ((uint32_t)g.i * g.ny + g.j) * 2u * x.P(2);
    const int64_t nx2 = 2LL * x.P(0) * g.ny * g.nz, ny2 = 2LL * x.P(1) * g.nx * g.nz, nz2 = 2LL * x.P(2) * g.nx * g.ny;
    auto pmask = [&](int ax, uint32_t upd) { return ax == 0 ? (sx >= 0 ? upd : 0u) : ax == 1 ? (sy >= 0 ? upd : 0u) : upd & zm; };
    auto pload = [&](int ax, int a, uint32_t m) {
        const float *f = x.psi_in(a);
        if (ax == 0) return Group::ld(f, px, m, x.vpsi(), nx2);
        if (ax == 1) return Group::ld(f, py, m, x.vpsi(), ny2);
        F4 r{};
#pragma unroll
        for (int e = 0; e < 4; e++)
            if (((m >> e) & 1) && FDTD_IN(pz + sz[e], nz2)) r.v[e] = f[pz + sz[e]];
        return r;
    };
    auto pstore = [&](int ax, int a, uint32_t m, const F4 &v) {
        float *f = x.psi_out(a);
        if (ax == 0) Group::st(f, px, m, x.vpsi(), v, nx2);
        else if (ax == 1) Group::st(f, py, m, x.vpsi(), v, ny2);
        else
#pragma unroll
            for (int e = 0; e < 4; e++)
                if (((m >> e) & 1) && FDTD_IN(pz + sz[e], nz2)) f[pz + sz[e]] = v.v[e];
    };
    // psi <- b psi + a d; v +- (coef cv) (km1 d + psi), on the cells m of one axis' slab
    auto term = [&](int st, int ax, uint32_t m, F4 &v, F4 &psi, const Window &w, const F4 &cv, bool add) {
        if (!m) return;
        const Tab T = x.tab(st, ax);
        float b = 0.f, a = 0.f, km1 = 0.f;
        if (ax != 2) {
            const int s = ax == 0 ? sx : sy;
            b = __ldg(T.b + s);
            a = __ldg(T.a + s);
            km1 = __ldg(T.km1 + s);
        }
#pragma unroll
        for (int e = 0; e < 4; e++) {
            if (!((m >> e) & 1)) continue;
            if (ax == 2) {
                b = __ldg(T.b + sz[e]);
                a = __ldg(T.a + sz[e]);
                km1 = __ldg(T.km1 + sz[e]);
            }
            const float d = diff4(w, e);
            psi.v[e] = fadd(fmul(b, psi.v[e]), fmul(a, d));
            const float t = fmul(fmul(x.coef(st), cv.v[e]), fadd(fmul(km1, d), psi.v[e]));
            v.v[e] = add ? fadd(v.v[e], t) : fsub(v.v[e], t);
        }
    };
    // component q from windows p and w (curl of p minus curl of w); CPML terms of the axes ax1
    // (window w1, psi array a1, added when add1) and then ax2
    struct Out {
        F4 v, s1, s2;
        uint32_t m1, m2;
    };
    auto comp = [&](int q, uint32_t upd, const Window &p, const Window &w, int ax1, int a1, const Window &w1, bool add1,
                    int ax2, int a2, const Window &w2) {
        Out o{Group::ld(x.fin(q), g.c, g.in, true, g.n), F4{}, F4{}, pmask(ax1, upd), pmask(ax2, upd)};
        const F4 cv = x.cv(q, g);
        if (o.m1) o.s1 = pload(ax1, a1, o.m1);
        if (o.m2) o.s2 = pload(ax2, a2, o.m2);
        F4 d27;
#pragma unroll
        for (int e = 0; e < 4; e++)
            d27.v[e] = fsub(fmul(27.0f, curl4(p.c.v[e], p.b.v[e], w.c.v[e], w.b.v[e])),
                            curl4(p.d.v[e], p.a.v[e], w.d.v[e], w.a.v[e]));
#pragma unroll
        for (int st = 0; st < NST; st++) {
#pragma unroll
            for (int e = 0; e < 4; e++)
                if ((upd >> e) & 1) o.v.v[e] = x.main(st, o.v.v[e], cv.v[e], d27.v[e]);
            term(st, ax1, o.m1, o.v, o.s1, w1, cv, add1);
            term(st, ax2, o.m2, o.v, o.s2, w2, cv, !add1);
        }
        return o;
    };
    auto copy = [&](int q) { return Out{Group::ld(x.fin(q), g.c, g.in, true, g.n), F4{}, F4{}, 0u, 0u}; };
    auto store = [&](int q, const Out &o, int ax1, int a1, int ax2, int a2) {
        if (o.m1) pstore(ax1, a1, o.m1, o.s1);
        if (o.m2) pstore(ax2, a2, o.m2, o.s2);
        Group::st(x.fout(q), g.c, g.in, true, o.v, g.n);
    };
    auto mine = [&](int q) { return !Ctx::SPLIT || only == q; };
    Out o;
    if (mine(0)) {
        if (jin && km) {
            const Window p = g.template rows<E, Ctx::RO>(x.g(2), g.Y), w = g.template along_z<E, Ctx::RO>(x.g(1));
            o = comp(0, km, p, w, 1, 3, p, E, 2, 4, w);
        } else {
            o = copy(0);
        }
        store(0, o, 1, 3, 2, 4);
    }
    if (mine(1)) {
        if (iin && km) {
            const Window p = g.template along_z<E, Ctx::RO>(x.g(0)), w = g.template rows<E, Ctx::RO>(x.g(2), g.X);
            o = comp(1, km, p, w, 0, 0, w, !E, 2, 5, p);
        } else {
            o = copy(1);
        }
        store(1, o, 0, 0, 2, 5);
    }
    if (mine(2)) {
        if (iin && jin) {
            const Window p = g.template rows<E, Ctx::RO>(x.g(1), g.X), w = g.template rows<E, Ctx::RO>(x.g(0), g.Y);
            o = comp(2, g.in, p, w, 0, 1, p, E, 1, 2, w);
        } else {
            o = copy(2);
        }
        store(2, o, 0, 1, 1, 2);
    }
}

}  // namespace sg
}  // namespace fdtd
