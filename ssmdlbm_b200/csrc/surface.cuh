// surface.cuh — boundary kernels.
//
// The reference applies, after its four bulk kernels and in this order
// (src/main.cu:165-169): water inflow at y = 0, oil inflow at z = 0, outflow
// at y = ny-1, outflow at z = nz-1, copy-periodic x.  Each writes
// post-stream population slots whose source cell is a ghost cell; in pull
// layout those slots live in the ghost cell itself, so every kernel here
// writes ghost-cell slots of the destination buffer only.  The kernels keep
// the reference's order because later ones read what earlier ones wrote
// (outflow z reads u on the y = ny-1 face, copy-periodic x copies slots and
// phi written by the outflows, copy-periodic y reads the x ghosts).
#pragma once

#include "common.cuh"
#include "noise.h"

namespace ssmd {

// Velocity c and weight of one direction, for code that picks it at run time.
struct Dir {
    float cx, cy, cz, w;
    int ix, iy, iz; // the same components as integers
};

constexpr uint64_t pack_axis(int axis) { // 2 bits per direction: c + 1
    uint64_t v = 0;
    for (int q = 0; q < 27; ++q)
        v |= (uint64_t)((axis == 0 ? cx27(q) : (axis == 1 ? cy27(q) : cz27(q))) + 1) << (2 * q);
    return v;
}

template <int Q>
__device__ __forceinline__ Dir direction(int q) {
    constexpr uint64_t X = pack_axis(0), Y = pack_axis(1), Z = pack_axis(2);
    Dir d;
    d.ix = (int)((X >> (2 * q)) & 3u) - 1;
    d.iy = (int)((Y >> (2 * q)) & 3u) - 1;
    d.iz = (int)((Z >> (2 * q)) & 3u) - 1;
    d.cx = float(d.ix);
    d.cy = float(d.iy);
    d.cz = float(d.iz);
    d.w = q == 0 ? VS<Q>::w(0) : (q <= 6 ? VS<Q>::w1 : (q <= 18 ? VS<Q>::w2 : VS<Q>::w3));
    return d;
}

// The boundary values' arithmetic is written out, one rounding per operation: a
// `a * b + c` left to the compiler is fused in an order that depends on what is
// constant around it, and a last bit at the inlet grows in the liquid column.  Which
// product of a sum of two enters fused (the other one is rounded first) is
// therefore a rule on the direction: these are the bits of direction-by-direction code
// with constant c.
__device__ __forceinline__ float two_products(float a, float x, float b, float y, bool second_fused) {
    return fmaf(second_fused ? b : a, second_fused ? y : x,
                __fmul_rn(second_fused ? a : b, second_fused ? x : y));
}

// Shifted equilibrium of direction d (D3Q19.cuh:133-140, D3Q27.cuh:147-154).
template <int Q>
__device__ __forceinline__ float feq_of(const Dir &d, float rho, float ux, float uy, float uz) {
    const float u2 = fmaf(uz, uz, fmaf(ux, ux, __fmul_rn(uy, uy)));
    const float uu = __fmul_rn(1.5f, u2);
    const float cu = __fmul_rn(3.0f, fmaf(d.cz, uz, fmaf(d.cx, ux, __fmul_rn(d.cy, uy))));
    float b = Q == 27 ? __fsub_rn(1.0f, uu) : fmaf(-1.5f, u2, 1.0f);
    b = fmaf(__fmul_rn(0.5f, cu), cu, __fadd_rn(b, cu));
    if constexpr (Q == 27) {
        const float cu3 = __fmul_rn(__fmul_rn(cu, cu), cu);
        b = __fadd_rn(b, fmaf(cu3, float(1.0 / 6.0), -__fmul_rn(uu, cu)));
    }
    return fmaf(__fmul_rn(d.w, rho), b, -d.w);
}

template <int Q, int q>
__device__ __forceinline__ float feq_dir(float rho, float ux, float uy, float uz) {
    constexpr Dir d{float(cx27(q)), float(cy27(q)), float(cz27(q)), VS<Q>::w(q), cx27(q), cy27(q), cz27(q)};
    return feq_of<Q>(d, rho, ux, uy, uz);
}

// Hermite non-equilibrium of direction d (D3Q19.cuh:142-161, D3Q27.cuh:156-185).
template <int Q>
__device__ __forceinline__ float fneq_of(const Dir &d, float pxx, float pyy, float pzz, float pxy, float pxz,
                                         float pyz, float ux, float uy, float uz) {
    const float cx = d.cx, cy = d.cy, cz = d.cz; // -1, 0, 1: products with them are exact
    const float kx = cx * cx - kCs2, ky = cy * cy - kCs2, kz = cz * cz - kCs2;
    float h = fmaf(kz, pzz, two_products(kx, pxx, ky, pyy, d.ix == 0 && d.iy != 0));
    h = fmaf(2.0f, fmaf(cy * cz, pyz, fmaf(cx * cz, pxz, __fmul_rn(cx * cy, pxy))), h);
    if constexpr (Q == 27) {
        const float ux2 = 2.0f * ux, uy2 = 2.0f * uy, uz2 = 2.0f * uz;
        const float c0 = kx * cy, c1 = kx * cz;
        float s = two_products(c0, fmaf(ux2, pxy, __fmul_rn(pxx, uy)), c1, fmaf(ux2, pxz, __fmul_rn(pxx, uz)),
                               c0 < 0.0f && c1 > 0.0f);
        s = fmaf(ky * cx, fmaf(pyy, ux, __fmul_rn(uy2, pxy)), s);
        s = fmaf(ky * cz, fmaf(uy2, pyz, __fmul_rn(pyy, uz)), s);
        s = fmaf(kz * cx, fmaf(pzz, ux, __fmul_rn(uz2, pxz)), s);
        s = fmaf(kz * cy, fmaf(pzz, uy, __fmul_rn(uz2, pyz)), s);
        const float c6 = 6.0f * (cx * cy * cz);
        const float t = fmaf(uz, pxy, fmaf(ux, pyz, __fmul_rn(uy, pxz)));
        h = __fadd_rn(h, two_products(3.0f, s, c6, t, c6 > 0.0f));
    }
    return __fmul_rn(__fmul_rn(d.w, 4.5f), h);
}

__device__ __forceinline__ bool in_range(int v, int lo, int hi) { return v >= lo && v <= hi; }

// Oil inlet speed u_oil (1 + a N(seed, step, cell)), rounded step by step
// (no contraction) so that host code evaluating the same expression in FP32
// gets the same bits.
__device__ __forceinline__ float inlet_speed(const Physics &P, unsigned long long step, uint32_t cell) {
    const float n = float(ssmd_noise::gaussian(P.seed, step, cell, 0u));
    return __fmul_rn(P.u_oil, __fadd_rn(1.0f, __fmul_rn(P.noise_amp, n)));
}

// How the boundary launches are split.  A face has few cells and, with one
// thread per face cell doing every direction, a launch was ~700 instructions of
// straight-line code run once by a handful of warps, each direction's loads
// behind the store of the one before: 4-5 us of fetches and round trips whatever
// the lattice, 26 us for the x copies, whose every access is a sector of its
// own (101 x 75 x 203 crossflow, D3Q27 F16_G32: 45 us a step in five launches, 21
// in three as below; 64 x 64 x 128 jet 5.0 -> 3.0 us).  So every (face cell, population slot) has a thread of its own, the
// direction is picked at run time (the code is a ninth), and the two faces of an
// axis share a launch: inflow writes ghost plane 0 and reads plane 1, outflow
// writes plane n - 1 and reads plane n - 2 (axes with jets have n >= 6), so neither
// reads what the other writes.  The reference's order (above) is kept by pairs,
// (water inflow, outflow y) before (oil inflow, outflow z): oil inflow reads
// fluid cells only and writes plane z = 0, outflow y reads and writes at fluid
// z, so these two may change places.
constexpr int kFaceX = 32, kFaceY = 4; // a block's face cells
// population slots of a face (directions that leave it, then the macroscopic fields
// with the g slot) and of a copy pair (directions with a component along the axis, g,
// the fields)
template <int Q>
constexpr int kFaceDirs = Q == 27 ? 9 : 5;

// The directions whose component along `axis` is s (or, s = 0, is not zero), 5 bits each.
constexpr int axis_of(int axis, int q) { return axis == 0 ? cx27(q) : (axis == 1 ? cy27(q) : cz27(q)); }
template <int Q>
constexpr uint64_t face_list(int axis, int s) {
    uint64_t v = 0;
    int n = 0;
    for (int q = 0; q < Q; ++q)
        if (axis_of(axis, q) == s) v |= (uint64_t)q << (5 * n++);
    return v;
}

// Regularized inflow / outflow value of direction d for a ghost cell:
// f = f_eq(rho_b, u_b) + omco f_neq(Pi(fn), u(fn)) at fluid node fn.
template <int Q>
__device__ __forceinline__ float regularized(const Fields &F, const Dir &d, uint32_t fn, float rho, float ux, float uy,
                                             float uz, float omco) {
    const float feq = feq_of<Q>(d, rho, ux, uy, uz);
    const float fneq = fneq_of<Q>(d, F.pxx[fn], F.pyy[fn], F.pzz[fn], F.pxy[fn], F.pxz[fn], F.pyz[fn], F.ux[fn],
                                  F.uy[fn], F.uz[fn]);
    return fmaf(omco, fneq, feq);
}

// phi and u of the ghost pair (gL, gR) from the fluid cells (bR, bL) they repeat.
__device__ __forceinline__ void copy_ghost_fields(const Fields &F, uint32_t gL, uint32_t bR, uint32_t gR,
                                                  uint32_t bL) {
    const float p0 = F.phi[bR], p1 = F.phi[bL], x0 = F.ux[bR], x1 = F.ux[bL];
    const float y0 = F.uy[bR], y1 = F.uy[bL], z0 = F.uz[bR], z1 = F.uz[bL];
    F.phi[gL] = p0;
    F.phi[gR] = p1;
    F.ux[gL] = x0;
    F.ux[gR] = x1;
    F.uy[gL] = y0;
    F.uy[gR] = y1;
    F.uz[gL] = z0;
    F.uz[gR] = z1;
}

// Water inflow disc on y = 0 (BoundaryConditions.cuh:36-99).  Thread (x, z), slot k.
template <int Q, class TF, class TG>
__device__ __forceinline__ void bc_water_inflow_at(const StepArgs<TF, TG> &a, const int x, const int z, const int k) {
    const Geometry &G = a.geo;
    const Physics &P = a.phys;
    if (x >= (int)G.nx || z >= (int)G.nz) return;
    const float dx = float(x) - P.water_cx, dz = float(z) - P.water_cz;
    if (dx * dx + dz * dz > P.water_r2) return;
    const uint32_t b = cell_index(G, x, 0, z);
    const float uw = P.u_water;
    if (k == kFaceDirs<Q>) {
        a.fld.rho[b] = 1.0f;
        a.fld.phi[b] = 0.0f;
        a.fld.ux[b] = 0.0f;
        a.fld.uy[b] = uw;
        a.fld.uz[b] = 0.0f;
        Store<TG>::st(a.g_dst + slot(G, 3, b), 0.0f); // w_3 * phi (1 + 4 u_y) with phi = 0
        return;
    }
    const int q = (int)((face_list<Q>(1, 1) >> (5 * k)) & 31u);
    const Dir d = direction<Q>(q);
    const int xx = axis_nb(x + d.ix, G.nx, G.bcx == BC_PERIODIC);
    const int zz = axis_nb(z + d.iz, G.nz, G.bcz == BC_PERIODIC);
    if (xx < 0 || zz < 0) return; // outside the lattice (the reference reads out of bounds)
    Store<TF>::st(a.f_dst + slot(G, q, b),
                  regularized<Q>(a.fld, d, cell_index(G, xx, 1, zz), 1.0f, 0.0f, uw, 0.0f, P.omco_water));
}

// Oil inflow disc on z = 0 (BoundaryConditions.cuh:101-168).  Thread (x, y), slot k.
template <int Q, class TF, class TG>
__device__ __forceinline__ void bc_oil_inflow_at(const StepArgs<TF, TG> &a, const int x, const int y, const int k) {
    const Geometry &G = a.geo;
    const Physics &P = a.phys;
    if (x >= (int)G.nx || y >= (int)G.ny) return;
    const float dx = float(x) - P.oil_cx, dy = float(y) - P.oil_cy;
    if (dx * dx + dy * dy > P.oil_r2) return;
    const uint32_t b = cell_index(G, x, y, 0);
    float uin = P.u_oil;
    if (P.noise_amp != 0.0f) {
        uin = inlet_speed(P, a.status->step, b);
    }
    if (k == kFaceDirs<Q>) {
        a.fld.rho[b] = 1.0f;
        a.fld.phi[b] = 1.0f;
        a.fld.ux[b] = 0.0f;
        a.fld.uy[b] = 0.0f;
        a.fld.uz[b] = uin;
        Store<TG>::st(a.g_dst + slot(G, 5, b), kW7_1 * 1.0f * (1.0f + 4.0f * uin));
        return;
    }
    const int q = (int)((face_list<Q>(2, 1) >> (5 * k)) & 31u);
    const Dir d = direction<Q>(q);
    const int xx = axis_nb(x + d.ix, G.nx, G.bcx == BC_PERIODIC);
    const int yy = axis_nb(y + d.iy, G.ny, G.bcy == BC_PERIODIC);
    if (xx < 0 || yy < 0 || !in_range(xx, G.x_lo, G.x_hi) || !in_range(yy, G.y_lo, G.y_hi)) return;
    Store<TF>::st(a.f_dst + slot(G, q, b),
                  regularized<Q>(a.fld, d, cell_index(G, xx, yy, 1), 1.0f, 0.0f, 0.0f, uin, P.omco_oil));
}

// Outflow on y = ny-1 (BoundaryConditions.cuh:170-233).  Thread (x, z), slot k.
template <int Q, class TF, class TG>
__device__ __forceinline__ void bc_outflow_y_at(const StepArgs<TF, TG> &a, const int x, const int z, const int k) {
    const Geometry &G = a.geo;
    if (!in_range(x, G.x_lo, G.x_hi) || !in_range(z, G.z_lo, G.z_hi)) return;
    const uint32_t b = cell_index(G, x, G.ny - 1, z);
    const uint32_t i1 = cell_index(G, x, G.ny - 2, z);
    const Fields &F = a.fld;
    const float ux = F.ux[i1], uy = F.uy[i1], uz = F.uz[i1], rho = F.rho[i1];
    if (k == kFaceDirs<Q>) {
        const float phi = F.phi[i1];
        F.rho[b] = rho;
        F.phi[b] = phi;
        F.ux[b] = ux;
        F.uy[b] = uy;
        F.uz[b] = uz;
        Store<TG>::st(a.g_dst + slot(G, 4, b), kW7_1 * phi * (1.0f - 4.0f * uy));
        return;
    }
    const int q = (int)((face_list<Q>(1, -1) >> (5 * k)) & 31u);
    const Dir d = direction<Q>(q);
    const int xx = axis_nb(x + d.ix, G.nx, G.bcx == BC_PERIODIC);
    const int zz = axis_nb(z + d.iz, G.nz, G.bcz == BC_PERIODIC);
    if (xx < 0 || zz < 0 || !in_range(xx, G.x_lo, G.x_hi) || !in_range(zz, G.z_lo, G.z_hi)) return;
    Store<TF>::st(a.f_dst + slot(G, q, b),
                  regularized<Q>(F, d, cell_index(G, xx, G.ny - 2, zz), rho, ux, uy, uz, a.phys.omco_ref));
}

// Outflow on z = nz-1 (BoundaryConditions.cuh:235-293).  Thread (x, y), slot k.
template <int Q, class TF, class TG>
__device__ __forceinline__ void bc_outflow_z_at(const StepArgs<TF, TG> &a, const int x, const int y, const int k) {
    const Geometry &G = a.geo;
    if (!in_range(x, G.x_lo, G.x_hi) || !in_range(y, G.y_lo, G.y_hi)) return;
    const uint32_t b = cell_index(G, x, y, G.nz - 1);
    const uint32_t i1 = cell_index(G, x, y, G.nz - 2);
    const Fields &F = a.fld;
    const float ux = F.ux[i1], uy = F.uy[i1], uz = F.uz[i1], rho = F.rho[i1];
    if (k == kFaceDirs<Q>) {
        const float phi = F.phi[i1];
        F.rho[b] = rho;
        F.phi[b] = phi;
        F.ux[b] = ux;
        F.uy[b] = uy;
        F.uz[b] = uz;
        Store<TG>::st(a.g_dst + slot(G, 6, b), kW7_1 * phi * (1.0f - 4.0f * uz));
        return;
    }
    const int q = (int)((face_list<Q>(2, -1) >> (5 * k)) & 31u);
    const Dir d = direction<Q>(q);
    // no fluid-range check here, as in the reference (ghost nodes allowed)
    const int xx = axis_nb(x + d.ix, G.nx, G.bcx == BC_PERIODIC);
    const int yy = axis_nb(y + d.iy, G.ny, G.bcy == BC_PERIODIC);
    if (xx < 0 || yy < 0) return;
    Store<TF>::st(a.f_dst + slot(G, q, b),
                  regularized<Q>(F, d, cell_index(G, xx, yy, G.nz - 2), rho, ux, uy, uz, a.phys.omco_ref));
}

// Copy-periodic x (BoundaryConditions.cuh:295-349).  Thread (y, z), all y, z; slot k.
// Push slot (1, y, z) <- (nx-2, y, z) for c_x > 0 is pull slot
// (0, y-c_y, z-c_z) <- (nx-3, y-c_y, z-c_z); c_x < 0 likewise with
// (nx-1, .) <- (2, .).  Slots whose pull home leaves the lattice are never
// read by a fluid cell and are skipped.
template <int Q, class TF, class TG>
__device__ __forceinline__ void bc_copy_x_at(const StepArgs<TF, TG> &a, const int y, const int z, const int k) {
    const Geometry &G = a.geo;
    if (y >= (int)G.ny || z >= (int)G.nz) return;
    const int nx = G.nx;
    constexpr int D = kFaceDirs<Q>;
    if (k < 2 * D) {
        const int q = (int)(((k < D ? face_list<Q>(0, 1) : face_list<Q>(0, -1)) >> (5 * (k < D ? k : k - D))) & 31u);
        const Dir d = direction<Q>(q);
        const int hy = axis_nb(y - d.iy, G.ny, G.bcy == BC_PERIODIC), hz = axis_nb(z - d.iz, G.nz, G.bcz == BC_PERIODIC);
        if (hy < 0 || hz < 0) return;
        const int to = k < D ? 0 : nx - 1;
        const int from = k < D ? nx - 3 : 2;
        TF *f = a.f_dst;
        f[slot(G, q, cell_index(G, to, hy, hz))] = f[slot(G, q, cell_index(G, from, hy, hz))];
        return;
    }
    const uint32_t gL = cell_index(G, 0, y, z), gR = cell_index(G, nx - 1, y, z);
    if (k == 2 * D) {
        TG *g = a.g_dst;
        const TG v1 = g[slot(G, 1, cell_index(G, nx - 3, y, z))], v2 = g[slot(G, 2, cell_index(G, 2, y, z))];
        g[slot(G, 1, gL)] = v1;
        g[slot(G, 2, gR)] = v2;
        return;
    }
    const uint32_t bL = cell_index(G, 1, y, z), bR = cell_index(G, nx - 2, y, z);
    copy_ghost_fields(a.fld, gL, bR, gR, bL);
}

// Copy-periodic y: the same rule as copy-periodic x applied to y (the
// reference only has the x version; this completes the x,y-periodic jet box).
// Thread (x, z), all x, z; slot k.
template <int Q, class TF, class TG>
__device__ __forceinline__ void bc_copy_y_at(const StepArgs<TF, TG> &a, const int x, const int z, const int k) {
    const Geometry &G = a.geo;
    if (x >= (int)G.nx || z >= (int)G.nz) return;
    const int ny = G.ny;
    constexpr int D = kFaceDirs<Q>;
    if (k < 2 * D) {
        const int q = (int)(((k < D ? face_list<Q>(1, 1) : face_list<Q>(1, -1)) >> (5 * (k < D ? k : k - D))) & 31u);
        const Dir d = direction<Q>(q);
        const int hx = axis_nb(x - d.ix, G.nx, G.bcx == BC_PERIODIC), hz = axis_nb(z - d.iz, G.nz, G.bcz == BC_PERIODIC);
        if (hx < 0 || hz < 0) return;
        const int to = k < D ? 0 : ny - 1;
        const int from = k < D ? ny - 3 : 2;
        TF *f = a.f_dst;
        f[slot(G, q, cell_index(G, hx, to, hz))] = f[slot(G, q, cell_index(G, hx, from, hz))];
        return;
    }
    const uint32_t gL = cell_index(G, x, 0, z), gR = cell_index(G, x, ny - 1, z);
    if (k == 2 * D) {
        TG *g = a.g_dst;
        const TG v3 = g[slot(G, 3, cell_index(G, x, ny - 3, z))], v4 = g[slot(G, 4, cell_index(G, x, 2, z))];
        g[slot(G, 3, gL)] = v3;
        g[slot(G, 4, gR)] = v4;
        return;
    }
    const uint32_t bL = cell_index(G, x, 1, z), bR = cell_index(G, x, ny - 2, z);
    copy_ghost_fields(a.fld, gL, bR, gR, bL);
}

// ---- launches ------------------------------------------------------------------
enum : int { BK_JET_Y = 0, BK_JET_Z, BK_COPY_X, BK_COPY_Y };

// Faces of a launch, and slots of each.
template <int K>
constexpr int kFaces = K == BK_JET_Y || K == BK_JET_Z ? 2 : 1;
template <int Q, int K>
constexpr int kSlots = K == BK_JET_Y || K == BK_JET_Z ? kFaceDirs<Q> + 1 : 2 * kFaceDirs<Q> + 2;

// Grid of one boundary launch over faces of at most n0 x n1 cells of `count`
// lattices: blocks of kFaceX x kFaceY face cells, blockIdx.x the tiles along the
// first axis times the slots of the faces.  (Several slots per thread in a loop, so
// that all blocks of a large face are resident at once, lost to the round trips
// that then follow one another: 256 x 256 face 5.6 -> 7.4 us, crossflow 21 -> 26.  The one
// loss: three 128 x 128 x 512 D3Q27 FP32 jets on streams of their own, whose bulk blocks
// fill every SM, take 484 us for each step instead of 480; one alone in a replayed graph
// takes 450 instead of 456.  One thread per cell there brought the 484 to 481 and the 450
// to 459.)
template <int Q, int K>
inline dim3 face_grid(uint32_t n0, uint32_t n1, unsigned count = 1) {
    return dim3((n0 + kFaceX - 1) / kFaceX * (kFaces<K> * kSlots<Q, K>), (n1 + kFaceY - 1) / kFaceY, count);
}

template <int Q, int K, class TF, class TG>
__device__ __forceinline__ void bc_face(const StepArgs<TF, TG> &a) {
    const Geometry &G = a.geo;
    const int tiles = (int)gridDim.x / (kFaces<K> * kSlots<Q, K>);
    const int s = (int)blockIdx.x / tiles; // slot of the first face, then of the second
    const int i0 = ((int)blockIdx.x - s * tiles) * kFaceX + (int)threadIdx.x;
    const int i1 = (int)blockIdx.y * kFaceY + (int)threadIdx.y;
    constexpr int N = kSlots<Q, K>;
    if constexpr (K == BK_JET_Y) {
        if (G.bcy != BC_JET) return;
        if (s < N) bc_water_inflow_at<Q>(a, i0, i1, s);
        else bc_outflow_y_at<Q>(a, i0, i1, s - N);
    } else if constexpr (K == BK_JET_Z) {
        if (G.bcz != BC_JET) return;
        if (s < N) bc_oil_inflow_at<Q>(a, i0, i1, s);
        else bc_outflow_z_at<Q>(a, i0, i1, s - N);
    } else if constexpr (K == BK_COPY_X) {
        if (G.bcx == BC_COPY) bc_copy_x_at<Q>(a, i0, i1, s);
    } else {
        if (G.bcy == BC_COPY) bc_copy_y_at<Q>(a, i0, i1, s);
    }
}

template <int Q, class TF, class TG, int K>
__global__ void __launch_bounds__(kFaceX * kFaceY) bc_kernel(const StepArgs<TF, TG> a) {
    bc_face<Q, K>(a);
}

} // namespace ssmd
