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

// Velocity c and weight of one direction.
struct Dir {
    float cx, cy, cz, w;
    int ix, iy, iz; // the same components as integers
};

template <int Q>
__host__ __device__ constexpr Dir dir_of(int q) {
    return Dir{float(cx27(q)), float(cy27(q)), float(cz27(q)), VS<Q>::w(q), cx27(q), cy27(q), cz27(q)};
}

// Component of a direction picked at run time along `axis`.
constexpr int axis_of(int axis, int q) { return axis == 0 ? cx27(q) : (axis == 1 ? cy27(q) : cz27(q)); }
constexpr uint64_t pack_axis(int axis) { // 2 bits per direction: c + 1
    uint64_t v = 0;
    for (int q = 0; q < 27; ++q) v |= (uint64_t)(axis_of(axis, q) + 1) << (2 * q);
    return v;
}
template <int AXIS>
__device__ __forceinline__ int component(int q) {
    constexpr uint64_t V = pack_axis(AXIS);
    return (int)((V >> (2 * q)) & 3u) - 1;
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
    constexpr Dir d = dir_of<Q>(q);
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

// How the boundary launches are split.  A face has few cells.  With one thread
// per face cell doing every direction, a launch was ~700 instructions of
// straight-line code run once by a handful of warps, each direction's loads
// behind the store of the one before: 4-5 us of fetches and round trips whatever
// the lattice, 26 us for the x copies, whose every access is a sector of its
// own.  So
//  - a jet face cell has three threads, each with one row of up to three
//    directions (regularized_row), all its loads in flight at once;
//  - a copied pair has a thread per population slot, the direction picked at run time;
//  - the two faces of an axis share a launch: inflow writes ghost plane 0 and
//    reads plane 1, outflow writes plane n - 1 and reads plane n - 2 (axes with jets
//    have n >= 6), so neither reads what the other writes.
// us a launch on B200, one thread per face cell -> now: jet faces of 64 x 64 x 128
// D3Q19 FP32 5.0 -> 3.5, 128 x 128 x 512 D3Q27 FP32 6.6 -> 4.5, 256 x 256 x 1024 D3Q19
// FP32 5.9 -> 4.6, 24 jets at once 16 -> 12; x copies of a 101 x 75 x 203 crossflow
// (D3Q27 F16_G32) 25 -> 13, its boundaries altogether 44 in five launches -> 21 in three.
// The reference's order (above) is kept by pairs, (water inflow, outflow y)
// before (oil inflow, outflow z): oil inflow reads fluid cells only and writes
// plane z = 0, outflow y reads and writes at fluid z, so these two may change
// places.
constexpr int kFaceX = 32, kFaceY = 4; // a block's face cells
// directions that leave a face; a copied pair has the slots of both, one for g and
// one for the fields
template <int Q>
constexpr int kFaceDirs = Q == 27 ? 9 : 5;

// The directions whose component along `axis` is s (or, s = 0, is not zero), 5 bits each.
template <int Q>
constexpr uint64_t face_list(int axis, int s) {
    uint64_t v = 0;
    int n = 0;
    for (int q = 0; q < Q; ++q)
        if (axis_of(axis, q) == s) v |= (uint64_t)q << (5 * n++);
    return v;
}

// Regularized inflow / outflow values of one row of directions for the ghost cell b
// of face cell (x, i1), f = f_eq(rho_b, u_b) + omco f_neq(Pi(fn), u(fn)) at fluid
// node fn: the directions with component S along AXIS (1: y, 2: z) and ROW along
// the face's second axis.  FLUID: only where fn is a fluid cell (otherwise: inside
// the lattice).  All loads come before the first store.
template <int Q, int AXIS, int S, int ROW, bool FLUID, class TF, class TG>
__device__ __forceinline__ void regularized_row(const StepArgs<TF, TG> &a, int x, int i1, uint32_t b, float rho,
                                                float ux, float uy, float uz, float omco) {
    const Geometry &G = a.geo;
    const Fields &F = a.fld;
    const int j = AXIS == 1 ? axis_nb(i1 + ROW, G.nz, G.bcz == BC_PERIODIC)
                            : axis_nb(i1 + ROW, G.ny, G.bcy == BC_PERIODIC);
    if (j < 0 || (FLUID && !(AXIS == 1 ? in_range(j, G.z_lo, G.z_hi) : in_range(j, G.y_lo, G.y_hi)))) return;
    const int plane = S > 0 ? 1 : (int)(AXIS == 1 ? G.ny : G.nz) - 2;
    const uint32_t row = AXIS == 1 ? cell_index(G, 0, plane, j) : cell_index(G, 0, j, plane);
    float v[3][9];
    bool ok[3];
    unroll<0, 3>([&](auto k) {
        constexpr int K = decltype(k)::value, q = AXIS == 1 ? q27(K - 1, S, ROW) : q27(K - 1, ROW, S);
        if constexpr (q < Q) {
            const int xx = axis_nb(x + K - 1, G.nx, G.bcx == BC_PERIODIC);
            ok[K] = xx >= 0 && (!FLUID || in_range(xx, G.x_lo, G.x_hi));
            if (ok[K]) {
                const uint32_t fn = row + (uint32_t)xx;
                v[K][0] = F.pxx[fn], v[K][1] = F.pyy[fn], v[K][2] = F.pzz[fn];
                v[K][3] = F.pxy[fn], v[K][4] = F.pxz[fn], v[K][5] = F.pyz[fn];
                v[K][6] = F.ux[fn], v[K][7] = F.uy[fn], v[K][8] = F.uz[fn];
            }
        }
    });
    unroll<0, 3>([&](auto k) {
        constexpr int K = decltype(k)::value, q = AXIS == 1 ? q27(K - 1, S, ROW) : q27(K - 1, ROW, S);
        if constexpr (q < Q) {
            if (ok[K]) {
                constexpr Dir d = dir_of<Q>(q);
                const float feq = feq_of<Q>(d, rho, ux, uy, uz);
                const float fneq = fneq_of<Q>(d, v[K][0], v[K][1], v[K][2], v[K][3], v[K][4], v[K][5], v[K][6],
                                              v[K][7], v[K][8]);
                Store<TF>::st(a.f_dst + slot(G, q, b), fmaf(omco, fneq, feq));
            }
        }
    });
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

// Water inflow disc on y = 0 (BoundaryConditions.cuh:36-99).  Thread (x, z), row of directions.
template <int Q, int ROW, class TF, class TG>
__device__ __forceinline__ void bc_water_inflow_at(const StepArgs<TF, TG> &a, const int x, const int z) {
    const Geometry &G = a.geo;
    const Physics &P = a.phys;
    if (x >= (int)G.nx || z >= (int)G.nz) return;
    const float dx = float(x) - P.water_cx, dz = float(z) - P.water_cz;
    if (dx * dx + dz * dz > P.water_r2) return;
    const uint32_t b = cell_index(G, x, 0, z);
    const float uw = P.u_water;
    // (a node outside the lattice, which the reference reads out of bounds, is left out)
    regularized_row<Q, 1, 1, ROW, false>(a, x, z, b, 1.0f, 0.0f, uw, 0.0f, P.omco_water);
    if constexpr (ROW == 0) {
        a.fld.rho[b] = 1.0f;
        a.fld.phi[b] = 0.0f;
        a.fld.ux[b] = 0.0f;
        a.fld.uy[b] = uw;
        a.fld.uz[b] = 0.0f;
        Store<TG>::st(a.g_dst + slot(G, 3, b), 0.0f); // w_3 * phi (1 + 4 u_y) with phi = 0
    }
}

// Oil inflow disc on z = 0 (BoundaryConditions.cuh:101-168).  Thread (x, y), row of directions.
template <int Q, int ROW, class TF, class TG>
__device__ __forceinline__ void bc_oil_inflow_at(const StepArgs<TF, TG> &a, const int x, const int y) {
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
    regularized_row<Q, 2, 1, ROW, true>(a, x, y, b, 1.0f, 0.0f, 0.0f, uin, P.omco_oil);
    if constexpr (ROW == 0) {
        a.fld.rho[b] = 1.0f;
        a.fld.phi[b] = 1.0f;
        a.fld.ux[b] = 0.0f;
        a.fld.uy[b] = 0.0f;
        a.fld.uz[b] = uin;
        Store<TG>::st(a.g_dst + slot(G, 5, b), kW7_1 * 1.0f * (1.0f + 4.0f * uin));
    }
}

// Outflow on y = ny-1 (BoundaryConditions.cuh:170-233).  Thread (x, z), row of directions.
template <int Q, int ROW, class TF, class TG>
__device__ __forceinline__ void bc_outflow_y_at(const StepArgs<TF, TG> &a, const int x, const int z) {
    const Geometry &G = a.geo;
    if (!in_range(x, G.x_lo, G.x_hi) || !in_range(z, G.z_lo, G.z_hi)) return;
    const uint32_t b = cell_index(G, x, G.ny - 1, z);
    const uint32_t i1 = cell_index(G, x, G.ny - 2, z);
    const Fields &F = a.fld;
    const float ux = F.ux[i1], uy = F.uy[i1], uz = F.uz[i1], rho = F.rho[i1];
    const float phi = ROW == 0 ? F.phi[i1] : 0.f;
    regularized_row<Q, 1, -1, ROW, true>(a, x, z, b, rho, ux, uy, uz, a.phys.omco_ref);
    if constexpr (ROW == 0) {
        F.rho[b] = rho;
        F.phi[b] = phi;
        F.ux[b] = ux;
        F.uy[b] = uy;
        F.uz[b] = uz;
        Store<TG>::st(a.g_dst + slot(G, 4, b), kW7_1 * phi * (1.0f - 4.0f * uy));
    }
}

// Outflow on z = nz-1 (BoundaryConditions.cuh:235-293).  Thread (x, y), row of directions.
template <int Q, int ROW, class TF, class TG>
__device__ __forceinline__ void bc_outflow_z_at(const StepArgs<TF, TG> &a, const int x, const int y) {
    const Geometry &G = a.geo;
    if (!in_range(x, G.x_lo, G.x_hi) || !in_range(y, G.y_lo, G.y_hi)) return;
    const uint32_t b = cell_index(G, x, y, G.nz - 1);
    const uint32_t i1 = cell_index(G, x, y, G.nz - 2);
    const Fields &F = a.fld;
    const float ux = F.ux[i1], uy = F.uy[i1], uz = F.uz[i1], rho = F.rho[i1];
    const float phi = ROW == 0 ? F.phi[i1] : 0.f;
    // no fluid-range check here, as in the reference (ghost nodes allowed)
    regularized_row<Q, 2, -1, ROW, false>(a, x, y, b, rho, ux, uy, uz, a.phys.omco_ref);
    if constexpr (ROW == 0) {
        F.rho[b] = rho;
        F.phi[b] = phi;
        F.ux[b] = ux;
        F.uy[b] = uy;
        F.uz[b] = uz;
        Store<TG>::st(a.g_dst + slot(G, 6, b), kW7_1 * phi * (1.0f - 4.0f * uz));
    }
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
        const int hy = axis_nb(y - component<1>(q), G.ny, G.bcy == BC_PERIODIC);
        const int hz = axis_nb(z - component<2>(q), G.nz, G.bcz == BC_PERIODIC);
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
        const int hx = axis_nb(x - component<0>(q), G.nx, G.bcx == BC_PERIODIC);
        const int hz = axis_nb(z - component<2>(q), G.nz, G.bcz == BC_PERIODIC);
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

// Faces of a launch, and threads per cell of each: the rows of directions of a jet
// face, the slots of a copied pair.
template <int K>
constexpr int kFaces = K == BK_JET_Y || K == BK_JET_Z ? 2 : 1;
template <int Q, int K>
constexpr int kSlots = K == BK_JET_Y || K == BK_JET_Z ? 3 : 2 * kFaceDirs<Q> + 2;

// Grid of one boundary launch over faces of at most n0 x n1 cells of `count`
// lattices: blocks of kFaceX x kFaceY face cells, blockIdx.x the tiles along the
// first axis times the slots of the faces.
// A thread per (cell, slot) on jet faces too is a little shorter on an idle device
// (the launches above: 3.2, 3.9, 5.5, 16 us) but 2560 blocks for a 128 x 128 face, and
// among other lattices' kernels, which fill every SM, their instructions and places
// count: three 128 x 128 x 512 D3Q27 FP32 jets on their own streams took 467 us a step
// each, with rows 464, with one thread per cell 464; one alone in a replayed graph 455.5,
// 456.7 and 459.3.  All inflow rows in one thread: 38.4 instead of 37.1 us a step on 64 x
// 64 x 128.  For the copies, several slots per thread in a loop lost to the round trips
// that follow one another (crossflow 21 -> 26 us).
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
    if constexpr (K == BK_JET_Y) {
        if (G.bcy != BC_JET) return;
        switch (s) {
        case 0: bc_water_inflow_at<Q, -1>(a, i0, i1); break;
        case 1: bc_water_inflow_at<Q, 0>(a, i0, i1); break;
        case 2: bc_water_inflow_at<Q, 1>(a, i0, i1); break;
        case 3: bc_outflow_y_at<Q, -1>(a, i0, i1); break;
        case 4: bc_outflow_y_at<Q, 0>(a, i0, i1); break;
        default: bc_outflow_y_at<Q, 1>(a, i0, i1); break;
        }
    } else if constexpr (K == BK_JET_Z) {
        if (G.bcz != BC_JET) return;
        switch (s) {
        case 0: bc_oil_inflow_at<Q, -1>(a, i0, i1); break;
        case 1: bc_oil_inflow_at<Q, 0>(a, i0, i1); break;
        case 2: bc_oil_inflow_at<Q, 1>(a, i0, i1); break;
        case 3: bc_outflow_z_at<Q, -1>(a, i0, i1); break;
        case 4: bc_outflow_z_at<Q, 0>(a, i0, i1); break;
        default: bc_outflow_z_at<Q, 1>(a, i0, i1); break;
        }
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
