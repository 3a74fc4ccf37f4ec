// reduce.cuh — FP64 global reductions over the fluid cells.
//
// Deterministic two-pass sum: pass 1 leaves one partial per block in a
// scratch array, pass 2 folds the partials in a fixed order, so the result
// does not depend on block scheduling.
#pragma once

#include "common.cuh"

namespace ssmd {

constexpr int kRedThreads = 256;
constexpr int kRedVals = 10; // phi, phi_next, mass, mx, my, mz, kinetic, umax, nonfinite, cells

// Value k (7 a maximum, the others sums) over the lanes of a warp, in every lane.
__device__ __forceinline__ double warp_fold(int k, double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double t = __shfl_xor_sync(0xffffffffu, v, o);
        v = k == 7 ? fmax(v, t) : v + t;
    }
    return v;
}

// Pass 1 by columns: a warp takes 32 neighbouring x of one row and marches along
// kRedPlanes z planes, so a cell costs no division and its loads (the five
// fields and seven populations) are coalesced and independent of the plane
// before.  The largest speed is kept squared (sqrt is monotonic and correctly
// rounded: the same bits).  On 128 x 128 x 512 cells (FP32 g: 403 MB; caches flushed
// before the launch) 73 us, 85 % of the measured copy bandwidth; one cell per thread
// in linear order, its coordinates from two divisions and a FP64 square root per
// cell, took 224.
constexpr int kRedPlanes = 16;

template <class TG>
__global__ void __launch_bounds__(kRedThreads) reduce_pass1(Geometry G, Fields F, const TG *__restrict__ g,
                                                            double *partials) {
    __shared__ double sm[kRedVals][kRedThreads / 32];
    double v[kRedVals] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
    double u2max = 0.0;
    const bool px = G.bcx == BC_PERIODIC, py = G.bcy == BC_PERIODIC, pz = G.bcz == BC_PERIODIC;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t segs = (G.nx + 31u) / 32u, cols = segs * G.ny;
    const uint32_t nz = (uint32_t)(G.z_hi - G.z_lo + 1), chunks = (nz + kRedPlanes - 1) / kRedPlanes;
    const uint64_t units = (uint64_t)cols * chunks;
    const TG *gq[7];
#pragma unroll
    for (int q = 0; q < 7; ++q) gq[q] = g + (uint64_t)q * G.cells;
    for (uint64_t w = (uint64_t)blockIdx.x * (kRedThreads / 32) + (threadIdx.x >> 5); w < units;
         w += (uint64_t)gridDim.x * (kRedThreads / 32)) {
        const uint32_t zc = (uint32_t)(w / cols), col = (uint32_t)(w - (uint64_t)zc * cols);
        const uint32_t yu = col / segs;
        const int y = (int)yu, x = (int)((col - yu * segs) * 32u + lane);
        if (x < G.x_lo || x > G.x_hi || y < G.y_lo || y > G.y_hi) continue;
        const int z0 = G.z_lo + (int)zc * kRedPlanes, z1 = min(z0 + kRedPlanes - 1, G.z_hi);
        // steps to the x and y neighbours (wrapped on periodic axes); the z ones per plane
        const uint32_t xm = px && x == 0 ? G.nx - 1u : 0u - 1u, xp = px && x == (int)G.nx - 1 ? 1u - G.nx : 1u;
        const uint32_t ym = py && y == 0 ? G.nxy - G.nx : 0u - G.nx, yp = py && y == (int)G.ny - 1 ? G.nx - G.nxy : G.nx;
        uint32_t c = cell_index(G, x, y, z0);
#pragma unroll 2
        for (int z = z0; z <= z1; ++z, c += G.nxy) {
            const uint32_t zm = pz && z == 0 ? (uint32_t)G.cells - G.nxy : 0u - G.nxy;
            const uint32_t zp = pz && z == (int)G.nz - 1 ? G.nxy - (uint32_t)G.cells : G.nxy;
            const float rho_f = F.rho[c], ux_f = F.ux[c], uy_f = F.uy[c], uz_f = F.uz[c], phi_f = F.phi[c];
            const float g0 = Store<TG>::ld(gq[0] + c), g1 = Store<TG>::ld(gq[1] + (uint32_t)(c + xm));
            const float g2 = Store<TG>::ld(gq[2] + (uint32_t)(c + xp)), g3 = Store<TG>::ld(gq[3] + (uint32_t)(c + ym));
            const float g4 = Store<TG>::ld(gq[4] + (uint32_t)(c + yp)), g5 = Store<TG>::ld(gq[5] + (uint32_t)(c + zm));
            const float g6 = Store<TG>::ld(gq[6] + (uint32_t)(c + zp));
            const double rho = rho_f, ux = ux_f, uy = uy_f, uz = uz_f, phi = phi_f;
            const double pn = ((((((double)g0 + (double)g1) + (double)g2) + (double)g3) + (double)g4) + (double)g5) + (double)g6;
            const double u2 = ux * ux + uy * uy + uz * uz;
            const bool bad = !(isfinite(rho) && isfinite(u2) && isfinite(phi) && isfinite(pn));
            v[0] += phi;
            v[1] += pn;
            v[2] += rho;
            v[3] += rho * ux;
            v[4] += rho * uy;
            v[5] += rho * uz;
            v[6] += 0.5 * rho * u2;
            if (!bad) u2max = fmax(u2max, u2);
            v[8] += bad ? 1.0 : 0.0;
            v[9] += 1.0;
        }
    }
    v[7] = sqrt(u2max);
#pragma unroll
    for (int k = 0; k < kRedVals; ++k) {
        const double t = warp_fold(k, v[k]);
        if (lane == 0) sm[k][threadIdx.x >> 5] = t;
    }
    __syncthreads();
    const int k = threadIdx.x;
    if (k < kRedVals) {
        double t = sm[k][0];
        for (int w = 1; w < kRedThreads / 32; ++w) t = k == 7 ? fmax(t, sm[k][w]) : t + sm[k][w];
        partials[(uint64_t)k * gridDim.x + blockIdx.x] = t;
    }
}

// Pass 2: warp k folds value k's partials (one block; 9.3 us as a tree over shared
// memory, 5.0 now, caches flushed).
constexpr int kFoldThreads = 32 * kRedVals;
static __global__ void __launch_bounds__(kFoldThreads) reduce_pass2(const double *partials, int nparts,
                                                                    double *out) {
    const int k = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double v = 0.0;
#pragma unroll 8
    for (int i = lane; i < nparts; i += 32) {
        const double p = partials[(uint64_t)k * nparts + i];
        v = k == 7 ? fmax(v, p) : v + p;
    }
    v = warp_fold(k, v);
    if (lane == 0) out[k] = v;
}

} // namespace ssmd
