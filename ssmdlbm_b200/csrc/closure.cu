// closure.cu — features, training targets and application of the learned closure.
//
// The closure runs the plain method on a 2x coarser lattice and corrects it
// per cell: an eddy viscosity nu_t added to nu(phi), and a factor on the
// surface tension.  Training data come from the solver's own fine runs:
// ssmd_closure_filter box-filters a fine lattice onto the coarse one (the
// resolved fields, the subgrid stress and the fine interface area density),
// ssmd_closure_targets turns them into the two targets, and
// ssmd_closure_features computes the network inputs from any lattice's
// macroscopic fields, so filtered fine data and a live coarse run are
// described by the same numbers.  Derivatives are central differences;
// exact-periodic axes wrap, the others clamp at the faces.
#include <cuda_runtime.h>

#include "closure.cuh"
#include "host.cuh"

using namespace ssmd;
using namespace ssmd::host;
using namespace ssmd::closure;

namespace {

// A block's 256 x 12 features go through shared memory: a thread's 48 bytes as
// three 16-byte stores there, then the block's 12 KB in one coalesced run (each thread
// writing its own row, twelve 4-byte stores 48 bytes apart across a warp, took 49 us on
// 64 x 64 x 256 cells; now 22).
constexpr int kFeatThreads = 256;
__global__ void __launch_bounds__(kFeatThreads)
    features_kernel(Grid g, const float *__restrict__ rho, const float *__restrict__ ux, const float *__restrict__ uy,
                    const float *__restrict__ uz, const float *__restrict__ phi, float nu_w, float nu_dow,
                    float *__restrict__ feat) {
    __shared__ __align__(16) float sf[kFeatThreads * SSMD_MLP_IN];
    const int64_t cells = (int64_t)g.nx * g.ny * g.nz;
    const int64_t base = blockIdx.x * (int64_t)kFeatThreads;
    const int n = (int)(cells - base < kFeatThreads ? cells - base : kFeatThreads);
    if ((int)threadIdx.x < n) {
        float f[SSMD_MLP_IN];
        closure::cell_features(g, rho, ux, uy, uz, phi, nu_w, nu_dow, base + threadIdx.x, f);
        float4 *row = reinterpret_cast<float4 *>(sf + threadIdx.x * SSMD_MLP_IN);
#pragma unroll
        for (int k = 0; k < SSMD_MLP_IN / 4; ++k) row[k] = make_float4(f[4 * k], f[4 * k + 1], f[4 * k + 2], f[4 * k + 3]);
    }
    __syncthreads();
    float *dst = feat + base * SSMD_MLP_IN;
    if ((reinterpret_cast<uintptr_t>(feat) & 15u) == 0) { // (a block's run is a multiple of 16 bytes)
        for (int k = threadIdx.x; k < n * SSMD_MLP_IN / 4; k += kFeatThreads)
            reinterpret_cast<float4 *>(dst)[k] = reinterpret_cast<const float4 *>(sf)[k];
    } else {
        for (int k = threadIdx.x; k < n * SSMD_MLP_IN; k += kFeatThreads) dst[k] = sf[k];
    }
}

// One thread per coarse cell: means over the 2 x 2 x 2 fine block, in FP64.  A
// block's two cells along x are loaded as one float2 where the field is 8-byte
// aligned (fine rows have even lengths), the neighbours phi's gradient needs once
// each, all by 32-bit cell indices (per-value loads with 64-bit index arithmetic took
// 74 us on 128 x 128 x 512 fine cells; now 61, bound by the FP64 conversions, sums and square
// roots, 49 us without the last; 80 registers for three blocks per SM: 84 take 76 us, 64 take 66).
__device__ __forceinline__ float2 pair_at(const float *__restrict__ a, uint32_t c, bool aligned) {
    if (aligned) return __ldg(reinterpret_cast<const float2 *>(a + c));
    return make_float2(__ldg(a + c), __ldg(a + c + 1));
}

__global__ void __launch_bounds__(256, 3)
    filter_kernel(Grid fg, Grid cg, const float *__restrict__ rho, const float *__restrict__ ux,
                  const float *__restrict__ uy, const float *__restrict__ uz, const float *__restrict__ phi,
                  float *__restrict__ coarse, float *__restrict__ tau, float *__restrict__ area) {
    const uint32_t cells = (uint32_t)cg.nx * cg.ny * cg.nz;
    const uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (t >= cells) return;
    const uint32_t i = (uint32_t)t;
    const uint32_t zy = i / cg.nx, X = i - zy * cg.nx, Z = zy / cg.ny, Y = zy - Z * cg.ny;
    const uint32_t nx = fg.nx, nxy = nx * (uint32_t)fg.ny;
    const uint32_t c0 = 2 * X + nx * (2 * Y) + nxy * (2 * Z); // the block's first fine cell
    const bool aligned = ((reinterpret_cast<uintptr_t>(rho) | reinterpret_cast<uintptr_t>(ux) |
                           reinterpret_cast<uintptr_t>(uy) | reinterpret_cast<uintptr_t>(uz) |
                           reinterpret_cast<uintptr_t>(phi)) & 7u) == 0;
    // phi of the block, p[k][j] its row pairs, and of the cells beside it along each
    // axis (wrapped on periodic axes, the face's own cell otherwise)
    const uint32_t bx0 = X > 0 ? c0 - 1 : (fg.px ? c0 + nx - 1 : c0);
    const uint32_t bx1 = X + 1 < (uint32_t)cg.nx ? c0 + 2 : (fg.px ? c0 + 2 - nx : c0 + 1);
    const uint32_t by0 = Y > 0 ? c0 - nx : (fg.py ? c0 + nxy - nx : c0);
    const uint32_t by1 = Y + 1 < (uint32_t)cg.ny ? c0 + 2 * nx : (fg.py ? c0 + 2 * nx - nxy : c0 + nx);
    const uint32_t total = nxy * (uint32_t)fg.nz;
    const uint32_t bz0 = Z > 0 ? c0 - nxy : (fg.pz ? c0 + total - nxy : c0);
    const uint32_t bz1 = Z + 1 < (uint32_t)cg.nz ? c0 + 2 * nxy : (fg.pz ? c0 + 2 * nxy - total : c0 + nxy);
    float2 p[2][2], y0[2], y1[2], z0[2], z1[2];
    float x0[2][2], x1[2][2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            p[k][j] = pair_at(phi, c0 + j * nx + k * nxy, aligned);
            x0[k][j] = __ldg(phi + (uint32_t)(bx0 + j * nx + k * nxy));
            x1[k][j] = __ldg(phi + (uint32_t)(bx1 + j * nx + k * nxy));
        }
        y0[k] = pair_at(phi, by0 + k * nxy, aligned);
        y1[k] = pair_at(phi, by1 + k * nxy, aligned);
        z0[k] = pair_at(phi, bz0 + k * nx, aligned); // (index: row of the block)
        z1[k] = pair_at(phi, bz1 + k * nx, aligned);
    }
    double m[5] = {0, 0, 0, 0, 0}, uu[6] = {0, 0, 0, 0, 0, 0}, a = 0.0;
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const uint32_t c = c0 + j * nx + k * nxy;
            const float2 r2 = pair_at(rho, c, aligned), ux2 = pair_at(ux, c, aligned), uy2 = pair_at(uy, c, aligned),
                         uz2 = pair_at(uz, c, aligned);
#pragma unroll
            for (int l = 0; l < 2; ++l) {
                auto of = [&](const float2 &v) { return l == 0 ? v.x : v.y; };
                const float u0 = of(ux2), u1 = of(uy2), u2 = of(uz2);
                m[0] += of(r2);
                m[1] += u0;
                m[2] += u1;
                m[3] += u2;
                m[4] += of(p[k][j]);
                uu[0] += (double)u0 * u0;
                uu[1] += (double)u1 * u1;
                uu[2] += (double)u2 * u2;
                uu[3] += (double)u0 * u1;
                uu[4] += (double)u0 * u2;
                uu[5] += (double)u1 * u2;
                const float gx = 0.5f * (l == 0 ? p[k][j].y - x0[k][j] : x1[k][j] - p[k][j].x);
                const float gy = 0.5f * (j == 0 ? of(p[k][1]) - of(y0[k]) : of(y1[k]) - of(p[k][0]));
                const float gz = 0.5f * (k == 0 ? of(p[1][j]) - of(z0[j]) : of(z1[j]) - of(p[0][j]));
                a += sqrt((double)gx * gx + (double)gy * gy + (double)gz * gz);
            }
        }
    for (int q = 0; q < 5; ++q) m[q] *= 0.125;
    for (int q = 0; q < 6; ++q) uu[q] *= 0.125;
    const uint64_t n = cells;
    for (int q = 0; q < 5; ++q) coarse[q * n + i] = (float)m[q];
    tau[0 * n + i] = (float)(uu[0] - m[1] * m[1]);
    tau[1 * n + i] = (float)(uu[1] - m[2] * m[2]);
    tau[2 * n + i] = (float)(uu[2] - m[3] * m[3]);
    tau[3 * n + i] = (float)(uu[3] - m[1] * m[2]);
    tau[4 * n + i] = (float)(uu[4] - m[1] * m[3]);
    tau[5 * n + i] = (float)(uu[5] - m[2] * m[3]);
    area[i] = (float)(0.125 * a);
}

// Neighbours by 32-bit indices found once per cell (closure::faces), each pair of
// results in one 8-byte store (64-bit index arithmetic for each of 24 loads: 33 us on 64 x
// 64 x 256 cells; now 17).
__global__ void targets_kernel(Grid g, const float *__restrict__ cf, const float *__restrict__ tau,
                               const float *__restrict__ area, float nut_max, float *__restrict__ targets,
                               float *__restrict__ weights) {
    const uint64_t cells = (uint64_t)g.nx * g.ny * g.nz;
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i >= cells) return;
    const closure::Faces n6 = closure::faces(g, (uint32_t)i);
    const float *ux = cf + 1 * cells, *uy = cf + 2 * cells, *uz = cf + 3 * cells, *phi = cf + 4 * cells;
    auto diff = [&](const float *v, uint32_t p, uint32_t m) { return 0.5f * (__ldg(v + p) - __ldg(v + m)); };
    float d[3][3];
    const float *u3[3] = {ux, uy, uz};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        d[a][0] = diff(u3[a], n6.xp, n6.xm);
        d[a][1] = diff(u3[a], n6.yp, n6.ym);
        d[a][2] = diff(u3[a], n6.zp, n6.zm);
    }
    const float t[3][3] = {{tau[0 * cells + i], tau[3 * cells + i], tau[4 * cells + i]},
                           {tau[3 * cells + i], tau[1 * cells + i], tau[5 * cells + i]},
                           {tau[4 * cells + i], tau[5 * cells + i], tau[2 * cells + i]}};
    const float tr = (t[0][0] + t[1][1] + t[2][2]) * (1.0f / 3.0f);
    float num = 0.f, den = 0.f;
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            const float s = 0.5f * (d[a][b] + d[b][a]);
            num += (t[a][b] - (a == b ? tr : 0.f)) * s;
            den += s * s;
        }
    // signed: negative values (backscatter) are kept, the coarse run bounds them
    const float nut = fminf(fmaxf(-num / (2.0f * den + 1e-12f), -nut_max), nut_max);
    const float gx = diff(phi, n6.xp, n6.xm), gy = diff(phi, n6.yp, n6.ym), gz = diff(phi, n6.zp, n6.zm);
    const float gm = sqrtf(gx * gx + gy * gy + gz * gz);
    float cs = 1.0f;
    if (gm >= 1e-2f) cs = fminf(fmaxf(2.0f * area[i] / gm, 0.25f), 4.0f);
    const float ph = phi[i];
    const float w1 = 4.0f * ph * (1.0f - ph) + 0.01f;
    if (((reinterpret_cast<uintptr_t>(targets) | reinterpret_cast<uintptr_t>(weights)) & 7u) == 0) {
        reinterpret_cast<float2 *>(targets)[i] = make_float2(nut, cs);
        reinterpret_cast<float2 *>(weights)[i] = make_float2(1.0f, w1);
    } else {
        targets[2 * i + 0] = nut;
        targets[2 * i + 1] = cs;
        weights[2 * i + 0] = 1.0f;
        weights[2 * i + 1] = w1;
    }
}

// nu_t is bounded below by -nu(phi)/2 (feature 11), so the total viscosity
// stays at least half the molecular one and the relaxation rate below 2.
__global__ void apply_kernel(int64_t cells, const float *out, const float *feat, float nut_max, float *nut,
                             float *cs) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= cells) return;
    const float lo = fmaxf(-0.5f * feat[i * SSMD_MLP_IN + 11], -nut_max);
    nut[i] = fminf(fmaxf(out[2 * i + 0], lo), nut_max);
    cs[i] = fminf(fmaxf(out[2 * i + 1], 0.25f), 4.0f);
}

unsigned blocks_for(int64_t n) { return (unsigned)((n + 255) / 256); }

} // namespace

extern "C" int ssmd_closure_features(const ssmd_params *p, const LBMFields *fields, float *features,
                                     ssmd_stream_t stream) {
    if (int e = ssmd_validate(p)) return e;
    if (!fields || !fields->rho || !fields->ux || !fields->uy || !fields->uz || !fields->phi || !features)
        return fail(SSMD_ERR_INVALID_ARGUMENT, "null argument");
    const Grid g = grid_of(*p);
    const int64_t cells = (int64_t)g.nx * g.ny * g.nz;
    features_kernel<<<blocks_for(cells), kFeatThreads, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        g, fields->rho, fields->ux, fields->uy, fields->uz, fields->phi, p->nu_water, p->nu_oil - p->nu_water,
        features);
    return cuda_check(cudaGetLastError(), "features launch");
}

extern "C" int ssmd_closure_filter(const ssmd_params *fine, const LBMFields *fine_fields, float *coarse, float *tau,
                                   float *area, ssmd_stream_t stream) {
    if (int e = ssmd_validate(fine)) return e;
    if (!fine_fields || !fine_fields->rho || !fine_fields->ux || !fine_fields->uy || !fine_fields->uz ||
        !fine_fields->phi || !coarse || !tau || !area)
        return fail(SSMD_ERR_INVALID_ARGUMENT, "null argument");
    if ((fine->nx | fine->ny | fine->nz) & 1u)
        return fail(SSMD_ERR_INVALID_ARGUMENT, "filtering needs even lattice sizes (%u x %u x %u)", fine->nx,
                    fine->ny, fine->nz);
    const Grid fg = grid_of(*fine);
    Grid cg = fg;
    cg.nx /= 2;
    cg.ny /= 2;
    cg.nz /= 2;
    const int64_t cells = (int64_t)cg.nx * cg.ny * cg.nz;
    filter_kernel<<<blocks_for(cells), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        fg, cg, fine_fields->rho, fine_fields->ux, fine_fields->uy, fine_fields->uz, fine_fields->phi, coarse, tau,
        area);
    return cuda_check(cudaGetLastError(), "filter launch");
}

extern "C" int ssmd_closure_targets(const ssmd_params *coarse, const float *coarse_fields, const float *tau,
                                    const float *area, float nut_max, float *targets, float *weights,
                                    ssmd_stream_t stream) {
    if (int e = ssmd_validate(coarse)) return e;
    if (!coarse_fields || !tau || !area || !targets || !weights)
        return fail(SSMD_ERR_INVALID_ARGUMENT, "null argument");
    const Grid g = grid_of(*coarse);
    const int64_t cells = (int64_t)g.nx * g.ny * g.nz;
    targets_kernel<<<blocks_for(cells), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        g, coarse_fields, tau, area, nut_max, targets, weights);
    return cuda_check(cudaGetLastError(), "targets launch");
}

extern "C" int ssmd_closure_apply(const ssmd_params *coarse, const float *net, const float *features, float *out,
                                  float *nut, float *sigma_scale, float nut_max, ssmd_stream_t stream) {
    if (int e = ssmd_validate(coarse)) return e;
    if (!net || !features || !out || !nut || !sigma_scale) return fail(SSMD_ERR_INVALID_ARGUMENT, "null argument");
    const int64_t cells = (int64_t)coarse->nx * coarse->ny * coarse->nz;
    if (int e = ssmd_mlp_forward(net, features, cells, out, stream)) return e;
    apply_kernel<<<blocks_for(cells), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(cells, out, features,
                                                                                        nut_max, nut, sigma_scale);
    return cuda_check(cudaGetLastError(), "closure apply launch");
}
