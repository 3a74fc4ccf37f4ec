// stats.cu — jet statistics on the device: centreline profile and droplets.
//
// The reference writes raw phi / rho fields only (src/main.cu:121-145) and
// leaves statistics to offline post-processing; its optional running means
// (src/derivedFields/operators/timeAverage.cuh:37-82) are the closest
// counterpart.  These kernels read the macroscopic arrays, so they need a
// step with SSMD_STEP_STORE_MACROS (or the initial state) first.
//
//   centreline: for every z, the mean of u_z and of phi over the (one, two
//     or four) cells nearest the oil nozzle axis (x, y) = (oil_cx, oil_cy), FP64.
//   droplets: connected components of {fluid cells with phi > threshold}
//     under 6-neighbour connectivity (exact-periodic axes wrap), labelled with
//     a lock-free union-find: every label points at a smaller or equal index,
//     unions hook the larger root under the smaller one with atomicMin
//     (the GPU union-find of Playne and Hawick, IEEE TPDS 2018), then every
//     label leads to its root (the smallest index of the component).
//     Per component: cell count, FP64 sum of phi (the "volume"), and whether
//     it touches the first fluid plane above the oil inlet.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>

#include "host.cuh"

using namespace ssmd;
using namespace ssmd::host;

namespace {

constexpr uint32_t kBG = 0xFFFFFFFFu;

struct DropScratch {
    uint32_t *label;  // per cell: a smaller or equal cell of its component; kBG: background
    uint32_t *cells;  // the foreground cells, unordered
    uint32_t *count;  // per root: its component's cells, then its entry in the list
    double *volume;   // per root
    uint32_t *n_out;  // components found; n_out[1]: foreground cells
    ssmd_droplet *list;
    int max_list;
};

__device__ __forceinline__ bool fluid_cell(const Geometry &G, int x, int y, int z) {
    return x >= G.x_lo && x <= G.x_hi && y >= G.y_lo && y <= G.y_hi && z >= G.z_lo && z <= G.z_hi;
}

__global__ void centreline_kernel(Geometry G, Fields F, float cx, float cy, double *uz_out, double *phi_out) {
    const int z = blockIdx.x * blockDim.x + threadIdx.x;
    if (z >= (int)G.nz) return;
    const int x0 = (int)floorf(cx), x1 = (int)ceilf(cx);
    const int y0 = (int)floorf(cy), y1 = (int)ceilf(cy);
    double su = 0.0, sp = 0.0;
    int n = 0;
    for (int y = y0; y <= y1; ++y)
        for (int x = x0; x <= x1; ++x) {
            if (x < 0 || y < 0 || x >= (int)G.nx || y >= (int)G.ny) continue;
            const uint32_t c = cell_index(G, x, y, z);
            su += (double)F.uz[c];
            sp += (double)F.phi[c];
            ++n;
        }
    uz_out[z] = n ? su / n : 0.0;
    phi_out[z] = n ? sp / n : 0.0;
}

// Labels, and the list of foreground cells: the kernels that follow visit only
// those (a jet fills a few per cent of its lattice).  A block takes kCclCells
// consecutive cells and reserves its part of the list with one atomic.  The
// accumulators are cleared where a cell may become a root.  On 128 x 128 x 512 cells
// labelling, clearing four arrays and scanning the lattice in each of four kernels took 201 us
// (41 + 76 + 59 + 25); with the list 69 (20 + 28 + 15 + 3 + 3).
constexpr int kCclThreads = 256, kCclPer = 8, kCclCells = kCclThreads * kCclPer;

__global__ void __launch_bounds__(kCclThreads) ccl_init(Geometry G, const float *__restrict__ phi, float thr, DropScratch S) {
    __shared__ uint32_t s_warp[kCclThreads / 32], s_base;
    const uint64_t base = (uint64_t)blockIdx.x * kCclCells;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    float v[kCclPer];
#pragma unroll
    for (int k = 0; k < kCclPer; ++k) {
        const uint64_t i = base + (uint64_t)k * kCclThreads + threadIdx.x;
        v[k] = i < G.cells ? phi[i] : thr;
    }
    uint32_t on = 0, mine = 0; // this thread's foreground cells, and their number
#pragma unroll
    for (int k = 0; k < kCclPer; ++k) {
        const uint64_t i = base + (uint64_t)k * kCclThreads + threadIdx.x;
        const uint32_t c = (uint32_t)i;
        bool fg = i < G.cells && v[k] > thr, first = false;
        if (fg) {
            const uint32_t zy = c / G.nx;
            const int x = (int)(c - zy * G.nx), z = (int)(zy / G.ny), y = (int)(zy - (uint32_t)z * G.ny);
            fg = fluid_cell(G, x, y, z);
            first = x == 0;
        }
        // the label of a run of foreground cells of a row, within the warp's 32 cells: its first
        const uint32_t run = __ballot_sync(0xffffffffu, fg);
        const uint32_t starts = run & (~(run << 1) | __ballot_sync(0xffffffffu, fg && first));
        if (i < G.cells) S.label[c] = fg ? c - (lane - (31u - __clz(starts & (0xffffffffu >> (31u - lane))))) : kBG;
        if (fg) {
            on |= 1u << k;
            ++mine;
            S.count[c] = 0u;
            S.volume[c] = 0.0;
        }
    }
    // exclusive scan of `mine` over the block
    uint32_t scan = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, scan, o);
        if (lane >= (uint32_t)o) scan += t;
    }
    if (lane == 31u) s_warp[warp] = scan;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0;
        for (int w = 0; w < kCclThreads / 32; ++w) {
            const uint32_t k = s_warp[w];
            s_warp[w] = t;
            t += k;
        }
        s_base = t ? atomicAdd(S.n_out + 1, t) : 0u;
    }
    __syncthreads();
    uint32_t at = s_base + s_warp[warp] + scan - mine;
#pragma unroll
    for (int k = 0; k < kCclPer; ++k)
        if (on & (1u << k)) S.cells[at++] = (uint32_t)(base + (uint64_t)k * kCclThreads + threadIdx.x);
}

__device__ __forceinline__ uint32_t find_root(const uint32_t *L, uint32_t a) {
    uint32_t p = ((volatile const uint32_t *)L)[a];
    while (p != a) {
        a = p;
        p = ((volatile const uint32_t *)L)[a];
    }
    return a;
}

__device__ __forceinline__ void unite(uint32_t *L, uint32_t a, uint32_t b) {
    // bounded: each retry strictly lowers the label at one of the two roots
    for (int guard = 0; guard < (1 << 20); ++guard) {
        a = find_root(L, a);
        b = find_root(L, b);
        if (a == b) return;
        if (a > b) {
            const uint32_t t = a;
            a = b;
            b = t;
        }
        const uint32_t old = atomicMin(&L[b], a);
        if (old == b) return;
        b = old;
    }
}

// Unions with the next cell along x, y and z, left out where they follow from
// others: along x inside a run that ccl_init labelled, along y and z where the pair
// one x to the left is foreground too (it is united, and both its cells are with ours).
// With every foreground pair united (long chains on a few labels) this took 63 us,
// now 28.
__global__ void ccl_union(Geometry G, DropScratch S) {
    const uint32_t total = S.n_out[1];
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < total; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t c = S.cells[i];
        const uint32_t zy = c / G.nx;
        const int x = (int)(c - zy * G.nx), z = (int)(zy / G.ny), y = (int)(zy - (uint32_t)z * G.ny);
        const bool left = x > 0 && S.label[c - 1] != kBG;
        const bool per[3] = {G.bcx == BC_PERIODIC, G.bcy == BC_PERIODIC, G.bcz == BC_PERIODIC};
        const int n[3] = {(int)G.nx, (int)G.ny, (int)G.nz};
        for (int d = 0; d < 3; ++d) {
            int q[3] = {x, y, z};
            q[d] += 1;
            const bool wraps = q[d] >= n[d];
            if (wraps) {
                if (!per[d]) continue;
                q[d] -= n[d];
            }
            if (d == 0 && !wraps && (c & 31u) != 31u) continue; // the run's label, or no neighbour
            const uint32_t j = cell_index(G, q[0], q[1], q[2]);
            if (S.label[j] == kBG) continue; // (background or outside the fluid region)
            if (d > 0 && left && S.label[j - 1] != kBG) continue;
            unite(S.label, c, j);
        }
    }
}

// Cells and volume per root.  Neighbouring entries of the list mostly belong to
// one component: a warp whose cells all do adds its sums with one atomic each (a
// jet's one component took an atomic per cell on one address).
__global__ void ccl_accumulate(Geometry G, const float *__restrict__ phi, DropScratch S) {
    const uint32_t total = S.n_out[1];
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint32_t lane = threadIdx.x & 31u;
    for (uint64_t i0 = blockIdx.x * (uint64_t)blockDim.x + (threadIdx.x & ~31u); i0 < total; i0 += stride) { // (warp-uniform)
        const uint64_t i = i0 + lane;
        const bool on = i < total;
        uint32_t r = 0;
        double vol = 0.0;
        if (on) {
            const uint32_t c = S.cells[i];
            r = find_root(S.label, c);
            vol = (double)phi[c];
        }
        const uint32_t active = __ballot_sync(0xffffffffu, on);
        const uint32_t r0 = __shfl_sync(0xffffffffu, r, 0); // (lane 0 is on whenever any lane is)
        if (__all_sync(0xffffffffu, !on || r == r0)) {
            for (int o = 16; o > 0; o >>= 1) vol += __shfl_xor_sync(0xffffffffu, vol, o);
            if (lane == 0) {
                atomicAdd(&S.count[r0], (uint32_t)__popc(active));
                atomicAdd(&S.volume[r0], vol);
            }
        } else if (on) {
            atomicAdd(&S.count[r], 1u);
            atomicAdd(&S.volume[r], vol);
        }
    }
}

// A list entry per root; its index replaces the root's count (max_list when the
// list is full), for ccl_touch.
__global__ void ccl_collect(DropScratch S) {
    const uint32_t total = S.n_out[1];
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < total; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t c = S.cells[i];
        if (S.label[c] != c) continue;
        const uint32_t slot_i = atomicAdd(S.n_out, 1u);
        const uint32_t cells = S.count[c];
        S.count[c] = slot_i;
        if (slot_i >= (uint32_t)S.max_list) continue;
        ssmd_droplet d;
        d.root = c;
        d.cells = cells;
        d.volume = S.volume[c];
        d.touches_inlet = 0u;
        d.reserved = 0u;
        S.list[slot_i] = d;
    }
}

// Components with a cell in the first fluid plane.
__global__ void ccl_touch(Geometry G, DropScratch S) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= G.nxy) return;
    const uint32_t c = (uint32_t)G.z_lo * G.nxy + i;
    if (S.label[c] == kBG) return;
    const uint32_t slot_i = S.count[find_root(S.label, c)];
    if (slot_i < (uint32_t)S.max_list) S.list[slot_i].touches_inlet = 1u;
}

size_t round256(size_t b) { return (b + 255) & ~(size_t)255; }

// Phase-field populations that cross the boundary of the fluid region in the
// step just taken.  In the pull layout fluid cell x gathers direction q from
// slot q of x - c_q, so phi enters from ghost slots (q, x - c_q) and leaves
// through the fluid slots (q, x) whose x + c_q is a ghost cell.  FP64 sums;
// with the collision conserving phi per cell this closes the budget
// sum phi^{n+1} = sum phi^n + inflow - outflow.
// Only the fluid cells beside a ghost layer take part, so only those planes are
// visited: blockIdx.y = 2 axis + side, first index along the face's first axis (scanning
// every cell for them took 82 us on 128 x 128 x 512 cells; the faces take 4.6).
template <class TG>
__global__ void phase_flux_kernel(Geometry G, const TG *g, double *acc) {
    __shared__ double s_in[256], s_out[256];
    double in = 0.0, out = 0.0;
    const int axis = (int)blockIdx.y >> 1, side = (int)blockIdx.y & 1;
    const bool per = axis == 0 ? G.bcx == BC_PERIODIC : (axis == 1 ? G.bcy == BC_PERIODIC : G.bcz == BC_PERIODIC);
    if (per) return; // (the whole block)
    const int lo[3] = {G.x_lo, G.y_lo, G.z_lo}, hi[3] = {G.x_hi, G.y_hi, G.z_hi};
    const uint32_t step[3] = {1u, G.nx, G.nxy};
    const int a0 = axis == 0 ? 1 : 0, a1 = axis == 2 ? 1 : 2;
    const uint32_t n0 = (uint32_t)(hi[a0] - lo[a0] + 1), n1 = (uint32_t)(hi[a1] - lo[a1] + 1);
    const int q_out = 2 * axis + (side ? 1 : 2), q_in = 2 * axis + (side ? 2 : 1); // 1:+x 2:-x 3:+y 4:-y 5:+z 6:-z
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < (uint64_t)n0 * n1;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t i1 = (uint32_t)(i / n0), i0 = (uint32_t)(i - (uint64_t)i1 * n0);
        const uint32_t c = (uint32_t)(side ? hi[axis] : lo[axis]) * step[axis] + (lo[a0] + i0) * step[a0] +
                           (lo[a1] + i1) * step[a1];
        const uint32_t ghost = side ? c + step[axis] : c - step[axis];
        in += (double)Store<TG>::ld(g + slot(G, q_in, ghost));
        out += (double)Store<TG>::ld(g + slot(G, q_out, c));
    }
    s_in[threadIdx.x] = in;
    s_out[threadIdx.x] = out;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) {
            s_in[threadIdx.x] += s_in[threadIdx.x + w];
            s_out[threadIdx.x] += s_out[threadIdx.x + w];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        atomicAdd(&acc[0], s_in[0]);
        atomicAdd(&acc[1], s_out[0]);
    }
}

} // namespace

extern "C" int ssmd_centreline(const ssmd_params *p, const LBMFields *fields, double *uz_out, double *phi_out,
                               ssmd_stream_t stream) {
    if (int e = ssmd_validate(p)) return e;
    if (!fields || !fields->uz || !fields->phi || !uz_out || !phi_out)
        return fail(SSMD_ERR_INVALID_ARGUMENT, "null argument");
    const Geometry G = make_geometry(*p);
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    centreline_kernel<<<(G.nz + 127) / 128, 128, 0, st>>>(G, make_fields(*fields), p->oil_cx, p->oil_cy, uz_out,
                                                         phi_out);
    return cuda_check(cudaGetLastError(), "centreline launch");
}

extern "C" size_t ssmd_droplets_scratch_bytes(const ssmd_params *p, int32_t max_droplets) {
    if (!p || max_droplets < 0) return 0;
    const size_t n = (size_t)p->nx * p->ny * p->nz;
    return round256(n * 4) * 3 + round256(n * 8) + 256 + round256((size_t)max_droplets * sizeof(ssmd_droplet));
}

extern "C" int ssmd_droplets(const ssmd_params *p, const LBMFields *fields, float threshold, void *scratch,
                             size_t scratch_bytes, ssmd_droplet *out, int32_t max_droplets, int32_t *n_out,
                             ssmd_stream_t stream) {
    if (int e = ssmd_validate(p)) return e;
    if (!fields || !fields->phi || !scratch || !out || !n_out || max_droplets <= 0)
        return fail(SSMD_ERR_INVALID_ARGUMENT, "null argument");
    if (scratch_bytes < ssmd_droplets_scratch_bytes(p, max_droplets))
        return fail(SSMD_ERR_INVALID_ARGUMENT, "scratch_bytes %zu < required %zu", scratch_bytes,
                    ssmd_droplets_scratch_bytes(p, max_droplets));
    const Geometry G = make_geometry(*p);
    const size_t n = G.cells;
    char *s = static_cast<char *>(scratch);
    DropScratch S{};
    S.label = reinterpret_cast<uint32_t *>(s);
    s += round256(n * 4);
    S.cells = reinterpret_cast<uint32_t *>(s);
    s += round256(n * 4);
    S.count = reinterpret_cast<uint32_t *>(s);
    s += round256(n * 4);
    S.volume = reinterpret_cast<double *>(s);
    s += round256(n * 8);
    S.n_out = reinterpret_cast<uint32_t *>(s);
    s += 256;
    S.list = reinterpret_cast<ssmd_droplet *>(s);
    S.max_list = max_droplets;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (int e = cuda_check(cudaMemsetAsync(S.n_out, 0, 2 * sizeof(uint32_t), st), "droplet counters")) return e;
    ccl_init<<<(unsigned)((n + kCclCells - 1) / kCclCells), kCclThreads, 0, st>>>(G, fields->phi, threshold, S);
    const unsigned nb = (unsigned)std::min<size_t>((n + 255) / 256, 8 * 148); // (grid-stride over the list)
    ccl_union<<<nb, 256, 0, st>>>(G, S);
    ccl_accumulate<<<nb, 256, 0, st>>>(G, fields->phi, S);
    ccl_collect<<<nb, 256, 0, st>>>(S);
    ccl_touch<<<(G.nxy + 255) / 256, 256, 0, st>>>(G, S);
    if (int e = cuda_check(cudaGetLastError(), "droplet kernels")) return e;
    // the number found and the first entries in one read (the list follows its header)
    constexpr int kFirst = 256;
    const int32_t first = max_droplets < kFirst ? max_droplets : kFirst;
    alignas(16) char head[256 + kFirst * sizeof(ssmd_droplet)];
    if (int e = cuda_check(cudaMemcpyAsync(head, S.n_out, 256 + (size_t)first * sizeof(ssmd_droplet),
                                           cudaMemcpyDeviceToHost, st),
                           "droplet list"))
        return e;
    if (int e = cuda_check(cudaStreamSynchronize(st), "droplet sync")) return e;
    uint32_t found = 0;
    std::memcpy(&found, head, sizeof found);
    const int32_t k = (int32_t)(found < (uint32_t)max_droplets ? found : (uint32_t)max_droplets);
    std::memcpy(out, head + 256, sizeof(ssmd_droplet) * (size_t)std::min(k, first));
    if (k > first) {
        if (int e = cuda_check(cudaMemcpyAsync(out + first, S.list + first, sizeof(ssmd_droplet) * (size_t)(k - first),
                                               cudaMemcpyDeviceToHost, st),
                               "droplet list"))
            return e;
        if (int e = cuda_check(cudaStreamSynchronize(st), "droplet sync")) return e;
    }
    *n_out = (int32_t)found;
    return found > (uint32_t)max_droplets
               ? fail(SSMD_ERR_INVALID_ARGUMENT, "%u droplets found, only %d returned", found, max_droplets)
               : SSMD_OK;
}

extern "C" int ssmd_phase_flux(const ssmd_params *p, const LBMFields *fields, uint64_t steps_done, double *inflow,
                               double *outflow, ssmd_stream_t stream) {
    if (int e = ssmd_validate(p)) return e;
    if (int e = check_fields(*p, fields)) return e;
    if (!inflow || !outflow) return fail(SSMD_ERR_INVALID_ARGUMENT, "null output");
    const Geometry G = make_geometry(*p);
    const void *g = (steps_done & 1ull) == 0ull ? fields->g : p->g_alt;
    double *acc = reinterpret_cast<double *>(static_cast<char *>(p->workspace) + kPartialOff);
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (int e = cuda_check(cudaMemsetAsync(acc, 0, 2 * sizeof(double), st), "flux clear")) return e;
    const uint64_t face = std::max({(uint64_t)G.nx * G.ny, (uint64_t)G.nx * G.nz, (uint64_t)G.ny * G.nz});
    const dim3 nb((unsigned)std::min<uint64_t>((face + 255) / 256, 512), 6);
    switch (p->storage) {
    case SSMD_STORAGE_F32: phase_flux_kernel<float><<<nb, 256, 0, st>>>(G, static_cast<const float *>(g), acc); break;
    case SSMD_STORAGE_F16: phase_flux_kernel<__half><<<nb, 256, 0, st>>>(G, static_cast<const __half *>(g), acc); break;
    case SSMD_STORAGE_F16_G32: // g as float
        phase_flux_kernel<float><<<nb, 256, 0, st>>>(G, static_cast<const float *>(g), acc);
        break;
    default: { // BF16 runs keep g in half
        using TG = phase_t<__nv_bfloat16>;
        phase_flux_kernel<TG><<<nb, 256, 0, st>>>(G, static_cast<const TG *>(g), acc);
        break;
    }
    }
    if (int e = cuda_check(cudaGetLastError(), "flux launch")) return e;
    double h[2] = {0.0, 0.0};
    if (int e = cuda_check(cudaMemcpyAsync(h, acc, sizeof h, cudaMemcpyDeviceToHost, st), "flux copy")) return e;
    if (int e = cuda_check(cudaStreamSynchronize(st), "flux sync")) return e;
    *inflow = h[0];
    *outflow = h[1];
    return SSMD_OK;
}
