// mlp.cu — the learned closure's per-cell network on the 5th-generation tensor cores.
//
// Network: 12 features -> 64 -> 64 -> 2 outputs, GELU after the two hidden
// layers in its tanh form, gelu(z) = z/2 (1 + tanh(sqrt(2/pi) (z + 0.044715
// z^3))) (Hendrycks & Gimpel, "Gaussian Error Linear Units", 2016), with
// tanh from the SFU (tanh.approx.f32, absolute error about 2^-11, below the
// bf16 rounding of the hidden activations that follows), features
// standardised by stored mean / inverse std, outputs p = scale * r + offset
// with r the last layer's raw output.  A persistent CTA loops over tiles of 128
// cells, weights staged once per CTA; inference: 128 threads, thread i <-> cell row i
// of the tile; training: 512 threads, four per row (mlp_train_kernel):
//   X [128 x 16] (bf16, K padded 12 -> 16)   z1 = X W1^T      (tcgen05, N = 64, K = 16)
//   H1 = gelu(z1 + b1) [128 x 64] bf16        z2 = H1 W2^T     (4 MMAs of K = 16)
//   H2 = gelu(z2 + b2) [128 x 64] bf16        r  = H2 W3^T     (N padded 2 -> 16)
// The epilogues read the accumulators back with tcgen05.ld (inference: the next 16
// columns in flight while the current 16 are processed), add the bias,
// apply GELU on pairs of columns with packed FP32 arithmetic (fma.rn.f32x2
// and friends, sm_100) and write the next layer's bf16 operand.  Inference
// stages W2 and W3 halved and its epilogues write 2 gelu(z), one multiply
// fewer per value: the products, hence every result, are the same bit for
// bit (scaling by 2 commutes with each rounding).
// Inference (forward, and the fused closure refresh that computes the
// features from the macroscopic fields and applies the outputs) keeps one
// 64-column accumulator (z1, z2 and r in turn: each is dead once its
// epilogue has read it) and one activation tile (X, H1, H2 in turn: each is
// dead once the MMA reading it has completed), 29 KB of shared memory and 64
// TMEM columns per CTA, so seven CTAs share an SM and hide each other's MMA
// round trips.
// Training (ssmd_mlp_grad) keeps z1 and z2 for the backward pass:
//   L = (1/n) sum_i sum_k w_ik (r_ik - (t_ik - offset_k) / scale_k)^2,
// dH2 = dR W3 and dZ2 = dH2 gelu'(z2 + b2) on the CUDA cores (N = 2 is too
// narrow for an MMA), dH1 = dZ2 W2 on the tensor cores, dZ1 = dH1 gelu'(z1 +
// b1); the weight and bias gradients (sums over a tile's 128 rows) on the
// tensor cores too: two MMAs per tile whose K is the tile's rows read the same
// row-wise tiles X, H1, H2, dZ1, dZ2, dR as MN-major operands and accumulate
// dW2^T, dW3^T (G1) and dW1^T with the bias gradients (G2, through a column of
// ones in X) in TMEM across the CTA's tiles; they run while the next tile
// begins.  The CTA's sums are then either added across CTAs with
// atomics (ssmd_mlp_grad) or written as one row per CTA and summed in CTA
// order by a second kernel (ssmd_mlp_grad_ws: the same bits on every run).  Every
// wait on an MMA is bounded: on timeout the CTA records bit 0 of the status word,
// frees its TMEM and returns.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "adam.cuh"
#include "closure.cuh"
#include "host.cuh"
#include "umma.cuh"

using namespace ssmd;
using namespace ssmd::host;

namespace {

constexpr int kIn = SSMD_MLP_IN, kK1 = 16, kH = SSMD_MLP_HIDDEN, kOut = SSMD_MLP_OUT, kN3 = 16;
constexpr int kRows = 128, kThreadsMlp = 128;
constexpr int kTrainGroups = 4, kThreadsTrain = kTrainGroups * kRows; // training: 16 columns of a row per thread
constexpr int oW1 = 0, oB1 = oW1 + kH * kK1, oW2 = oB1 + kH, oB2 = oW2 + kH * kH, oW3 = oB2 + kH,
              oB3 = oW3 + kOut * kH, kParams = oB3 + kOut;
constexpr int oMean = kParams, oInvStd = oMean + kIn, oScale = oInvStd + kIn, oOffset = oScale + kOut,
              kNet = oOffset + kOut;
static_assert(kParams == SSMD_MLP_PARAMS, "parameter layout");
static_assert(kNet == SSMD_MLP_NET_FLOATS, "network layout");

enum : int { kFwd = 0, kTrain = 1, kRefresh = 2 };

// TMEM columns: training keeps z1 (0-63) and z2 (64-127) for the backward
// pass, r at 128-143, dH1 at 192-255 and the CTA's weight-gradient sums
// across its tiles at 256-335 (G1) and 336-479 (G2); inference puts z1, z2
// and r in turn on columns 0-63.
template <int MODE>
constexpr uint32_t tmem_cols() { return MODE == kTrain ? 512u : 64u; }
template <int MODE>
constexpr uint32_t col_z2() { return MODE == kTrain ? 64u : 0u; }
template <int MODE>
constexpr uint32_t col_r() { return MODE == kTrain ? 128u : 0u; }
constexpr uint32_t cZ1 = 0, cDH1 = 192, cG1 = 256, cG2 = 336;
constexpr int kGB = 2 * kH + 16;   // columns of the gradient tile: dZ1, dZ2, dR (2 of 16)
constexpr uint64_t kMmaWaitNs = 1000000000ull;

// shared-memory map (bytes from an aligned base: 1024 bytes for training,
// 128 for inference; the no-swizzle operand layout needs 16).  Training, all
// bf16, 8 x 8 core matrices of 128 bytes, a row group of 8 rows after the other:
//   X, twice [128 x 16]: columns 0-11 the features, 12 ones, 13-15 zero (this
//       tile's and the next's: the gradient MMA reads the one while the other is written)
//   HH [128 x 128]: H1 (columns 0-63), H2 (64-127)
//   DZ [128 x 144]: dZ1 (0-63), dZ2 (64-127), dR (128-129), zeros
// Each is a K-major operand (rows M) of the layers' MMAs and, with its rows as K, an
// MN-major one of the gradient MMAs: G1 = HH^T DZ[:, 64..143] holds dW2^T and dW3^T, G2 =
// X^T DZ holds dW1^T and, in its ones row, the three bias gradients (G2's M = 128
// reads columns 16-127 past X: their products land in accumulator rows nobody
// reads).  (Transposed copies of all six, 270 two-byte stores per row with
// 4-way bank conflicts, were 4000 of the 14 000 cycles of a tile and 55 KB more.)
constexpr uint32_t sXT = 0, kXBytes = kRows * kK1 * 2, sHH = 2 * kXBytes, sDZ = sHH + kRows * 2 * kH * 2,
                   sW1T = sDZ + kRows * kGB * 2, sW3T = sW1T + kH * kK1 * 2, sW2T = sW3T + kN3 * kH * 2,
                   sDY = sW2T + kH * kH * 2;
constexpr uint32_t kXGroup = kK1 / 8 * 128, kHGroup = 2 * kH / 8 * 128, kDGroup = kGB / 8 * 128; // a row group's bytes
// (the last K step's second row group of the second X buffer, and 128 columns from there)
static_assert(kXBytes + (kRows / 8 - 1) * kXGroup + 128 / 8 * 128 <= sDZ, "G2's reads past X stay inside X and HH");
template <int MODE>
struct Layout {
    static constexpr bool T = MODE == kTrain;
    // inference: W1, W3, W2, then one activation tile that holds X, H1, H2 in turn
    static constexpr uint32_t sW1 = T ? sW1T : 0, sW3 = T ? sW3T : 2048, sH1 = 12288, sW2 = T ? sW2T : 4096, sH2 = sH1,
                              sX = sH1;
    static constexpr uint32_t big = T ? sDY + kRows * kOut * 4 : sH1 + kRows * kH * 2;
    static constexpr uint32_t b1 = big, b2 = b1 + kH * 4, b3 = b2 + kH * 4, w3f = b3 + 16,
                              norm = w3f + (T ? kOut * kH * 4 : 0), bar = norm + 32 * 4, slot = bar + 8,
                              abort = slot + 4, end = abort + 4;
    static constexpr uint32_t align = T ? 1024 : 128;
    static constexpr size_t bytes = end + align; // + alignment slack of the dynamic base
};

// Everything a launch needs (one struct for the three modes).
struct MlpArgs {
    const float *net;
    const float *feat;   // kFwd, kTrain: n x 12 features
    const float *target; // kTrain
    const float *weight; // kTrain (may be null)
    const int64_t *rows; // kTrain: row i of the batch is row rows[i] of feat, target, weight (null: row i)
    int64_t n_rows;      // kTrain: rows of feat, target, weight
    int64_t n;
    float *out;          // kFwd: n x 2
    float *grad;         // kTrain: atomics into grad, or null with partials
    float *partials;     // kTrain deterministic: one row of kParams + 1 per CTA
    double *loss;        // kTrain (atomic path)
    closure::Grid g;     // kRefresh: the lattice and its macroscopic fields
    const float *rho, *ux, *uy, *uz, *phi;
    float nu_w, nu_dow, nut_max;
    float *nut, *cs;     // kRefresh outputs
};

__device__ unsigned int g_mlp_status;

// GELU, tanh form: u = sqrt(2/pi) z (1 + 0.044715 z^2), gelu = z/2 + z/2 tanh(u)
constexpr float kG0 = 0.7978845608028654f;           // sqrt(2 / pi)
constexpr float kG1 = 0.7978845608028654f * 0.044715f;

__device__ __forceinline__ float tanh_sfu(float x) {
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// gelu of two columns at once: u = z fma(kG1, z^2, kG0), h = z/2,
// gelu = fma(h, tanh(u), h), elementwise with packed FP32 (fma.rn.f32x2 etc.);
// TWICE: 2 gelu(z) = fma(z, tanh(u), z).
template <bool TWICE = false>
__device__ __forceinline__ float2 gelu2(float2 z) {
    const float2 p = __ffma2_rn(__fmul2_rn(z, z), make_float2(kG1, kG1), make_float2(kG0, kG0));
    const float2 u = __fmul2_rn(z, p);
    const float2 t = make_float2(tanh_sfu(u.x), tanh_sfu(u.y));
    if constexpr (TWICE) return __ffma2_rn(z, t, z);
    const float2 hz = __fmul2_rn(z, make_float2(0.5f, 0.5f));
    return __ffma2_rn(hz, t, hz);
}
// d gelu / dz = (1 + t)/2 + z/2 (1 - t^2) du/dz,  du/dz = sqrt(2/pi) (1 + 3 * 0.044715 z^2)
__device__ __forceinline__ float gelu_grad(float z) {
    const float z2 = z * z;
    const float t = tanh_sfu(z * fmaf(kG1, z2, kG0));
    const float du = fmaf(3.0f * kG1, z2, kG0);
    return fmaf(0.5f * z * du, fmaf(-t, t, 1.0f), fmaf(0.5f, t, 0.5f));
}

__device__ __forceinline__ uint32_t pack2(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&h);
}

// Store 8 consecutive values (k0 .. k0 + 7) of row r of an R x K bf16 tile.
__device__ __forceinline__ void st8(unsigned char *tile, int r, int k0, int K, const float *v) {
    uint4 u;
    u.x = pack2(v[0], v[1]);
    u.y = pack2(v[2], v[3]);
    u.z = pack2(v[4], v[5]);
    u.w = pack2(v[6], v[7]);
    *reinterpret_cast<uint4 *>(tile + umma::kmajor_offset(r, k0, K)) = u;
}


// Copy a [ROWS x K] block of fp32 weights (row stride K), times `scale` (a
// power of two), into a bf16 tile of ROWS_PAD rows (extra rows and the columns from KV on
// zero).  A thread converts 8 values of a row and
// stores them at once, and all its loads are in flight together: a CTA's
// set-up is one round trip, not one per element of a thread (training kernel
// on 65 536 rows, 4 tiles a CTA: 3 us of 43; forward of 1 M rows, 8 tiles a CTA: 75 ->
// 67; refresh of 96 x 96 x 384 cells: 238 -> 229).
template <int ROWS, int ROWS_PAD, int K, int THREADS, int KV = K>
__device__ __forceinline__ void load_weights(unsigned char *tile, const float *src, int tid, float scale = 1.0f) {
    constexpr int CHUNKS = ROWS_PAD * (K / 8);
#pragma unroll
    for (int c0 = 0; c0 < CHUNKS; c0 += THREADS) {
        const int c = c0 + tid;
        if (CHUNKS % THREADS != 0 && c >= CHUNKS) break;
        const int r = c / (K / 8), k0 = 8 * (c % (K / 8));
        float v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = r < ROWS && k0 + i < KV ? __ldg(src + r * K + k0 + i) * scale : 0.f;
        st8(tile, r, k0, K, v);
    }
}

// Bounded wait on the MMA barrier by every thread, then a block-wide vote.
__device__ __forceinline__ bool wait_mma(uint64_t *bar, uint32_t phase, volatile uint32_t *abort_flag) {
    if (!mbar_wait_bounded(bar, phase, kMmaWaitNs)) *abort_flag = 1u;
    __syncthreads();
    const bool ok = *abort_flag == 0u;
    if (ok) umma::fence_after_sync();
    return ok;
}

// Bias + GELU of 16 accumulator columns v (columns c0 .. c0 + 15 of the layer)
// into columns t0 .. t0 + 15 of row r of a bf16 tile of K columns (TWICE: 2 gelu, for a
// next layer staged with halved weights).
template <bool TWICE, int K>
__device__ __forceinline__ void gelu16(const float (&v)[16], const float *bias, int c0, unsigned char *tile, int r,
                                       int t0) {
    uint32_t pk[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float4 b = *reinterpret_cast<const float4 *>(bias + c0 + 4 * i);
        const float2 g0 = gelu2<TWICE>(__fadd2_rn(make_float2(v[4 * i], v[4 * i + 1]), make_float2(b.x, b.y)));
        const float2 g1 = gelu2<TWICE>(__fadd2_rn(make_float2(v[4 * i + 2], v[4 * i + 3]), make_float2(b.z, b.w)));
        pk[2 * i] = pack2(g0.x, g0.y);
        pk[2 * i + 1] = pack2(g1.x, g1.y);
    }
    *reinterpret_cast<uint4 *>(tile + umma::kmajor_offset(r, t0, K)) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
    *reinterpret_cast<uint4 *>(tile + umma::kmajor_offset(r, t0 + 8, K)) = make_uint4(pk[4], pk[5], pk[6], pk[7]);
}

// Inference epilogue of a 64-column accumulator: the TMEM load of columns
// 16 (c + 1) .. 16 c + 31 is in flight while columns 16 c .. 16 c + 15 are processed.
__device__ __forceinline__ void hidden_epilogue(uint32_t taddr, const float *bias, unsigned char *tile, int r) {
    uint32_t nxt[16];
    umma::tmem_ld16_issue(taddr, nxt);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        float v[16];
        umma::tmem_ld_wait16(nxt);
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(nxt[i]);
        if (c < 3) umma::tmem_ld16_issue(taddr + 16 * (c + 1), nxt);
        gelu16<true, kH>(v, bias, 16 * c, tile, r, 16 * c);
    }
}

// Training epilogue of columns 16 grp .. 16 grp + 15, into HH from column t0 on.
__device__ __forceinline__ void hidden_epilogue16(uint32_t taddr, const float *bias, unsigned char *hh, int r, int grp,
                                                  int t0) {
    float v[16];
    umma::tmem_ld16(taddr + 16 * grp, v);
    gelu16<false, 2 * kH>(v, bias, 16 * grp, hh, r, t0 + 16 * grp);
}

// The 12 standardised features of one row into x[16] (columns 12-15 zero);
// kRefresh also returns feature 11, nu(phi), for the bound on nu_t.
template <int MODE>
__device__ __forceinline__ void load_row(const MlpArgs &a, const float *norm, int64_t row, bool valid, float (&x)[kK1],
                                         float &nu_phi) {
#pragma unroll
    for (int i = 0; i < kK1; ++i) x[i] = 0.f;
    nu_phi = 0.f;
    if (!valid) return;
    float f[kIn];
    if constexpr (MODE == kRefresh) {
        closure::cell_features(a.g, a.rho, a.ux, a.uy, a.uz, a.phi, a.nu_w, a.nu_dow, row, f);
    } else if ((reinterpret_cast<uintptr_t>(a.feat) & 15u) == 0) {
        const float4 *p = reinterpret_cast<const float4 *>(a.feat + row * kIn); // 48-byte rows: 16-byte aligned
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const float4 v = __ldg(p + q);
            f[4 * q] = v.x;
            f[4 * q + 1] = v.y;
            f[4 * q + 2] = v.z;
            f[4 * q + 3] = v.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < kIn; ++i) f[i] = __ldg(a.feat + row * kIn + i);
    }
    nu_phi = f[11];
#pragma unroll
    for (int i = 0; i < kIn; ++i) x[i] = (f[i] - norm[i]) * norm[kIn + i];
}

template <int MODE>
__global__ void __launch_bounds__(kThreadsMlp, 7) mlp_kernel(const MlpArgs a) {
    static_assert(MODE == kFwd || MODE == kRefresh, "training has its own kernel");
    using L = Layout<MODE>;
    extern __shared__ unsigned char smem_raw[];
    unsigned char *sm = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + (L::align - 1)) &
                                                          ~(uintptr_t)(L::align - 1));
    const int tid = threadIdx.x, warp = tid >> 5;
    const float *net = a.net;
    const int64_t n = a.n;
    float *b1 = reinterpret_cast<float *>(sm + L::b1);
    float *b2 = reinterpret_cast<float *>(sm + L::b2);
    float *b3 = reinterpret_cast<float *>(sm + L::b3);
    float *norm = reinterpret_cast<float *>(sm + L::norm);
    uint64_t *bar = reinterpret_cast<uint64_t *>(sm + L::bar);
    uint32_t *slot = reinterpret_cast<uint32_t *>(sm + L::slot);
    volatile uint32_t *abort_flag = reinterpret_cast<volatile uint32_t *>(sm + L::abort);

    // ---- set-up: TMEM, barrier, weights
    if (warp == 0) umma::tmem_alloc(slot, tmem_cols<MODE>());
    if (tid == 0) {
        mbar_init(bar, 1);
        *abort_flag = 0u;
        fence_barrier_init();
    }
    // W2 and W3 are fed with 2 gelu(z): halved weights, the same products
    load_weights<kH, kH, kK1, kThreadsMlp>(sm + L::sW1, net + oW1, tid);
    load_weights<kH, kH, kH, kThreadsMlp>(sm + L::sW2, net + oW2, tid, 0.5f);
    load_weights<kOut, kN3, kH, kThreadsMlp>(sm + L::sW3, net + oW3, tid, 0.5f);
    for (int e = tid; e < kH; e += kThreadsMlp) {
        b1[e] = net[oB1 + e];
        b2[e] = net[oB2 + e];
    }
    if (tid < kOut) b3[tid] = net[oB3 + tid];
    if (tid < kNet - kParams) norm[tid] = net[kParams + tid];
    __syncthreads();

    const int r = tid;
    const uint32_t sbase = smem_addr(sm);
    uint32_t phase = 0;
    bool ok = true;
    const int64_t tiles = (n + kRows - 1) / kRows;
    uint32_t tmem = 0, lane_base = 0;

    for (int64_t tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
        const int64_t row = tile * kRows + r;
        const bool valid = row < n;
        float nu_phi;
        {
            float x[kK1];
            load_row<MODE>(a, norm, row, valid, x, nu_phi);
            st8(sm + L::sX, r, 0, kK1, x);
            st8(sm + L::sX, r, 8, kK1, x + 8);
        }
        fence_proxy_async(); // generic-proxy smem writes -> visible to the tensor core
        umma::fence_before_sync();
        __syncthreads(); // also: every TMEM read and MMA of the previous tile is complete
        tmem = *slot;
        lane_base = tmem + ((uint32_t)(warp * 32) << 16);

        // ---- layer 1
        if (tid == 0) {
            umma::fence_after_sync();
            umma::mma_bf16(tmem + cZ1, umma::smem_desc(sbase + L::sX, 128, 256),
                           umma::smem_desc(sbase + L::sW1, 128, 256), umma::idesc_bf16(128, kH), false);
            umma::commit(bar);
        }
        ok = wait_mma(bar, phase, abort_flag);
        phase ^= 1u;
        if (!ok) break;
        hidden_epilogue(lane_base + cZ1, b1, sm + L::sH1, r);
        fence_proxy_async();
        umma::fence_before_sync();
        __syncthreads();

        // ---- layer 2
        if (tid == 0) {
            umma::fence_after_sync();
            for (int ks = 0; ks < kH / 16; ++ks)
                umma::mma_bf16(tmem + col_z2<MODE>(), umma::smem_desc(sbase + L::sH1 + 256 * ks, 128, 1024),
                               umma::smem_desc(sbase + L::sW2 + 256 * ks, 128, 1024), umma::idesc_bf16(128, kH),
                               ks > 0);
            umma::commit(bar);
        }
        ok = wait_mma(bar, phase, abort_flag);
        phase ^= 1u;
        if (!ok) break;
        hidden_epilogue(lane_base + col_z2<MODE>(), b2, sm + L::sH2, r);
        fence_proxy_async();
        umma::fence_before_sync();
        __syncthreads();

        // ---- layer 3 (N padded to 16; rows 2..15 of W3 are zero)
        if (tid == 0) {
            umma::fence_after_sync();
            for (int ks = 0; ks < kH / 16; ++ks)
                umma::mma_bf16(tmem + col_r<MODE>(), umma::smem_desc(sbase + L::sH2 + 256 * ks, 128, 1024),
                               umma::smem_desc(sbase + L::sW3 + 256 * ks, 128, 1024), umma::idesc_bf16(128, kN3),
                               ks > 0);
            umma::commit(bar);
        }
        ok = wait_mma(bar, phase, abort_flag);
        phase ^= 1u;
        if (!ok) break;
        float rr[kOut];
        {
            float v[2];
            umma::tmem_ld2(lane_base + col_r<MODE>(), v);
            rr[0] = v[0] + b3[0];
            rr[1] = v[1] + b3[1];
        }
        if constexpr (MODE == kFwd) {
            if (valid)
                *reinterpret_cast<float2 *>(a.out + row * kOut) =
                    make_float2(fmaf(norm[2 * kIn + 0], rr[0], norm[2 * kIn + 2]),
                                fmaf(norm[2 * kIn + 1], rr[1], norm[2 * kIn + 3]));
        } else {
            // the closure's bounds (ssmd_closure_apply): nu_t >= max(-nu(phi)/2, -nut_max)
            if (valid) {
                const float p0 = fmaf(norm[2 * kIn + 0], rr[0], norm[2 * kIn + 2]);
                const float p1 = fmaf(norm[2 * kIn + 1], rr[1], norm[2 * kIn + 3]);
                const float lo = fmaxf(-0.5f * nu_phi, -a.nut_max);
                a.nut[row] = fminf(fmaxf(p0, lo), a.nut_max);
                a.cs[row] = fminf(fmaxf(p1, 0.25f), 4.0f);
            }
        }
    }

    // ---- tear-down: every TMEM read is complete before the warp frees it
    umma::fence_before_sync();
    __syncthreads();
    if (!ok && tid == 0) atomicOr(&g_mlp_status, 1u);
    if (warp == 0) umma::tmem_dealloc(*slot, tmem_cols<MODE>());
}

// What a training thread holds of one row before its tile begins: features
// 4 grp .. 4 grp + 3 (groups 0-2), targets and weights.
struct TrainRow {
    float4 f;
    float t0, t1, w0, w1;
    bool valid;
};

// Training: 512 threads per CTA, one CTA per SM (512 TMEM columns).  Thread (grp,
// r) handles row r and, of every 64-column layer, columns 16 grp .. 16 grp + 15.  The
// kernel is a chain of MMA round trips and epilogues per tile; with one thread
// per row (4 warps per SM, one per scheduler) the epilogues' ~5000 instructions
// ran at the latency of one warp: 15 us a tile, 62 us for 65 536 rows; with four
// threads per row 40, the gather included, and 28 with the gradient MMAs reading
// row-wise tiles (see the shared-memory map) and a row's index loaded a tile ahead of
// the row.  The rows of a mini-batch are read through their indices (a.rows), the
// next tile's while this one's layers run: gathering them first took three launches
// and 50 us of the 128 us step.  Every value and every sum is in the order of one
// thread per row: the same bits.
__global__ void __launch_bounds__(kThreadsTrain, 1) mlp_train_kernel(const MlpArgs a) {
    using L = Layout<kTrain>;
    extern __shared__ unsigned char smem_raw[];
    unsigned char *sm = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + (L::align - 1)) &
                                                          ~(uintptr_t)(L::align - 1));
    const int tid = threadIdx.x, warp = tid >> 5;
    const int r = tid & (kRows - 1), grp = tid / kRows;
    const float *net = a.net;
    const int64_t n = a.n;
    float *b1 = reinterpret_cast<float *>(sm + L::b1);
    float *b2 = reinterpret_cast<float *>(sm + L::b2);
    float *b3 = reinterpret_cast<float *>(sm + L::b3);
    float *w3f = reinterpret_cast<float *>(sm + L::w3f);
    float *norm = reinterpret_cast<float *>(sm + L::norm);
    uint64_t *bar = reinterpret_cast<uint64_t *>(sm + L::bar);
    uint32_t *slot = reinterpret_cast<uint32_t *>(sm + L::slot);
    volatile uint32_t *abort_flag = reinterpret_cast<volatile uint32_t *>(sm + L::abort);
    const int64_t tiles = (n + kRows - 1) / kRows;

    // the source row of this thread's row of a tile; -1: none
    auto source = [&](int64_t tile) -> int64_t {
        const int64_t row = tile * kRows + r;
        if (row >= n) return -1;
        if (!a.rows) return row;
        const int64_t s = __ldg(a.rows + row);
        if (s >= 0 && s < a.n_rows) return s;
        if (grp == 0) atomicOr(&g_mlp_status, 2u);
        return -1;
    };
    const bool aligned = (reinterpret_cast<uintptr_t>(a.feat) & 15u) == 0; // 48-byte rows: 16-byte aligned
    auto fetch = [&](int64_t s) -> TrainRow {
        TrainRow d;
        d.f = make_float4(0.f, 0.f, 0.f, 0.f);
        d.t0 = d.t1 = d.w0 = d.w1 = 0.f;
        d.valid = s >= 0;
        if (!d.valid) return d;
        if (grp < kIn / 4) {
            const float *p = a.feat + s * kIn + 4 * grp;
            if (aligned) d.f = __ldg(reinterpret_cast<const float4 *>(p));
            else d.f = make_float4(__ldg(p), __ldg(p + 1), __ldg(p + 2), __ldg(p + 3));
        }
        d.t0 = a.target[s * kOut + 0];
        d.t1 = a.target[s * kOut + 1];
        d.w0 = a.weight ? a.weight[s * kOut + 0] : 1.0f;
        d.w1 = a.weight ? a.weight[s * kOut + 1] : 1.0f;
        return d;
    };
    // (a row's index is loaded a tile before the row itself: two round trips, neither waited for)
    TrainRow cur = fetch((int64_t)blockIdx.x < tiles ? source(blockIdx.x) : -1);
    int64_t nsrc = (int64_t)blockIdx.x + gridDim.x < tiles ? source((int64_t)blockIdx.x + gridDim.x) : -1;

    // ---- set-up: TMEM, barrier, weights
    if (warp == 0) umma::tmem_alloc(slot, tmem_cols<kTrain>());
    if (tid == 0) {
        mbar_init(bar, 1);
        *abort_flag = 0u;
        fence_barrier_init();
    }
    load_weights<kH, kH, kK1, kThreadsTrain, kIn>(sm + L::sW1, net + oW1, tid); // (X's column 12 is the gradients' ones)
    load_weights<kH, kH, kH, kThreadsTrain>(sm + L::sW2, net + oW2, tid);
    load_weights<kOut, kN3, kH, kThreadsTrain>(sm + L::sW3, net + oW3, tid);
    if (tid < kH) {
        b1[tid] = net[oB1 + tid];
        b2[tid] = net[oB2 + tid];
    }
    if (tid < kOut * kH) w3f[tid] = net[oW3 + tid];
    if (tid < kOut) b3[tid] = net[oB3 + tid];
    if (tid < kNet - kParams) norm[tid] = net[kParams + tid];
    if (grp == 0) { // the columns of DZ that no tile writes: 130-143 (128-129 with every tile)
        *reinterpret_cast<uint4 *>(sm + sDZ + umma::kmajor_offset(r, 2 * kH, kGB)) = make_uint4(0u, 0u, 0u, 0u);
        *reinterpret_cast<uint4 *>(sm + sDZ + umma::kmajor_offset(r, 2 * kH + 8, kGB)) = make_uint4(0u, 0u, 0u, 0u);
    }
    __syncthreads();

    const uint32_t sbase = smem_addr(sm);
    uint32_t phase = 0;
    bool ok = true;
    // the weight-gradient MMAs of a tile run while the next tile begins: the commit
    // of that tile's first MMA covers them, before anything they read is written
    bool gfirst = true;
    uint32_t xbuf = 0;
    float lsum = 0.f;
    const uint32_t tmem = *slot;
    const uint32_t lane_base = tmem + ((uint32_t)((warp & 3) * 32) << 16);

    for (int64_t tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
        const uint32_t sX = sXT + xbuf * kXBytes;
        {
            // group 3 writes columns 12-15: one, zeros
            float x[4];
            const float f[4] = {cur.f.x, cur.f.y, cur.f.z, cur.f.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
                x[i] = grp == kIn / 4 ? (i == 0 ? 1.0f : 0.f)
                                      : (cur.valid ? (f[i] - norm[4 * grp + i]) * norm[kIn + 4 * grp + i] : 0.f);
            *reinterpret_cast<uint2 *>(sm + sX + umma::kmajor_offset(r, 4 * grp, kK1)) =
                make_uint2(pack2(x[0], x[1]), pack2(x[2], x[3]));
        }
        fence_proxy_async(); // generic-proxy smem writes -> visible to the tensor core
        umma::fence_before_sync();
        __syncthreads(); // also: every TMEM read of the previous tile is complete

        // ---- layer 1
        if (tid == 0) {
            umma::fence_after_sync();
            umma::mma_bf16(tmem + cZ1, umma::smem_desc(sbase + sX, 128, kXGroup),
                           umma::smem_desc(sbase + L::sW1, 128, 256), umma::idesc_bf16(128, kH), false);
            umma::commit(bar);
        }
        const TrainRow nxt = fetch(nsrc);
        nsrc = tile + 2 * (int64_t)gridDim.x < tiles ? source(tile + 2 * (int64_t)gridDim.x) : -1;
        ok = wait_mma(bar, phase, abort_flag);
        phase ^= 1u;
        if (!ok) break;
        hidden_epilogue16(lane_base + cZ1, b1, sm + sHH, r, grp, 0);
        fence_proxy_async();
        umma::fence_before_sync();
        __syncthreads();

        // ---- layer 2
        if (tid == 0) {
            umma::fence_after_sync();
            for (int ks = 0; ks < kH / 16; ++ks)
                umma::mma_bf16(tmem + col_z2<kTrain>(), umma::smem_desc(sbase + sHH + 256 * ks, 128, kHGroup),
                               umma::smem_desc(sbase + L::sW2 + 256 * ks, 128, 1024), umma::idesc_bf16(128, kH),
                               ks > 0);
            umma::commit(bar);
        }
        ok = wait_mma(bar, phase, abort_flag);
        phase ^= 1u;
        if (!ok) break;
        hidden_epilogue16(lane_base + col_z2<kTrain>(), b2, sm + sHH, r, grp, kH);
        fence_proxy_async();
        umma::fence_before_sync();
        __syncthreads();

        // ---- layer 3 (N padded to 16; rows 2..15 of W3 are zero)
        if (tid == 0) {
            umma::fence_after_sync();
            for (int ks = 0; ks < kH / 16; ++ks)
                umma::mma_bf16(tmem + col_r<kTrain>(), umma::smem_desc(sbase + sHH + kH / 8 * 128 + 256 * ks, 128, kHGroup),
                               umma::smem_desc(sbase + L::sW3 + 256 * ks, 128, 1024), umma::idesc_bf16(128, kN3),
                               ks > 0);
            umma::commit(bar);
        }
        ok = wait_mma(bar, phase, abort_flag);
        phase ^= 1u;
        if (!ok) break;
        float rr[kOut];
        {
            float v[2];
            umma::tmem_ld2(lane_base + col_r<kTrain>(), v);
            rr[0] = v[0] + b3[0];
            rr[1] = v[1] + b3[1];
        }
        // ---- loss and dL/dr (each of a row's threads; group 0 keeps the sum)
        float d0 = 0.f, d1 = 0.f;
        if (cur.valid) {
            const float inv_n = 1.0f / (float)n;
            const float t0 = (cur.t0 - norm[2 * kIn + 2]) / norm[2 * kIn + 0];
            const float t1 = (cur.t1 - norm[2 * kIn + 3]) / norm[2 * kIn + 1];
            const float e0 = rr[0] - t0, e1 = rr[1] - t1;
            lsum += cur.w0 * e0 * e0 + cur.w1 * e1 * e1;
            d0 = 2.0f * cur.w0 * e0 * inv_n;
            d1 = 2.0f * cur.w1 * e1 * inv_n;
        }
        if (grp == 0) *reinterpret_cast<uint32_t *>(sm + sDZ + umma::kmajor_offset(r, 2 * kH, kGB)) = pack2(d0, d1); // dR
        // ---- dZ2 = (dR W3) * gelu'(z2 + b2)
        {
            float v[16];
            umma::tmem_ld16(lane_base + col_z2<kTrain>() + 16 * grp, v);
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const int j = 16 * grp + i;
                const float dh = fmaf(d0, w3f[j], d1 * w3f[kH + j]);
                v[i] = dh * gelu_grad(v[i] + b2[j]);
            }
            st8(sm + sDZ, r, kH + 16 * grp, kGB, v);
            st8(sm + sDZ, r, kH + 16 * grp + 8, kGB, v + 8);
        }
        fence_proxy_async();
        umma::fence_before_sync();
        __syncthreads();
        // ---- dH1 = dZ2 W2 (B: W2 with its outputs o as K, MN-major)
        if (tid == 0) {
            umma::fence_after_sync();
            for (int ks = 0; ks < kH / 16; ++ks)
                umma::mma_bf16(tmem + cDH1, umma::smem_desc(sbase + sDZ + kH / 8 * 128 + 256 * ks, 128, kDGroup),
                               umma::smem_desc(sbase + L::sW2 + 2048 * ks, 1024, 128),
                               umma::idesc_bf16(128, kH, false, true), ks > 0);
            umma::commit(bar);
        }
        ok = wait_mma(bar, phase, abort_flag);
        phase ^= 1u;
        if (!ok) break;
        {
            float dh[16], z[16];
            umma::tmem_ld16(lane_base + cDH1 + 16 * grp, dh);
            umma::tmem_ld16(lane_base + cZ1 + 16 * grp, z);
#pragma unroll
            for (int i = 0; i < 16; ++i) dh[i] *= gelu_grad(z[i] + b1[16 * grp + i]);
            st8(sm + sDZ, r, 16 * grp, kGB, dh); // dZ1
            st8(sm + sDZ, r, 16 * grp + 8, kGB, dh + 8);
        }
        fence_proxy_async();
        umma::fence_before_sync();
        __syncthreads();
        // ---- weight and bias gradients of this tile, summed over its 128
        // rows (the MMAs' K) into the CTA's accumulators G1 and G2:
        //   G1 [128 x 80]  += HH^T DZ[:, 64..143]: rows 0-63 dW2^T, rows 64-127 cols 64-65 dW3^T
        //   G2 [128 x 144] += X^T DZ: rows 0-11 cols 0-63 dW1^T; row 12: db1, db2, db3
        if (tid == 0) {
            umma::fence_after_sync();
            for (int ks = 0; ks < kRows / 16; ++ks)
                umma::mma_bf16(tmem + cG1, umma::smem_desc(sbase + sHH + 2 * kHGroup * ks, kHGroup, 128),
                               umma::smem_desc(sbase + sDZ + kH / 8 * 128 + 2 * kDGroup * ks, kDGroup, 128),
                               umma::idesc_bf16(128, kGB - kH, true, true), !gfirst || ks > 0);
            for (int ks = 0; ks < kRows / 16; ++ks)
                umma::mma_bf16(tmem + cG2, umma::smem_desc(sbase + sX + 2 * kXGroup * ks, kXGroup, 128),
                               umma::smem_desc(sbase + sDZ + 2 * kDGroup * ks, kDGroup, 128),
                               umma::idesc_bf16(128, kGB, true, true), !gfirst || ks > 0);
        }
        xbuf ^= 1u;
        gfirst = false;
        cur = nxt;
    }
    if (ok && !gfirst) {
        if (tid == 0) umma::commit(bar); // the last tile's gradient MMAs
        ok = wait_mma(bar, phase, abort_flag);
    }

    if (ok) {
        // atomics into grad, or this CTA's row of the deterministic workspace
        float *dst = a.partials ? a.partials + (size_t)blockIdx.x * (kParams + 1) : a.grad;
        auto put = [&](int k, float v) {
            if (a.partials) dst[k] = v;
            else atomicAdd(&dst[k], v);
        };
        // the thread of row m reads row m of the accumulators, group g columns
        // 16 g .. 16 g + 15 of G1 and every fourth 16 of G2
        const int m = r;
        if (!gfirst) {
            float v[16];
            if (m < kH) { // dW2[o][m] = G1[m][o]
                umma::tmem_ld16(lane_base + cG1 + 16 * grp, v);
#pragma unroll
                for (int i = 0; i < 16; ++i) put(oW2 + (16 * grp + i) * kH + m, v[i]);
            } else if (grp == 0) { // dW3[k][m - 64] = G1[m][64 + k]
                umma::tmem_ld16(lane_base + cG1 + kH, v);
                put(oW3 + 0 * kH + (m - kH), v[0]);
                put(oW3 + 1 * kH + (m - kH), v[1]);
            }
            if ((warp & 3) == 0) { // warp-collective loads: lanes 0-11 dW1, lane 12 the biases
                umma::tmem_ld16(lane_base + cG2 + 16 * grp, v);
                if (m < kK1) {
#pragma unroll
                    for (int i = 0; i < 16; ++i) put(oW1 + (16 * grp + i) * kK1 + m, m < kIn ? v[i] : 0.f); // dW1[o][m]
                }
                if (m == kIn) {
#pragma unroll
                    for (int i = 0; i < 16; ++i) put(oB1 + 16 * grp + i, v[i]);
                }
                umma::tmem_ld16(lane_base + cG2 + kH + 16 * grp, v);
                if (m == kIn) {
#pragma unroll
                    for (int i = 0; i < 16; ++i) put(oB2 + 16 * grp + i, v[i]);
                }
                if (grp == 0) {
                    float w[2];
                    umma::tmem_ld2(lane_base + cG2 + 2 * kH, w);
                    if (m == kIn) {
                        put(oB3 + 0, w[0]);
                        put(oB3 + 1, w[1]);
                    }
                }
            }
        } else { // a CTA without tiles adds zeros
            for (int e = tid; e < kParams; e += kThreadsTrain) put(e, 0.f);
        }
        float l = lsum;
        for (int off = 16; off > 0; off >>= 1) l += __shfl_xor_sync(0xffffffffu, l, off);
        if (a.partials) {
            float *wl = reinterpret_cast<float *>(sm + sDY); // group 0's per-warp losses, summed in warp order
            __syncthreads();
            if ((tid & 31) == 0 && grp == 0) wl[warp] = l;
            __syncthreads();
            if (tid == 0) dst[kParams] = ((wl[0] + wl[1]) + wl[2]) + wl[3];
        } else if ((tid & 31) == 0 && grp == 0) {
            atomicAdd(a.loss, (double)l / (double)n);
        }
    } else if (tid == 0) { // no sums: the gradient of this call is not to be used
        if (a.partials) a.partials[(size_t)blockIdx.x * (kParams + 1) + kParams] = aborted_mark();
        else atomicAdd(a.loss, (double)aborted_mark());
    }

    // ---- tear-down: every TMEM read is complete before the warp frees it
    umma::fence_before_sync();
    __syncthreads();
    if (!ok && tid == 0) atomicOr(&g_mlp_status, 1u);
    if (warp == 0) umma::tmem_dealloc(tmem, tmem_cols<kTrain>());
}

__global__ void adam_kernel(float *__restrict__ p, const float *__restrict__ g, float *__restrict__ m,
                            float *__restrict__ v, int count, float lr, float beta1, float beta2, float eps,
                            float corr1, float corr2) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    adam_update(p[i], g[i], m[i], v[i], lr, beta1, beta2, eps, corr1, corr2);
}

__global__ void average_kernel(float *__restrict__ avg, const float *__restrict__ p, int count, float decay) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    avg[i] = average_update(avg[i], p[i], decay);
}

// The kernel and threads per CTA of a mode.
template <int MODE>
auto kernel_of() {
    if constexpr (MODE == kTrain) return mlp_train_kernel;
    else return mlp_kernel<MODE>;
}
template <int MODE>
constexpr int kThreadsOf = MODE == kTrain ? kThreadsTrain : kThreadsMlp;

// Resident CTAs per SM of a mode and the SM count, computed once per mode and
// device from the device's limits: shared memory (with the per-block
// reservation), registers (allocated per warp in multiples of 8 per thread),
// threads, blocks, and TMEM (every resident CTA must get its columns without
// waiting in tcgen05.alloc).  On sm_100a with CUDA 12.9 the occupancy query
// returns 1 for these kernels, where the hardware holds 7 (ncu's
// launch__occupancy_limit_shared_mem), so it is not used.
template <int MODE>
int launch_shape(size_t smem, int &per_sm, int &sms) {
    static thread_local int cached_dev = -1, c_per_sm = 1, c_sms = 148;
    int dev = 0;
    if (int e = cuda_check(cudaGetDevice(&dev), "cudaGetDevice")) return e;
    if (dev != cached_dev) {
        if (int e = cuda_check(cudaFuncSetAttribute(kernel_of<MODE>(), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                    (int)smem),
                               "mlp smem attribute"))
            return e;
        cudaFuncAttributes fa{};
        if (int e = cuda_check(cudaFuncGetAttributes(&fa, kernel_of<MODE>()), "mlp attributes")) return e;
        auto attr = [&](cudaDeviceAttr a, int fallback) {
            int v = 0;
            return (cudaDeviceGetAttribute(&v, a, dev) == cudaSuccess && v > 0) ? v : fallback;
        };
        const int m = attr(cudaDevAttrMultiProcessorCount, 148);
        const int smem_sm = attr(cudaDevAttrMaxSharedMemoryPerMultiprocessor, 233472);
        const int reserved = attr(cudaDevAttrReservedSharedMemoryPerBlock, 1024);
        const int regs_sm = attr(cudaDevAttrMaxRegistersPerMultiprocessor, 65536);
        const int threads_sm = attr(cudaDevAttrMaxThreadsPerMultiProcessor, 2048);
        const int blocks_sm = attr(cudaDevAttrMaxBlocksPerMultiprocessor, 32);
        const int regs_warp = ((fa.numRegs + 7) / 8) * 8 * 32;
        const int warps = kThreadsOf<MODE> / 32;
        int n = smem_sm / ((int)smem + fa.sharedSizeBytes + reserved);
        n = std::min(n, regs_sm / (regs_warp * warps));
        n = std::min(n, threads_sm / kThreadsOf<MODE>);
        n = std::min(n, blocks_sm);
        n = std::min(n, (int)(512u / tmem_cols<MODE>()));
        c_per_sm = n > 0 ? n : 1;
        c_sms = m;
        cached_dev = dev;
    }
    per_sm = c_per_sm;
    sms = c_sms;
    return SSMD_OK;
}

template <int MODE>
int launch(MlpArgs a, cudaStream_t st, int max_ctas = 0, const AdamArgs &ad = AdamArgs{}) {
    // training: one CTA per SM (it allocates all 512 TMEM columns; 120 KB of shared
    // memory keep a second one away, whose allocation would wait for the first to end)
    const size_t smem = MODE == kTrain ? (Layout<MODE>::bytes > (size_t)120 * 1024 ? Layout<MODE>::bytes
                                                                                     : (size_t)120 * 1024)
                                       : Layout<MODE>::bytes;
    int per_sm = 1, sms = 148;
    if (int e = launch_shape<MODE>(smem, per_sm, sms)) return e;
    const int64_t tiles = (a.n + kRows - 1) / kRows;
    int64_t slots = (int64_t)sms * per_sm;
    if (max_ctas > 0 && slots > max_ctas) slots = max_ctas;
    const unsigned blocks = (unsigned)(tiles < slots ? tiles : slots);
    kernel_of<MODE>()<<<blocks, kThreadsOf<MODE>, smem, st>>>(a);
    if (int e = cuda_check(cudaGetLastError(), "mlp launch")) return e;
    if (MODE == kTrain && a.partials) {
        grad_sum_kernel<kParams><<<(kParams + 1 + 31) / 32, kSumThreads, 0, st>>>(a.partials, (int)blocks, a.n, a.grad,
                                                                                 a.loss, ad);
        return cuda_check(cudaGetLastError(), "gradient sum launch");
    }
    return SSMD_OK;
}

} // namespace

extern "C" int ssmd_mlp_forward(const float *net, const float *features, int64_t n, float *out,
                                ssmd_stream_t stream) {
    if (!net || !features || !out || n < 0) return fail(SSMD_ERR_INVALID_ARGUMENT, "null argument or n < 0");
    if (n == 0) return SSMD_OK;
    if (n > (int64_t)0x7FFFFFFF * kRows) return fail(SSMD_ERR_INVALID_ARGUMENT, "too many rows");
    if ((reinterpret_cast<uintptr_t>(out) & 7u) != 0) return fail(SSMD_ERR_INVALID_ARGUMENT, "out must be 8-byte aligned");
    MlpArgs a{};
    a.net = net;
    a.feat = features;
    a.n = n;
    a.out = out;
    return launch<kFwd>(a, reinterpret_cast<cudaStream_t>(stream));
}

extern "C" int ssmd_mlp_grad(const float *net, const float *features, const float *targets, const float *weights,
                             int64_t n, float *grad, double *loss, ssmd_stream_t stream) {
    if (!net || !features || !targets || !grad || !loss || n <= 0)
        return fail(SSMD_ERR_INVALID_ARGUMENT, "null argument or n <= 0");
    if (n > (int64_t)0x7FFFFFFF * kRows) return fail(SSMD_ERR_INVALID_ARGUMENT, "too many rows");
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (int e = cuda_check(cudaMemsetAsync(grad, 0, sizeof(float) * kParams, st), "grad clear")) return e;
    if (int e = cuda_check(cudaMemsetAsync(loss, 0, sizeof(double), st), "loss clear")) return e;
    MlpArgs a{};
    a.net = net;
    a.feat = features;
    a.target = targets;
    a.weight = weights;
    a.n = n;
    a.grad = grad;
    a.loss = loss;
    return launch<kTrain>(a, st);
}

extern "C" size_t ssmd_mlp_grad_workspace_bytes(void) {
    return sizeof(float) * (size_t)kMaxGradCtas * (kParams + 1);
}

extern "C" int ssmd_mlp_grad_ws(const float *net, const float *features, const float *targets, const float *weights,
                                int64_t n, float *grad, double *loss, float *workspace, size_t workspace_bytes,
                                ssmd_stream_t stream) {
    if (!net || !features || !targets || !grad || !loss || !workspace || n <= 0)
        return fail(SSMD_ERR_INVALID_ARGUMENT, "null argument or n <= 0");
    if (n > (int64_t)0x7FFFFFFF * kRows) return fail(SSMD_ERR_INVALID_ARGUMENT, "too many rows");
    if (workspace_bytes < ssmd_mlp_grad_workspace_bytes())
        return fail(SSMD_ERR_INVALID_ARGUMENT, "workspace_bytes %zu < required %zu", workspace_bytes,
                    ssmd_mlp_grad_workspace_bytes());
    MlpArgs a{};
    a.net = net;
    a.feat = features;
    a.target = targets;
    a.weight = weights;
    a.n = n;
    a.grad = grad;
    a.loss = loss;
    a.partials = workspace;
    return launch<kTrain>(a, reinterpret_cast<cudaStream_t>(stream), kMaxGradCtas);
}

extern "C" int ssmd_mlp_train_step(float *net, const float *features, const float *targets, const float *weights,
                                   int64_t n_rows, const int64_t *rows, int64_t batch, float *grad, double *loss,
                                   float *m, float *v, int64_t t, float lr, float beta1, float beta2, float eps,
                                   float *avg, float decay, float *workspace, size_t workspace_bytes,
                                   ssmd_stream_t stream) {
    if (!net || !features || !targets || !rows || !grad || !loss || !m || !v || !workspace || n_rows <= 0 || batch <= 0 ||
        t <= 0)
        return fail(SSMD_ERR_INVALID_ARGUMENT, "null argument, n_rows <= 0, batch <= 0 or t <= 0");
    if (batch > (int64_t)0x7FFFFFFF * kRows) return fail(SSMD_ERR_INVALID_ARGUMENT, "too many rows");
    if (avg && !(decay >= 0.0f && decay <= 1.0f)) return fail(SSMD_ERR_INVALID_ARGUMENT, "decay outside [0, 1]");
    if (workspace_bytes < ssmd_mlp_grad_workspace_bytes())
        return fail(SSMD_ERR_INVALID_ARGUMENT, "workspace_bytes %zu < required %zu", workspace_bytes,
                    ssmd_mlp_grad_workspace_bytes());
    MlpArgs a{};
    a.net = net;
    a.feat = features;
    a.target = targets;
    a.weight = weights;
    a.rows = rows;
    a.n_rows = n_rows;
    a.n = batch;
    a.grad = grad;
    a.loss = loss;
    a.partials = workspace;
    AdamArgs ad{net, m, v, avg, lr, beta1, beta2, eps, (float)(1.0 - pow((double)beta1, (double)t)),
                (float)(1.0 - pow((double)beta2, (double)t)), decay};
    return launch<kTrain>(a, reinterpret_cast<cudaStream_t>(stream), kMaxGradCtas, ad);
}

extern "C" int ssmd_closure_refresh(const ssmd_params *coarse, const LBMFields *fields, const float *net,
                                    float nut_max, float *nut, float *sigma_scale, ssmd_stream_t stream) {
    if (int e = ssmd_validate(coarse)) return e;
    if (!fields || !fields->rho || !fields->ux || !fields->uy || !fields->uz || !fields->phi || !net || !nut ||
        !sigma_scale)
        return fail(SSMD_ERR_INVALID_ARGUMENT, "null argument");
    MlpArgs a{};
    a.net = net;
    a.n = (int64_t)coarse->nx * coarse->ny * coarse->nz;
    a.g = closure::grid_of(*coarse);
    a.rho = fields->rho;
    a.ux = fields->ux;
    a.uy = fields->uy;
    a.uz = fields->uz;
    a.phi = fields->phi;
    a.nu_w = coarse->nu_water;
    a.nu_dow = coarse->nu_oil - coarse->nu_water;
    a.nut_max = nut_max;
    a.nut = nut;
    a.cs = sigma_scale;
    return launch<kRefresh>(a, reinterpret_cast<cudaStream_t>(stream));
}

extern "C" int ssmd_mlp_adam(float *net, const float *grad, float *m, float *v, int64_t t, float lr, float beta1,
                             float beta2, float eps, ssmd_stream_t stream) {
    if (!net || !grad || !m || !v || t <= 0) return fail(SSMD_ERR_INVALID_ARGUMENT, "null argument or t <= 0");
    const float corr1 = (float)(1.0 - pow((double)beta1, (double)t));
    const float corr2 = (float)(1.0 - pow((double)beta2, (double)t));
    adam_kernel<<<(kParams + 255) / 256, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        net, grad, m, v, kParams, lr, beta1, beta2, eps, corr1, corr2);
    return cuda_check(cudaGetLastError(), "adam launch");
}

extern "C" int ssmd_mlp_average(float *avg, const float *net, float decay, ssmd_stream_t stream) {
    if (!avg || !net || !(decay >= 0.0f && decay <= 1.0f))
        return fail(SSMD_ERR_INVALID_ARGUMENT, "null argument or decay outside [0, 1]");
    average_kernel<<<(kParams + 255) / 256, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(avg, net, kParams,
                                                                                              decay);
    return cuda_check(cudaGetLastError(), "average launch");
}

extern "C" int ssmd_mlp_status(uint32_t *status) {
    if (!status) return fail(SSMD_ERR_INVALID_ARGUMENT, "null argument");
    unsigned int v = 0;
    if (int e = cuda_check(cudaMemcpyFromSymbol(&v, g_mlp_status, sizeof v), "mlp status")) return e;
    *status = v;
    return SSMD_OK;
}
