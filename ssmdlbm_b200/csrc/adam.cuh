// adam.cuh — what follows the closure network's per-CTA gradient rows: their sum,
// the Adam step and the weight average.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace ssmd {

constexpr int kMaxGradCtas = 256; // rows of the deterministic gradient workspace

// A CTA whose MMA wait ran out writes this NaN as its row's loss and nothing else.
// Arithmetic gives the NaN 0x7fffffff, so no sum of a CTA can be taken for it.
constexpr uint32_t kAbortedRow = 0x7fc0ab07u;
__device__ __forceinline__ float aborted_mark() { return __uint_as_float(kAbortedRow); }

__device__ __forceinline__ void adam_update(float &p, float gi, float &m, float &v, float lr, float beta1, float beta2,
                                            float eps, float corr1, float corr2) {
    // (explicit fma: the kernels that share this round alike)
    m = fmaf(1.0f - beta1, gi, beta1 * m);
    v = fmaf((1.0f - beta2) * gi, gi, beta2 * v);
    p -= lr * (m / corr1) / (sqrtf(v / corr2) + eps);
}
__device__ __forceinline__ float average_update(float avg, float p, float decay) {
    return fmaf(decay, avg - p, p); // decay avg + (1 - decay) p
}

// Adam step and weight average that follow a gradient (m null: none; avg null: none).
struct AdamArgs {
    float *net, *m, *v, *avg;
    float lr, beta1, beta2, eps, corr1, corr2, decay;
};

// Deterministic reduction of the per-CTA gradient rows, column k summed over the
// CTAs in CTA order (FP32, like the atomic path; the loss column in FP64), then
// the Adam step and the average on it.  A block takes 32 columns: its
// 8 warps bring the rows into shared memory, all in flight at once, and one
// warp adds them.  (A thread per column that loaded its rows one after the other:
// 8.5 us, and 4 us more for Adam and the average in launches of their own; now 4.6 us
// for all three.)
// Where a row is marked aborted there is no gradient: grad and loss become NaN, and
// net, m, v and avg stay as they are.
constexpr int kSumThreads = 256;
static_assert(kMaxGradCtas <= kSumThreads, "a thread looks at one row's mark");
template <int PARAMS>
__global__ void __launch_bounds__(kSumThreads)
    grad_sum_kernel(const float *__restrict__ partials, int ctas, int64_t n, float *__restrict__ grad,
                    double *__restrict__ loss, const AdamArgs ad) {
    __shared__ float s[kMaxGradCtas][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int k = blockIdx.x * 32 + lane;
    // Adam's operands are on their way while the rows come in
    const bool step = warp == 0 && k < PARAMS;
    const float m0 = step && ad.m ? ad.m[k] : 0.f, v0 = step && ad.m ? ad.v[k] : 0.f;
    const float p0 = step && ad.net ? ad.net[k] : 0.f, a0 = step && ad.avg ? ad.avg[k] : 0.f;
    const bool mark = (int)threadIdx.x < ctas &&
                      __float_as_uint(__ldg(partials + (size_t)threadIdx.x * (PARAMS + 1) + PARAMS)) == kAbortedRow;
    float row[kMaxGradCtas / (kSumThreads / 32)];
#pragma unroll
    for (int i = 0; i < kMaxGradCtas / (kSumThreads / 32); ++i) {
        const int b = warp + i * (kSumThreads / 32);
        row[i] = b < ctas && k <= PARAMS ? __ldg(partials + (size_t)b * (PARAMS + 1) + k) : 0.f;
    }
#pragma unroll
    for (int i = 0; i < kMaxGradCtas / (kSumThreads / 32); ++i) s[warp + i * (kSumThreads / 32)][lane] = row[i];
    const bool aborted = __syncthreads_or(mark); // also: the rows are in shared memory
    if (warp != 0) return;
    if (aborted) {
        if (k < PARAMS) grad[k] = aborted_mark();
        else if (k == PARAMS) *loss = (double)aborted_mark();
        return;
    }
    if (k < PARAMS) {
        float g = 0.f;
#pragma unroll 8
        for (int b = 0; b < ctas; ++b) g += s[b][lane];
        grad[k] = g;
        float p = p0;
        if (ad.m) {
            float m = m0, v = v0;
            adam_update(p, g, m, v, ad.lr, ad.beta1, ad.beta2, ad.eps, ad.corr1, ad.corr2);
            ad.net[k] = p;
            ad.m[k] = m;
            ad.v[k] = v;
        }
        if (ad.avg) ad.avg[k] = average_update(a0, p, ad.decay);
    } else if (k == PARAMS) {
        double l = 0.0;
        for (int b = 0; b < ctas; ++b) l += (double)s[b][lane];
        *loss = l / (double)n;
    }
}

} // namespace ssmd
