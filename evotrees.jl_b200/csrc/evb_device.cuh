// Device helpers shared by the training and the inference kernels.
#pragma once
#include "evb_internal.cuh"
#include <float.h>

// ---------------------------------------------------------------------------------- scalar loss math
__device__ __forceinline__ float sigmoidf_(float x) { return 1.0f / (1.0f + expf(-x)); }             // loss.jl:249-251
__device__ __forceinline__ float softplusf_(float x) { return fmaxf(x, 0.0f) + log1pf(expf(-fabsf(x))); } // loss.jl:257-260

// pred[:, i] += leaf with the loss-specific clamps of predict! (src/predict.jl:1-62)
__device__ __forceinline__ void pred_add(int loss, int K, float *p, const float *leaf) {
    if (loss == EVB_LOGLOSS) {
        for (int k = 0; k < K; ++k) p[k] = fminf(fmaxf(p[k] + leaf[k], -15.0f), 15.0f);
    } else if (loss == EVB_GAUSSIAN_MLE || loss == EVB_LOGISTIC_MLE) {
        for (int t = 0; t < K / 2; ++t) {
            p[2 * t] += leaf[2 * t];
            p[2 * t + 1] = fmaxf(-15.0f, p[2 * t + 1] + leaf[2 * t + 1]);
        }
    } else if (loss == EVB_MLOGLOSS) {
        float m = -INFINITY;
        for (int k = 0; k < K; ++k) { p[k] += leaf[k]; m = fmaxf(m, p[k]); }
        for (int k = 0; k < K; ++k) p[k] = fmaxf(-15.0f, p[k] - m);
    } else {
        for (int k = 0; k < K; ++k) p[k] += leaf[k];
    }
}

__device__ __forceinline__ int traverse(const uint32_t *packed, const uint8_t *xrow) {
    int nid = 1;
    uint32_t pk = packed[0];
    while ((pk >> 24) & 1u) {
        const uint32_t x = xrow[pk & 0xffffu], bin = (pk >> 16) & 0xffu;
        const bool cond = ((pk >> 25) & 1u) ? (x <= bin) : (x == bin);
        nid = (nid << 1) + (cond ? 0 : 1); // nid = nid << 1 + !cond (src/predict.jl:7)
        pk = packed[nid - 1];
    }
    return nid;
}


// ---------------------------------------------------------------------------------- split scan and partition
__device__ __forceinline__ double warp_incl_scan(double v, int lane) {
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        double t = __shfl_up_sync(0xffffffffu, v, d);
        if (lane >= d) v += t;
    }
    return v;
}
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
    return v;
}
__device__ __forceinline__ long long warp_sum(long long v) {
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
    return v;
}
__device__ __forceinline__ int warp_incl_scan_i(int v, int lane) {
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        int t = __shfl_up_sync(0xffffffffu, v, d);
        if (lane >= d) v += t;
    }
    return v;
}
// Counts arrivals: what the arriving thread (and threads it has synchronised with) wrote before is visible to whoever sees the count.
// One release-acquire operation instead of fences on both sides of a relaxed one, each of which waits for L2 (0.5 us).
__device__ __forceinline__ uint32_t arrive(uint32_t *count) {
    uint32_t v;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(v) : "l"(count) : "memory");
    return v;
}
// a / b for operands that quot_ok lets through: the quotient by a reciprocal from Newton's iteration, corrected by its exact remainder
// (P. Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990).  It is the division's
// unless b's bits are all ones, the method's known exception: a power of two by such a number is one unit in the last place too small.
// tests/test_quotients_gpu.py: random pairs, those whose quotients lie closest to the middle of two numbers, the ends of the range.  The division
// of the language checks its range with a branch of its own, so that quotients are worked out one after the other (four: 521 clocks, 130
// each); these overlap.
__device__ __forceinline__ double quot(double a, double b) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(b));
    r = fma(r, fma(-b, r, 1.0), r); // 1e-6, 1e-12 ..
    r = fma(r, fma(-b, r, 1.0), r);
    const double q = a * r;
    return fma(fma(-b, q, a), r, q);
}
// a < 2^600, b < 2^300 (neither infinite nor a NaN).  Small a need no test: a is the square of a sum of float32 gradients, a whole number of units of 2^-213 or more, so it is
// zero or far above 2^-600, and quotient, reciprocal and the last bit of the remainder (2^-104 a) are normal numbers.  (Below 2^-600 the last bits
// may be wrong; a test for that cost 100k x 10 about one percent.)
__device__ __forceinline__ bool quot_ok(double a, double b) { return a < 0x1p600 && b < 0x1p300; }
// both sides of a candidate split (src/split.jl:1)
__device__ __forceinline__ double terms_gh(double gl, double hl, double wl, double gr, double hr, double wr, double lambda, double L2) {
    const double a = gl * gl, b = fmax(DBL_EPSILON, hl + lambda * wl + L2), c = gr * gr, d = fmax(DBL_EPSILON, hr + lambda * wr + L2);
    if (quot_ok(a, b) && quot_ok(c, d)) return quot(a, b) * 0.5 + quot(c, d) * 0.5;
    return a / b / 2.0 + c / d / 2.0;
}
__device__ __forceinline__ double term_gh(double g, double h, double w, double lambda, double L2) {
    return g * g / fmax(DBL_EPSILON, h + lambda * w + L2) / 2.0; // src/split.jl:1
}
__device__ __forceinline__ bool goes_left(uint32_t pk, uint32_t x) { // split_set! predicate (fit-utils.jl:173, 291)
    const uint32_t bin = (pk >> 16) & 0xffu;
    return ((pk >> 25) & 1u) ? (x <= bin) : (x == bin);
}

// ---------------------------------------------------------------------------------- gradients, metrics
// Gradient record of one row: the channels whose sums the histograms hold, in the reference's order g_1..g_K, h_1..h_K, w
// (`cache.∇`, src/init.jl:173).  Left out: w when no weights were given (it is 1) and, for mse, the hessians (h = 2w is
// rebuilt from the sums of w): `elided`.
struct AlphaSet { float a[8]; }; // a[0]: alpha of the quantile loss; a[0..K-1]: alphas of the multiquantile loss
__device__ __forceinline__ void grad_row(int loss, int K, bool elided, const float *p, const void *y, int ycols, long long i, float w, float *rec,
                                         const AlphaSet &al) {
    const float alpha = al.a[0];
    if (loss == EVB_MSE) {
        const float *yf = (const float *)y + (size_t)i * ycols;
        for (int k = 0; k < K; ++k) {
            rec[k] = 2.0f * (p[k] - yf[k]) * w;
            if (!elided) rec[K + k] = 2.0f * w;
        }
    } else if (loss == EVB_LOGLOSS) {
        const float *yf = (const float *)y + (size_t)i * ycols;
        for (int k = 0; k < K; ++k) {
            const float s = sigmoidf_(p[k]);
            rec[k] = (s - yf[k]) * w;
            rec[K + k] = s * (1.0f - s) * w;
        }
    } else if (loss == EVB_MLOGLOSS) {
        const uint32_t yi = ((const uint32_t *)y)[i];
        float isum = 0.0f;
        for (int k = 0; k < K; ++k) isum += expf(p[k]);
        for (int k = 0; k < K; ++k) {
            const float prob = expf(p[k]) / isum;
            rec[k] = (((uint32_t)(k + 1) == yi) ? prob - 1.0f : prob) * w;
            rec[K + k] = prob * (1.0f - prob) * w;
        }
    } else if (loss == EVB_MULTIQUANTILE) { // one target, one quantile per output row (src/loss.jl:160-172)
        const float yi = ((const float *)y)[i];
        for (int k = 0; k < K; ++k) {
            const float d = yi - p[k];
            rec[k] = (d > 0.0f ? al.a[k] : al.a[k] - 1.0f) * w;
            rec[K + k] = d;
        }
    } else if (loss == EVB_QUANTILE) { // quantile_grad_diff, src/loss.jl:93-98: the second slot keeps the raw residual
        const float *yf = (const float *)y + (size_t)i * ycols;
        for (int k = 0; k < K; ++k) {
            const float d = yf[k] - p[k];
            rec[k] = (d > 0.0f ? alpha : alpha - 1.0f) * w;
            rec[K + k] = d;
        }
    } else if (loss == EVB_MAE || loss == EVB_CRED_VAR || loss == EVB_CRED_STD) { // src/loss.jl:86-91
        const float *yf = (const float *)y + (size_t)i * ycols;
        for (int k = 0; k < K; ++k) {
            const float d = yf[k] - p[k];
            rec[k] = d * w;
            rec[K + k] = (loss == EVB_MAE ? 0.0f : d * d) * w;
        }
    } else if (loss == EVB_POISSON || loss == EVB_GAMMA || loss == EVB_TWEEDIE) { // src/loss.jl:65-84
        const float *yf = (const float *)y + (size_t)i * ycols;
        for (int k = 0; k < K; ++k) {
            const float pr = expf(p[k]), yk = yf[k];
            float g, h;
            if (loss == EVB_POISSON) { g = pr - yk; h = pr; }
            else if (loss == EVB_GAMMA) { g = 2.0f * (1.0f - yk / pr); h = 2.0f * yk / pr; }
            else { // rho = 1.5: pred^(2-rho) = sqrt(pred), pred^(1-rho) = 1 / sqrt(pred)
                const float a = sqrtf(pr), b = 1.0f / a;
                g = 2.0f * (a - yk * b);
                h = 2.0f * (0.5f * a + 0.5f * yk * b);
            }
            rec[k] = g * w;
            rec[K + k] = h * w;
        }
    } else if (loss == EVB_LOGISTIC_MLE) { // src/loss.jl:207-217
        const int Y = K / 2;
        const float *yf = (const float *)y + (size_t)i * ycols;
        for (int t = 0; t < Y; ++t) {
            const float loc = p[2 * t], sr = p[2 * t + 1];
            const float scale = softplusf_(sr), ds = sigmoidf_(sr);
            const float z = (yf[t] - loc) / scale, th = tanhf(z / 2.0f);
            rec[2 * t] = -th / scale * w;
            rec[2 * t + 1] = (1.0f - z * th) * ds / scale * w;
            rec[2 * Y + 2 * t] = 1.0f / (3.0f * scale * scale) * w;
            rec[2 * Y + 2 * t + 1] = (3.14159274f * 3.14159274f + 3.0f) / 9.0f * (ds / scale) * (ds / scale) * w;
        }
    } else { // EVB_GAUSSIAN_MLE
        const int Y = K / 2;
        const float *yf = (const float *)y + (size_t)i * ycols;
        for (int t = 0; t < Y; ++t) {
            const float loc = p[2 * t], sr = p[2 * t + 1];
            const float scale = softplusf_(sr), ds = sigmoidf_(sr);
            const float resid = loc - yf[t];
            const float s2 = scale * scale;
            rec[2 * t] = resid / s2 * w;
            rec[2 * t + 1] = (1.0f - resid * resid / s2) * ds / scale * w;
            rec[2 * Y + 2 * t] = 1.0f / s2 * w;
            rec[2 * Y + 2 * t + 1] = 2.0f * (ds / scale) * (ds / scale) * w;
        }
    }
}
// Per-row metric value in float, as `_metric_value` / `_mle2p_metric_value` / `mlogloss` compute it
// (src/metrics.jl:1-110): the caller multiplies by w and accumulates in double.
__device__ __forceinline__ float metric_row(int metric, int K, const float *p, const void *y, int ycols, long long i, float w, const AlphaSet &al) {
    const float alpha = al.a[0];
    if (metric == EVB_METRIC_MLOGLOSS) {
        const uint32_t yi = ((const uint32_t *)y)[i];
        float isum = 0.0f;
        for (int k = 0; k < K; ++k) isum += expf(p[k]);
        return w * (logf(isum) - p[yi - 1]);
    }
    const float *yf = (const float *)y + (size_t)i * ycols;
    if (metric == EVB_METRIC_MULTIQUANTILE) { // src/metrics.jl:120-141
        float acc = 0.0f;
        for (int k = 0; k < K; ++k) acc += al.a[k] * fmaxf(yf[0] - p[k], 0.0f) + (1.0f - al.a[k]) * fmaxf(p[k] - yf[0], 0.0f);
        return w * acc / (float)K;
    }
    if (metric == EVB_METRIC_GAUSSIAN_MLE || metric == EVB_METRIC_LOGISTIC_MLE) {
        const int Y = K / 2;
        float acc = 0.0f;
        for (int t = 0; t < Y; ++t) {
            const float scale = softplusf_(p[2 * t + 1]), d = yf[t] - p[2 * t];
            if (metric == EVB_METRIC_GAUSSIAN_MLE) acc += -(logf(scale) + d * d / (2.0f * scale * scale));
            else { const float az = fabsf(d / scale); acc += -logf(scale) - az - 2.0f * log1pf(expf(-az)); } // src/metrics.jl:84-89
        }
        return w * acc / (float)Y;
    }
    float acc = 0.0f;
    for (int k = 0; k < K; ++k) {
        const float pk = p[k], yk = yf[k];
        if (metric == EVB_METRIC_MSE) acc += (pk - yk) * (pk - yk);
        else if (metric == EVB_METRIC_MAE) acc += fabsf(pk - yk);
        else if (metric == EVB_METRIC_QUANTILE) acc += alpha * fmaxf(yk - pk, 0.0f) + (1.0f - alpha) * fmaxf(pk - yk, 0.0f); // src/metrics.jl:4-6
        else if (metric == EVB_METRIC_LOGLOSS) { const float s = sigmoidf_(pk); acc += -yk * logf(s) + (yk - 1.0f) * logf(1.0f - s); }
        else if (metric == EVB_METRIC_POISSON) { // src/metrics.jl:13-17; eps(1f-7)
            const float pr = expf(pk);
            acc += 2.0f * (yk * logf(yk / pr + 7.1054274e-15f) + pr - yk);
        } else if (metric == EVB_METRIC_GAMMA) { const float pr = expf(pk); acc += 2.0f * (logf(pr / yk) + yk / pr - 1.0f); }
        else { // tweedie, rho = 1.5 (src/metrics.jl:24-28)
            const float pr = expf(pk), a = sqrtf(pr);
            acc += 2.0f * (sqrtf(yk) / -0.5f / 0.5f - yk * (1.0f / a) / -0.5f + a / 0.5f);
        }
    }
    return w * acc / (float)K;
}
static inline AlphaSet evb_alpha_set(const evb_handle *h) {
    AlphaSet s;
    for (int k = 0; k < 8; ++k) s.a[k] = (float)h->p.alphas[k];
    if (h->p.loss != EVB_MULTIQUANTILE) s.a[0] = (float)h->p.alpha;
    return s;
}
// A copy node of the graph would cost 5 to 10 us between the kernels of two trees; these stores cost nothing.
__device__ __forceinline__ void publish(const uint4 *src, uint4 *dst, int n) {
    for (int i = threadIdx.x; i < n; i += blockDim.x) dst[i] = src[i];
}
