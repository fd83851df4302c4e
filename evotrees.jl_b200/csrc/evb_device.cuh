// Device helpers shared by the training and the inference kernels.
#pragma once
#include "evb_internal.cuh"

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

