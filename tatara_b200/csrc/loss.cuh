// The loss of one position and its sum over a block, shared by the tail kernels
// (pointwise/loss_wdl.rs:63-88, pointwise/loss_wrm.rs:99-180).
#pragma once
#include "common.cuh"

#define L1_SQR_SCALE (127.0f / 128.0f)

static __device__ __forceinline__ float sigmoidf_(float x) { return 1.0f / (1.0f + expf(-x)); }

// the extended WRM loss's per-position weight (loss_wrm / wrm_weight_sum, native_kernels.cu:455-458, 538-543)
static __device__ __forceinline__ float wrm_weight(const LossParams& lp, float target_wrm) {
    const float wb = (target_wrm - 0.5f) * (target_wrm - 0.5f) * target_wrm * (1.0f - target_wrm);
    return 1.0f + (powf(2.0f, lp.w1) - 1.0f) * powf(wb, lp.w2);
}

// returns the position's contribution to the reported loss sum (err^2 for the plain losses) and its output gradient
static __device__ __forceinline__ double loss_point(const LossParams& lp, float out, float score, float wdl, float* dy) {
    if (lp.kind == 0) {
        const float p = sigmoidf_(out * lp.scale);
        const float ys = sigmoidf_(score * lp.scale);
        const float y = lp.lambda * wdl + (1.0f - lp.lambda) * ys;
        const float err = p - y;
        *dy = 2.0f * err * p * (1.0f - p) * lp.scale * lp.norm;
        return (double)err * (double)err;
    }
    const float pt = (score - lp.target_offset) / lp.target_scaling;
    const float pmt = (-score - lp.target_offset) / lp.target_scaling;
    const float target_wrm = 0.5f * (1.0f + sigmoidf_(pt) - sigmoidf_(pmt));
    const float target = lp.lambda * wdl + (1.0f - lp.lambda) * target_wrm;
    const float scorenet = out * lp.nnue2score;
    const float q = sigmoidf_((scorenet - lp.in_offset) / lp.in_scaling);
    const float qm = sigmoidf_((-scorenet - lp.in_offset) / lp.in_scaling);
    const float qf = 0.5f * (1.0f + q - qm);
    const float err = qf - target;
    if (!lp.extended) {
        *dy = err * (lp.nnue2score / lp.in_scaling) * (q * (1.0f - q) + qm * (1.0f - qm)) * lp.norm;
        return (double)err * (double)err;
    }
    // loss_wrm, extended branch (native_kernels.cu:454-474): |err|^pow_exp, asymmetry above the target, weights
    // normalised by their sum over the batch (which replaces the per-position normaliser)
    const float weight = wrm_weight(lp, target_wrm);
    const float asym = qf > target ? 1.0f + lp.qp_asymmetry : 1.0f;
    const float abs_err = fabsf(err);
    const float abs_pow = powf(abs_err, lp.pow_exp - 1.0f);
    const float signed_pow = err < 0.0f ? -abs_pow : abs_pow;
    const float inv_wsum = (float)(1.0 / *lp.weight_sum);
    const float pred_grad = 0.5f * (lp.nnue2score / lp.in_scaling) * (q * (1.0f - q) + qm * (1.0f - qm));
    *dy = (weight * inv_wsum) * (asym * lp.pow_exp * signed_pow) * pred_grad;
    return (double)(asym * powf(abs_err, lp.pow_exp) * weight * lp.n_pos * inv_wsum);
}

// sum of err^2 over the block in f64, one partial per block (fixed order: no atomics)
static __device__ __forceinline__ void block_loss_partial(double v, double* partials) {
    __shared__ double s_w[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v += __shfl_down_sync(0xffffffffu, v, d);
    if (lane == 0) s_w[w] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        const int nw = (blockDim.x + 31) >> 5;
        for (int i = 0; i < nw; ++i) t += s_w[i];
        partials[blockIdx.x] = t;
    }
}
