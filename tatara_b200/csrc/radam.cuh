// The optimizer's arithmetic on four adjacent parameters (radam_step, native_kernels.cu:1291; pointwise/radam_step.rs:116-156),
// for the kernels of opt_kernels.cu.
#pragma once
#include "common.cuh"

#include <cuda_fp16.h>

static __device__ __forceinline__ unsigned ok_pack_h2(float lo, float hi) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const unsigned*>(&h);
}
static __device__ __forceinline__ float2 ok_unpack_h2(unsigned pair) { return __half22float2(*reinterpret_cast<const __half2*>(&pair)); }
static __device__ __forceinline__ uint2 pack_h4(float4 v) { return make_uint2(ok_pack_h2(v.x, v.y), ok_pack_h2(v.z, v.w)); }

// Four moments of one float4 of parameters.  fp32 state: as stored.  fp16 state (radam_step_f16state,
// native_kernels.cu:1127-1181): stored = clamp(value * scale) rounded to fp16; read back as stored / scale.  The update
// itself uses the unrounded new moments; the scales are powers of two, so scaling is exact.
template <bool HS>
static __device__ __forceinline__ float4 load_moment(const void* base, size_t i4, float inv_scale, bool streaming) {
    if (HS) {
        const uint2* p = static_cast<const uint2*>(base) + i4;
        const uint2 u = streaming ? __ldcs(p) : *p;
        const float2 a = ok_unpack_h2(u.x), b = ok_unpack_h2(u.y);
        return make_float4(a.x * inv_scale, a.y * inv_scale, b.x * inv_scale, b.y * inv_scale);
    }
    const float4* p = static_cast<const float4*>(base) + i4;
    return streaming ? __ldcs(p) : *p;
}
static __device__ __forceinline__ float clamp_h(float x, bool both) {
    x = x > 65504.0f ? 65504.0f : x;  // comparisons keep a NaN, as the reference does
    if (both) x = x < -65504.0f ? -65504.0f : x;
    return x;
}
template <bool HS>
static __device__ __forceinline__ void store_moment(void* base, size_t i4, float4 val, float scale, bool both, bool streaming) {
    if (HS) {
        const float4 q = make_float4(clamp_h(val.x * scale, both), clamp_h(val.y * scale, both), clamp_h(val.z * scale, both),
                                     clamp_h(val.w * scale, both));
        uint2* p = static_cast<uint2*>(base) + i4;
        if (streaming) __stcs(p, pack_h4(q)); else *p = pack_h4(q);
    } else {
        float4* p = static_cast<float4*>(base) + i4;
        if (streaming) __stcs(p, val); else *p = val;
    }
}
// rounded before it is added to anything (see radam_one)
static __device__ __forceinline__ float4 scale4(float4 g, float k) {
    return make_float4(__fmul_rn(g.x, k), __fmul_rn(g.y, k), __fmul_rn(g.z, k), __fmul_rn(g.w, k));
}

// Of a sum of two products one is rounded before it is added.  Which one is part of the results (AdamW's first steps turn a last bit
// into a visible difference after a few steps), so it is written out for every kernel and not left to the compiler, which chose
// by what stood around the call.  The forms are those of the first kernels as they were compiled.
//   moments, RADAM_OLD_FUSED: fma(beta, old, rounded new term), else fma(new factor, gradient, rounded beta * old)
//   weights, RADAM_STEP_FUSED: p * decay rounded, then fma(-rate, value, .), else fma(p, decay, -rounded rate * value);
//   RADAM_STEP_DENOM: the former where the value is divided by the root of the second moment, RADAM_STEP_LERP: on look-ahead steps
enum { RADAM_OLD_FUSED = 1, RADAM_STEP_FUSED = 2, RADAM_STEP_DENOM = 4, RADAM_STEP_LERP = 8 };
enum {
    RADAM_SMALL = RADAM_OLD_FUSED | RADAM_STEP_DENOM,  // the small groups
    RADAM_TABLE = RADAM_OLD_FUSED | RADAM_STEP_LERP,   // the FT table without a factorizer
    RADAM_FACT = 0,                                    // with one
    RADAM_FACT_LAST = RADAM_STEP_FUSED                 // with one: of a virtual row every fourth column
};

static __device__ __forceinline__ float radam_rate(const OptScalars& sc) { return __fmul_rn(sc.lr, sc.step_size); }
static __device__ __forceinline__ float radam_decay(const OptScalars& sc, float rate) { return __fmaf_rn(-sc.decay, rate, 1.0f); }

template <int FORM>
static __device__ __forceinline__ float radam_one(float p, float& m, float& v, float g, const OptScalars& sc, float rate,
                                                   float decay_mul) {
    const float gm = 1.0f - sc.beta1, gv = __fmul_rn(1.0f - sc.beta2, g);
    const float mi = (FORM & RADAM_OLD_FUSED) ? __fmaf_rn(sc.beta1, m, __fmul_rn(gm, g)) : __fmaf_rn(gm, g, __fmul_rn(sc.beta1, m));
    const float vi = (FORM & RADAM_OLD_FUSED) ? __fmaf_rn(sc.beta2, v, __fmul_rn(gv, g)) : __fmaf_rn(gv, g, __fmul_rn(sc.beta2, v));
    m = mi;
    v = vi;
    float val = mi;
    if (sc.denom != 0) val = __fdiv_rn(val, __fadd_rn(__fsqrt_rn(vi), sc.eps));
    const bool step_fused = (FORM & RADAM_STEP_FUSED) || ((FORM & RADAM_STEP_DENOM) && sc.denom != 0) || ((FORM & RADAM_STEP_LERP) && sc.lerp != 0);
    p = step_fused ? __fmaf_rn(-rate, val, __fmul_rn(p, decay_mul)) : __fmaf_rn(p, decay_mul, -__fmul_rn(rate, val));
    p = p < sc.min_w ? sc.min_w : p;
    p = p > sc.max_w ? sc.max_w : p;
    return p;
}

// FORM of the first three, LAST of the fourth
template <int FORM, int LAST = FORM>
static __device__ __forceinline__ float4 radam_four(float4 p, float4& m, float4& v, float4 g, const OptScalars& sc,
                                                     float rate, float decay_mul) {
    float4 r;
    r.x = radam_one<FORM>(p.x, m.x, v.x, g.x, sc, rate, decay_mul);
    r.y = radam_one<FORM>(p.y, m.y, v.y, g.y, sc, rate, decay_mul);
    r.z = radam_one<FORM>(p.z, m.z, v.z, g.z, sc, rate, decay_mul);
    r.w = radam_one<LAST>(p.w, m.w, v.w, g.w, sc, rate, decay_mul);
    return r;
}

static __device__ __forceinline__ float4 lerp_four(float4 w, float4 s, float alpha) {
    const float oma = 1.0f - alpha;
    return make_float4(alpha * w.x + oma * s.x, alpha * w.y + oma * s.y, alpha * w.z + oma * s.z, alpha * w.w + oma * s.w);
}
