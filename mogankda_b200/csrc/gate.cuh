// Gate activations and their derivatives.
#pragma once
#include "common.cuh"

namespace mkda {

// natural-log decay for one element; s = x + dt_bias, E = exp(A_log), lb = lower bound (< 0)
__device__ __forceinline__ float gate_value(int mode, float s, float E, float lb) {
    if (mode == MKDA_GATE_GDN) return fmaxf(-E * softplusf_(s), lb);
    if (mode == MKDA_GATE_KIMI) return lb * sigmoidf_(E * s);
    if (mode == MKDA_GATE_EDA) return lb + (-lb) * expf_(-(E / fabsf(lb)) * softplusf_(s));
    return s;
}
// d gate / d s  and  d gate / d A_log
__device__ __forceinline__ void gate_grad(int mode, float s, float E, float lb, float& ds, float& dA) {
    if (mode == MKDA_GATE_GDN) {
        const float sp = softplusf_(s);
        const float keep = (-E * sp >= lb) ? 1.f : 0.f;    // clamp passes no gradient
        ds = keep * (-E) * sigmoidf_(s);
        dA = keep * (-E) * sp;
    } else if (mode == MKDA_GATE_KIMI) {
        const float u = E * s, sg = sigmoidf_(u), d = lb * sg * (1.f - sg);
        ds = d * E;
        dA = d * u;
    } else if (mode == MKDA_GATE_EDA) {
        const float sp = softplusf_(s), c = E / fabsf(lb), w = expf_(-c * sp), d = lb * w * c;
        ds = d * sigmoidf_(s);
        dA = d * sp;
    } else {
        ds = 1.f;
        dA = 0.f;
    }
}

}  // namespace mkda
