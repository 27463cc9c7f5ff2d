// Activation functions shared by the layer and model kernels.
#pragma once
#include "common.cuh"

namespace lampa {

__device__ __forceinline__ float sigmoidf_(float x) { return __fdividef(1.f, 1.f + __expf(-x)); }
// log(1 + e^x) as max(x, 0) + log1p(e^-|x|); the log1p is the hardware log above 0.01 (absolute
// error 2e-7) and its cubic Taylor polynomial below.  torch switches to x above 20, where the
// two agree to fp32 rounding.
__device__ __forceinline__ float softplusf_(float x) {
    const float e = __expf(-fabsf(x));
    const float l = e > 0.01f ? __logf(1.f + e) : e * (1.f - e * (0.5f - e * (1.f / 3.f)));
    return fmaxf(x, 0.f) + l;
}

// x Phi(x).  erfc(z) = (1 + a1 z + ... + a6 z^6)^-16 (Abramowitz & Stegun 7.1.28, error below 3e-7) on |x| / sqrt(2):
// one reciprocal and ten multiply-adds, where erff costs twice that; the negative side comes out as 0.5 x erfc, without
// the cancellation of 1 + erf.  Largest absolute difference from the exact function 7e-7.
__device__ __forceinline__ float geluf_(float x) {
    const float z = fabsf(x) * 0.70710678f;
    float p = 0.0000430638f;
    p = fmaf(p, z, 0.0002765672f);
    p = fmaf(p, z, 0.0001520143f);
    p = fmaf(p, z, 0.0092705272f);
    p = fmaf(p, z, 0.0422820123f);
    p = fmaf(p, z, 0.0705230784f);
    p = fmaf(p, z, 1.f);
    p *= p; p *= p; p *= p; p *= p;                       // overflows where erfc is far below the smallest float: 0
    const float h = __fdividef(0.5f, p);
    return x * (x < 0.f ? h : 1.f - h);
}

}  // namespace lampa
