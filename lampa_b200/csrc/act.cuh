// Activation functions shared by the layer and model kernels.
#pragma once
#include "common.cuh"

namespace lampa {

__device__ __forceinline__ float sigmoidf_(float x) { return __fdividef(1.f, 1.f + __expf(-x)); }
// log(1 + e^x) as max(x, 0) + log1p(e^-|x|).  log1p(e) = e P(e) on [0, 1] with P the degree-8 Chebyshev fit of log1p(e) / e:
// relative error 2e-7 in fp32 and no branch (the hardware log below its accuracy limit needed one, which diverges in
// nearly every warp).  torch switches to x above 20, where the two agree to fp32 rounding.
__device__ __forceinline__ float softplusf_(float x) {
    const float e = __expf(-fabsf(x));
    float p = 0.005253457929939032f;
    p = fmaf(p, e, -0.02958850748836994f);
    p = fmaf(p, e, 0.07836166769266129f);
    p = fmaf(p, e, -0.13674770295619965f);
    p = fmaf(p, e, 0.19111430644989014f);
    p = fmaf(p, e, -0.24844369292259216f);
    p = fmaf(p, e, 0.33319270610809326f);
    p = fmaf(p, e, -0.49999502301216125f);
    p = fmaf(p, e, 1.f);
    return fmaf(p, e, fmaxf(x, 0.f));
}

__device__ __forceinline__ float rcp_approx(float x) {      // one instruction; for arguments of moderate size
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
    return y;
}
// sigmoid with the bare reciprocal: 1 + e^-x is at least 1, so the range handling of __fdividef has nothing to do
__device__ __forceinline__ float sigmoid_fast(float x) { return rcp_approx(1.f + __expf(-x)); }

// Two fp32 values in one 64-bit register and the packed arithmetic on them: one issue slot for two operations.
struct F2 { uint64_t v; };
__device__ __forceinline__ F2 f2(float lo, float hi) { F2 r; asm("mov.b64 %0, {%1, %2};\n" : "=l"(r.v) : "f"(lo), "f"(hi)); return r; }
__device__ __forceinline__ F2 f2(float x) { return f2(x, x); }
__device__ __forceinline__ void f2_get(F2 a, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;\n" : "=f"(lo), "=f"(hi) : "l"(a.v)); }
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) { F2 r; asm("fma.rn.f32x2 %0, %1, %2, %3;\n" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v)); return r; }
__device__ __forceinline__ F2 mul2(F2 a, F2 b) { F2 r; asm("mul.rn.f32x2 %0, %1, %2;\n" : "=l"(r.v) : "l"(a.v), "l"(b.v)); return r; }
__device__ __forceinline__ F2 add2(F2 a, F2 b) { F2 r; asm("add.rn.f32x2 %0, %1, %2;\n" : "=l"(r.v) : "l"(a.v), "l"(b.v)); return r; }

// x Phi(x) of two values.  erfc(z) = (1 + a1 z + ... + a6 z^6)^-16 (Abramowitz & Stegun 7.1.28, error below 3e-7) with
// z = |x| / sqrt(2); x Phi(x) = max(x, 0) - |x| erfc(z) / 2, which has no cancellation on either side.  19 instructions
// for the pair; erff costs more than that for one.  Largest absolute difference from the exact function 7e-7.
__device__ __forceinline__ void gelu_pair(float x0, float x1, float& y0, float& y1) {
    const F2 z = f2(fabsf(x0) * 0.70710678f, fabsf(x1) * 0.70710678f);
    F2 p = f2(0.0000430638f);
    p = fma2(p, z, f2(0.0002765672f));
    p = fma2(p, z, f2(0.0001520143f));
    p = fma2(p, z, f2(0.0092705272f));
    p = fma2(p, z, f2(0.0422820123f));
    p = fma2(p, z, f2(0.0705230784f));
    p = fma2(p, z, f2(1.f));
    p = mul2(p, p); p = mul2(p, p); p = mul2(p, p); p = mul2(p, p);      // infinite where erfc is far below the smallest float
    float p0, p1;
    f2_get(p, p0, p1);
    f2_get(fma2(mul2(z, f2(-0.70710678f)), f2(rcp_approx(p0), rcp_approx(p1)), f2(fmaxf(x0, 0.f), fmaxf(x1, 0.f))), y0, y1);
}

}  // namespace lampa
