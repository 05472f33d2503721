// tanh of scores under a soft cap, for the kernels of the mixed heads (attention_mixed_mma.cu, attention_mixed_token.cu).
#pragma once

namespace kl {

// tanh(x) for |x| <= CAP_SMALL: x + x^3 R(x^2) with R of degree four, fitted for the relative error of tanh (4.7e-9 of it with these float32
// coefficients; in 32 bits 0.76 units in the last place).  Scores under a soft cap lie there as a rule, and this takes seven instructions and no branch.
constexpr float CAP_SMALL = 0.6f;
__device__ __forceinline__ float cap_tanh(float x) {
    const float u = x * x;
    float r = fmaf(-5.895158275961876e-3f, u, 2.0795971155166626e-2f);
    r = fmaf(r, u, -5.3783830255270004e-2f);
    r = fmaf(r, u, 0.13331924378871918f);
    r = fmaf(r, u, -0.33333298563957214f);
    return fmaf(x * u, r, x);
}
// v times (c + rest), which together are scale / cap, rounded once; of an infinite or huge one the leading product (tanh is 1 far before that)
__device__ __forceinline__ float cap_quotient(float v, float c, float rest) {
    const float x = v * c;
    return fabsf(x) < 64.f ? fmaf(v, c, v * rest) : x;
}
// the same of a score whose leading product is at most CAP_SMALL
__device__ __forceinline__ float cap_small_quotient(float v, float c, float rest) { return fmaf(v, c, v * rest); }

// scale / cap as the sum of two numbers (0 without a cap)
inline void cap_parts(float scale, float cap, float& c, float& rest) {
    const double q = cap > 0.f ? (double)scale / (double)cap : 0.0;
    c = (float)q;
    rest = (float)(q - (double)c);
}

}  // namespace kl
