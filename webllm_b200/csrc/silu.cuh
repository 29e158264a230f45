// silu of one value, for the epilogue that takes it over many (gemm_pair.cu).
#pragma once

namespace wb {

// g / (1 + e^-g) in f32. An epilogue has 128 of these per thread and item, and few issue slots to do them in, so every instruction counts:
//   * e^a = 2^t with t = a log2(e) rounded, which the hardware's 2^x takes over its whole range, times 1 + r ln(2) for what the rounding
//     left off, r = a log2(e) - t: exact in an fma but for log2(e)'s own second part. (t alone is good to 2^-17 at a = 88.)
//   * one approximate reciprocal of the denominator and one Newton step on it. The step is on the reciprocal and not on the quotient,
//     which may be infinite.
// The exponent is held within +-88: above, 1 + e^-g is 1; below, the denominator is beyond 2^126, where the reciprocal is flushed to 0,
// which the true quotient rounds to in fp16 whatever it is multiplied with. NaN comes through g. 14 instructions, two of them on the special
// function unit; with expf and two fast quotients 2048 x 896 -> 2 x 4864 took 53.6 us, without any silu 44.
__device__ __forceinline__ float silu(float g)
{
    const float a = fmaxf(fminf(-g, 88.f), -88.f);
    constexpr float kLog2e = 1.44269502f, kLog2eRest = 1.92596303e-8f, kLn2 = 0.693147182f;  // log2(e) in two parts, ln(2)
    const float t = a * kLog2e, r = fmaf(a, kLog2eRest, fmaf(a, kLog2e, -t));
    float e, q;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(t));
    const float d = fmaf(e, r * kLn2, e) + 1.f;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(q) : "f"(d));
    return g * fmaf(fmaf(-d, q, 1.f), q, q);
}

}  // namespace wb
