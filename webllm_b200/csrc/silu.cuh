// silu of one value, for the epilogue that takes it over many (gemm_pair.cu).
#pragma once

namespace wb {

// g / (1 + e^-g) in f32, as exact as the formula written out (silu_mul_kernel, qwen_ops.cu, which this takes the place of from 129 rows
// on): against 64 bits over +-12 both are at most 3.35 units of 2^-24 off, rms 0.75. The `/` operator costs a range check and a branch for
// each of a thread's 128 values, which then run one after the other. Here it is an approximate reciprocal, the quotient by it and
// one step on its residual, which an fma gives exactly. The ends:
//   * from g = -87.3 on the denominator is beyond 2^126, where the reciprocal is flushed to 0, which the true quotient rounds to in fp16
//     whatever it is multiplied with; the exponent is held at 88 so that the denominator stays finite.
//   * for g = infinity the residual is no number, which the maximum takes off: the quotient stays infinite. NaN comes through it.
// 2048 x 896 -> 2 x 4864, a layer of the 0.5B-shaped model: 124.1 us; with 2^x of a product and the remainder of its rounding in place of
// expf, and the Newton step on the reciprocal, 123.3, but up to 4.4 units off and rms 0.91; with 2^x and both remainders (rms 0.67) 126.4.
__device__ __forceinline__ float silu(float g)
{
    const float d = 1.f + expf(fminf(-g, 88.f));
    float q;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(q) : "f"(d));
    const float p = g * q;
    return fmaf(fmaxf(fmaf(-p, d, g), -3.40282347e38f), q, p);
}

}  // namespace wb
