// silu of one value, for the epilogue that takes it over many (gemm_pair.cu).
#pragma once

namespace wb {

// g / (1 + e^-g) in f32. The fast quotient (within 2 ulp) with one step of iterative refinement: its residual, exact in an fma,
// divided again. The `/` operator costs a range check and a branch for each of a thread's 128 values, which then run one after
// the other (75 us -> 67 us at 2048 x 896 -> 2 x 4864). The range is known here: 1 <= d, and from 2^126 on, where d is held at
// e^88, the fast quotient is 0, which the true one rounds to in fp16 whatever it is multiplied with.
__device__ __forceinline__ float silu(float g)
{
    const float d = 1.f + expf(fminf(-g, 88.f));
    const float q = __fdividef(g, d);
    return g == INFINITY ? g : q + __fdividef(fmaf(-q, d, g), d);
}

}  // namespace wb
