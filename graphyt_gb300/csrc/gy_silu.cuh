// gy_silu.cuh -- the surrogate's activation, z / (1 + exp(-z)), without the division's branches.
#pragma once

namespace gy {

// a / d for a divisor d >= 1, without the division's branch for the other divisors, so that the
// compiler can interleave the activations of a row: the hardware reciprocal and Markstein's
// correction of the quotient by its remainder (IBM J. Res. Dev. 34, 1990).  With d = 1 + __expf(-z),
// over all 2^32 z from -87 up: 1 / d has the division's bits, and z / d differs in its last bit at two
// z, at none once rounded to BF16.  Past d = 2^126, where the reciprocal is zero, so is the result
// (at most 1.1e-36 in truth).
// The remainder is negated, so that a quotient of -0 stays -0, and is NaN where a or d is infinite:
// fminf makes it finite there, and the result is a for a = +inf and zero for an overflowed d.  A NaN
// in a or d reaches the result by the quotient.
__device__ __forceinline__ float div_ge1(float a, float d)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    const float q = a * r;
    return fmaf(-fminf(fmaf(d, q, -a), 3.4e38f), r, q);
}

__device__ __forceinline__ float silu(float z) { return div_ge1(z, 1.0f + __expf(-z)); }

}  // namespace gy
