// x / (1 + exp(-x)), the same bits as that division for every fp32 x, without a branch.
//
// The compiler's division has a branch for the ends of the range, so that the values of a thread that finishes several came one after
// the other: 12000 clocks between two gate/up tiles of 256 rows in the prefill GEMM, 1500 with an approximate division.  That one alone
// is two units in the last place off: one fp32 value in forty came out differently, and one fp16 result in ten thousand.  So the
// quotient by an approximate reciprocal is corrected once by its own remainder, which a fused multiply-add gives exactly (Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor", 1990); compared with the division over all 2^32
// arguments.  Gate/up 5120 x 17408 at 512 rows: 141.4 us, with the approximation alone 140.4; at 77 rows 43.9 and 43.7.
#pragma once

#include <cuda_runtime.h>

namespace xb {

__device__ __forceinline__ float silu(float x) {
    const float y = 1.0f + expf(-x);
    // divisors above 2^126 have no normal reciprocal: a power of two, taken out again behind it (quotients stay above 2^-122)
    const float s = x < -40.0f ? 0x1p-64f : 1.0f;
    const float ys = y * s;
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(ys));
    const float q = x * r;
    const float rem = fmaf(-q, ys, x);
    // (no remainder: the quotient stands, -0 too.  NaN: x or y is not finite, and the quotient is what the division gives)
    return (fabsf(rem) > 0.0f ? fmaf(rem, r, q) : q) * s;
}

}  // namespace xb
