// The Uncharted 2 filmic curve of gamma_correction.frag:20-74, normalised by its value at the white point.
#pragma once

#include "common.cuh"

namespace phe_gb300 {

// gamma_correction.frag:35-43 constants; products of constants are folded in float as GLSL does.
constexpr float kU2A = 0.25f, kU2B = 0.25f, kU2C = 0.105f, kU2D = 0.20f, kU2E = 0.025f, kU2F = 0.25f;
constexpr float kU2CB = kU2C * kU2B, kU2DE = kU2D * kU2E, kU2DF = kU2D * kU2F, kU2EF = kU2E / kU2F;
constexpr float kU2White = (11.2f * (kU2A * 11.2f + kU2CB) + kU2DE) / (11.2f * (kU2A * 11.2f + kU2B) + kU2DF) - kU2EF;
constexpr float kU2WhiteInv = 1.0f / kU2White;

// n / d rounded to nearest, for |n|, |d| and the quotient far from the ends of the exponent range: the
// quotient's approximation n * r corrected with its fused residual (Markstein, IBM J. Res. Dev. 34, 1990), r the
// rounded reciprocal of d.
__device__ __forceinline__ float divide_in_range(float n, float d, float r)
{
	const float q = __fmul_rn(n, r);
	return __fmaf_rn(__fmaf_rn(-d, q, n), r, q);
}

// u2(x) / u2(W) of the filmic curve. It is a function of one float, and tests/cpp/filmic_test.cu compares it with
// the divisions as written for every float below the bound: the same bits.
constexpr float kFilmicBound = 1.0e15f;   // the numerator and denominator stay below 2^100
__device__ __forceinline__ float filmic_over_white(float x)
{
	const float num = __fadd_rn(__fmul_rn(x, __fadd_rn(__fmul_rn(kU2A, x), kU2CB)), kU2DE);
	const float den = __fadd_rn(__fmul_rn(x, __fadd_rn(__fmul_rn(kU2A, x), kU2B)), kU2DF);
	if (x < kFilmicBound)
		return divide_in_range(__fsub_rn(divide_in_range(num, den, reciprocal_in_range(den)), kU2EF), kU2White, kU2WhiteInv);
	return __fdiv_rn(__fsub_rn(__fdiv_rn(num, den), kU2EF), kU2White);
}

} // namespace phe_gb300
