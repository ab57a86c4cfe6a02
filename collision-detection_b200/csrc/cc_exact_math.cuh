// a / sqrt(s) in double with IEEE results (sqrt, then the division, each
// correctly rounded) as one short branch-free sequence.
//
// The exact MPR normalizes four vectors per iteration, and sqrt and
// __drcp_rn, correctly rounded for every input, end in branches on rare
// operands: two of them never overlap (measured on B200, one warp: sqrt 93
// cycles, reciprocal 76, and two independent ones take twice that), while a
// dependent FP64 multiply-add is 9 cycles and independent ones overlap. Here
// one seed serves the root and its reciprocal, the rare operands are told by
// one flag that the caller tests once, and two normalizations side by side
// cost little more than one.
//
// With r1 = (1 + rho) / sqrt(s), |rho| <= 1.6 * 2^-53:
//  * seed: rsqrt.approx.ftz.f64, relative error below 2^-20 (every upper word
//    of [1, 4) checked on B200), then one step of the third-order iteration
//    r0 * (1 + e/2 + 3/8 e^2), e = 1 - s r0^2, the binomial series of
//    (1 - e)^(-1/2): its truncation is 5/16 e^3 < 2^-58, its roundings
//    0.5 + 1 units of 2^-53.
//  * root: l0 = s r1, l = l0 + (s - l0^2) r1/2 (Newton's step for s - l^2 = 0).
//    Before its last rounding l is within 10.2 * 2^-106 of sqrt(s),
//    relatively. A root that lies that close to the midpoint of two doubles
//    satisfies S 2^54 - M^2 = D for its integer significands with |D| < 84;
//    tests/test_exact_rounding.py lists all solutions and every r1 in the
//    bound, and the result is the correctly rounded root for all of them.
//  * reciprocal of l: two of Newton's steps y + y (1 - l y) from r1. With
//    delta the error of y, one step lands l delta^2 below 1/l (and the rounding
//    of its residual within 2^-106), so it rounds wrongly only where 2^106 - D
//    factors into the significand of l and an odd 54-bit midpoint for a small D
//    (Markstein, IBM J. Res. Dev. 34(1), 1990); the first step is then one unit
//    off at most and the second one right, but for the significand of all
//    ones, which the flag sends to the caller's slow path. The same test runs
//    all of these significands.
//  * quotients: q0 = a r1, corrected once with r1 (faithful) and once with the
//    correctly rounded reciprocal (Markstein's theorem, as in quot_rcp).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace cc {

// s in [2^-200, 2^200] and l's significand not all ones: the steps above hold
// without underflow or overflow.
struct InvRoot {
	double l;   // RN(sqrt(s))
	double y;   // RN(1 / l)
	double r;   // 1 / sqrt(s) within 1.6 * 2^-53
	bool ok;
};

__device__ __forceinline__ InvRoot inv_root(double s) {
	InvRoot o;
	double r0;
	asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r0) : "d"(s));
	const double g = s * r0;
	const double e = fma(-g, r0, 1.0);
	o.r = fma(r0 * e, fma(0.375, e, 0.5), r0);
	const double l0 = s * o.r;
	o.l = fma(fma(-l0, l0, s), 0.5 * o.r, l0);
	const double y1 = fma(o.r, fma(-o.l, o.r, 1.0), o.r);
	o.y = fma(y1, fma(-o.l, y1, 1.0), y1);
	const uint32_t hi = (uint32_t)__double2hiint(s);
	o.ok = (hi - 0x33700000u <= 0x4C700000u - 0x33700000u) & ((uint32_t)__double2loint(o.l) != 0xffffffffu);
	return o;
}

// a / l for the root above; a zero or |a| >= 2^-700 (quot_large).
__device__ __forceinline__ double quot_root(double a, const InvRoot &v) {
	const double q0 = a * v.r;
	const double q1 = -fma(-fma(-v.l, q0, a), v.r, -q0);
	return -fma(-fma(-v.l, q1, a), v.y, -q1);
}
// All magnitudes at least 2^-700.
__device__ __forceinline__ bool quot_large(double x, double y, double z) {
	const auto mag = [](double a) { return (uint32_t)__double2hiint(a) & 0x7fffffffu; };
	return min(min(mag(x), mag(y)), mag(z)) >= 0x14300000u;
}

}  // namespace cc
