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
//    tests/test_exact_root.py lists all solutions and every r1 in the
//    bound, and the result is the correctly rounded root for all of them.
//  * reciprocal of l: two of Newton's steps y + y (1 - l y) from r1. With
//    delta the error of y, one step lands l delta^2 below 1/l (and the rounding
//    of its residual within 2^-106), so it rounds wrongly only where 2^106 - D
//    factors into the significand of l and an odd 54-bit midpoint for a small D
//    (Markstein, IBM J. Res. Dev. 34(1), 1990); the first step is then one unit
//    off at most and the second one right, but for the significand of all
//    ones, l = 2^(k+1) (1 - 2^-53): its reciprocal 2^-(k+1) (1 + 2^-53 + ...) lies
//    just above a midpoint and rounds to 2^-(k+1) (1 + 2^-52), put together from
//    l's exponent. (Unit vectors of unrotated bodies come with s = 1 - 2^-53, so
//    it is usual.) The same test runs all of these significands,
//    tests/test_exact_root_ones.py that one.
//  * quotients: q0 = a r1, corrected once with r1 (faithful) and once with the
//    correctly rounded reciprocal (Markstein's theorem, as in quot_rcp).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace cc {

// ok: s in [2^-200, 2^200], so the steps above hold without underflow or overflow.
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
	const uint32_t lhi = (uint32_t)__double2hiint(o.l);
	const bool ones = ((lhi | 0xfff00000u) & (uint32_t)__double2loint(o.l)) == 0xffffffffu;
	o.y = __hiloint2double(ones ? (int)(0x7fdfffffu - lhi) : __double2hiint(o.y), ones ? 1 : __double2loint(o.y));
	const uint32_t hi = (uint32_t)__double2hiint(s);
	o.ok = hi - 0x33700000u <= 0x4C700000u - 0x33700000u;
	return o;
}

// a / l for the root above; a zero (which keeps its sign) or |a| > 2^-700 (quot_ok).
__device__ __forceinline__ double quot_root(double a, const InvRoot &v) {
	const double q0 = a * v.r;
	const double q1 = -fma(-fma(-v.l, q0, a), v.r, -q0);
	return -fma(-fma(-v.l, q1, a), v.y, -q1);
}
// Upper word of 2 |a|'s bits, minus one: all ones for a zero.
__device__ __forceinline__ uint32_t size_or_zero(double a) {
	return (uint32_t)((2ull * (unsigned long long)__double_as_longlong(a) - 1ull) >> 32);
}
constexpr uint32_t kSizeOfZero = 0xffffffffu;
// All of them zero or above 2^-700. Zeros are usual: every direction along an axis of
// an unrotated body has two. (As the slow path's work, with axis directions of
// cylinders and the all-ones root above: 488K pairs of 40K unrotated bodies, boxes
// 485 us and mixed types 778; so 330 and 353. 177K pairs with ten unrotated boulders
// 421 and 232; turned bodies, 402K pairs, 445 and 422.)
__device__ __forceinline__ bool quot_ok(uint32_t x, uint32_t y, uint32_t z) { return min(min(x, y), z) >= 0x28600000u; }
__device__ __forceinline__ bool quot_ok(double x, double y, double z) {
	return quot_ok(size_or_zero(x), size_or_zero(y), size_or_zero(z));
}

}  // namespace cc
