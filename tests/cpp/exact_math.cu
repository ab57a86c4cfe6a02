// inv_root, quot_root (collision-detection_b200/csrc/cc_exact_math.cuh) on the device,
// against the device's correctly rounded sqrt, reciprocal and division bit for bit, and
// the bound on the seed that their derivation starts from, over every upper word of
// [1, 4) (the seed depends on no other bits but the exponent's, which scales it).
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "cc_exact_math.cuh"

namespace {

__device__ unsigned long long g_bad, g_ok, g_example;

__device__ unsigned long long bits(double x) { return (unsigned long long)__double_as_longlong(x); }
__device__ void fail(unsigned long long what) {
	if (atomicAdd(&g_bad, 1ull) == 0) g_example = what;
}
__device__ unsigned long long next(unsigned long long &s) {  // SplitMix64
	unsigned long long z = (s += 0x9E3779B97F4A7C15ull);
	z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
	z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
	return z ^ (z >> 31);
}

// Upper words of [1, 4): 2^21 of them, each with lower words 0, all ones and one drawn.
__global__ void k_seed() {
	const unsigned w = blockIdx.x * blockDim.x + threadIdx.x;  // grid: 2^21 threads
	unsigned long long r = w;
	const unsigned low[3] = {0u, 0xffffffffu, (unsigned)next(r)};
	for (int q = 0; q < 3; q++) {
		const double s = __hiloint2double((int)(0x3FF00000u + w), (int)low[q]);
		double r0;
		asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r0) : "d"(s));
		// |r0 sqrt(s) - 1| < 2^-20, by e = 1 - s r0^2 (about twice it; the product's own roundings are below 2^-51)
		const double e = fma(-s * r0, r0, 1.0);
		if (!(fabs(e) < 0x1.fffp-20)) fail(bits(s));
		else atomicAdd(&g_ok, 1ull);
	}
}

__device__ void check(double s, double a) {
	const cc::InvRoot v = cc::inv_root(s);
	if (!v.ok) return;
	atomicAdd(&g_ok, 1ull);
	const double l = __dsqrt_rn(s);
	if (bits(v.l) != bits(l)) fail(bits(s));
	if (bits(v.y) != bits(__drcp_rn(l))) fail(bits(s));
	if (cc::quot_ok(a, a, a) && fabs(a) <= 2.0 * l && bits(cc::quot_root(a, v)) != bits(__ddiv_rn(a, l))) fail(bits(a));
}

// Drawn operands over the whole range of `ok`; lengths next to 1 and to powers of two;
// squares of drawn numbers (exact roots) and their neighbours; numerators of every size
// down to the limit, zeros of either sign among them.
__global__ void k_check(unsigned long long seed, int per) {
	unsigned long long r = seed + (unsigned long long)(blockIdx.x * blockDim.x + threadIdx.x) * 0x632BE59BD9B4E019ull;
	for (int q = 0; q < per; q++) {
		const unsigned long long m = next(r), k = next(r);
		double s = __longlong_as_double((long long)((m & 0xFFFFFFFFFFFFFull) | ((unsigned long long)(1023 - 200 + k % 400) << 52)));
		if (q % 4 == 1) s = __longlong_as_double((long long)(0x3FF0000000000000ull + (m % 4097) - 2048));
		if (q % 4 == 2) {
			const double t = __longlong_as_double((long long)((m & 0xFFFFFFFF000000ull) >> (k % 25) | ((unsigned long long)(1023 - 90 + k % 180) << 52)) & 0x7FFFFFFFFFFFFFFFll);
			s = __longlong_as_double(__double_as_longlong(t * t) + (long long)(k >> 32) % 3 - 1);
		}
		if (q % 4 == 3) s = __longlong_as_double((long long)(((unsigned long long)(1023 - 199 + k % 398) << 52) + (m % 9) - 4));
		const double l = sqrt(s);
		const unsigned long long d = next(r);
		double a = l * ((double)(long long)d * 0x1p-63);
		if (d % 8 == 1) a = ldexp(a, -(int)((d >> 8) % 600));
		if (d % 8 == 2) a = (d >> 8) & 1 ? 0.0 : -0.0;
		if (d % 8 == 3) a = (d >> 8) & 1 ? l : -l;
		check(s, a);
	}
}

// The roots whose significand is all ones, at every exponent in range.
__global__ void k_ones() {
	const int k = (int)(blockIdx.x * blockDim.x + threadIdx.x) - 100;  // grid: 201 blocks of one
	const double s = ldexp(1.0 - 0x1p-53, 2 * k);
	const double l = ldexp(1.0 - 0x1p-53, k);
	const cc::InvRoot v = cc::inv_root(s);
	if (!v.ok) return;
	if (bits(v.l) != bits(l)) fail(bits(s));
	unsigned long long r = (unsigned long long)k;
	for (int q = 0; q < 20000; q++) check(s, l * ((double)(long long)next(r) * 0x1p-63));
}

bool report(const char *what, unsigned long long at_least) {
	unsigned long long bad = 0, ok = 0, ex = 0;
	const bool ran = cudaDeviceSynchronize() == cudaSuccess && cudaMemcpyFromSymbol(&bad, g_bad, 8) == cudaSuccess &&
	                 cudaMemcpyFromSymbol(&ok, g_ok, 8) == cudaSuccess && cudaMemcpyFromSymbol(&ex, g_example, 8) == cudaSuccess;
	const bool good = ran && bad == 0 && ok >= at_least;
	printf("%s: %s, %llu checked, %llu differ (first: %016llx)\n", what, good ? "TEST PASSED" : "TEST FAILED", ok, bad, ex);
	const unsigned long long zero = 0;
	cudaMemcpyToSymbol(g_bad, &zero, 8);
	cudaMemcpyToSymbol(g_ok, &zero, 8);
	return good;
}

}  // namespace

int main() {
	k_seed<<<(1u << 21) / 256, 256>>>();
	bool good = report("seed", 3ull << 21);
	k_check<<<1024, 256>>>(1, 200);
	good = report("root, reciprocal, quotients", 40000000) && good;
	k_ones<<<201, 1>>>();
	good = report("significands of all ones", 3900000) && good;
	return good ? 0 : 1;
}
