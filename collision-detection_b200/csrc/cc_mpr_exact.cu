// The narrowphase's exact variant: the reference's MPR (CollideAndFindPoint,
// src/narrowphase/Narrowphase.cu:122-314, inside function_MPR_Store :316-423)
// with its arithmetic in double: world coordinates, every direction normalized
// as v / sqrt(v.v), the reference's operation order. This translation unit is
// compiled with -fmad=false, so every product and sum rounds separately, as in
// the reference's host build with real = double: contacts equal the FP64
// oracle's, rounded to float on output.
//
// A pair runs on two neighbouring lanes: the even one evaluates the support
// map of shape A, the odd one that of shape B, and both keep the portal (the
// same arithmetic on the same operands). An iteration ("trip") of a warp
// evaluates one support pair for each of its running pairs and updates their
// portals, as in cc_mpr.cuh. What bounds it is the chain of dependent FP64
// operations of the longest pairs (about 40 trips; half of the pairs that
// reach the refinement run to its cap), so the trip is built to be short:
//  * the two supports side by side on two lanes: one sequence of instructions
//    instead of two (ptxas does not interleave two independent FP64 chains of
//    one lane, and a lone warp issues them at 3.5 cycles an instruction);
//  * normalizations by inv_root / quot_root (cc_exact_math.cuh), one range
//    flag each, instead of sqrt, reciprocal and per-component range branches;
//  * one straight support sequence for spheres, ellipsoids, boxes and
//    cylinders. Operands are selected by type and the two long parts (the
//    normalization that ellipsoids and cylinders share, the ellipsoid's second
//    one) run only if a lane of the warp needs them, so lanes of different
//    types share every instruction instead of taking turns. RECT, CONE and
//    TRIANGLEMESH, and operands outside the range of the fast normalizations,
//    take the general support() of cc_mpr.cuh.
//  * pairs wait for one another at their two costly turns: those that end
//    with a contact park until kBatch of the warp's pairs have nothing to do
//    (or none runs), and then the parked ones are finished and the idle lanes
//    take new pairs together.
#include <algorithm>

#include "cc_exact_math.cuh"
#include "cc_mpr.cuh"

namespace cc {

namespace {
using namespace mpr;
constexpr int kNT = 64;
// Pairs of a warp that have to be done before the warp turns to them (of 16;
// 195,000 pairs: 239 us with 6, 241 with 8; 306 with 12 before the last changes).
constexpr int kBatch = 6;

__device__ __forceinline__ D3 pick(bool c, D3 a, D3 b) { return mk(c ? a.x : b.x, c ? a.y : b.y, c ? a.z : b.z); }

// The rare paths as calls, so that the instructions of a trip lie together.
__device__ __noinline__ D3 unit_rare(double x, double y, double z) { return unit<double, true>(mk(x, y, z)); }

// unit<double, true> bit for bit where ok stays true.
__device__ __forceinline__ D3 unit_fast(D3 a, bool &ok) {
	const InvRoot v = inv_root(dotp(a, a));
	ok &= v.ok & quot_ok(a.x, a.y, a.z);
	return mk(quot_root(a.x, v), quot_root(a.y, v), quot_root(a.z, v));
}
__device__ __forceinline__ D3 unit_x(D3 a) {
	bool ok = true;
	D3 q = unit_fast(a, ok);
	if (!ok) q = unit_rare(a.x, a.y, a.z);
	return q;
}
// a / sqrt(a.a) in double with IEEE results, without the square root and the
// reciprocal when a.a lies within 2^20 units in the last place of 1 (a vector
// normalized once already). With s = a.a whose bits are bits(1) + e:
//  * sqrt(s) has the bits bits(1) + floor(e / 2). For s = 1 + t, sqrt(s) lies
//    strictly below 1 + t/2 (concavity) and above 1 + t/2 - t^2/8. Above 1
//    (t = e 2^-52) 1 + t/2 is representable for even e and a midpoint for odd
//    e; below 1 (t = e 2^-53, spacing 2^-53) the same holds with the halved
//    spacing. Either way the correctly rounded root is the representable
//    number at or just below 1 + t/2, t^2/8 being far below half a spacing.
//  * RN(1 / l) for l with the bits bits(1) + f: for f >= 0, 1/l lies above
//    1 - f 2^-52 (representable, bits(1) - 2f) by less than f^2 2^-104, under
//    half the spacing 2^-53 below 1; for f < 0, 1/l lies strictly above
//    1 - f 2^-53, which is representable (bits(1) - f/2) for even f and a
//    midpoint for odd f, so RN gives bits(1) + ceil(-f / 2) = bits(1) -
//    floor(f / 2).
// The quotients start from a itself (l differs from 1 by at most 2^-32, so
// a + (a - l a) y is faithful) and are corrected once more (Markstein), so the
// result is bit for bit unit<double, true>(a) where ok stays true; every
// component a zero or at least 2^-900.
__device__ __forceinline__ D3 again_fast(D3 a, bool &ok) {
	const double s = dotp(a, a);
	const int e = __double2loint(s), f = e >> 1;  // e fits 32 bits; f = floor(e / 2)
	const int g = f >= 0 ? -2 * f : -(f >> 1);
	constexpr int kOneHi = 0x3FF00000, kNear = 1 << 20;
	const double l = __hiloint2double(kOneHi + (f >> 31), f), y = __hiloint2double(kOneHi + (g >> 31), g);
	const auto quot = [&](double x) {
		const double q1 = -fma(-fma(-l, x, x), y, -x);
		return -fma(-fma(-l, q1, x), y, -q1);
	};
	ok &= ((uint32_t)(e + kNear) <= 2u * kNear) & (__double2hiint(s) == kOneHi + (e >> 31));
	return mk(quot(a.x), quot(a.y), quot(a.z));
}
// One shape of a pair. Y holds the factors of its local support point: B
// (ellipsoid, box), B.x three times (sphere), (B.x, B.y, B.x) (cylinder).
// fast: support_fast applies (the four types, with factors that keep its
// operands far from underflow).
struct Side {
	int type;
	bool fast;
	D3 X, Y;         // centre, factors (RECT, CONE: B; TRIANGLEMESH: vertices 0 and 1)
	D3 r0, r1, r2;   // rotation rows (TRIANGLEMESH: r0 = vertex 2)
};
__device__ __forceinline__ bool usual(double x) { return (fabs(x) >= 0x1p-40) & (fabs(x) <= 0x1p40); }
__device__ __forceinline__ Side side_of(const Shape<double> &s) {
	Side o = {s.type, true, s.X, s.Y, s.r0, s.r1, s.r2};
	if (s.type == SPHERE) {
		o.Y = mk(s.Y.x, s.Y.x, s.Y.x);
	} else if (s.type == CYLINDER) {
		o.Y.z = s.Y.x;
		o.fast = usual(s.Y.x) & usual(s.Y.y);
	} else if (s.type == ELLIPSOID) {
		o.fast = usual(s.Y.x) & usual(s.Y.y) & usual(s.Y.z);
	} else if (s.type != BOX) {
		o.fast = false;
	}
	return o;
}
// The shape again, for support() and centre() (which do not read the factors
// that side_of replaced).
__device__ __forceinline__ Shape<double> shape_of(const Side &s) {
	Shape<double> o;
	o.type = s.type;
	o.X = s.X; o.Y = s.Y;
	o.r0 = s.r0; o.r1 = s.r1; o.r2 = s.r2;
	return o;
}
__device__ __forceinline__ D3 centre_of(const Side &s) { return centre(shape_of(s)); }

// What the warp's lanes need of the support sequence (bits of `need`).
constexpr uint32_t kNeedUnit = 1, kNeedEllipsoid = 2;
__device__ __forceinline__ uint32_t side_need(int type) {
	return type == ELLIPSOID ? kNeedUnit | kNeedEllipsoid : (type == CYLINDER ? kNeedUnit : 0u);
}
__device__ __forceinline__ double with_sign_of(double b, double x) {  // sgn(x) b for x != 0
	return __hiloint2double(__double2hiint(b) ^ (__double2hiint(x) & 0x80000000), __double2loint(b));
}

__device__ __noinline__ D3 support_rare(Side s, D3 d) { return support<double, true>(shape_of(s), d); }
// support<double, true>(s, d) bit for bit where ok stays true; need: the union
// over the warp. The signs that box and cylinder take are sign bits; where the
// direction in the shape's frame has a zero, the sign is zero and they take the
// product with it.
__device__ __forceinline__ D3 support_fast(const Side &s, D3 d, uint32_t need, bool &ok) {
	const bool cyl = s.type == CYLINDER, ell = s.type == ELLIPSOID, box = s.type == BOX;
	const D3 n = mcol(s.r0, s.r1, s.r2, d);
	const uint32_t nx = size_or_zero(n.x), ny = size_or_zero(n.y), nz = size_or_zero(n.z);
	ok &= s.fast & quot_ok(nx, ny, nz);
	D3 u = n, e = n;
	if (need & kNeedUnit) {  // ellipsoid: n / |n|; cylinder: (n.x, 0, n.z) / |.|
		const bool uses = cyl | ell;
		D3 w = mk(n.x, cyl ? 0.0 : n.y, n.z);
		const double s2 = dotp(w, w);
		const bool axis = cyl & (s2 == 0.0);  // along the cylinder's axis: (0, sgn(n.y) B.y, 0)
		w.x = axis ? 0.0 : w.x;
		w.z = axis ? 0.0 : w.z;
		const InvRoot v = inv_root(axis ? 1.0 : s2);
		u = pick(uses, mk(quot_root(w.x, v), quot_root(w.y, v), quot_root(w.z, v)), n);
		ok &= !uses | v.ok;
	}
	if (need & kNeedEllipsoid) {  // B B u / |B u|
		const D3 bn = mulv(s.Y, u), bbn = mulv(mulv(s.Y, s.Y), u);
		const InvRoot v = inv_root(dotp(bn, bn));
		e = mk(quot_root(bbn.x, v), quot_root(bbn.y, v), quot_root(bbn.z, v));
		ok &= !ell | v.ok;
	}
	// sphere: B.x n; box: sgn(n) B; cylinder: (B.x u.x, sgn(n.y) B.y, B.x u.z)
	const uint32_t sign = box ? 0x7fffffffu : 0xffffffffu;  // sgn(-0) is +0
	const auto plain = [&](double x) { return __hiloint2double(__double2hiint(x) & sign, __double2loint(x)); };
	const D3 t = mulv(s.Y, mk(plain(u.x), plain(u.y), plain(u.z)));
	const D3 l = mk(box & (nx != kSizeOfZero) ? with_sign_of(s.Y.x, n.x) : (ell ? e.x : t.x),
	                (box | cyl) & (ny != kSizeOfZero) ? with_sign_of(s.Y.y, n.y) : (ell ? e.y : t.y),
	                box & (nz != kSizeOfZero) ? with_sign_of(s.Y.z, n.z) : (ell ? e.z : t.z));
	return add(mrow(s.r0, s.r1, s.r2, l), s.X);
}
__device__ __forceinline__ D3 shfl_partner(uint32_t mask, D3 a) {
	return mk(__shfl_xor_sync(mask, a.x, 1), __shfl_xor_sync(mask, a.y, 1), __shfl_xor_sync(mask, a.z, 1));
}

struct Pair {
	uint32_t index;
	int st, it;  // state; iterations of the current phase
	bool hit, mesh;  // a side is a TRIANGLEMESH (no envelope, :378-380)
	Side s;      // this lane's shape: A (even lane) or B (odd lane)
	D3 v0, v1, v2, v3;
	D3 n;  // direction of the next support pair (post stage: the normal, with the contact point in v1)
};

// This lane's support points behind the portal's three vertices (v11, v21, v31
// or v12, v22, v32), read only when a contact is finished: in shared memory,
// so that an iteration stores the new one with three stores instead of nine
// selects among 18 registers.
struct LanePoints {
	double *p;  // this lane's column of [3 vertices][3 coordinates][kNT]
	__device__ __forceinline__ void put(int vertex, D3 a) const {
		double *q = p + vertex * (3 * kNT);
		q[0] = a.x; q[kNT] = a.y; q[2 * kNT] = a.z;
	}
	__device__ __forceinline__ D3 get(int vertex) const {
		const double *q = p + vertex * (3 * kNT);
		return mk(q[0], q[kNT], q[2 * kNT]);
	}
};

__device__ __forceinline__ double side_sign(double x, bool odd) {  // direction of support(A, -d), support(B, d)
	return __hiloint2double(__double2hiint(x) ^ (odd ? 0 : (int)0x80000000), __double2loint(x));
}

// This lane's support point of a trip (support(A, -d), support(B, d)): w is
// normalized to d, once more when refining, with the unit normal left in L.n.
__device__ __forceinline__ D3 trip(Pair &L, D3 w, bool refines, bool odd, uint32_t need) {
	bool ok = true;
	D3 d = unit_fast(w, ok);
	if (refines) {
		L.n = d;
		d = again_fast(d, ok);
	}
	D3 p = support_fast(L.s, mk(side_sign(d.x, odd), side_sign(d.y, odd), side_sign(d.z, odd)), need, ok);
	if (!ok) {
		d = unit_rare(w.x, w.y, w.z);
		if (refines) {
			L.n = d;
			d = unit_rare(d.x, d.y, d.z);
		}
		p = support_rare(L.s, pick(odd, d, neg(d)));
	}
	return p;
}

// A refinement's portal update (:240-311) with the new normal in L.n and the
// support points p (this lane's) and p2 (its partner's).
__device__ __forceinline__ void refine_update(Pair &L, D3 p, D3 p2, bool odd, const LanePoints &pts) {
	L.it++;
	L.hit |= dotp(L.n, L.v1) >= 0.0;
	const D3 v = sub(pick(odd, p, p2), pick(odd, p2, p));
	const double delta = dotp(sub(v, L.v3), L.n);
	const double depth = dotp(v, L.n);
	const double s41 = dotp(crossp(v, L.v1), L.v0), s42 = dotp(crossp(v, L.v2), L.v0),
	             s43 = dotp(crossp(v, L.v3), L.v0);
	const bool end = (delta <= 1e-20) | (depth <= 0.0) | (L.it > kMaxIter);
	if (end) {
		L.st = L.hit ? kParked : kIdle;
		return;
	}
	const bool to3 = (s41 < 0.0) & !(s42 < 0.0), to2 = !(s41 < 0.0) & (s43 < 0.0), to1 = !(to3 | to2);
	pts.put(to3 ? 2 : (to2 ? 1 : 0), p);
	L.v1 = pick(to1, v, L.v1);
	L.v2 = pick(to2, v, L.v2);
	L.v3 = pick(to3, v, L.v3);
}

// finish_refine (cc_mpr.cuh): the contact point; the normal stays in L.n.
// Called by the lanes of `mask`.
__device__ __forceinline__ void finish(Pair &L, const LanePoints &pts, uint32_t mask) {
	const D3 v1 = L.v1, v2 = L.v2, v3 = L.v3, v0 = L.v0, n = L.n;
	double b0 = dotp(crossp(v1, v2), v3);
	double b1 = dotp(crossp(v3, v2), v0);
	double b2 = dotp(crossp(v0, v1), v3);
	double b3 = dotp(crossp(v2, v1), v0);
	double sum = b0 + b1 + b2 + b3;
	if (sum <= 0.0) {
		b0 = 0.0;
		b1 = dotp(crossp(v2, v3), n);
		b2 = dotp(crossp(v3, v1), n);
		b3 = dotp(crossp(v1, v2), n);
		sum = b1 + b2 + b3;
	}
	const double inv = 1.0 / sum;
	const D3 p = add(add(add(scl(b0, centre_of(L.s)), scl(b1, pts.get(0))), scl(b2, pts.get(1))), scl(b3, pts.get(2)));
	const D3 pq = add(p, shfl_partner(mask, p));
	L.v1 = mk(pq.x * inv * 0.5, pq.y * inv * 0.5, pq.z * inv * 0.5);
	L.n = unit_x(n);
	L.st = kPost;
}

// State update of the phases before and after the refinement.
__device__ __forceinline__ void other_update(Pair &L, D3 p, D3 p2, bool odd, const LanePoints &pts, float envelope,
                                             const long long *pairs, const uint32_t *ID, const NpScratch &sc) {
	const D3 v = sub(pick(odd, p, p2), pick(odd, p2, p));
	const bool miss = dotp(v, L.n) <= 0.0;
	if (L.st == kS1) {  // :146-171
		L.v1 = v;
		pts.put(0, p);
		L.n = crossp(v, L.v0);
		L.st = kS2;
		if (miss) {
			L.st = kIdle;
		} else if (is_zero(L.n)) {
			L.n = unit_x(sub(v, L.v0));
			const D3 s12 = add(p, p2);
			L.v1 = mk(s12.x * 0.5, s12.y * 0.5, s12.z * 0.5);
			L.st = kPost;
		}
	} else if (L.st == kS2) {  // :173-191
		L.v2 = v;
		L.n = crossp(sub(L.v1, L.v0), sub(v, L.v0));
		if (dotp(L.n, L.v0) > 0.0) {  // the new vertex becomes the first
			pts.put(1, pts.get(0));
			pts.put(0, p);
			L.v2 = L.v1;
			L.v1 = v;
			L.n = neg(L.n);
		} else {
			pts.put(1, p);
		}
		L.it = 1;
		L.hit = false;
		L.st = miss ? kIdle : kDisc;
	} else if (L.st == kDisc) {  // :201-232
		L.v3 = v;
		const double s13 = dotp(crossp(L.v1, v), L.v0), s32 = dotp(crossp(v, L.v2), L.v0);
		if (miss) {
			L.st = kIdle;
		} else if (s13 < 0.0) {
			pts.put(1, p);
			L.v2 = v;
			L.n = crossp(sub(L.v1, L.v0), sub(v, L.v0));
		} else if (s32 < 0.0) {
			pts.put(0, p);
			L.v1 = v;
			L.n = crossp(sub(v, L.v0), sub(L.v2, L.v0));
		} else {
			pts.put(2, p);
			L.st = kRefine;
			L.it = 0;
		}
		if (L.st == kDisc && L.it++ > kMaxIter) L.st = kIdle;
	} else {  // kPost :404-406
		const D3 N = L.n, p0 = L.v1;
		const D3 q = add(scl(dotp(sub(p, p0), N), N), p0), q2 = add(scl(dotp(sub(p2, p0), N), N), p0);
		if (!odd) {
			const uint64_t key = (uint64_t)pairs[L.index];
			write_contact(L.index, L.mesh ? 0.0 : (double)envelope, mk(0.0, 0.0, 0.0), neg(N), q, q2,
			              __ldg(ID + (uint32_t)(key >> 32)), __ldg(ID + (uint32_t)key), sc);
		}
		L.st = kIdle;
	}
}

// Starts pair i (:338-397; start_pair of cc_mpr.cuh) on the lanes of `mask`,
// each loading its own shape. Sphere-sphere pairs and skipped pairs end here.
__device__ __forceinline__ void start(Pair &L, uint32_t i, bool odd, uint32_t mask, uint64_t n, const int32_t *T,
                                      const float *A, const float *B, const float *C, const float *R,
                                      const uint32_t *ID, uint64_t nb, const uint8_t *active, const float *pos,
                                      const float *rot, float envelope, const long long *pairs, const NpScratch &sc) {
	const uint64_t key = (uint64_t)pairs[i];
	const uint64_t sh64 = odd ? key & 0xffffffffull : key >> 32;
	bool good = sh64 < n;
	const uint32_t sh = good ? (uint32_t)sh64 : 0u;
	uint32_t id = n ? __ldg(ID + sh) : 0u;
	good &= id < nb;
	if (!odd) {
		sc.pairs[i] = key;
		sc.flag[i] = 0u;
	}
	const bool bad = !good | (bool)__shfl_xor_sync(mask, !good, 1);
	if (bad & !odd) atomicOr(sc.err, (uint32_t)kErrBadIndex);
	const bool act = good && active[good ? id : 0u];
	const bool act2 = __shfl_xor_sync(mask, act, 1);
	const uint32_t id2 = __shfl_xor_sync(mask, id, 1);
	const bool live = !bad & (act | act2) & (id != id2);  // :344-349
	Shape<double> s;
	s.type = SPHERE;
	s.X = s.Y = s.r0 = s.r1 = s.r2 = mk(0.0, 0.0, 0.0);
	if (live) s = load_shape<double>(sh, id, T, A, B, C, R, pos, rot, mk(0.0, 0.0, 0.0));
	const int type2 = __shfl_xor_sync(mask, s.type, 1);
	const D3 c = centre(s), c2 = shfl_partner(mask, c);
	const double r2 = __shfl_xor_sync(mask, s.Y.x, 1);
	const D3 x2 = shfl_partner(mask, s.X);
	if (!live) return;
	if (s.type == SPHERE && type2 == SPHERE) {  // :382-397
		if (odd) return;
		const D3 rel = sub(x2, s.X);
		const double d2 = dotp(rel, rel);
		const double ra = s.Y.x, rb = r2;
		const double cd = ra + rb;
		if (!(d2 <= cd * cd)) return;
		const D3 N = unit_x(rel);
		write_contact(i, (double)envelope, mk(0.0, 0.0, 0.0), N, add(s.X, scl(ra, N)), sub(x2, scl(rb, N)), id, id2, sc);
		return;
	}
	// CollideAndFindPoint :137-144
	L.index = i;
	L.s = side_of(s);
	L.mesh = (s.type == TRIANGLEMESH) | (type2 == TRIANGLEMESH);
	L.v0 = sub(pick(odd, c, c2), pick(odd, c2, c));
	if (is_zero(L.v0)) L.v0 = mk(1.0, 0.0, 0.0);
	L.n = neg(L.v0);
	L.st = kS1;
}

__global__ void __launch_bounds__(kNT, 6) k_mpr_exact(uint64_t P_cap, const unsigned long long *P_dev, uint64_t n,
                                                    const int32_t *__restrict__ T, const float *__restrict__ A,
                                                    const float *__restrict__ B, const float *__restrict__ C,
                                                    const float *__restrict__ R, const uint32_t *__restrict__ ID,
                                                    uint64_t nb, const uint8_t *__restrict__ active,
                                                    const float *__restrict__ pos, const float *__restrict__ rot,
                                                    float envelope, const long long *__restrict__ pairs,
                                                    NpScratch sc) {
	const uint64_t P = P_dev ? min(P_cap, (uint64_t)*P_dev) : P_cap;
	uint32_t *queue = sc.queue;
	const uint32_t lane = threadIdx.x & 31, lt = (1u << lane) - 1u;
	const bool odd = lane & 1;
	// pairs a warp holds: as few as take all of them at once over the grid's
	// warps; the warps' first pairs are fixed, the queue starts behind them
	const uint64_t warps = (uint64_t)gridDim.x * (kNT / 32);
	const uint32_t width = (uint32_t)min((P + warps - 1) / warps, (uint64_t)16);
	const uint64_t first = warps * width;
	uint64_t j = ((uint64_t)blockIdx.x * (kNT / 32) + (threadIdx.x >> 5)) * width + (lane >> 1);
	const uint32_t batch = min((uint32_t)kBatch, width);
	__shared__ double points[3 * 3 * kNT];
	const LanePoints pts = {points + threadIdx.x};
	Pair L;
	L.st = kIdle;
	bool fresh = true, drained = false;  // before the first fill; the queue is exhausted (warp-uniform)
	while (true) {
		const bool wants = L.st == kIdle && !drained && (lane >> 1) < width;
		const uint32_t idle = __ballot_sync(0xffffffffu, wants), parked = __ballot_sync(0xffffffffu, L.st == kParked);
		uint32_t runs = __ballot_sync(0xffffffffu, L.st != kIdle && L.st != kParked);
		if (!(idle | parked | runs)) break;
		if (!runs || (uint32_t)__popc(idle | parked) >= 2 * batch) {
			if (idle) {  // new pairs for the idle lanes, one atomic per warp
				const uint32_t cnt = __popc(idle) >> 1;
				if (!fresh) {
					uint32_t base = 0;
					const int leader = __ffs(idle) - 1;
					if ((int)lane == leader) base = atomicAdd(queue, cnt);
					base = __shfl_sync(0xffffffffu, base, leader);
					j = first + base + (__popc(idle & lt) >> 1);
					drained = first + base + cnt >= P;
				} else {
					drained = first >= P;
				}
				fresh = false;
				const bool take = wants && j < P;
				const uint32_t mask = __ballot_sync(0xffffffffu, take);
				if (take)
					start(L, (uint32_t)j, odd, mask, n, T, A, B, C, R, ID, nb, active, pos, rot, envelope, pairs, sc);
			}
			if (L.st == kParked) finish(L, pts, parked);
		}
		// trips until enough pairs have ended (or only parked ones are left)
		const int stop = drained ? 0 : 2 * ((int)width - (int)batch);  // lanes that may still run when the loop ends
		bool running = L.st != kIdle && L.st != kParked;
		const uint32_t need = __reduce_or_sync(0xffffffffu, running ? side_need(L.s.type) : 0u);
		while (true) {
			runs = __ballot_sync(0xffffffffu, running);
			if (__popc(runs) <= stop) break;
			const uint32_t others = __ballot_sync(0xffffffffu, running && L.st != kRefine);
			if (drained && !others) {  // refinements only, and no more pairs to come: the same trip without the other states
				while (runs) {
					if (L.st == kRefine) {
						const D3 w = crossp(sub(L.v2, L.v1), sub(L.v3, L.v1));
						const D3 p = trip(L, w, true, odd, need);
						refine_update(L, p, shfl_partner(runs, p), odd, pts);
					}
					runs = __ballot_sync(0xffffffffu, L.st == kRefine);
				}
				break;
			}
			if (running) {
				const bool refines = L.st == kRefine;
				D3 w = L.n;
				if (refines) w = crossp(sub(L.v2, L.v1), sub(L.v3, L.v1));  // :240-253
				const D3 p = trip(L, w, refines, odd, need);
				const D3 p2 = shfl_partner(runs, p);
				if (refines) refine_update(L, p, p2, odd, pts);
				else if (others) other_update(L, p, p2, odd, pts, envelope, pairs, ID, sc);
				running = L.st != kIdle && L.st != kParked;
			}
		}
	}
	pdl_wait();  // beside the pair sort: this kernel ends after it
}
}  // namespace

int mpr_exact_resident_blocks() {
	static const int b = [] {
		int v = 0;
		if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, k_mpr_exact, kNT, 0) != cudaSuccess || v < 1) v = 1;
		return v;
	}();
	return b;
}

void launch_mpr_exact(unsigned grid, uint64_t P_cap, const unsigned long long *P_dev, uint64_t n, const int32_t *T,
                      const float *A, const float *B, const float *C, const float *R, const uint32_t *ID, uint64_t nb,
                      const uint8_t *active, const float *pos, const float *rot, float envelope,
                      const long long *pairs, const NpScratch &sc, cudaStream_t s, bool beside) {
	// Beside the pair sort: its blocks, a cooperative launch, are all resident once
	// this kernel starts, the two share no data, and this one ends after it. Else a
	// plain launch, and no early start of what follows either: blocks that become
	// resident among a neighbour's spread unevenly, and few warps of FP64 chains run
	// as slow as the fullest SM (3.4K pairs of 130K bodies: a step of 99 us with the
	// MPR's blocks launched early, 86 without; 2K pairs of 1K bodies: 91 us with its
	// successor's launched early, 85 without).
	if (beside)
		launch_pdl<true>(k_mpr_exact, dim3(grid), dim3(kNT), 0, s, P_cap, P_dev, n, T, A, B, C, R, ID, nb, active, pos, rot,
		                 envelope, pairs, sc);
	else
		k_mpr_exact<<<grid, kNT, 0, s>>>(P_cap, P_dev, n, T, A, B, C, R, ID, nb, active, pos, rot, envelope, pairs, sc);
}

}  // namespace cc
