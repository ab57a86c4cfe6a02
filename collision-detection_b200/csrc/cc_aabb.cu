// AABB generation: AABBGenerator::GenerateAABB of the reference
// (src/aabb/AABBGenerator.cu:84-188) as one sm_100a kernel, one thread per
// shape, optionally fused with the broadphase's first pass (scene bounds,
// extent sums and input validation) so the pipeline reads each shape once.
// Compiled with -fmad=false: results are bit-identical to the reference's
// host build.
#include <algorithm>

#include "cc_common.cuh"
#include "cc_internal.h"
#include "cc_math.cuh"
#include "cc_stats.cuh"

namespace cc {

namespace {
constexpr int kNT = 256;

__device__ __forceinline__ float3 ld3(const float *p, uint64_t i) {
	return f3(__ldg(p + 3 * i), __ldg(p + 3 * i + 1), __ldg(p + 3 * i + 2));
}
__device__ __forceinline__ float4 ld4(const float *p, uint64_t i) {
	return __ldg(reinterpret_cast<const float4 *>(p) + i);
}
__device__ __forceinline__ float smin(float a, float b) { return (b < a) ? b : a; }  // std::min
__device__ __forceinline__ float smax(float a, float b) { return (a < b) ? b : a; }  // std::max

// function_ComputeAABB (AABBGenerator.cu:84-116). Returns false for the types
// the reference skips (:110-111): nothing is written for them.
__device__ __forceinline__ bool shape_aabb(uint64_t i, const int32_t *T, const float *A, const float *B,
                                           const float *C, const float *R, const uint32_t *ID, uint64_t nb,
                                           const float *pos, const float *rot, float3 &mn, float3 &mx,
                                           uint32_t *err) {
	const int type = __ldg(T + i);
	const uint32_t id = __ldg(ID + i);
	if (id >= nb) {
		atomicOr(err, (uint32_t)kErrBadIndex);
		return false;
	}
	float3 a = ld3(A, i), b = ld3(B, i);
	const float3 position = ld3(pos, id);
	const float4 brot = ld4(rot, id);
	const float4 lrot = ld4(R, i);
	// A zero local offset rotates to (+-0, +-0, +-0) and an identity local
	// rotation leaves body_rot unchanged up to the sign of zero terms; neither
	// sign survives (p +- r rounds the same, |R| drops it), so skipping that
	// arithmetic gives bit-identical boxes.
	const bool a_zero = a.x == 0.f && a.y == 0.f && a.z == 0.f;
	const bool r_ident = lrot.x == 1.f && lrot.y == 0.f && lrot.z == 0.f && lrot.w == 0.f;
	if (type == SPHERE) {  // :96-98, ComputeAABBSphere :11-14
		const float3 p = a_zero ? position : qrot(a, brot) + position;
		const float3 r = f3(b.x, b.x, b.x);
		mn = p - r;
		mx = p + r;
		return true;
	}
	if (type == CONE) {  // :103-107: the reference treats type 5 as a triangle
		const float4 rotation = qmul(brot, lrot);
		const float3 c = ld3(C, i);
		a = qrot(a + position, rotation);
		b = qrot(b + position, rotation);
		const float3 cc = qrot(c + position, rotation);
		mn = f3(smin(a.x, smin(b.x, cc.x)), smin(a.y, smin(b.y, cc.y)), smin(a.z, smin(b.z, cc.z)));
		mx = f3(smax(a.x, smax(b.x, cc.x)), smax(a.y, smax(b.y, cc.y)), smax(a.z, smax(b.z, cc.z)));
		return true;
	}
	if (type == ELLIPSOID || type == BOX || type == CYLINDER) {  // :108-109, ComputeAABBBox :25-35
		const Rot m = rot_rows(r_ident ? brot : qmul(brot, lrot));
		const float3 half = f3(dot(abs3(m.r0), b), dot(abs3(m.r1), b), dot(abs3(m.r2), b));
		const float3 p = a_zero ? position : qrot(a, brot) + position;
		mn = p - half;
		mx = p + half;
		return true;
	}
	return false;
}

// Persistent: each thread walks shapes blockIdx*kNT + tid, step gridDim*kNT,
// keeping its share of the bounds in registers, so the block reduces once.
template <bool kStats>
__global__ void __launch_bounds__(kNT) k_aabb(uint64_t n, const int32_t *__restrict__ T, const float *__restrict__ A,
                                               const float *__restrict__ B, const float *__restrict__ C,
                                               const float *__restrict__ R, const uint32_t *__restrict__ ID,
                                               uint64_t nb, const float *__restrict__ pos,
                                               const float *__restrict__ rot, float *__restrict__ aabb,
                                               DevStats *stats, uint32_t *err, PlanArgs pa, ZeroList zero) {
	pdl_begin();
	zero_ranges(zero);
	float3 bmn = f3(INFINITY, INFINITY, INFINITY), bmx = f3(-INFINITY, -INFINITY, -INFINITY);
	float3 esum = f3(0.f, 0.f, 0.f);  // extent sum for the grid tuner's mean box size
	bool have = false;
	uint32_t e = 0, ecnt = 0;
	for (uint64_t i = (uint64_t)blockIdx.x * kNT + threadIdx.x; i < n; i += (uint64_t)gridDim.x * kNT) {
		float3 mn, mx;
		if (shape_aabb(i, T, A, B, C, R, ID, nb, pos, rot, mn, mx, err)) {
			float *o = aabb + 3 * i, *o2 = aabb + 3 * (i + n);
			o[0] = mn.x; o[1] = mn.y; o[2] = mn.z;
			o2[0] = mx.x; o2[1] = mx.y; o2[2] = mx.z;
		} else if (kStats) {  // skipped shape: the broadphase sees the caller's old values
			const float *o = aabb + 3 * i, *o2 = aabb + 3 * (i + n);
			mn = f3(o[0], o[1], o[2]);
			mx = f3(o2[0], o2[1], o2[2]);
		}
		if constexpr (kStats) {
			if (!finite3(mn) || !finite3(mx)) e |= kErrNonFinite;
			if (mn.x > mx.x || mn.y > mx.y || mn.z > mx.z) e |= kErrInverted;
			bmn = f3(fminf(bmn.x, mn.x), fminf(bmn.y, mn.y), fminf(bmn.z, mn.z));
			bmx = f3(fmaxf(bmx.x, mx.x), fmaxf(bmx.y, mx.y), fmaxf(bmx.z, mx.z));
			esum = esum + (mx - mn);
			ecnt++;
			have = true;
		}
	}
	if constexpr (kStats) accumulate_stats<kNT>(bmn, bmx, have, stats, pa, e, esum, ecnt);
}
// ---------------------------------------------------------------- batches
// The front of a batch pass as one kernel: scene and global body id of every
// shape, its box, the scenes' bounds and, by the last block, their plans and
// the first cells of their grids. kGather: the scenes lie in their own
// allocations (src) and are copied into the concatenated arrays (dst) on the
// way; otherwise `all` holds the concatenated arrays.
//
// Each block takes a run of neighbouring tiles, so it meets few scenes: bounds
// and extents stay in registers and go to the scene's accumulators once per
// block and scene. (As separate kernels, every warp of the bounds pass sent ten
// atomics to the same few words: 122 us of a 700K-shape pass of 16 scenes, and
// the gather, lookup and box passes read and wrote the shapes three times.)
struct Bounds {
	float3 mn, mx, ext;
	uint32_t e, cnt;
	__device__ __forceinline__ void clear() {
		mn = f3(INFINITY, INFINITY, INFINITY);
		mx = f3(-INFINITY, -INFINITY, -INFINITY);
		ext = f3(0.f, 0.f, 0.f);
		e = cnt = 0;
	}
	__device__ __forceinline__ void add(float3 lo, float3 hi) {
		if (!finite3(lo) || !finite3(hi)) e |= kErrNonFinite;
		if (lo.x > hi.x || lo.y > hi.y || lo.z > hi.z) e |= kErrInverted;
		mn = f3(fminf(mn.x, lo.x), fminf(mn.y, lo.y), fminf(mn.z, lo.z));
		mx = f3(fmaxf(mx.x, hi.x), fmaxf(mx.y, hi.y), fmaxf(mx.z, hi.z));
		ext = ext + (hi - lo);
		cnt++;
	}
};
// The warp's bounds of scene s into its accumulators (all lanes).
__device__ __forceinline__ void warp_flush(const Bounds &b, SceneStats *sst, uint32_t s, uint32_t *err) {
	const float mn[3] = {b.mn.x, b.mn.y, b.mn.z}, mx[3] = {b.mx.x, b.mx.y, b.mx.z};
	const float ext[3] = {b.ext.x, b.ext.y, b.ext.z};
	const uint32_t cnt = __reduce_add_sync(0xffffffffu, b.cnt), e = __reduce_or_sync(0xffffffffu, b.e);
	const uint32_t lane = threadIdx.x & 31;
	if (!cnt) return;
	SceneStats &t = sst[s];
#pragma unroll
	for (int d = 0; d < 3; d++) {
		const uint32_t lo = __reduce_min_sync(0xffffffffu, b.cnt ? f2ord(mn[d]) : 0xffffffffu);
		const uint32_t hi = __reduce_max_sync(0xffffffffu, b.cnt ? f2ord(mx[d]) : 0u);
		const float sum = warp_sum(ext[d]);
		if (lane == 0) {
			atomicMax(&t.bmin_inv[d], ~lo);
			atomicMax(&t.bmax[d], hi);
			atomicAdd(&t.ext_sum[d], (double)sum);
		}
	}
	if (lane == 0) {
		atomicAdd(&t.count, (unsigned long long)cnt);
		if (e) {
			atomicOr(&t.err, e);
			atomicOr(err, e);
		}
	}
}
// The largest s in [lo, S) with off[s] <= i (off nondecreasing, off[lo] <= i).
__device__ __forceinline__ uint32_t scene_at(const unsigned long long *off, uint32_t lo, uint32_t S, uint64_t i) {
	uint32_t hi = S;
	while (hi - lo > 1) {
		const uint32_t mid = (lo + hi) >> 1;
		if (__ldg(off + mid) <= i) lo = mid;
		else hi = mid;
	}
	return lo;
}

template <bool kGather>
__global__ void __launch_bounds__(kNT) k_batch_front(uint64_t n, uint64_t nb, uint32_t S,
                                                      const unsigned long long *__restrict__ shape_off,
                                                      const unsigned long long *__restrict__ body_off, SceneSrc all,
                                                      const SceneSrc *__restrict__ src, SceneDst dst,
                                                      uint32_t *__restrict__ scene_of, uint32_t *__restrict__ gid,
                                                      float *__restrict__ aabb, DevStats *stats, SceneStats *sst,
                                                      PlanArgs pa, Plan *plans, uint32_t *__restrict__ cell_base,
                                                      ZeroList zero) {
	pdl_begin();
	zero_ranges(zero);
	const uint64_t step = (uint64_t)gridDim.x * kNT;
	if constexpr (kGather) {
		for (uint64_t i = (uint64_t)blockIdx.x * kNT + threadIdx.x; i < nb; i += step) {
			const uint32_t s = scene_at(body_off, 0, S, i);
			const uint64_t j = i - __ldg(body_off + s);
			const SceneSrc &c = src[s];
#pragma unroll
			for (int d = 0; d < 3; d++) dst.pos[3 * i + d] = c.pos[3 * j + d];
			reinterpret_cast<float4 *>(dst.rot)[i] = reinterpret_cast<const float4 *>(c.rot)[j];
			dst.active[i] = c.active[j];
		}
	}
	const uint64_t tiles = (n + kNT - 1) / kNT, per = (tiles + gridDim.x - 1) / gridDim.x;
	const uint64_t t0 = min(tiles, blockIdx.x * per), t1 = min(tiles, t0 + per);
	Bounds acc;
	acc.clear();
	uint32_t hint = t0 < t1 ? scene_at(shape_off, 0, S, t0 * kNT) : 0u;  // scene of the tile's first shape
	for (uint64_t t = t0; t < t1; t++) {
		const uint64_t i = t * kNT + threadIdx.x, last = min(n, (t + 1) * kNT) - 1;
		const bool have = i < n, one = __ldg(shape_off + hint + 1) > last;  // the tile lies in scene `hint`
		uint32_t s = hint;
		if (!one && have) s = scene_at(shape_off, hint, S, i);
		float3 mn = f3(0.f, 0.f, 0.f), mx = mn;
		if (have) {
			const uint64_t s0 = __ldg(shape_off + s), b0 = __ldg(body_off + s), nb_s = __ldg(body_off + s + 1) - b0;
			SceneSrc c;
			if constexpr (kGather) {
				c = src[s];
			} else {
				c = {all.T + s0, all.A + 3 * s0, all.B + 3 * s0, all.C + 3 * s0, all.R + 4 * s0, all.ID + s0,
				     all.pos + 3 * b0, all.rot + 4 * b0, nullptr};
			}
			const uint64_t j = i - s0;
			const uint32_t id = __ldg(c.ID + j);
			scene_of[i] = s;
			gid[i] = id < nb_s ? (uint32_t)(b0 + id) : 0xffffffffu;  // shape_aabb reports the others
			if constexpr (kGather) {
				const int type = __ldg(c.T + j);
				dst.T[i] = type;
				dst.ID[i] = id;
				reinterpret_cast<float4 *>(dst.R)[i] = ld4(c.R, j);
#pragma unroll
				for (int d = 0; d < 3; d++) {
					dst.A[3 * i + d] = __ldg(c.A + 3 * j + d);
					dst.B[3 * i + d] = __ldg(c.B + 3 * j + d);
				}
				if (type == CONE || type == TRIANGLEMESH)  // the only ones whose C is read
#pragma unroll
					for (int d = 0; d < 3; d++) dst.C[3 * i + d] = __ldg(c.C + 3 * j + d);
			}
			float *o = aabb + 3 * i, *o2 = aabb + 3 * (i + n);
			if (shape_aabb(j, c.T, c.A, c.B, c.C, c.R, c.ID, nb_s, c.pos, c.rot, mn, mx, &stats->err)) {
				o[0] = mn.x; o[1] = mn.y; o[2] = mn.z;
				o2[0] = mx.x; o2[1] = mx.y; o2[2] = mx.z;
			} else {  // skipped shape: the broadphase sees the caller's old values
				mn = f3(o[0], o[1], o[2]);
				mx = f3(o2[0], o2[1], o2[2]);
			}
		}
		if (one) {
			if (have) acc.add(mn, mx);
			continue;
		}
		// the run of the scene up to here ends; this tile's shapes scene by scene
		warp_flush(acc, sst, hint, &stats->err);
		acc.clear();
		uint32_t todo = __ballot_sync(0xffffffffu, have);
		while (todo) {
			const uint32_t sw = __shfl_sync(0xffffffffu, s, __ffs(todo) - 1);
			Bounds b;
			b.clear();
			if (have && s == sw) b.add(mn, mx);
			warp_flush(b, sst, sw, &stats->err);
			todo &= ~__ballot_sync(0xffffffffu, have && s == sw);
		}
		hint = last + 1 < n ? scene_at(shape_off, hint, S, last + 1) : hint;
	}
	warp_flush(acc, sst, hint, &stats->err);
	__shared__ bool s_last;
	__shared__ uint32_t scan[40];
	__threadfence();
	__syncthreads();
	if (threadIdx.x == 0) s_last = atomicAdd(&stats->blocks_done, 1u) == gridDim.x - 1;
	__syncthreads();
	if (!s_last) return;
	__threadfence();
	uint64_t run = 0;
	for (uint32_t q = 0; q < S; q += kNT) {
		const uint32_t s = q + threadIdx.x;
		Plan p;
		memset(&p, 0, sizeof(p));
		if (s < S) {
			const uint64_t n_s = shape_off[s + 1] - shape_off[s];
			if (n_s) {
				const SceneStats &t = sst[s];
				const unsigned long long cnt = __ldcg(&t.count);
				uint32_t lo[3], hi[3];
				double mean[3];
				for (int d = 0; d < 3; d++) {
					lo[d] = __ldcg(&t.bmin_inv[d]);
					hi[d] = __ldcg(&t.bmax[d]);
					mean[d] = __ldcg(&t.ext_sum[d]) / (double)(cnt ? cnt : 1);
				}
				GridParams g = pa.gp;
				g.g_max = batch_scene_cells(n_s);
				p = make_plan(lo, hi, __ldcg(&t.err), mean, g, pa.gx, pa.gy, pa.gz, n_s);
				if (!p.valid) p.G = 0;
			}
			plans[s] = p;
		}
		uint32_t total;
		const uint32_t before = block_excl_scan<uint32_t, kNT>(p.G, scan, &total);
		if (s < S) cell_base[s] = (uint32_t)(run + before);
		run += total;
	}
	if (threadIdx.x == 0) {
		cell_base[S] = (uint32_t)run;
		stats->cells = run;
	}
}

template <class K>
int resident_blocks(K kernel) {
	int b = 0;
	if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kernel, kNT, 0) != cudaSuccess || b < 1) b = 1;
	return b;
}
}  // namespace

void launch_aabb(uint64_t n, const int32_t *T, const float *A, const float *B, const float *C, const float *R,
                 const uint32_t *ID, uint64_t nb, const float *pos, const float *rot, float *aabb, DevStats *stats,
                 uint32_t *err, const GridParams &gp, const int grid[3], cudaStream_t s, const ZeroList &zero) {
	if (n == 0) return;
	// persistent grid: as many blocks as are resident at once
	static const int per_sm[2] = {resident_blocks(k_aabb<false>), resident_blocks(k_aabb<true>)};
	const unsigned blocks =
	    (unsigned)std::min<uint64_t>((n + kNT - 1) / kNT, (uint64_t)kNumSMs * per_sm[stats ? 1 : 0]);
	PlanArgs pa;
	pa.gp = gp;
	pa.gx = grid ? grid[0] : 1;
	pa.gy = grid ? grid[1] : 1;
	pa.gz = grid ? grid[2] : 1;
	pa.n = n;
	if (stats)
		launch_pdl(k_aabb<true>, dim3(blocks), dim3(kNT), 0, s, n, T, A, B, C, R, ID, nb, pos, rot, aabb, stats, err, pa, zero);
	else
		launch_pdl(k_aabb<false>, dim3(blocks), dim3(kNT), 0, s, n, T, A, B, C, R, ID, nb, pos, rot, aabb, nullptr, err, pa, zero);
}

void launch_batch_front(uint64_t n, uint64_t nb, uint32_t S, const unsigned long long *shape_off,
                        const unsigned long long *body_off, const SceneSrc &all, const SceneSrc *src, const SceneDst &dst,
                        uint32_t *scene_of, uint32_t *gid, float *aabb, DevStats *stats, SceneStats *sst,
                        const GridParams &gp, const int grid[3], Plan *plans, uint32_t *cell_base, cudaStream_t s,
                        const ZeroList &zero) {
	if (n == 0) return;
	static const int per_sm[2] = {resident_blocks(k_batch_front<false>), resident_blocks(k_batch_front<true>)};
	const unsigned blocks = (unsigned)std::min<uint64_t>((n + kNT - 1) / kNT, (uint64_t)kNumSMs * per_sm[src ? 1 : 0]);
	PlanArgs pa;
	pa.gp = gp;
	pa.gx = grid[0];
	pa.gy = grid[1];
	pa.gz = grid[2];
	pa.n = n;
	launch_pdl(src ? k_batch_front<true> : k_batch_front<false>, dim3(blocks), dim3(kNT), 0, s, n, nb, S, shape_off, body_off,
	           all, src, dst, scene_of, gid, aabb, stats, sst, pa, plans, cell_base, zero);
}

}  // namespace cc
