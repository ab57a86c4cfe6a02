// Uniform-grid broadphase (the reference's Broadphase::detectPossibleCollisions,
// src/broadphase/Broadphase.cu:344-545) as sm_100a kernels.
//
// Pair path, scenes without crowded cells (the rule is cc_ctx::chain_state):
//   k_bounds        scene bounds + extent sums + validation     (Broadphase.cu:368-376)
//   k_link          in-place shift by fabs(min) (:379-386), one 32-byte entry per
//                   (cell, body) linked into its cell's chain
//   k_walk          closed AABB overlap (:237) of every entry with the entries
//                   behind it in the chain, emitted from the home cell (below)
// Pair path, crowded scenes:
//   k_bounds, then k_count  in-place shift by fabs(min) (:379-386) + per-cell
//                   counts on the search grid
//   scan            cell offsets (decoupled look-back)
//   k_scatter       cell-ordered (AABB, body) entries
//   k_pair_test     (cells of many entries: k_dense_order, k_dense_test)
//                   closed AABB overlap (:237) of every entry with the later
//                   entries of its cell; a pair is emitted only from its home
//                   cell (the cell holding the larger of the two min corners on
//                   every axis, a point of both boxes and so of both cell
//                   ranges), so each overlapping pair appears exactly once and no
//                   unique pass is needed (replaces :484-533)
// Both:
//   scan            per-owner offsets (owner = smaller index)
//   k_owner_scatter bucket pairs by owner; k_segsort sorts each bucket
//                   -> the sorted, duplicate-free int64 list of :522-535
//
// Two overlapping boxes always share a cell of ANY grid built from a monotone
// cell map (float subtraction, multiplication and truncation are monotone), and
// the reference re-tests every candidate on the shifted boxes, so its pair list
// is exactly {(a,b): a<b, closed overlap of the shifted boxes}: the search grid
// here is chosen for speed, independent of the caller's bins per axis.
//
// Bin-list path (on request): the reference's own sorted (bin, body) list on
// the caller's grid, with its HashMin truncation and unclamped linear index
// (:125-200, :428-480), for parity checks.
//
// Compiled with -fmad=false (the shift and the bin scale must round exactly as
// the reference's host build does).
#include <algorithm>
#include <atomic>
#include <climits>
#include <cstdlib>

#include "cc_common.cuh"
#include "cc_internal.h"
#include "cc_math.cuh"
#include "cc_stats.cuh"

namespace cc {

namespace {
constexpr int kNT = 256;

__device__ __forceinline__ float3 ld3p(const float *p, uint64_t i) { return f3(p[3 * i], p[3 * i + 1], p[3 * i + 2]); }

// A block's kNT boxes, staged through shared memory with 16-byte loads: the
// min corners of boxes [i0, i0+kNT) are 3*kNT contiguous floats at aabb+3*i0
// and the max corners the same at aabb+3*(n+i0). stage[0..3kNT) = mins,
// stage[3kNT..6kNT) = maxs. Vector accesses are used when both runs are
// 16-byte aligned and complete; otherwise scalar ones.
__device__ __forceinline__ bool tile_vec_ok(const float *aabb, uint64_t n, uint64_t i0) {
	return i0 + kNT <= n && ((reinterpret_cast<uintptr_t>(aabb + 3 * i0) & 15) == 0) &&
	       ((reinterpret_cast<uintptr_t>(aabb + 3 * (n + i0)) & 15) == 0);
}
// The same for 32-byte vector accesses.
__device__ __forceinline__ bool tile_vec_ok32(const float *aabb, uint64_t n, uint64_t i0) {
	return i0 + kNT <= n && ((reinterpret_cast<uintptr_t>(aabb + 3 * i0) & 31) == 0) &&
	       ((reinterpret_cast<uintptr_t>(aabb + 3 * (n + i0)) & 31) == 0);
}
__device__ __forceinline__ void load_tile_aabb(const float *__restrict__ aabb, uint64_t n, uint64_t i0, float *stage) {
	if (tile_vec_ok(aabb, n, i0)) {
		const float4 *lo = reinterpret_cast<const float4 *>(aabb + 3 * i0);
		const float4 *hi = reinterpret_cast<const float4 *>(aabb + 3 * (n + i0));
		float4 *st = reinterpret_cast<float4 *>(stage);
		for (int k = threadIdx.x; k < 3 * kNT / 4; k += kNT) {
			st[k] = lo[k];
			st[3 * kNT / 4 + k] = hi[k];
		}
	} else {
		const uint64_t m = i0 < n ? min((uint64_t)kNT, n - i0) : 0;
		for (int k = threadIdx.x; k < 3 * (int)m; k += kNT) {
			stage[k] = aabb[3 * i0 + k];
			stage[3 * kNT + k] = aabb[3 * (n + i0) + k];
		}
	}
}
__device__ __forceinline__ void store_tile_aabb(float *__restrict__ aabb, uint64_t n, uint64_t i0, const float *stage) {
	if (tile_vec_ok(aabb, n, i0)) {
		float4 *lo = reinterpret_cast<float4 *>(aabb + 3 * i0);
		float4 *hi = reinterpret_cast<float4 *>(aabb + 3 * (n + i0));
		const float4 *st = reinterpret_cast<const float4 *>(stage);
		for (int k = threadIdx.x; k < 3 * kNT / 4; k += kNT) {
			lo[k] = st[k];
			hi[k] = st[3 * kNT / 4 + k];
		}
	} else {
		const uint64_t m = i0 < n ? min((uint64_t)kNT, n - i0) : 0;
		for (int k = threadIdx.x; k < 3 * (int)m; k += kNT) {
			aabb[3 * i0 + k] = stage[k];
			aabb[3 * (n + i0) + k] = stage[3 * kNT + k];
		}
	}
}

// Search-grid cell of a shifted coordinate: monotone in v.
__device__ __forceinline__ int cell_of(float v, float lo, float inv, int dim) {
	float t = (v - lo) * inv;
	int c = (int)fminf(fmaxf(t, 0.f), (float)(dim - 1));
	return c;
}
struct CellRange {
	int c0[3], c1[3];
};
__device__ __forceinline__ CellRange cell_range(const Plan &p, float3 mn, float3 mx) {
	CellRange r;
	r.c0[0] = cell_of(mn.x, p.lo[0], p.inv[0], p.dim[0]);
	r.c0[1] = cell_of(mn.y, p.lo[1], p.inv[1], p.dim[1]);
	r.c0[2] = cell_of(mn.z, p.lo[2], p.inv[2], p.dim[2]);
	r.c1[0] = cell_of(mx.x, p.lo[0], p.inv[0], p.dim[0]);
	r.c1[1] = cell_of(mx.y, p.lo[1], p.inv[1], p.dim[1]);
	r.c1[2] = cell_of(mx.z, p.lo[2], p.inv[2], p.dim[2]);
	return r;
}
__device__ __forceinline__ uint32_t pack_cell(int x, int y, int z) {
	return (uint32_t)x | ((uint32_t)y << 10) | ((uint32_t)z << 20);
}
__global__ void __launch_bounds__(kNT) k_bounds(uint64_t n, const float *__restrict__ aabb, DevStats *stats,
                                                 PlanArgs pa, ZeroList zero) {
	zero_ranges(zero);
	const uint64_t i = (uint64_t)blockIdx.x * kNT + threadIdx.x;
	float3 mn = f3(0.f, 0.f, 0.f), mx = mn;
	const bool have = i < n;
	if (have) {
		mn = ld3p(aabb, i);
		mx = ld3p(aabb, i + n);
	}
	accumulate_stats_one<kNT>(mn, mx, have, stats, pa);
}

// The plan again for another search grid (the boxes may be shifted already).
__global__ void k_replan(DevStats *stats, PlanArgs pa) {
	pa.gx = stats->plan.grid[0];
	pa.gy = stats->plan.grid[1];
	pa.gz = stats->plan.grid[2];
	store_plan(stats, pa);
}

// The plan a shape is searched with: the block's staged plan (one scene) or
// its scene's plan (batch).
template <bool kBatch>
__device__ __forceinline__ const Plan &plan_of(const Plan &sp, const SceneMap &sm, uint64_t shape, uint32_t &base) {
	if constexpr (kBatch) {
		const uint32_t s = __ldg(sm.scene_of + shape);
		base = __ldg(sm.cell_base + s);
		return sm.plans[s];
	} else {
		base = 0;
		return sp;
	}
}
__device__ __forceinline__ uint32_t cell_index(const Plan &p, uint32_t base, int x, int y, int z) {
	return base + (uint32_t)x + (uint32_t)p.dim[0] * ((uint32_t)y + (uint32_t)p.dim[1] * z);
}

// The plan of the block's shapes [i0, i0 + kNT) into shared memory (sp, base),
// with a barrier. A batch's tile may span scenes: returns false then, and each
// shape takes its own (plan_of).
template <bool kBatch>
__device__ __forceinline__ bool tile_plan(uint64_t n, uint64_t i0, const DevStats *stats, const SceneMap &sm, Plan &sp,
                                          uint32_t &base) {
	const Plan *from = &stats->plan;
	bool one = true;
	base = 0;
	if constexpr (kBatch) {
		const uint32_t s0 = __ldg(sm.scene_of + i0), s1 = __ldg(sm.scene_of + min(i0 + kNT, n) - 1);
		one = s0 == s1;
		from = sm.plans + s0;
		base = __ldg(sm.cell_base + s0);
	}
	if (one && threadIdx.x < sizeof(Plan) / 4)
		reinterpret_cast<uint32_t *>(&sp)[threadIdx.x] = reinterpret_cast<const uint32_t *>(from)[threadIdx.x];
	__syncthreads();
	return one;
}

// The block's boxes [i0, i0 + kNT) shifted in place by fabs(min) (:382-386), in
// `stage` on return (after a barrier). one: they share the plan sp. shift 0:
// they are shifted already.
template <bool kBatch>
__device__ __forceinline__ void load_shifted_tile(uint64_t n, float *__restrict__ aabb, uint64_t i0, const Plan &sp,
                                                  const SceneMap &sm, float *stage, int shift, bool one) {
	if (!shift || (one && !sp.valid)) {
		load_tile_aabb(aabb, n, i0, stage);
		__syncthreads();
		return;
	}
	if (one && tile_vec_ok32(aabb, n, i0)) {
		// in-place shift by fabs(min) (:382-386) on 32-byte vectors, in
		// registers on the way to shared memory: thread k < 96 takes floats
		// [8k, 8k + 8) of the min-corner run, thread 96 + k those of the
		// max-corner run; float 8k + j is component (2k + j) mod 3
		const int t = threadIdx.x;
		if (t < 3 * kNT / 4) {
			const int k = t < 3 * kNT / 8 ? t : t - 3 * kNT / 8;
			float *run = t < 3 * kNT / 8 ? aabb + 3 * i0 : aabb + 3 * (n + i0);
			const int r = (2 * k) % 3;
			const float o0 = sp.origin[r], o1 = sp.origin[r == 2 ? 0 : r + 1], o2 = sp.origin[r == 0 ? 2 : r - 1];
			float4 a, b;
			ld_global_v8(run + 8 * k, a, b);
			a = make_float4(a.x + o0, a.y + o1, a.z + o2, a.w + o0);
			b = make_float4(b.x + o1, b.y + o2, b.z + o0, b.w + o1);
			st_global_v8(run + 8 * k, a, b);
			float4 *st = reinterpret_cast<float4 *>(stage) + (t < 3 * kNT / 8 ? 0 : 3 * kNT / 4);
			st[2 * k] = a;
			st[2 * k + 1] = b;
		}
		__syncthreads();
	} else {
		load_tile_aabb(aabb, n, i0, stage);
		__syncthreads();
		// element by element
		if (kBatch && !one) {
			for (int k = threadIdx.x; k < 6 * kNT; k += kNT) {
				const uint64_t shape = i0 + (uint64_t)((k % (3 * kNT)) / 3);
				if (shape < n) {
					const Plan &p = sm.plans[__ldg(sm.scene_of + shape)];
					if (p.valid) stage[k] = stage[k] + p.origin[k % 3];
				}
			}
		} else {
			for (int k = threadIdx.x; k < 6 * kNT; k += kNT) stage[k] = stage[k] + sp.origin[k % 3];
		}
		__syncthreads();
		store_tile_aabb(aabb, n, i0, stage);
	}
}

template <bool kBatch>
__global__ void __launch_bounds__(kNT) k_count(uint64_t n, float *__restrict__ aabb, DevStats *stats,
                                                uint32_t *__restrict__ cell_count, uint32_t *__restrict__ owner_count,
                                                SceneMap sm, int oshift, uint32_t *__restrict__ owner_cursor, int shift) {
	pdl_begin();
	__shared__ Plan sp;
	__shared__ __align__(16) float stage[6 * kNT];  // read and written as float4
	const uint64_t i0 = (uint64_t)blockIdx.x * kNT;
	uint32_t base0;
	const bool one = tile_plan<kBatch>(n, i0, stats, sm, sp, base0);
	if (!kBatch && !sp.valid) return;  // invalid input: nothing is modified
	load_shifted_tile<kBatch>(n, aabb, i0, sp, sm, stage, shift, one);
	const uint64_t i = i0 + threadIdx.x;
	if (i >= n) return;
	const float3 mn = f3(stage[3 * threadIdx.x], stage[3 * threadIdx.x + 1], stage[3 * threadIdx.x + 2]);
	const float *hs = stage + 3 * kNT;
	const float3 mx = f3(hs[3 * threadIdx.x], hs[3 * threadIdx.x + 1], hs[3 * threadIdx.x + 2]);
	if ((i & ((1ull << oshift) - 1)) == 0) {  // the first body of its owner bucket
		owner_count[i >> oshift] = 0u;
		if (owner_cursor) owner_cursor[i >> oshift] = 0u;
	}
	uint32_t base = base0;
	const Plan &p = one ? sp : plan_of<kBatch>(sp, sm, i, base);
	if (kBatch && !p.valid) return;
	const CellRange r = cell_range(p, mn, mx);
	if ((uint64_t)(r.c1[0] - r.c0[0] + 1) * (r.c1[1] - r.c0[1] + 1) * (r.c1[2] - r.c0[2] + 1) > kWideCells) stats->wide = 1u;
	for (int z = r.c0[2]; z <= r.c1[2]; z++)
		for (int y = r.c0[1]; y <= r.c1[1]; y++)
			for (int x = r.c0[0]; x <= r.c1[0]; x++) atomicAdd(&cell_count[cell_index(p, base, x, y, z)], 1u);
}
// Cell-ordered entries: one thread per body, a cursor atomic per covered cell.
template <bool kBatch>
__global__ void __launch_bounds__(kNT) k_scatter(uint64_t n, const float *__restrict__ aabb, const DevStats *stats,
                                                  const uint32_t *__restrict__ cell_start,
                                                  uint32_t *__restrict__ cursor, float4 *__restrict__ entries,
                                                  uint64_t cap, uint32_t *err, SceneMap sm,
                                                  unsigned long long *__restrict__ cs) {
	pdl_begin();
	__shared__ Plan sp;
	__shared__ __align__(16) float stage[6 * kNT];  // read and written as float4
	if (threadIdx.x < sizeof(Plan) / 4)
		reinterpret_cast<uint32_t *>(&sp)[threadIdx.x] = reinterpret_cast<const uint32_t *>(&stats->plan)[threadIdx.x];
	const uint64_t i0 = (uint64_t)blockIdx.x * kNT;
	load_tile_aabb(aabb, n, i0, stage);
	__syncthreads();
	const uint64_t i = i0 + threadIdx.x;
	if ((!kBatch && !sp.valid) || i >= n) return;
	const float3 mn = f3(stage[3 * threadIdx.x], stage[3 * threadIdx.x + 1], stage[3 * threadIdx.x + 2]);
	const float *hs = stage + 3 * kNT;
	const float3 mx = f3(hs[3 * threadIdx.x], hs[3 * threadIdx.x + 1], hs[3 * threadIdx.x + 2]);
	uint32_t base;
	const Plan &p = plan_of<kBatch>(sp, sm, i, base);
	if (kBatch && !p.valid) return;
	const CellRange r = cell_range(p, mn, mx);
	bool over = false;
	const float4 elo = make_float4(mn.x, mn.y, mn.z, __uint_as_float((uint32_t)i));
	const auto put = [&](uint64_t slot, uint32_t packed) {
		if (slot < cap) {  // one 32-byte store (entries are 32-byte aligned)
			st_global_v8(reinterpret_cast<float *>(entries + 2 * slot), elo,
			             make_float4(mx.x, mx.y, mx.z, __uint_as_float(packed)));
		} else {
			over = true;
		}
	};
	// a slot in cell c: start + cursor, from one packed 64-bit atomic when the
	// scan wrote the packed words, else a start load and a cursor atomic
	const auto take = [&](uint32_t c) -> uint64_t {
		if (cs) {
			const unsigned long long w = atomicAdd(cs + c, 1ull);
			return (w >> 32) + (w & 0xffffffffull);
		}
		return (uint64_t)cell_start[c] + atomicAdd(&cursor[c], 1u);
	};
	const int nx = r.c1[0] - r.c0[0] + 1, ny = r.c1[1] - r.c0[1] + 1, nz = r.c1[2] - r.c0[2] + 1;
	if (nx <= 2 && ny <= 2 && nz <= 2) {
		// up to 2x2x2 cells (nearly every box): the offset loads and cursor
		// atomics of all its cells are issued before any result is used, so a
		// thread waits one memory round trip instead of one per cell
		uint32_t cell[8], packed[8], slot[8];
#pragma unroll
		for (int q = 0; q < 8; q++) {
			const int x = r.c0[0] + (q & 1), y = r.c0[1] + ((q >> 1) & 1), z = r.c0[2] + (q >> 2);
			cell[q] = cell_index(p, base, x, y, z);
			packed[q] = pack_cell(x, y, z);
		}
#pragma unroll
		for (int q = 0; q < 8; q++)
			if ((q & 1) < nx && ((q >> 1) & 1) < ny && (q >> 2) < nz)
				slot[q] = (uint32_t)take(cell[q]);
#pragma unroll
		for (int q = 0; q < 8; q++)
			if ((q & 1) < nx && ((q >> 1) & 1) < ny && (q >> 2) < nz) put(slot[q], packed[q]);
	} else {
		for (int z = r.c0[2]; z <= r.c1[2]; z++)
			for (int y = r.c0[1]; y <= r.c1[1]; y++)
				for (int x = r.c0[0]; x <= r.c1[0]; x++) {
					const uint32_t c = cell_index(p, base, x, y, z);
					put(take(c), pack_cell(x, y, z));
				}
	}
	if (over) atomicOr(err, (uint32_t)kErrCapacity);
}

// Each entry is tested against the later entries of its cell; a warp takes
// 32 entries and deals their tests out evenly over its lanes (so a warp's
// rounds follow the SUM of its entries' partner counts, not 32 x the largest). A warp's 32 entries and the kWin - 32 that follow them are
// staged in shared memory with coalesced 16-byte loads (cells hold a handful
// of entries, so the inner loop almost never leaves the window); loops are
// warp-uniform so the emission can be warp-aggregated: found pairs collect in
// a per-warp shared buffer that is flushed with one counter atomic per
// kOutBuf - 31 pairs or more (dense scenes emit billions of pairs).
constexpr int kWinDefault = 96;  // window (entries per warp staged in shared memory); tunable: 64, 96, 128
constexpr int kOutBuf = 128;

__device__ __forceinline__ void flush_pairs(unsigned long long *buf, uint32_t cnt, uint32_t lane,
                                            unsigned long long *pair_counter, unsigned long long *pairs,
                                            uint64_t pair_cap) {
	unsigned long long start = 0;
	if (lane == 0) start = atomicAdd(pair_counter, (unsigned long long)cnt);
	start = __shfl_sync(0xffffffffu, start, 0);
	for (uint32_t k = lane; k < cnt; k += 32) {
		const unsigned long long pos = start + k;
		if (pos < pair_cap) pairs[pos] = buf[k];
	}
	__syncwarp();
}

template <bool kBatch, int kWin>
__global__ void __launch_bounds__(kNT, 5) k_pair_test(const DevStats *stats, const uint32_t *__restrict__ cell_start,
                                                    const float4 *__restrict__ entries,
                                                    uint64_t entry_cap, uint32_t *__restrict__ owner_count,
                                                    unsigned long long *__restrict__ pairs, uint64_t pair_cap,
                                                    unsigned long long *pair_counter, SceneMap sm, DenseItem *dense,
                                                    uint64_t dense_cap, unsigned long long *dense_count,
                                                    unsigned long long *mask_words,
                                                    uint32_t *err, uint32_t dense_cell, int oshift) {
	pdl_begin();
	__shared__ Plan sp;
	__shared__ float4 win_all[kNT / 32][2 * kWin];
	__shared__ unsigned long long out_all[kNT / 32][kOutBuf];
	__shared__ uint32_t owned_s[kNT];  // pairs owned by each lane's entry in the current window
	if (threadIdx.x < sizeof(Plan) / 4)
		reinterpret_cast<uint32_t *>(&sp)[threadIdx.x] = reinterpret_cast<const uint32_t *>(&stats->plan)[threadIdx.x];
	__syncthreads();
	if (!kBatch && !sp.valid) return;
	float4 *win = win_all[threadIdx.x >> 5];
	unsigned long long *obuf = out_all[threadIdx.x >> 5];
	uint32_t ocnt = 0;  // pairs in obuf (warp-uniform)
	const uint64_t E = min((uint64_t)stats->entries, entry_cap);
	const uint32_t lane = threadIdx.x & 31;
	const uint32_t lt = (1u << lane) - 1u;
	const uint64_t warps = (uint64_t)gridDim.x * (kNT / 32);
	for (uint64_t base = ((uint64_t)blockIdx.x * (kNT / 32) + (threadIdx.x >> 5)) * 32; base < E; base += warps * 32) {
		// stage entries [base, base + kWin) of this warp
		const uint32_t nwin = (uint32_t)min((uint64_t)kWin, E - base);
		__syncwarp();
		// asynchronous 16-byte copies straight into shared memory: all of the
		// window's loads are in flight at once and hold no registers
		for (uint32_t k = lane; k < 2 * nwin; k += 32) cp_async16(win + k, entries + 2 * base + k);
		cp_async_wait_all();
		__syncwarp();
		const uint64_t e = base + lane;
		const bool valid = e < E;
		float4 alo = make_float4(0.f, 0.f, 0.f, 0.f), ahi = alo;
		int my_n = 0;
		int cx = 0, cy = 0, cz = 0;
		const uint32_t ida = valid ? __float_as_uint(win[2 * lane].w) : 0u;
		uint32_t cbase;
		const Plan &pl = plan_of<kBatch>(sp, sm, ida, cbase);
		if (valid) {
			alo = win[2 * lane];
			ahi = win[2 * lane + 1];
			const uint32_t pc = __float_as_uint(ahi.w);
			cx = pc & 1023; cy = (pc >> 10) & 1023; cz = (pc >> 20) & 1023;
			const uint32_t c = cell_index(pl, cbase, cx, cy, cz);
			const uint64_t beg = cell_start[c];
			const uint64_t end = min((uint64_t)cell_start[c + 1], entry_cap);
			my_n = (int)(end > e + 1 ? end - e - 1 : 0);
			if (end - beg > dense_cell) {
				if (dense) {  // left to k_dense_test
					my_n = 0;
					if (e == beg) {
						const uint32_t k = (uint32_t)(end - beg), chunks = (k + kNT - 1) / kNT;
						const unsigned long long at = atomicAdd(dense_count, (unsigned long long)chunks);
						unsigned long long words = 0;
						for (uint32_t q = 0; q < chunks; q++) words += dense_mask_words(k, q * kNT);
						words = atomicAdd(mask_words, words);
						for (uint32_t q = 0; q < chunks; q++) {
							if (at + q < dense_cap) dense[at + q] = DenseItem{c, q * kNT, words};
							else atomicOr(err, (uint32_t)kErrCapacity);
							words += dense_mask_words(k, q * kNT);
						}
					}
				} else if (e == beg) {
					// no dense-cell kernel this call (the last found no dense
					// cell): tested here, and counted so the next call has one
					atomicAdd(dense_count, 1ull);
				}
			}
		}
		float lo0 = pl.lo[0], lo1 = pl.lo[1], lo2 = pl.lo[2];
		float iv0 = pl.inv[0], iv1 = pl.inv[1], iv2 = pl.inv[2];
		int d0 = pl.dim[0], d1 = pl.dim[1], d2 = pl.dim[2];

		// the warp's sum(my_n) tests, dealt out 32 per round: test k belongs to
		// the lane a with pre[a] <= k < pre[a] + my_n[a] (pre: exclusive scan)
		int pre = my_n;
#pragma unroll
		for (int o = 1; o < 32; o <<= 1) {
			const int v = __shfl_up_sync(0xffffffffu, pre, o);
			if ((int)lane >= o) pre += v;
		}
		const int total = __shfl_sync(0xffffffffu, pre, 31);
		pre -= my_n;
		owned_s[threadIdx.x] = 0;
		__syncwarp();
		for (int k0 = 0; k0 < total; k0 += 32) {
			const int k = k0 + (int)lane;
			int a = 0;
#pragma unroll
			for (int step = 16; step > 0; step >>= 1) {
				const int v = __shfl_sync(0xffffffffu, pre, a + step);
				if (v <= k) a += step;
			}
			const int t = k - __shfl_sync(0xffffffffu, pre, a);
			if constexpr (kBatch) {  // entries of one warp may come from different scenes
				lo0 = __shfl_sync(0xffffffffu, pl.lo[0], a);
				lo1 = __shfl_sync(0xffffffffu, pl.lo[1], a);
				lo2 = __shfl_sync(0xffffffffu, pl.lo[2], a);
				iv0 = __shfl_sync(0xffffffffu, pl.inv[0], a);
				iv1 = __shfl_sync(0xffffffffu, pl.inv[1], a);
				iv2 = __shfl_sync(0xffffffffu, pl.inv[2], a);
				d0 = __shfl_sync(0xffffffffu, pl.dim[0], a);
				d1 = __shfl_sync(0xffffffffu, pl.dim[1], a);
				d2 = __shfl_sync(0xffffffffu, pl.dim[2], a);
			}
			bool emit = false;
			unsigned long long key = 0;
			uint32_t other_owner = 0xffffffffu;
			if (k < total) {
				const float4 plo = win[2 * a], phi = win[2 * a + 1];
				const uint32_t pc = __float_as_uint(phi.w);
				const int px = pc & 1023, py = (pc >> 10) & 1023, pz = (pc >> 20) & 1023;
				const uint32_t loc = (uint32_t)a + 1 + (uint32_t)t;  // partner's position in the window
				float4 blo, bhi;
				if (loc < nwin) {
					blo = win[2 * loc];
					bhi = win[2 * loc + 1];
				} else {
					const uint64_t q = base + loc;
					blo = entries[2 * q];
					bhi = entries[2 * q + 1];
				}
				if (plo.x <= bhi.x && blo.x <= phi.x && plo.y <= bhi.y && blo.y <= phi.y && plo.z <= bhi.z &&
				    blo.z <= phi.z) {
					// home cell: the cell holding the larger min corner on every
					// axis (a point of both boxes, so of both cell ranges); few
					// boxes overlap in sparse cells, so it is evaluated per pair
					const bool hx = cell_of(fmaxf(plo.x, blo.x), lo0, iv0, d0) == px;
					const bool hy = cell_of(fmaxf(plo.y, blo.y), lo1, iv1, d1) == py;
					const bool hz = cell_of(fmaxf(plo.z, blo.z), lo2, iv2, d2) == pz;
					if (hx && hy && hz) {
						const uint32_t ia = __float_as_uint(plo.w), idb = __float_as_uint(blo.w);
						const uint32_t lo = min(ia, idb), hi = max(ia, idb);
						key = ((unsigned long long)lo << 32) | hi;
						emit = true;
						if (lo == ia) atomicAdd(&owned_s[(threadIdx.x & ~31u) + a], 1u);
						else other_owner = lo;
					}
				}
			}
			const uint32_t b = __ballot_sync(0xffffffffu, emit);
			if (b) {
				const uint32_t nb = __popc(b);
				if (ocnt + nb > kOutBuf) {
					flush_pairs(obuf, ocnt, lane, pair_counter, pairs, pair_cap);
					ocnt = 0;
				}
				if (emit) {
					obuf[ocnt + __popc(b & lt)] = key;
					if (other_owner != 0xffffffffu) atomicAdd(&owner_count[other_owner >> oshift], 1u);
				}
				ocnt += nb;
				__syncwarp();
			}
		}
		__syncwarp();
		const uint32_t owned = owned_s[threadIdx.x];
		if (owned) atomicAdd(&owner_count[ida >> oshift], owned);
	}
	if (ocnt) flush_pairs(obuf, ocnt, lane, pair_counter, pairs, pair_cap);
}

// ---------------------------------------------------------------- chained search
// For scenes without crowded cells: the entries of a cell form a linked list
// through the entry array instead of a sorted run, which takes the cell counts,
// their scan and the scatter out of the search. A body's first entry is its
// own slot i (written in order); the entries for further cells go to slots from
// n up, taken per block, with their body in extra_body. An entry is one 32-byte
// record: (min.xyz, next), (max.xyz, packed cell), next = 1 + the slot that
// headed the cell's chain before it, 0 at the end.
// Stage times (us), sorted cells (count + scan + scatter + pair test) -> chains
// (link + walk): 16,384 spheres 39 -> 20, 130K mixed shapes 49 -> 24, 1M 109 ->
// 64, a batch of 1.4M shapes 160 -> 97, a heap of 50K (20 entries a cell) 60 ->
// 49. Crowded cells are the other way round (a chain is one lane's serial walk,
// a sorted cell full warps' work), hence kChainLong.
//
// Bound by barriers and the chain heads' atomics (ncu at 1M: 40 % issue, 8 MB of
// sectors each way are the boxes' shift): the first cell's exchange is under way
// while the block collects the further ones as work items, so that lanes with
// one cell (60 % of the boxes) do not wait for those with eight (38 -> 34 us).
template <bool kBatch>
__global__ void __launch_bounds__(kNT) k_link(uint64_t n, float *__restrict__ aabb, DevStats *stats,
                                               uint32_t *__restrict__ head, float4 *__restrict__ entries, uint64_t cap,
                                               uint32_t *__restrict__ extra_body, uint32_t *__restrict__ owner_count,
                                               SceneMap sm, int oshift, uint32_t *__restrict__ owner_cursor, int shift) {
	pdl_begin();
	__shared__ Plan sp;
	__shared__ __align__(16) float stage[6 * kNT];  // read and written as float4
	__shared__ uint32_t s_first[kNT], s_cell[kNT], s_items, s_wide;
	__shared__ uint16_t s_item[7 * kNT];
	__shared__ unsigned long long s_base;
	if (threadIdx.x == 0) s_items = s_wide = 0;
	const uint64_t i0 = (uint64_t)blockIdx.x * kNT;
	uint32_t base0;
	const bool one = tile_plan<kBatch>(n, i0, stats, sm, sp, base0);
	if (!kBatch && !sp.valid) return;  // invalid input: nothing is modified
	load_shifted_tile<kBatch>(n, aabb, i0, sp, sm, stage, shift, one);
	const uint64_t i = i0 + threadIdx.x;
	const bool have = i < n;
	const float3 mn = f3(stage[3 * threadIdx.x], stage[3 * threadIdx.x + 1], stage[3 * threadIdx.x + 2]);
	const float *hs = stage + 3 * kNT;
	const float3 mx = f3(hs[3 * threadIdx.x], hs[3 * threadIdx.x + 1], hs[3 * threadIdx.x + 2]);
	if (have && (i & ((1ull << oshift) - 1)) == 0) {  // the first body of its owner bucket
		owner_count[i >> oshift] = 0u;
		if (owner_cursor) owner_cursor[i >> oshift] = 0u;
	}
	uint32_t base = base0;
	const Plan &p = one ? sp : plan_of<kBatch>(sp, sm, have ? i : n - 1, base);
	CellRange r;
	int nx = 1, ny = 1, nz = 1;
	bool live = have && (!kBatch || p.valid);
	if (live) {
		r = cell_range(p, mn, mx);
		nx = r.c1[0] - r.c0[0] + 1;
		ny = r.c1[1] - r.c0[1] + 1;
		nz = r.c1[2] - r.c0[2] + 1;
		if ((uint64_t)nx * ny * nz > kChainCells) {  // the search is redone on sorted cells
			atomicOr(&stats->err, (uint32_t)kErrLongChain);
			live = false;
		}
	}
	const auto put = [&](uint64_t slot, float3 lo, float3 hi, uint32_t next, uint32_t packed) {
		st_global_v8(reinterpret_cast<float *>(entries + 2 * slot), make_float4(lo.x, lo.y, lo.z, __uint_as_float(next)),
		             make_float4(hi.x, hi.y, hi.z, __uint_as_float(packed)));
	};
	uint32_t next = 0, first = 0, cell = 0;
	if (live) {
		first = pack_cell(r.c0[0], r.c0[1], r.c0[2]);
		cell = cell_index(p, base, r.c0[0], r.c0[1], r.c0[2]);
		if (i < cap) next = atomicExch(head + cell, (uint32_t)i + 1u);
	}
	// the further cells of boxes within 2x2x2 (nearly all) become work items of
	// the block, (thread, cell offset), so that they too are written by full warps
	const bool small = live && nx <= 2 && ny <= 2 && nz <= 2;
	const uint32_t more = live ? (uint32_t)(nx * ny * nz) - 1u : 0u;
	const uint32_t incl = warp_incl_scan(small ? more : 0u);
	uint32_t at = 0;
	if ((threadIdx.x & 31) == 31 && incl) at = atomicAdd(&s_items, incl);
	at = __shfl_sync(0xffffffffu, at, 31) + incl - (small ? more : 0u);
	s_first[threadIdx.x] = first;
	s_cell[threadIdx.x] = cell;
	uint32_t wide = 0;
	if (small) {
		for (int q = 1; q < 8; q++)
			if ((q & 1) < nx && ((q >> 1) & 1) < ny && (q >> 2) < nz) s_item[at++] = (uint16_t)(threadIdx.x | (q << 8));
	} else if (more) {
		wide = atomicAdd(&s_wide, more);
	}
	if (have && i < cap) put(i, mn, mx, next, first);  // not live: an entry in no chain
	__syncthreads();
	const uint32_t items = s_items;
	if (threadIdx.x == 0) s_base = items + s_wide ? n + atomicAdd(&stats->extra, (unsigned long long)items + s_wide) : n;
	__syncthreads();
	const uint64_t slot0 = s_base;
	for (uint32_t k = threadIdx.x; k < items; k += kNT) {
		const uint32_t w = s_item[k], t = w & 255u, dx = (w >> 8) & 1u, dy = (w >> 9) & 1u, dz = w >> 10;
		uint32_t b2;
		const Plan &pt = one ? sp : plan_of<kBatch>(sp, sm, i0 + t, b2);
		const uint64_t slot = slot0 + k;
		if (slot < cap) {
			const uint32_t c = s_cell[t] + dx + (uint32_t)pt.dim[0] * (dy + (uint32_t)pt.dim[1] * dz);
			const uint32_t prev = atomicExch(head + c, (uint32_t)slot + 1u);
			put(slot, f3(stage[3 * t], stage[3 * t + 1], stage[3 * t + 2]), f3(hs[3 * t], hs[3 * t + 1], hs[3 * t + 2]), prev,
			    s_first[t] + (dx | (dy << 10) | (dz << 20)));
			extra_body[slot - n] = (uint32_t)(i0 + t);
		}
	}
	if (more && !small) {
		uint64_t slot = slot0 + items + wide;
		for (int z = r.c0[2]; z <= r.c1[2]; z++)
			for (int y = r.c0[1]; y <= r.c1[1]; y++)
				for (int x = r.c0[0]; x <= r.c1[0]; x++) {
					if (x == r.c0[0] && y == r.c0[1] && z == r.c0[2]) continue;
					if (slot < cap) {
						put(slot, mn, mx, atomicExch(head + cell_index(p, base, x, y, z), (uint32_t)slot + 1u), pack_cell(x, y, z));
						extra_body[slot - n] = (uint32_t)i;
					}
					slot++;
				}
	}
}

// Before the walk on a context that knows nothing of its scenes: does any cell
// hold more than kChainLong entries? (The walk then returns at once.)
__global__ void __launch_bounds__(kNT) k_chain_check(DevStats *stats, uint64_t g_max, const uint32_t *__restrict__ head,
                                                      const float4 *__restrict__ entries, uint64_t cap) {
	pdl_begin();
	const uint64_t G = min(g_max, (uint64_t)stats->cells);
	for (uint64_t c = (uint64_t)blockIdx.x * kNT + threadIdx.x; c < G; c += (uint64_t)gridDim.x * kNT) {
		uint32_t at = head[c], len = 0;
		while (at && at <= cap && len <= kChainLong) {
			at = __float_as_uint(entries[2 * (uint64_t)(at - 1)].w);
			len++;
		}
		if (len > kChainLong) {
			atomicAdd(&stats->dense_items, 1ull);
			atomicOr(&stats->err, (uint32_t)kErrLongChain);
		}
	}
}

// Every entry is tested against the entries behind it in its cell's chain: each
// pair of a cell once, whichever of the two was linked later. Bound by the
// chain's dependent loads (an L2 round trip each; the records of 1M bodies fit
// the L2): the warp's next entries are loaded while the present ones walk (five
// blocks per SM: 30 us at 1M; six, which spill, 32; four 31.5). Pairs are
// emitted as in k_pair_test: from the home cell, through a per-warp buffer.
constexpr uint32_t kChainMost = 4096;
template <bool kBatch>
__global__ void __launch_bounds__(kNT, 5) k_walk(uint64_t n, DevStats *stats, const float4 *__restrict__ entries,
                                                  uint64_t cap, const uint32_t *__restrict__ extra_body,
                                                  uint32_t *__restrict__ owner_count,
                                                  unsigned long long *__restrict__ pairs, uint64_t pair_cap, SceneMap sm,
                                                  int oshift) {
	pdl_begin();
	__shared__ Plan sp;
	__shared__ unsigned long long out_all[kNT / 32][kOutBuf];
	__shared__ uint32_t s_stop;
	if (threadIdx.x < sizeof(Plan) / 4)
		reinterpret_cast<uint32_t *>(&sp)[threadIdx.x] = reinterpret_cast<const uint32_t *>(&stats->plan)[threadIdx.x];
	const uint64_t total = n + stats->extra;
	if (threadIdx.x == 0) s_stop = __ldcg(&stats->err) & kErrLongChain;  // only the check sets it before this kernel's walk
	if (blockIdx.x == 0 && threadIdx.x == 0) stats->entries = total;
	__syncthreads();
	if ((!kBatch && !sp.valid) || s_stop) return;
	unsigned long long *obuf = out_all[threadIdx.x >> 5];
	uint32_t ocnt = 0;  // pairs in obuf (warp-uniform)
	const uint64_t E = min(total, cap);
	const uint32_t lane = threadIdx.x & 31, lt = (1u << lane) - 1u;
	const auto body_of = [&](uint64_t slot) { return slot < n ? (uint32_t)slot : __ldg(extra_body + (slot - n)); };
	const uint64_t warps = (uint64_t)gridDim.x * (kNT / 32);
	const auto load = [&](uint64_t e, float4 &lo, float4 &hi) {
		lo.w = 0.f;  // no entry: nothing follows
		if (e < E) ld_global_v8(reinterpret_cast<const float *>(entries + 2 * e), lo, hi);
	};
	uint64_t e = ((uint64_t)blockIdx.x * (kNT / 32) + (threadIdx.x >> 5)) * 32 + lane;
	float4 nlo = make_float4(0.f, 0.f, 0.f, 0.f), nhi = nlo;
	load(e, nlo, nhi);
	for (; e - lane < E; e += warps * 32) {
		const float4 alo = nlo, ahi = nhi;
		load(e + warps * 32, nlo, nhi);  // the warp's next entries arrive while these walk
		uint32_t next = __float_as_uint(alo.w), hops = 0, owned = 0;
		while (__any_sync(0xffffffffu, next != 0u)) {
			bool emit = false;
			unsigned long long key = 0;
			if (next) {
				const uint64_t at = next - 1u;
				float4 blo, bhi;
				ld_global_v8(reinterpret_cast<const float *>(entries + 2 * at), blo, bhi);
				next = __float_as_uint(blo.w);
				if (++hops >= kChainLong && next) {
					if (hops == kChainLong) atomicAdd(&stats->dense_items, 1ull);
					if (hops >= kChainMost) {
						atomicOr(&stats->err, (uint32_t)kErrLongChain);
						next = 0u;
					}
				}
				if (alo.x <= bhi.x && blo.x <= ahi.x && alo.y <= bhi.y && blo.y <= ahi.y && alo.z <= bhi.z && blo.z <= ahi.z) {
					const uint32_t pc = __float_as_uint(ahi.w), ia = body_of(e);
					uint32_t cbase;
					const Plan &p = plan_of<kBatch>(sp, sm, ia, cbase);
					if (cell_of(fmaxf(alo.x, blo.x), p.lo[0], p.inv[0], p.dim[0]) == (int)(pc & 1023) &&
					    cell_of(fmaxf(alo.y, blo.y), p.lo[1], p.inv[1], p.dim[1]) == (int)((pc >> 10) & 1023) &&
					    cell_of(fmaxf(alo.z, blo.z), p.lo[2], p.inv[2], p.dim[2]) == (int)((pc >> 20) & 1023)) {
						const uint32_t ib = body_of(at);
						const uint32_t lo = min(ia, ib), hi = max(ia, ib);
						key = ((unsigned long long)lo << 32) | hi;
						emit = true;
						if (lo == ia) owned++;
						else atomicAdd(&owner_count[lo >> oshift], 1u);
					}
				}
			}
			const uint32_t b = __ballot_sync(0xffffffffu, emit);
			if (b) {
				const uint32_t nb = __popc(b);
				if (ocnt + nb > kOutBuf) {
					flush_pairs(obuf, ocnt, lane, &stats->pairs, pairs, pair_cap);
					ocnt = 0;
				}
				if (emit) obuf[ocnt + __popc(b & lt)] = key;
				ocnt += nb;
				__syncwarp();
			}
		}
		if (owned) atomicAdd(&owner_count[body_of(e) >> oshift], owned);
	}
	if (ocnt) flush_pairs(obuf, ocnt, lane, &stats->pairs, pairs, pair_cap);
}

// ---------------------------------------------------------------- small scenes
// Up to kAllPairsBodies bodies every box is tested against every later one: a
// search through cells is a chain of dependent loads (a heap of 1,000 bodies: link
// 4 us, walk 14), n^2 / 2 tests of boxes in shared memory are not. Steps
// with cells and with this, us, at 2 pairs a body and at 0.1: 500 bodies 83 and 71, 71
// and 70; 1,000 87 and 71, 71 and 70; 2,000 101 and 88, 72 and 70; 3,000 107 and 97,
// but 71 and 81.
__global__ void __launch_bounds__(kNT) k_shift(uint64_t n, float *__restrict__ aabb, const DevStats *stats,
                                                uint32_t *__restrict__ owner_count, uint32_t *__restrict__ cursor,
                                                uint32_t buckets, int shift) {
	pdl_begin();
	if (!stats->plan.valid) return;  // invalid input: nothing is modified
	const uint64_t k = (uint64_t)blockIdx.x * kNT + threadIdx.x;
	if (k < buckets) {
		owner_count[k] = 0u;
		if (cursor) cursor[k] = 0u;
	}
	if (shift && k < 6 * n) aabb[k] = aabb[k] + stats->plan.origin[k % 3];
}

constexpr int kAllCols = 64;
// Block (x, y): rows [256 x, 256 x + 256), one a thread, against columns
// [64 y, 64 y + 64).
__global__ void __launch_bounds__(kNT) k_all_pairs(uint32_t n, DevStats *stats, const float *__restrict__ aabb,
                                                    uint32_t *__restrict__ owner_count,
                                                    unsigned long long *__restrict__ pairs, uint64_t pair_cap, int oshift) {
	pdl_begin();
	__shared__ float4 lo[kAllCols], hi[kAllCols];
	if (!stats->plan.valid) return;
	if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) stats->entries = n;
	const uint32_t i = blockIdx.x * kNT + threadIdx.x, c0 = blockIdx.y * kAllCols;
	if (c0 + kAllCols <= blockIdx.x * kNT + 1) return;  // no later column
	const float *mx = aabb + 3 * (uint64_t)n;
	if (threadIdx.x < kAllCols) {
		const uint32_t j = c0 + threadIdx.x;
		lo[threadIdx.x] = j < n ? make_float4(aabb[3 * j], aabb[3 * j + 1], aabb[3 * j + 2], 0.f)
		                        : make_float4(INFINITY, INFINITY, INFINITY, 0.f);
		hi[threadIdx.x] = j < n ? make_float4(mx[3 * j], mx[3 * j + 1], mx[3 * j + 2], 0.f)
		                        : make_float4(-INFINITY, -INFINITY, -INFINITY, 0.f);
	}
	float3 a0 = f3(INFINITY, INFINITY, INFINITY), a1 = f3(-INFINITY, -INFINITY, -INFINITY);
	if (i < n) {
		a0 = f3(aabb[3 * i], aabb[3 * i + 1], aabb[3 * i + 2]);
		a1 = f3(mx[3 * i], mx[3 * i + 1], mx[3 * i + 2]);
	}
	__syncthreads();
	uint32_t m[2] = {0u, 0u};
#pragma unroll
	for (int h = 0; h < 2; h++)
#pragma unroll
		for (int q = 0; q < 32; q++) {
			const float4 b0 = lo[32 * h + q], b1 = hi[32 * h + q];
			const bool over = (a0.x <= b1.x) & (b0.x <= a1.x) & (a0.y <= b1.y) & (b0.y <= a1.y) & (a0.z <= b1.z) & (b0.z <= a1.z);
			m[h] |= over ? 1u << q : 0u;
		}
	unsigned long long hits = (unsigned long long)m[1] << 32 | m[0];
	if (i >= c0) hits = i - c0 >= kAllCols - 1 ? 0ull : hits & ~0ull << (i - c0 + 1);  // later columns only
	const uint32_t cnt = __popcll(hits), incl = warp_incl_scan(cnt), lane = threadIdx.x & 31;
	const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
	if (!total) return;
	unsigned long long at = 0;
	if (lane == 31) at = atomicAdd(&stats->pairs, (unsigned long long)total);
	at = __shfl_sync(0xffffffffu, at, 31) + incl - cnt;
	if (cnt) atomicAdd(&owner_count[i >> oshift], cnt);
	for (; hits; hits &= hits - 1, at++)
		if (at < pair_cap) pairs[at] = (unsigned long long)i << 32 | (c0 + (uint32_t)__ffsll((long long)hits) - 1u);
}

// In-place bitonic sort of m (a power of two) keys in shared memory by
// `nt` cooperating threads (thread t of them); sync() separates the steps.
template <class K, class Sync>
__device__ __forceinline__ void bitonic_shared(K *s, int m, int t, int nt, Sync sync) {
	for (int k = 2; k <= m; k <<= 1) {
		for (int j = k >> 1; j > 0; j >>= 1) {
			// compare-exchange q pairs (i, i + j), i with bit j clear: every thread busy
			for (int q = t; q < (m >> 1); q += nt) {
				const int i = ((q & ~(j - 1)) << 1) | (q & (j - 1));
				const int p = i + j;
				const bool up = (i & k) == 0;
				const K x = s[i], y = s[p];
				if ((x > y) == up) {
					s[i] = y;
					s[p] = x;
				}
			}
			sync();
		}
	}
}

// ---------------------------------------------------------------- dense cells
// Cells of more than dense_cell entries are listed as (cell, chunk of 256 rows)
// and tested here, every row against the later entries of its cell:
//   k_dense_order  the entries of a dense cell in ascending body order, so that
//                  a pair's owner is always its row and a row meets its
//                  partners in ascending order;
//   k_dense_test   (kEmit false) counts the pairs of every row, which gives the
//                  owner buckets' sizes;
//   k_dense_test   (kEmit true), once the buckets have their offsets, writes
//                  each row's pairs as one ascending run into its owner's bucket.
// A test is some fifteen instructions (tests of 32 columns become one mask per
// row, by sign bits, kept for the write where there is room), far cheaper than
// an unsorted list of all pairs and its scatter: at 4.2M clustered spheres (246M pairs) the test
// that emitted through warp votes took 9.7 ms and the scatter 3.3.
struct DenseTile {
	float4 lo[kNT], hi[kNT];  // (min, body), (max, not-home bits)
};
// Columns [c0, c0 + kNT) of the cell's entries at s0; those past k fit nothing.
__device__ __forceinline__ void load_columns(DenseTile &t, const float4 *__restrict__ entries, uint64_t s0, uint32_t c0,
                                             uint32_t k) {
	float4 l = make_float4(INFINITY, INFINITY, INFINITY, 0.f), h = make_float4(-INFINITY, -INFINITY, -INFINITY, 0.f);
	if (c0 + threadIdx.x < k) {
		l = entries[2 * (s0 + c0 + threadIdx.x)];
		h = entries[2 * (s0 + c0 + threadIdx.x) + 1];
	}
	t.lo[threadIdx.x] = l;
	t.hi[threadIdx.x] = h;
}
// Bit 31 - q: the row (alo, ahi) and column g + q overlap (closed, :237) and this
// cell is their home cell. All six differences max - min have clear sign bits
// exactly if the boxes overlap (x - x is +0, differences of floats never round
// to zero); an axis is at home if either box's min corner is in this cell, so
// the pair is not at home where both not-home bits are set.
__device__ __forceinline__ uint32_t test_columns(const DenseTile &t, uint32_t g, float4 alo, float4 ahi) {
	const uint32_t na = __float_as_uint(ahi.w);
	uint32_t miss = 0;
#pragma unroll
	for (int q = 0; q < 32; q++) {
		const float4 blo = t.lo[g + q], bhi = t.hi[g + q];
		const uint32_t s = __float_as_uint(bhi.x - alo.x) | __float_as_uint(ahi.x - blo.x) | __float_as_uint(bhi.y - alo.y) |
		                   __float_as_uint(ahi.y - blo.y) | __float_as_uint(bhi.z - alo.z) | __float_as_uint(ahi.z - blo.z) |
		                   (0u - (na & __float_as_uint(bhi.w)));
		miss = __funnelshift_l(s, miss, 1);
	}
	return ~miss;
}

// Entries of the dense cells in ascending body order, the cell code replaced by
// the row's not-home bits (an axis whose min corner lies in a lower cell). A
// cell of up to kOrderSeg entries is one block's bitonic sort of (body, place)
// in shared memory; larger cells rank each entry by counting smaller bodies,
// k / 14 instructions an entry (all cells that way: 1.1 ms at 4.2M spheres).
constexpr uint32_t kOrderSeg = 4096;
template <bool kBatch>
__global__ void __launch_bounds__(kNT) k_dense_order(const DevStats *stats, const uint32_t *__restrict__ cell_start,
                                                      const float4 *__restrict__ entries, uint64_t entry_cap,
                                                      float4 *__restrict__ sorted, uint32_t *__restrict__ sorted_body,
                                                      SceneMap sm, const DenseItem *__restrict__ dense, uint64_t dense_cap) {
	pdl_begin();
	__shared__ Plan sp;
	__shared__ __align__(16) unsigned long long keys[kOrderSeg];
	if (threadIdx.x < sizeof(Plan) / 4)
		reinterpret_cast<uint32_t *>(&sp)[threadIdx.x] = reinterpret_cast<const uint32_t *>(&stats->plan)[threadIdx.x];
	__syncthreads();
	const auto put = [&](uint64_t from, uint64_t to) {
		float4 lo, hi;
		ld_global_v8(reinterpret_cast<const float *>(entries + 2 * from), lo, hi);
		const uint32_t id = __float_as_uint(lo.w), pc = __float_as_uint(hi.w);
		uint32_t cb;
		const Plan &p = plan_of<kBatch>(sp, sm, id, cb);
		const uint32_t not_home = (uint32_t)(cell_of(lo.x, p.lo[0], p.inv[0], p.dim[0]) != (int)(pc & 1023)) |
		                          ((uint32_t)(cell_of(lo.y, p.lo[1], p.inv[1], p.dim[1]) != (int)((pc >> 10) & 1023)) << 1) |
		                          ((uint32_t)(cell_of(lo.z, p.lo[2], p.inv[2], p.dim[2]) != (int)((pc >> 20) & 1023)) << 2);
		hi.w = __uint_as_float(not_home);
		st_global_v8(reinterpret_cast<float *>(sorted + 2 * to), lo, hi);
		sorted_body[to] = id;
	};
	const uint64_t items = min((uint64_t)stats->dense_items, dense_cap);
	for (uint64_t it = blockIdx.x; it < items; it += gridDim.x) {
		const DenseItem w = dense[it];
		const uint64_t s0 = cell_start[w.cell], s1 = min((uint64_t)cell_start[w.cell + 1], entry_cap);
		const uint32_t k = (uint32_t)(s1 - s0);
		if (k <= kOrderSeg) {
			if (w.row) continue;  // the cell's first item takes it whole
			uint32_t m = 2;
			while (m < k) m <<= 1;
			__syncthreads();
			for (uint32_t i = threadIdx.x; i < m; i += kNT)
				keys[i] = i < k ? ((unsigned long long)__float_as_uint(entries[2 * (s0 + i)].w) << 32) | i : ~0ull;
			__syncthreads();
			bitonic_shared(keys, (int)m, threadIdx.x, kNT, [] { __syncthreads(); });
			for (uint32_t i = threadIdx.x; i < k; i += kNT) put(s0 + (uint32_t)keys[i], s0 + i);
			continue;
		}
		const uint32_t i = w.row + threadIdx.x;
		const uint32_t id = i < k ? __float_as_uint(entries[2 * (s0 + i)].w) : 0u;
		uint32_t *ids = reinterpret_cast<uint32_t *>(keys);
		uint32_t rank = 0;
		for (uint32_t c0 = 0; c0 < k; c0 += kNT) {
			__syncthreads();
			ids[threadIdx.x] = c0 + threadIdx.x < k ? __float_as_uint(entries[2 * (s0 + c0 + threadIdx.x)].w) : 0xffffffffu;
			__syncthreads();
			const uint4 *v = reinterpret_cast<const uint4 *>(ids);
#pragma unroll 8
			for (int q = 0; q < kNT / 4; q++) {
				const uint4 x = v[q];
				rank += (x.x < id) + (x.y < id) + (x.z < id) + (x.w < id);
			}
		}
		if (i < k) put(s0 + i, s0 + rank);
	}
}

// Where there is room the masks of the count are kept for the write (row by row,
// eight words a column tile); then k_dense_emit writes the item's pairs, else
// this kernel tests it again.
template <bool kEmit>
__global__ void __launch_bounds__(kNT) k_dense_test(DevStats *stats, const uint32_t *__restrict__ cell_start,
                                                     const float4 *__restrict__ sorted, uint64_t entry_cap,
                                                     uint32_t *__restrict__ owner_count, uint32_t *__restrict__ row_count,
                                                     const DenseItem *__restrict__ dense, uint64_t dense_cap, int oshift,
                                                     uint32_t *__restrict__ masks, uint64_t mask_cap,
                                                     const unsigned long long *__restrict__ owner_off,
                                                     unsigned long long *__restrict__ out) {
	pdl_begin();
	__shared__ DenseTile tile;
	__shared__ uint32_t words[kEmit ? 1 : kNT / 32][kNT];  // each thread's masks of the tile
	__shared__ unsigned long long s_pairs;
	// the list does not fit the output, or all masks were kept
	if (kEmit && (stats->np_n != stats->pairs || stats->mask_words <= mask_cap)) return;
	if (!kEmit) {
		if (threadIdx.x == 0) s_pairs = blockIdx.x == 0 ? stats->tmp_pairs : 0ull;  // the sparse cells' pairs count too
		__syncthreads();
	}
	const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x / 32;
	const uint64_t items = min((uint64_t)stats->dense_items, dense_cap);
	for (uint64_t it = blockIdx.x; it < items; it += gridDim.x) {
		const DenseItem w = dense[it];
		const uint64_t s0 = cell_start[w.cell], s1 = min((uint64_t)cell_start[w.cell + 1], entry_cap);
		const uint32_t k = (uint32_t)(s1 - s0), r0 = w.row, i = r0 + threadIdx.x;
		const bool kept = w.mask + dense_mask_words(k, r0) <= mask_cap;
		if (kEmit && kept) continue;
		uint32_t *mask = masks + w.mask + (uint64_t)threadIdx.x * dense_row_words(k, r0);
		float4 alo = make_float4(INFINITY, INFINITY, INFINITY, 0.f), ahi = make_float4(-INFINITY, -INFINITY, -INFINITY, 0.f);
		if (i < k) ld_global_v8(reinterpret_cast<const float *>(sorted + 2 * (s0 + i)), alo, ahi);
		const uint32_t a = __float_as_uint(alo.w);
		uint32_t cnt = 0;
		unsigned long long *to = out;  // of the row's next pair
		if (kEmit) {
			cnt = i < k ? row_count[s0 + i] : 0u;
			if (cnt) to += owner_off[a >> oshift] + atomicSub(&owner_count[a >> oshift], cnt) - cnt;
		}
		for (uint32_t c0 = r0; c0 < k; c0 += kNT) {
			__syncthreads();  // the previous tile is no longer read
			load_columns(tile, sorted, s0, c0, k);
			__syncthreads();
			const uint32_t groups = min((uint32_t)kNT, k - c0 + 31u) / 32u;
			// in the diagonal tile a warp's rows have no later column before their own group
			for (uint32_t g = c0 == r0 ? warp : 0u; g < groups; g++) {
				uint32_t hit = test_columns(tile, 32 * g, alo, ahi);
				if (c0 == r0 && g == warp) hit &= lane == 31 ? 0u : 0x7fffffffu >> lane;  // later columns only
				if constexpr (!kEmit) {
					cnt += __popc(hit);
					words[g][threadIdx.x] = hit;
				} else {
					while (hit) {
						const uint32_t q = __clz(hit);
						hit &= ~(0x80000000u >> q);
						*to++ = ((unsigned long long)a << 32) | __float_as_uint(tile.lo[32 * g + q].w);
					}
				}
			}
			if (!kEmit && kept && i < k) {  // the tile's eight words of this row (its own: no barrier)
				float f[8];
#pragma unroll
				for (uint32_t g = 0; g < 8; g++)
					f[g] = __uint_as_float(g < groups && (c0 != r0 || g >= warp) ? words[kEmit ? 0 : g][threadIdx.x] : 0u);
				st_global_v8(reinterpret_cast<float *>(mask + (c0 - r0) / 32), make_float4(f[0], f[1], f[2], f[3]),
				             make_float4(f[4], f[5], f[6], f[7]));
			}
		}
		if constexpr (!kEmit) {
			if (i < k) row_count[s0 + i] = cnt;
			if (cnt) atomicAdd(&owner_count[a >> oshift], cnt);
			const uint32_t sum = __reduce_add_sync(0xffffffffu, cnt);
			if (lane == 0 && sum) atomicAdd(&s_pairs, (unsigned long long)sum);
		}
	}
	if constexpr (!kEmit) {
		__syncthreads();
		if (threadIdx.x == 0 && s_pairs) atomicAdd(&stats->pairs, s_pairs);
	}
}

// The pairs of the items whose masks were kept: W lanes per row, a lane per mask
// word, so that a row's pairs are written together (a lane per row kept 300,000
// partly written lines under way and thrashed the L2: 5.8 ms at 4.2M spheres;
// 32 lanes for every row 2.4, most of them without a word).
template <int W>
__device__ __forceinline__ void emit_rows(unsigned long long *__restrict__ out, const uint32_t *__restrict__ body,
                                          const uint32_t *__restrict__ masks, uint32_t per, uint32_t cnt, uint32_t a,
                                          unsigned long long at) {
	const uint32_t lane = threadIdx.x & 31, sub = lane & (W - 1);
	const auto word = [&](uint32_t r, uint32_t g) { return g + sub < per ? __ldcs(masks + (uint64_t)r * per + g + sub) : 0u; };
	uint32_t ahead = word(lane / W, 0);
	for (uint32_t r0 = 0; r0 < 32; r0 += 32 / W) {
		const uint32_t r = r0 + lane / W;
		uint32_t hit = ahead;
		if (r0 + 32 / W < 32) ahead = word(r + 32 / W, 0);  // the next rows' words arrive meanwhile
		const uint32_t c = __shfl_sync(0xffffffffu, cnt, r);
		const unsigned long long key = (unsigned long long)__shfl_sync(0xffffffffu, a, r) << 32;
		unsigned long long *to = out + __shfl_sync(0xffffffffu, at, r);
		if (!c) hit = 0u;  // rows past the cell's end: words never written
		for (uint32_t g = 0; g < per; g += W) {
			if (g) hit = c ? word(r, g) : 0u;
			const uint32_t own = __popc(hit);
			uint32_t incl = own;
#pragma unroll
			for (int o = 1; o < W; o <<= 1) {
				const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o, W);
				if ((int)sub >= o) incl += t;
			}
			unsigned long long *p = to + (incl - own);
			while (hit) {
				const uint32_t q = __clz(hit);
				hit &= ~(0x80000000u >> q);
				*p++ = key | body[32 * (g + sub) + q];
			}
			if (g + W < per) to += __shfl_sync(0xffffffffu, incl, W - 1, W);
		}
	}
}
__global__ void __launch_bounds__(kNT) k_dense_emit(DevStats *stats, const uint32_t *__restrict__ cell_start,
                                                     const uint32_t *__restrict__ sorted_body, uint64_t entry_cap,
                                                     uint32_t *__restrict__ owner_count,
                                                     const uint32_t *__restrict__ row_count,
                                                     const DenseItem *__restrict__ dense, uint64_t dense_cap, int oshift,
                                                     const uint32_t *__restrict__ masks, uint64_t mask_cap,
                                                     const unsigned long long *__restrict__ owner_off,
                                                     unsigned long long *__restrict__ out) {
	pdl_begin();
	if (stats->np_n != stats->pairs) return;  // the list does not fit the output
	const uint32_t warp = threadIdx.x / 32;
	const uint64_t items = min((uint64_t)stats->dense_items, dense_cap);
	for (uint64_t it = blockIdx.x; it < items; it += gridDim.x) {
		const DenseItem w = dense[it];
		const uint64_t s0 = cell_start[w.cell], s1 = min((uint64_t)cell_start[w.cell + 1], entry_cap);
		const uint32_t k = (uint32_t)(s1 - s0), per = dense_row_words(k, w.row);
		if (w.mask + dense_mask_words(k, w.row) > mask_cap) continue;
		const uint32_t *body = sorted_body + s0 + w.row;
		const uint32_t i = w.row + threadIdx.x;
		const uint32_t cnt = i < k ? row_count[s0 + i] : 0u, a = i < k ? sorted_body[s0 + i] : 0u;
		unsigned long long at = 0;
		if (cnt) at = owner_off[a >> oshift] + atomicSub(&owner_count[a >> oshift], cnt) - cnt;
		if (!__any_sync(0xffffffffu, cnt != 0u)) continue;
		const uint32_t *mask = masks + w.mask + (uint64_t)(32 * warp) * per;
		if (per <= 8) emit_rows<8>(out, body, mask, per, cnt, a, at);
		else if (per <= 16) emit_rows<16>(out, body, mask, per, cnt, a, at);
		else emit_rows<32>(out, body, mask, per, cnt, a, at);
	}
}

// Bucket the unsorted pairs by owner bucket (the smaller index >> oshift). Their
// count comes from the device; if they exceed the scratch, or all pairs the
// output, nothing is written.
__global__ void __launch_bounds__(kNT) k_owner_scatter(DevStats *stats, const unsigned long long *tmp_n, uint64_t pair_cap,
                                                        uint64_t out_cap, const unsigned long long *__restrict__ tmp,
                                                        const unsigned long long *__restrict__ owner_off,
                                                        uint32_t *__restrict__ owner_count,
                                                        unsigned long long *__restrict__ out, int oshift) {
	pdl_begin();
	const unsigned long long all = stats->pairs, P = *tmp_n;  // P < all: the dense cells' pairs are not in tmp
	const bool fits = P <= pair_cap && all <= out_cap;
	if (blockIdx.x == 0 && threadIdx.x == 0) stats->np_n = fits ? all : 0ull;
	if (!fits) return;
	// lanes of a warp whose pairs share an owner take their slots with one
	// atomic (pair lists of dense cells arrive grouped by owner)
	const uint32_t lane = threadIdx.x & 31, lt = (1u << lane) - 1u;
	const uint64_t step = (uint64_t)gridDim.x * kNT;
	for (uint64_t t0 = (uint64_t)blockIdx.x * kNT + (threadIdx.x & ~31u); t0 < P; t0 += step) {
		const uint64_t t = t0 + lane;
		const bool valid = t < P;
		const unsigned long long key = valid ? tmp[t] : 0ull;
		const uint32_t a = valid ? (uint32_t)(key >> 32) >> oshift : 0xffffffffu;
		const uint32_t peers = __match_any_sync(0xffffffffu, a);
		const int leader = __ffs(peers) - 1;
		uint32_t base = 0;
		if (valid && (int)lane == leader) base = atomicSub(&owner_count[a], (uint32_t)__popc(peers));
		base = __shfl_sync(0xffffffffu, base, leader);
		if (valid) out[owner_off[a] + base - 1u - __popc(peers & lt)] = key;
	}
}

// Sort keys inside an owner bucket: 32-bit packings of the 64-bit pair keys
// that order like them (the bucket fixes the high bits of the owner).
struct KeyPack {
	int shift, kb;  // BpBuffers::owner_shift, key_bits
};
// kPack false: one owner per bucket (shift 0), the key is the partner half.
// The choice is a template parameter, resolved per kernel launch: a runtime
// test inside the register sorts' unrolled load and store loops made the
// warp-tier kernel almost twice as slow on the 16.7M clustered scene.
template <bool kPack>
__device__ __forceinline__ uint32_t pack_key(unsigned long long key, KeyPack kp) {
	const uint32_t b = (uint32_t)key;
	if constexpr (!kPack) {
		return b;
	} else {
		const uint32_t alo = (uint32_t)(key >> 32) & ((1u << kp.shift) - 1u);
		return (alo << kp.kb) | b;
	}
}
template <bool kPack>
__device__ __forceinline__ unsigned long long unpack_key(uint32_t v, uint32_t bucket, KeyPack kp) {
	if constexpr (!kPack) {
		return ((unsigned long long)bucket << 32) | v;
	} else {
		const uint32_t a = (bucket << kp.shift) | (v >> kp.kb);
		return ((unsigned long long)a << 32) | (v & ((1u << kp.kb) - 1u));
	}
}

constexpr int kTinySeg = 8;    // buckets sorted by one thread with a bubble network in registers
constexpr int kSmallSeg = 32;  // buckets sorted by one thread with a bitonic network in registers

// Compare-exchange of two keys held in registers (ascending).
__device__ __forceinline__ void cx(uint32_t &x, uint32_t &y) {
	const uint32_t a = x, b = y;
	x = min(a, b);
	y = max(a, b);
}
constexpr int kMidSeg = 1024;
constexpr int kBigSeg = 16384;

// One bucket of at most kSmallSeg keys sorted by one thread in registers, on the
// packed 32-bit keys: a bubble network up to kTinySeg keys, a bitonic network
// padded to kSmallSeg above (one load and one store round trip either way).
template <bool kPack>
__device__ __forceinline__ void sort_thread_bucket(unsigned long long *__restrict__ out, uint64_t beg, uint64_t len,
                                                   uint32_t a, KeyPack kp) {
	if (len > 1 && len <= kTinySeg) {
		uint32_t v[kTinySeg];
#pragma unroll
		for (int q = 0; q < kTinySeg; q++) v[q] = (uint64_t)q < len ? pack_key<kPack>(out[beg + q], kp) : 0xffffffffu;
#pragma unroll
		for (int r = 0; r < kTinySeg - 1; r++)
#pragma unroll
			for (int q = 0; q < kTinySeg - 1 - r; q++) cx(v[q], v[q + 1]);
#pragma unroll
		for (int q = 0; q < kTinySeg; q++)
			if ((uint64_t)q < len) out[beg + q] = unpack_key<kPack>(v[q], a, kp);
	} else if (len > kTinySeg && len <= kSmallSeg) {
		uint32_t v[kSmallSeg];
#pragma unroll
		for (int q = 0; q < kSmallSeg; q++) v[q] = (uint64_t)q < len ? pack_key<kPack>(out[beg + q], kp) : 0xffffffffu;
#pragma unroll
		for (int k = 2; k <= kSmallSeg; k <<= 1)
#pragma unroll
			for (int j = k >> 1; j > 0; j >>= 1)
#pragma unroll
				for (int i = 0; i < kSmallSeg; i++) {
					const int l = i ^ j;
					if (l > i) {
						if ((i & k) == 0) cx(v[i], v[l]);
						else cx(v[l], v[i]);
					}
				}
#pragma unroll
		for (int q = 0; q < kSmallSeg; q++)
			if ((uint64_t)q < len) out[beg + q] = unpack_key<kPack>(v[q], a, kp);
	}
}

// Sorts each owner bucket (all keys share the bucket's owners, n here is the
// bucket count): <= 32 keys by one thread, loaded into registers at once and
// sorted there by a static network on the packed keys (a bubble network up to
// 8 keys, a bitonic network padded to 32 above); longer buckets are listed for
// k_segsort_mid (<= 1024 keys, from the front of big_list) or k_segsort_big
// (<= 16384, from the back), which sort the packed 32-bit keys (pack_key).
template <bool kPack>
__global__ void __launch_bounds__(kNT) k_segsort(uint64_t n, const unsigned long long *__restrict__ owner_off,
                                                  unsigned long long *__restrict__ out, uint32_t *big_list,
                                                  uint64_t big_cap, DevStats *stats, KeyPack kp) {
	pdl_begin();
	if (stats->np_n != stats->pairs) return;  // the pairs were not emitted (uniform over the grid)
	const uint64_t a = (uint64_t)blockIdx.x * kNT + threadIdx.x;
	uint64_t len = 0;
	if (a < n) {
		const uint64_t beg = owner_off[a], end = owner_off[a + 1];
		len = end - beg;
		sort_thread_bucket<kPack>(out, beg, len, (uint32_t)a, kp);
	}
	const bool longer = len > kSmallSeg;
	const uint32_t wmax = __reduce_max_sync(0xffffffffu, longer ? (uint32_t)min(len, (uint64_t)0xffffffffu) : 0u);
	if ((threadIdx.x & 31) == 0 && wmax) atomicMax(&stats->max_segment, (unsigned long long)wmax);
	if (len > kBigSeg) atomicOr(&stats->err, (uint32_t)kErrSegmentTooLong);
	// list the longer buckets, one counter atomic per warp and tier
	const bool mid = longer && len <= kMidSeg, big = len > kMidSeg && len <= kBigSeg;
	const uint32_t lane = threadIdx.x & 31, lt = (1u << lane) - 1u;
#pragma unroll
	for (int tier = 0; tier < 2; tier++) {
		const bool want = tier == 0 ? mid : big;
		const uint32_t m = __ballot_sync(0xffffffffu, want);
		if (!m) continue;
		unsigned long long base = 0;
		if (lane == (uint32_t)(__ffs(m) - 1)) base = atomicAdd(tier == 0 ? &stats->big_segments : &stats->seg_big,
		                                                       (unsigned long long)__popc(m));
		base = __shfl_sync(0xffffffffu, base, __ffs(m) - 1);
		if (want) {
			const unsigned long long slot = base + __popc(m & lt);
			if (slot < big_cap) big_list[tier == 0 ? slot : big_cap - 1 - slot] = (uint32_t)a;
			else atomicOr(&stats->err, (uint32_t)kErrSegmentTooLong);
		}
	}
}

// Register bitonic sort of 32*K keys held by one warp, striped: key e = 32*r
// + lane sits in v[r] of that lane. Steps whose partner distance j is below 32
// exchange across lanes (shuffle), the others pair registers of the same lane
// (register distance j/32, resolved at compile time through a switch so that
// v stays in registers).
// el = the key index held in v[0] by this lane (the warp's first key +
// lane); the network sorts key e ascending where (e & k) == 0 in merge size k.
template <int K, int JR>
__device__ __forceinline__ void bitonic_reg_step(uint32_t (&v)[K], int el, int k) {
	if constexpr (JR < K) {
#pragma unroll
		for (int r = 0; r < K; r++)
			if ((r & JR) == 0) {
				const bool up = ((el + 32 * r) & k) == 0;
				const uint32_t x = v[r], y = v[r | JR];
				v[r] = up ? min(x, y) : max(x, y);
				v[r | JR] = up ? max(x, y) : min(x, y);
			}
	}
}
// One step of partner distance j < 32 * K (inside the warp's keys).
template <int K>
__device__ __forceinline__ void bitonic_warp_step(uint32_t (&v)[K], int el, int j, int k) {
	if (j < 32) {
		const bool lower = (el & j) == 0;
#pragma unroll
		for (int r = 0; r < K; r++) {
			const uint32_t o = __shfl_xor_sync(0xffffffffu, v[r], j);
			const bool up = ((el + 32 * r) & k) == 0;
			v[r] = (lower == up) ? min(v[r], o) : max(v[r], o);
		}
	} else {
		switch (j >> 5) {
		case 1: bitonic_reg_step<K, 1>(v, el, k); break;
		case 2: bitonic_reg_step<K, 2>(v, el, k); break;
		case 4: bitonic_reg_step<K, 4>(v, el, k); break;
		case 8: bitonic_reg_step<K, 8>(v, el, k); break;
		case 16: bitonic_reg_step<K, 16>(v, el, k); break;
		}
	}
}
template <int K>
__device__ __forceinline__ void bitonic_reg(uint32_t (&v)[K], int lane) {
	for (int k = 2; k <= 32 * K; k <<= 1)
		for (int j = k >> 1; j > 0; j >>= 1) bitonic_warp_step<K>(v, lane, j, k);
}
// One bucket of len <= 32*K keys: partner halves into registers (padding
// sorts last), sorted, written back with the owner in the high half.
template <int K, bool kPack>
__device__ __forceinline__ void sort_bucket_reg(unsigned long long *__restrict__ out, uint64_t beg, uint64_t len,
                                                uint32_t a, int lane, KeyPack kp) {
	uint32_t v[K];
#pragma unroll
	for (int r = 0; r < K; r++) {
		const uint64_t e = 32u * r + lane;
		v[r] = e < len ? pack_key<kPack>(out[beg + e], kp) : 0xffffffffu;
	}
	bitonic_reg<K>(v, lane);
#pragma unroll
	for (int r = 0; r < K; r++) {
		const uint64_t e = 32u * r + lane;
		if (e < len) out[beg + e] = unpack_key<kPack>(v[r], a, kp);
	}
}

// A bucket of 1025..2048 keys on a pair of warps (half = 0, 1), 1024 keys
// each, 32 per lane; the one step of partner distance 1024 exchanges through
// the pair's 8 KB of shared memory x, the pair synchronizing on its own
// named barrier `bar` (both warps run the same steps).
constexpr int kPairSeg = 2048;
__device__ __forceinline__ void pair_sync(int bar) { asm volatile("bar.sync %0, 64;" ::"r"(bar) : "memory"); }
template <bool kPack>
__device__ __forceinline__ void sort_bucket_pair(unsigned long long *__restrict__ out, uint64_t beg, uint64_t len,
                                                 uint32_t a, int half, int lane, uint32_t *x, int bar, KeyPack kp) {
	const int el = half * 1024 + lane;
	uint32_t v[32];
#pragma unroll
	for (int r = 0; r < 32; r++) {
		const uint64_t e = (uint64_t)el + 32u * r;
		v[r] = e < len ? pack_key<kPack>(out[beg + e], kp) : 0xffffffffu;
	}
	for (int k = 2; k <= kPairSeg; k <<= 1)
		for (int j = k >> 1; j > 0; j >>= 1) {
			if (j == 1024) {
#pragma unroll
				for (int r = 0; r < 32; r++) x[el + 32 * r] = v[r];
				pair_sync(bar);
				const bool lower = half == 0;
#pragma unroll
				for (int r = 0; r < 32; r++) {
					const uint32_t o = x[(el + 32 * r) ^ 1024];
					const bool up = ((el + 32 * r) & k) == 0;
					v[r] = (lower == up) ? min(v[r], o) : max(v[r], o);
				}
				pair_sync(bar);  // x is free again
			} else {
				bitonic_warp_step<32>(v, el, j, k);
			}
		}
#pragma unroll
	for (int r = 0; r < 32; r++) {
		const uint64_t e = (uint64_t)el + 32u * r;
		if (e < len) out[beg + e] = unpack_key<kPack>(v[r], a, kp);
	}
}

// Buckets that are a few ascending runs (the rows of a body in its dense cells,
// k_dense_emit) are merged instead of sorted: adjacent runs pairwise, every key
// placed by a binary search in the partner run, between two halves of shared
// memory. At 4.2M clustered spheres (246M pairs) the bitonic tiers alone take 3.8
// ms at 15 warp instructions a key, merges and what is left to them 2.9 ms.
// Returns false, with the bucket untouched, above kMaxRuns runs. NT threads
// work together, Sync separates the steps; buf holds 2 * cap keys.
constexpr uint32_t kMaxRuns = 32;
constexpr int kSearch = 2;  // 4.2M clustered spheres, the mid tier: one 3.34 ms, two 2.89, four 3.06, eight 3.77
struct Runs {
	uint32_t start[kMaxRuns + 2], count;
};
template <int NT, bool kPack, class Sync>
__device__ __forceinline__ bool merge_runs(unsigned long long *__restrict__ out, uint64_t beg, uint32_t len, uint32_t a,
                                           uint32_t t, uint32_t *buf, uint32_t cap, Runs &runs, KeyPack kp, Sync sync) {
	uint32_t *src = buf, *dst = buf + cap;
	if (t == 0) {
		runs.count = 1;
		runs.start[0] = 0;
	}
	for (uint32_t e0 = t; e0 < len; e0 += 8 * NT) {  // eight loads in flight
		unsigned long long v[8];
#pragma unroll
		for (int q = 0; q < 8; q++) v[q] = e0 + q * NT < len ? out[beg + e0 + q * NT] : 0ull;
#pragma unroll
		for (int q = 0; q < 8; q++)
			if (e0 + q * NT < len) src[e0 + q * NT] = pack_key<kPack>(v[q], kp);
	}
	sync();
	for (uint32_t e = t; e < len; e += NT)
		if (e && src[e] < src[e - 1]) {  // a run starts here; their order is restored below
			const uint32_t at = atomicAdd(&runs.count, 1u);
			if (at < kMaxRuns) runs.start[at] = e;
		}
	sync();
	uint32_t R = runs.count;
	if (R > kMaxRuns) return false;
	if (R == 1) return true;
	// starts in order (at most 32: one warp, rank by counting)
	const uint32_t mine = t < R ? runs.start[t] : 0xffffffffu;
	uint32_t rank = 0;
	if (t < R)
		for (uint32_t q = 0; q < R; q++) rank += runs.start[q] < mine;
	sync();
	if (t < R) runs.start[rank] = mine;
	if (t == 0) runs.start[R] = len;
	sync();
	while (R > 1) {
		for (uint32_t r = 0; r < R; r += 2) {
			const uint32_t s0 = runs.start[r], s1 = runs.start[r + 1], s2 = r + 1 < R ? runs.start[r + 2] : s1;
			// branch-free searches of kSearch keys side by side: a search is a chain of
			// shared loads
			const uint32_t longer = max(s1 - s0, s2 - s1);
			const uint32_t top = longer ? 1u << (31 - __clz((int)longer)) : 0u;
			for (uint32_t i0 = s0 + t; i0 < s2; i0 += kSearch * NT) {
				uint32_t key[kSearch], lo[kSearch], end[kSearch];
#pragma unroll
				for (int q = 0; q < kSearch; q++) {
					const uint32_t i = i0 + q * NT;
					key[q] = i < s2 ? src[i] : 0u;
					lo[q] = i < s1 ? s1 : s0;
					end[q] = i < s1 ? s2 : s1;
				}
				for (uint32_t step = top; step; step >>= 1)
#pragma unroll
					for (int q = 0; q < kSearch; q++)
						if (lo[q] + step <= end[q] && src[lo[q] + step - 1] < key[q]) lo[q] += step;
#pragma unroll
				for (int q = 0; q < kSearch; q++)
					if (i0 + q * NT < s2) dst[i0 + q * NT + lo[q] - s1] = key[q];  // place in its own run + smaller keys of the other
			}
		}
		const uint32_t half = (R + 1) / 2;
		const uint32_t next = t < half ? runs.start[2 * t] : 0u;
		sync();
		if (t < half) runs.start[t] = next;
		if (t == 0) runs.start[half] = len;
		R = half;
		uint32_t *x = src;
		src = dst;
		dst = x;
		sync();
	}
	for (uint32_t e = t; e < len; e += NT) out[beg + e] = unpack_key<kPack>(src[e], a, kp);
	return true;
}

// The buckets of the mid and big lists that merge: warps take buckets of up to
// kMidSeg keys, then blocks those of up to kMergeSeg. A merged bucket leaves its
// list (kDoneBucket); k_segsort_mid and k_segsort_big sort what is left.
constexpr uint32_t kMergeSeg = 8 * kMidSeg;
constexpr uint32_t kDoneBucket = 0xffffffffu;
template <bool kPack>
__global__ void __launch_bounds__(kNT) k_segsort_runs(const DevStats *stats, uint64_t big_cap, uint32_t *__restrict__ big_list,
                                                       const unsigned long long *__restrict__ owner_off,
                                                       unsigned long long *__restrict__ out, KeyPack kp) {
	pdl_begin();
	extern __shared__ uint32_t merge_buf[];  // 2 * kMergeSeg keys
	__shared__ Runs runs[kNT / 32];
	if (stats->np_n != stats->pairs) return;
	const uint32_t warp = threadIdx.x / 32, lane = threadIdx.x & 31;
	const uint64_t nmid = min((uint64_t)stats->big_segments, big_cap);
	for (uint64_t g = (uint64_t)blockIdx.x * (kNT / 32) + warp; g < nmid; g += (uint64_t)gridDim.x * (kNT / 32)) {
		const uint32_t a = big_list[g];
		const uint64_t beg = owner_off[a], len = owner_off[a + 1] - beg;
		const bool done = merge_runs<32, kPack>(out, beg, (uint32_t)len, a, lane, merge_buf + 2 * kMidSeg * warp, kMidSeg,
		                                        runs[warp], kp, [] { __syncwarp(); });
		__syncwarp();
		if (done && lane == 0) big_list[g] = kDoneBucket;
	}
	__syncthreads();
	const uint64_t nbig = min((uint64_t)stats->seg_big, big_cap);
	for (uint64_t g = blockIdx.x; g < nbig; g += gridDim.x) {
		const uint32_t a = big_list[big_cap - 1 - g];
		const uint64_t beg = owner_off[a], len = owner_off[a + 1] - beg;
		if (len > kMergeSeg) continue;
		const bool done = merge_runs<kNT, kPack>(out, beg, (uint32_t)len, a, threadIdx.x, merge_buf, kMergeSeg, runs[0], kp,
		                                         [] { __syncthreads(); });
		__syncthreads();
		if (done && threadIdx.x == 0) big_list[big_cap - 1 - g] = kDoneBucket;
	}
}

// Buckets of 33..1024 keys: one warp per bucket, sorted in registers
// (2..32 keys per lane by bucket size); then buckets of 1025..2048 keys
// (listed for k_segsort_big, which leaves them) on pairs of warps.
constexpr int kMidNT = 256;
template <bool kPack>
__global__ void __launch_bounds__(kMidNT, 2) k_segsort_mid(const DevStats *stats, uint64_t big_cap,
                                                         const uint32_t *__restrict__ big_list,
                                                         const unsigned long long *__restrict__ owner_off,
                                                         unsigned long long *__restrict__ out, KeyPack kp) {
	pdl_begin();
	if (stats->np_n != stats->pairs) return;
	const uint64_t nmid = min((uint64_t)stats->big_segments, big_cap);
	const int lane = threadIdx.x & 31;
	const uint64_t warps = (uint64_t)gridDim.x * (kMidNT / 32);
	for (uint64_t g = (uint64_t)blockIdx.x * (kMidNT / 32) + (threadIdx.x >> 5); g < nmid; g += warps) {
		const uint32_t a = big_list[g];
		if (a == kDoneBucket) continue;
		const uint64_t beg = owner_off[a], len = owner_off[a + 1] - beg;  // 33..1024, listed by k_segsort
		if (len <= 64) sort_bucket_reg<2, kPack>(out, beg, len, a, lane, kp);
		else if (len <= 128) sort_bucket_reg<4, kPack>(out, beg, len, a, lane, kp);
		else if (len <= 256) sort_bucket_reg<8, kPack>(out, beg, len, a, lane, kp);
		else if (len <= 512) sort_bucket_reg<16, kPack>(out, beg, len, a, lane, kp);
		else sort_bucket_reg<32, kPack>(out, beg, len, a, lane, kp);
	}
	__shared__ uint32_t xch[kMidNT / 64][kPairSeg];
	const uint64_t nbig = min((uint64_t)stats->seg_big, big_cap);
	const int pair = threadIdx.x >> 6, half = (threadIdx.x >> 5) & 1;
	const uint64_t npairs = (uint64_t)gridDim.x * (kMidNT / 64);
	for (uint64_t g = (uint64_t)blockIdx.x * (kMidNT / 64) + pair; g < nbig; g += npairs) {
		const uint32_t a = big_list[big_cap - 1 - g];
		if (a == kDoneBucket) continue;
		const uint64_t beg = owner_off[a], len = owner_off[a + 1] - beg;
		if (len > kPairSeg) continue;  // the block tier's (uniform over the pair)
		sort_bucket_pair<kPack>(out, beg, len, a, half, lane, xch[pair], 1 + pair, kp);
	}
}

// Buckets of 2049..16384 keys: one block per bucket (grid-stride over the
// device-side count), bitonic sort of the partner halves in 64 KB of
// dynamic shared memory.
template <bool kPack>
__global__ void __launch_bounds__(512) k_segsort_big(const DevStats *stats, uint64_t big_cap,
                                                      const uint32_t *__restrict__ big_list,
                                                      const unsigned long long *__restrict__ owner_off,
                                                      unsigned long long *__restrict__ out, KeyPack kp) {
	pdl_begin();
	extern __shared__ uint32_t s[];
	if (stats->np_n != stats->pairs) return;
	const uint64_t nbig = min((uint64_t)stats->seg_big, big_cap);
	for (uint64_t g = blockIdx.x; g < nbig; g += gridDim.x) {
		const uint32_t a = big_list[big_cap - 1 - g];
		if (a == kDoneBucket) continue;
		const uint64_t beg = owner_off[a], len = owner_off[a + 1] - beg;
		if (len <= kPairSeg) continue;  // sorted by warp pairs in k_segsort_mid (uniform over the block)
		int m = 1;
		while ((uint64_t)m < len) m <<= 1;
		for (int i = threadIdx.x; i < m; i += blockDim.x) s[i] = (uint64_t)i < len ? pack_key<kPack>(out[beg + i], kp) : 0xffffffffu;
		__syncthreads();
		bitonic_shared(s, m, threadIdx.x, blockDim.x, [] { __syncthreads(); });
		for (int i = threadIdx.x; (uint64_t)i < len; i += blockDim.x) out[beg + i] = unpack_key<kPack>(s[i], a, kp);
		__syncthreads();
	}
}

// ---------------------------------------------------------------- fused owner sort
// Pair lists far shorter than the body count (the owner shift then keeps about
// eight pairs per bucket, so there are few buckets): the owner scan, the
// bucketing and every bucket sort of the path above run as ONE cooperative
// kernel. Each block scans all bucket counts itself into shared memory (a few
// KB read from L2 per block; no scan launch), buckets its share of the pairs
// through per-bucket cursors (zeroed by k_count, so the counts stay intact
// while other blocks still scan them), waits at one grid barrier, and sorts
// the buckets: <= 32 keys per thread, 33..1024 per warp in registers,
// 1025..kFusedSeg per block in shared memory. A longer bucket sets
// kErrSegmentTooLong (the caller then sorts the whole list). The grid is short
// (128 blocks for 1M bodies) and latency-bound: 21 us there, under the MPR that
// runs beside it; the bound of 64 registers leaves the MPR's blocks
// their room.
constexpr int kFusedNT = 256;
constexpr int kFusedSeg = 4096;
constexpr uint32_t kFusedBuckets = 8191;  // offsets + block-tier keys are 48 KB; with the static words the launch opts in

template <bool kPack>
__global__ void __launch_bounds__(kFusedNT, 4) k_owner_sort_fused(DevStats *stats, uint64_t pair_cap, uint64_t out_cap,
                                                             const unsigned long long *__restrict__ tmp,
                                                             const uint32_t *__restrict__ owner_count,
                                                             uint32_t *__restrict__ cursor, uint32_t nbk,
                                                             unsigned long long *__restrict__ out, int oshift,
                                                             KeyPack kp, uint32_t *host_stats) {
	pdl_trigger();  // (every block is resident: a cooperative launch)
	extern __shared__ uint32_t fsm[];  // off[nbk + 1], then kFusedSeg keys of the block tier
	__shared__ unsigned long long scan_sm[40];
	uint32_t *off = fsm, *keys = fsm + nbk + 1;
	const unsigned long long P = stats->pairs;
	const bool fits = P <= pair_cap && P <= out_cap && P < 0xffffffffull;
	if (blockIdx.x == 0 && threadIdx.x == 0) stats->np_n = fits ? P : 0ull;
	if (!fits) return report_by_last(stats, host_stats);  // uniform over the grid: no block reaches the barrier
	// 1. exclusive scan of the bucket counts: coalesced loads into shared
	// memory (all in flight at once), then one contiguous run per thread
	copy_words_to_shared<kFusedNT>(off, owner_count, nbk);
	__syncthreads();
	const uint32_t per = (nbk + kFusedNT - 1) / kFusedNT;
	const uint32_t b0 = min(nbk, threadIdx.x * per), b1 = min(nbk, b0 + per);
	unsigned long long run = 0;
	for (uint32_t b = b0; b < b1; b++) run += off[b];
	unsigned long long total;
	unsigned long long excl = block_excl_scan<unsigned long long, kFusedNT>(run, scan_sm, &total);
	for (uint32_t b = b0; b < b1; b++) {
		const uint32_t c = off[b];
		off[b] = (uint32_t)excl;
		excl += c;
	}
	if (threadIdx.x == 0) off[nbk] = (uint32_t)total;
	__syncthreads();
	// 2. bucket the pairs (lanes of a warp with one bucket share one atomic)
	const uint32_t lane = threadIdx.x & 31, lt = (1u << lane) - 1u;
	const uint64_t step = (uint64_t)gridDim.x * kFusedNT;
	for (uint64_t t0 = (uint64_t)blockIdx.x * kFusedNT + (threadIdx.x & ~31u); t0 < P; t0 += step) {
		const uint64_t t = t0 + lane;
		const bool valid = t < P;
		const unsigned long long key = valid ? tmp[t] : 0ull;
		const uint32_t a = valid ? (uint32_t)(key >> 32) >> oshift : 0xffffffffu;
		const uint32_t peers = __match_any_sync(0xffffffffu, a);
		const int leader = __ffs(peers) - 1;
		uint32_t base = 0;
		if (valid && (int)lane == leader) base = atomicAdd(&cursor[a], (uint32_t)__popc(peers));
		base = __shfl_sync(0xffffffffu, base, leader);
		if (valid) out[(uint64_t)off[a] + base + __popc(peers & lt)] = key;
	}
	grid_barrier(reinterpret_cast<GridBarrier *>(stats->bar_emit), &stats->err);
	// 3. sort the buckets, three tiers
	const uint64_t gt = (uint64_t)blockIdx.x * kFusedNT + threadIdx.x;
	uint32_t longest = 0;
	for (uint64_t b = gt; b < nbk; b += step) {
		const uint32_t beg = off[b], len = off[b + 1] - beg;
		sort_thread_bucket<kPack>(out, beg, len, (uint32_t)b, kp);
		longest = max(longest, len);
	}
	longest = __reduce_max_sync(0xffffffffu, longest);
	if (lane == 0 && longest > kSmallSeg) atomicMax(&stats->max_segment, (unsigned long long)longest);
	if (lane == 0 && longest > kFusedSeg) atomicOr(&stats->err, (uint32_t)kErrSegmentTooLong);
	const uint64_t warps = step / 32;
	for (uint64_t b = gt / 32; b < nbk; b += warps) {
		const uint32_t beg = off[b], len = off[b + 1] - beg;  // uniform over the warp
		if (len <= kSmallSeg || len > kMidSeg) continue;
		if (len <= 64) sort_bucket_reg<2, kPack>(out, beg, len, (uint32_t)b, lane, kp);
		else if (len <= 128) sort_bucket_reg<4, kPack>(out, beg, len, (uint32_t)b, lane, kp);
		else if (len <= 256) sort_bucket_reg<8, kPack>(out, beg, len, (uint32_t)b, lane, kp);
		else if (len <= 512) sort_bucket_reg<16, kPack>(out, beg, len, (uint32_t)b, lane, kp);
		else sort_bucket_reg<32, kPack>(out, beg, len, (uint32_t)b, lane, kp);
	}
	for (uint64_t b = blockIdx.x; b < nbk; b += gridDim.x) {
		const uint32_t beg = off[b], len = off[b + 1] - beg;  // uniform over the block
		if (len <= kMidSeg || len > kFusedSeg) continue;
		int m = 1;
		while ((uint32_t)m < len) m <<= 1;
		for (int i = threadIdx.x; i < m; i += kFusedNT) keys[i] = (uint32_t)i < len ? pack_key<kPack>(out[beg + i], kp) : 0xffffffffu;
		__syncthreads();
		bitonic_shared(keys, m, threadIdx.x, kFusedNT, [] { __syncthreads(); });
		for (int i = threadIdx.x; (uint32_t)i < len; i += kFusedNT) out[beg + i] = unpack_key<kPack>(keys[i], (uint32_t)b, kp);
		__syncthreads();
	}
	report_by_last(stats, host_stats);
}

// ---------------------------------------------------------------- bin list
// float -> int as the reference's host build converts (x86 cvttss2si: NaN and
// out-of-range values give INT_MIN), HashMin Broadphase.cu:125-133.
__device__ __forceinline__ int32_t trunc_x86(float v) {
	if (!(v >= -2147483648.0f && v < 2147483648.0f)) return INT_MIN;
	return __float2int_rz(v);
}
struct RefRange {
	int32_t g0[3], g1[3];
};
__device__ __forceinline__ RefRange ref_range(const Plan &p, float3 mn, float3 mx) {
	RefRange r;
	r.g0[0] = trunc_x86(mn.x * p.invbin[0]);
	r.g0[1] = trunc_x86(mn.y * p.invbin[1]);
	r.g0[2] = trunc_x86(mn.z * p.invbin[2]);
	r.g1[0] = trunc_x86(mx.x * p.invbin[0]);
	r.g1[1] = trunc_x86(mx.y * p.invbin[1]);
	r.g1[2] = trunc_x86(mx.z * p.invbin[2]);
	return r;
}

// function_Count_AABB_BIN_Intersection (:150-154) on the shifted boxes.
__global__ void __launch_bounds__(kNT) k_ref_count(uint64_t n, const float *__restrict__ aabb, const DevStats *stats,
                                                    uint32_t *__restrict__ cnt) {
	__shared__ Plan sp;
	if (threadIdx.x < sizeof(Plan) / 4)
		reinterpret_cast<uint32_t *>(&sp)[threadIdx.x] = reinterpret_cast<const uint32_t *>(&stats->plan)[threadIdx.x];
	__syncthreads();
	const uint64_t i = (uint64_t)blockIdx.x * kNT + threadIdx.x;
	if (i >= n) return;
	const RefRange r = ref_range(sp, ld3p(aabb, i), ld3p(aabb, i + n));
	const uint32_t c = (uint32_t)(r.g1[0] - r.g0[0] + 1) * (uint32_t)(r.g1[1] - r.g0[1] + 1) *
	                   (uint32_t)(r.g1[2] - r.g0[2] + 1);
	cnt[i] = c;
}

// function_Store_AABB_BIN_Intersection (:172-195): x outer, z inner, bin id
// z*gy*gx + y*gx + x in uint arithmetic (Hash_Index :140-147); the key is
// (bin << 32) | body so a stable sort on the upper half gives :428-432.
__global__ void __launch_bounds__(kNT) k_ref_emit(uint64_t n, const float *__restrict__ aabb, DevStats *stats,
                                                   const unsigned long long *__restrict__ off,
                                                   unsigned long long *__restrict__ keys, uint64_t cap) {
	__shared__ Plan sp;
	if (threadIdx.x < sizeof(Plan) / 4)
		reinterpret_cast<uint32_t *>(&sp)[threadIdx.x] = reinterpret_cast<const uint32_t *>(&stats->plan)[threadIdx.x];
	__syncthreads();
	const uint64_t i = (uint64_t)blockIdx.x * kNT + threadIdx.x;
	if (i >= n) return;
	const RefRange r = ref_range(sp, ld3p(aabb, i), ld3p(aabb, i + n));
	const uint32_t gx = (uint32_t)sp.grid[0], gy = (uint32_t)sp.grid[1];
	uint64_t w = off[i];
	const uint64_t wend = off[i + 1];
	uint32_t mb = 0;
	for (uint32_t x = (uint32_t)r.g0[0]; x <= (uint32_t)r.g1[0]; x++)
		for (uint32_t y = (uint32_t)r.g0[1]; y <= (uint32_t)r.g1[1]; y++)
			for (uint32_t z = (uint32_t)r.g0[2]; z <= (uint32_t)r.g1[2] && w < wend; z++) {
				const uint32_t bin = z * gy * gx + y * gx + x;
				mb = max(mb, bin);
				if (w < cap) keys[w] = ((unsigned long long)bin << 32) | (uint32_t)i;
				w++;
			}
	atomicMax(&stats->max_bin, mb);
	if (w != wend) atomicOr(&stats->err, (uint32_t)kErrBinCount);
}

__global__ void __launch_bounds__(kNT) k_ref_flags(const unsigned long long *__restrict__ keys, uint64_t E,
                                                    uint32_t *__restrict__ flags) {
	const uint64_t e = (uint64_t)blockIdx.x * kNT + threadIdx.x;
	if (e >= E) return;
	flags[e] = (e == 0 || (keys[e] >> 32) != (keys[e - 1] >> 32)) ? 1u : 0u;
}

// reduce_by_key (:439-443) + inclusive scan of the run lengths (:476-480).
__global__ void __launch_bounds__(kNT) k_ref_split(const unsigned long long *__restrict__ keys, uint64_t E,
                                                    const uint32_t *__restrict__ run_pos, uint32_t *bin_number,
                                                    uint32_t *body_number, uint32_t *active_bins, uint32_t *bin_end,
                                                    uint64_t cap_a) {
	const uint64_t e = (uint64_t)blockIdx.x * kNT + threadIdx.x;
	if (e >= E) return;
	const unsigned long long k = keys[e];
	const uint32_t bin = (uint32_t)(k >> 32);
	if (bin_number) bin_number[e] = bin;
	if (body_number) body_number[e] = (uint32_t)k;
	const uint32_t r = run_pos[e + 1] - 1u;  // run index of this entry
	if (r < cap_a) {
		if (active_bins && run_pos[e] == r) active_bins[r] = bin;  // first entry of the run
		if (bin_end && (e + 1 == E || run_pos[e + 2] != run_pos[e + 1])) bin_end[r] = (uint32_t)(e + 1);
	}
}

inline unsigned blocks_for(uint64_t n) { return (unsigned)((n + kNT - 1) / kNT); }
}  // namespace

void launch_bounds(uint64_t n, const float *aabb, DevStats *stats, const GridParams &gp, const int grid[3],
                   cudaStream_t s, const ZeroList &zero) {
	PlanArgs pa;
	pa.gp = gp;
	pa.gx = grid[0];
	pa.gy = grid[1];
	pa.gz = grid[2];
	pa.n = n;
	if (n) k_bounds<<<blocks_for(n), kNT, 0, s>>>(n, aabb, stats, pa, zero);
}

void launch_replan(uint64_t n, const BpBuffers &b, const GridParams &gp, cudaStream_t s) {
	PlanArgs pa;
	pa.gp = gp;
	pa.n = n;
	k_replan<<<1, 1, 0, s>>>(b.stats, pa);
}

void launch_count(uint64_t n, float *aabb, const BpBuffers &b, cudaStream_t s, bool shift) {
	if (!n) return;
	const auto k = b.sm.plans ? k_count<true> : k_count<false>;
	launch_pdl(k, dim3(blocks_for(n)), dim3(kNT), 0, s, n, aabb, b.stats, b.cell_count, b.owner_count, b.sm, b.owner_shift,
	           b.owner_cursor, shift ? 1 : 0);
}

void launch_link(uint64_t n, float *aabb, const BpBuffers &b, cudaStream_t s, bool shift) {
	if (!n) return;
	const auto k = b.sm.plans ? k_link<true> : k_link<false>;
	launch_pdl(k, dim3(blocks_for(n)), dim3(kNT), 0, s, n, aabb, b.stats, b.cell_count, b.entries, b.entry_cap, b.extra_body,
	           b.owner_count, b.sm, b.owner_shift, b.owner_cursor, shift ? 1 : 0);
}

void launch_shift(uint64_t n, float *aabb, const BpBuffers &b, cudaStream_t s, bool shift) {
	launch_pdl(k_shift, dim3(blocks_for(6 * n)), dim3(kNT), 0, s, n, aabb, b.stats, b.owner_count, b.owner_cursor,
	           (uint32_t)owner_buckets(n, b.owner_shift), shift ? 1 : 0);
}

void launch_all_pairs(uint64_t n, const float *aabb, const BpBuffers &b, cudaStream_t s) {
	launch_pdl(k_all_pairs, dim3(blocks_for(n), (unsigned)((n + kAllCols - 1) / kAllCols)), dim3(kNT), 0, s, (uint32_t)n,
	           b.stats, aabb, b.owner_count, b.pairs_tmp, b.pair_cap, b.owner_shift);
}

void launch_chain_check(const BpBuffers &b, uint32_t g_max, cudaStream_t s) {
	launch_pdl(k_chain_check, dim3((unsigned)std::min<uint64_t>(blocks_for(g_max), kNumSMs * 8)), dim3(kNT), 0, s, b.stats,
	           (uint64_t)g_max, b.cell_count, b.entries, b.entry_cap);
}

void launch_walk(uint64_t n, const BpBuffers &b, uint64_t entries_hint, cudaStream_t s) {
	if (!n) return;
	const auto k = b.sm.plans ? k_walk<true> : k_walk<false>;
	static const int per_sm = [] {
		int v = 0;
		if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, k_walk<false>, kNT, 0) != cudaSuccess || v < 1) v = 1;
		return v;
	}();
	const unsigned grid = (unsigned)std::min<uint64_t>(std::max<uint64_t>(blocks_for(entries_hint), 1), (uint64_t)kNumSMs * per_sm);
	launch_pdl(k, dim3(grid), dim3(kNT), 0, s, n, b.stats, b.entries, b.entry_cap, b.extra_body, b.owner_count, b.pairs_tmp,
	           b.pair_cap, b.sm, b.owner_shift);
}

// ---------------------------------------------------------------- cell offsets
// The cell offsets as one cooperative launch (reduce, one grid barrier, scan):
// each block sums its contiguous chunk of the counts, waits at the barrier,
// adds up the sums of the blocks before it (at most kScanCoopBlocks words)
// and scans its chunk on top, zeroing the counts behind it for the scatter's
// cursors. The single-pass look-back scan spent 13 us of a 1M-body step here
// almost entirely waiting (1 % SM throughput): its tiles wait on one another
// at L2 latency, the barrier is one round trip for the whole grid.
constexpr int kCsNT = 256, kCsIPT = 4, kCsTile = kCsNT * kCsIPT;
__global__ void __launch_bounds__(kCsNT) k_scan_cells_coop(DevStats *stats, uint32_t g_max, uint32_t *__restrict__ counts,
                                                         uint32_t *__restrict__ start,
                                                         unsigned long long *__restrict__ bsum,
                                                         unsigned long long *__restrict__ cs) {
	__shared__ unsigned long long sm[40];
	const uint64_t n = min((uint64_t)g_max, (uint64_t)stats->cells);
	const uint64_t per = ((n + gridDim.x - 1) / gridDim.x + kCsTile - 1) / kCsTile * kCsTile;
	const uint64_t lo = min(n, (uint64_t)blockIdx.x * per), hi = min(n, lo + per);
	unsigned long long part = 0;
	for (uint64_t i0 = lo + threadIdx.x; i0 < hi; i0 += 8 * kCsNT) {  // 8 loads in flight
		uint32_t v[8];
#pragma unroll
		for (int q = 0; q < 8; q++) v[q] = i0 + q * kCsNT < hi ? counts[i0 + q * kCsNT] : 0u;
#pragma unroll
		for (int q = 0; q < 8; q++) part += v[q];
	}
	unsigned long long total;
	(void)block_excl_scan<unsigned long long, kCsNT>(part, sm, &total);
	if (threadIdx.x == 0) bsum[blockIdx.x] = total;
	grid_barrier(reinterpret_cast<GridBarrier *>(stats->bar_scan), &stats->err);
	unsigned long long before = 0;
	for (uint32_t j = threadIdx.x; j < blockIdx.x; j += kCsNT) before += __ldcg(bsum + j);
	unsigned long long run_total;
	(void)block_excl_scan<unsigned long long, kCsNT>(before, sm, &run_total);
	for (uint64_t t0 = lo; t0 < hi; t0 += kCsTile) {
		const uint64_t i = t0 + (uint64_t)threadIdx.x * kCsIPT;
		uint32_t v[kCsIPT] = {0u, 0u, 0u, 0u};
		const bool full = i + kCsIPT <= hi;
		if (full) {
			const uint4 q = *reinterpret_cast<const uint4 *>(counts + i);
			v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
			*reinterpret_cast<uint4 *>(counts + i) = make_uint4(0u, 0u, 0u, 0u);
		} else {
#pragma unroll
			for (int j = 0; j < kCsIPT; j++)
				if (i + j < hi) {
					v[j] = counts[i + j];
					counts[i + j] = 0u;
				}
		}
		unsigned long long tile_total;
		const unsigned long long excl =
		    block_excl_scan<unsigned long long, kCsNT>((unsigned long long)v[0] + v[1] + v[2] + v[3], sm, &tile_total);
		uint32_t o[kCsIPT];
		unsigned long long r = run_total + excl;
#pragma unroll
		for (int j = 0; j < kCsIPT; j++) {
			o[j] = (uint32_t)r;
			r += v[j];
		}
		if (full) {
			*reinterpret_cast<uint4 *>(start + i) = make_uint4(o[0], o[1], o[2], o[3]);
		} else {
#pragma unroll
			for (int j = 0; j < kCsIPT; j++)
				if (i + j < hi) start[i + j] = o[j];
		}
		if (cs) {
#pragma unroll
			for (int j = 0; j < kCsIPT; j++)
				if (i + j < hi) cs[i + j] = (unsigned long long)o[j] << 32;
		}
		run_total += tile_total;
	}
	// the block whose chunk ends the counts (block 0 when there are none)
	// writes the end offset and the entry total
	if (threadIdx.x == 0 && hi == n && (lo < hi || (n == 0 && blockIdx.x == 0))) {
		start[n] = (uint32_t)run_total;
		stats->entries = run_total;
	}
}

void launch_scan_cells(const BpBuffers &b, uint32_t g_max, cudaStream_t s) {
	// the scan leaves the counts zeroed: they are the scatter's cursors
	if (b.scan_bsum) {
		static const int per_sm = [] {
			int v = 0;
			if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, k_scan_cells_coop, kCsNT, 0) != cudaSuccess || v < 1) v = 1;
			return v;
		}();
		const unsigned grid = (unsigned)std::max<uint64_t>(
		    1, std::min<uint64_t>((uint64_t)g_max / (8 * kCsTile), std::min<uint64_t>((uint64_t)per_sm * kNumSMs,
		                                                                               kScanCoopBlocks)));
		DevStats *st = b.stats;
		uint32_t gm = g_max, *cnt = b.cell_count, *start = b.cell_start;
		unsigned long long *bs = b.scan_bsum, *cs = b.cell_cs;
		void *args[] = {&st, &gm, &cnt, &start, &bs, &cs};
		cudaLaunchCooperativeKernel((const void *)k_scan_cells_coop, dim3(grid), dim3(kCsNT), args, 0, s);
		return;
	}
	launch_scan_u32_to_u32(b.cell_count, g_max, b.cell_start, b.status, b.ticket, &b.stats->err, s, &b.stats->cells,
	                       &b.stats->entries, b.pre_zeroed, b.cell_count);
}

void launch_scatter(uint64_t n, const float *aabb, const BpBuffers &b, cudaStream_t s, bool packed) {
	if (!n) return;
	unsigned long long *cs = packed ? b.cell_cs : nullptr;
	if (b.sm.plans)
		launch_pdl(k_scatter<true>, dim3(blocks_for(n)), dim3(kNT), 0, s, n, aabb, b.stats, b.cell_start, b.cell_count,
		           b.entries, b.entry_cap, &b.stats->err, b.sm, cs);
	else
		launch_pdl(k_scatter<false>, dim3(blocks_for(n)), dim3(kNT), 0, s, n, aabb, b.stats, b.cell_start, b.cell_count,
		           b.entries, b.entry_cap, &b.stats->err, b.sm, cs);
}

template <bool kBatch, int kWin>
void pair_test_as(const BpBuffers &b, unsigned grid, cudaStream_t s) {
	launch_pdl((k_pair_test<kBatch, kWin>), dim3(grid), dim3(kNT), 0, s, b.stats, b.cell_start, b.entries, b.entry_cap, b.owner_count,
	                                               b.pairs_tmp, b.pair_cap, b.dense ? &b.stats->tmp_pairs : &b.stats->pairs, b.sm,
	                                               b.dense, b.dense_cap, &b.stats->dense_items, &b.stats->mask_words, &b.stats->err, b.dense_cell,
	                                               b.owner_shift);
}
template <bool kBatch>
void pair_test_window(const BpBuffers &b, unsigned grid, cudaStream_t s) {
	switch (b.pair_window) {
	case 64: pair_test_as<kBatch, 64>(b, grid, s); break;
	case 128: pair_test_as<kBatch, 128>(b, grid, s); break;
	default: pair_test_as<kBatch, kWinDefault>(b, grid, s); break;
	}
}

// Persistent blocks over the device-side work items of the dense cells.
template <class K>
unsigned dense_grid(K kernel) {
	int v = 0;
	if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, kernel, kNT, 0) != cudaSuccess || v < 1) v = 1;
	return (unsigned)kNumSMs * v;
}

void launch_pair_test(uint64_t n, const BpBuffers &b, uint64_t entries_hint, cudaStream_t s) {
	(void)n;
	uint64_t want = (entries_hint + kNT - 1) / kNT;
	const uint64_t per_sm = b.pair_blocks_per_sm > 0 ? (uint64_t)b.pair_blocks_per_sm : 8;
	unsigned grid = (unsigned)std::min<uint64_t>(std::max<uint64_t>(want, 1), (uint64_t)kNumSMs * per_sm);
	if (b.sm.plans)
		pair_test_window<true>(b, grid, s);
	else
		pair_test_window<false>(b, grid, s);
	if (!b.dense) return;
	static const unsigned g_order = dense_grid(k_dense_order<true>), g_test = dense_grid(k_dense_test<false>);
	launch_pdl(b.sm.plans ? k_dense_order<true> : k_dense_order<false>, dim3(g_order), dim3(kNT), 0, s, b.stats, b.cell_start, b.entries,
	           b.entry_cap, b.sorted, b.sorted_body, b.sm, b.dense, b.dense_cap);
	launch_pdl(k_dense_test<false>, dim3(g_test), dim3(kNT), 0, s, b.stats, b.cell_start, b.sorted, b.entry_cap, b.owner_count,
	           b.row_count, b.dense, b.dense_cap, b.owner_shift, b.masks, b.mask_cap, (const unsigned long long *)nullptr,
	           (unsigned long long *)nullptr);
}

void launch_scan_owner(uint64_t n, const BpBuffers &b, cudaStream_t s) {
	launch_scan_u32_to_u64(b.owner_count, owner_buckets(n, b.owner_shift), b.owner_off, b.status2 ? b.status2 : b.status,
	                       b.ticket2 ? b.ticket2 : b.ticket, &b.stats->err, s, nullptr, nullptr, b.pre_zeroed);
}

void launch_owner_scatter(uint64_t out_cap, unsigned long long *out, const BpBuffers &b, cudaStream_t s) {
	const uint64_t bound = std::min<uint64_t>(b.pair_cap, out_cap);
	const unsigned grid = (unsigned)std::min<uint64_t>(std::max<uint64_t>(blocks_for(bound), 1), (uint64_t)kNumSMs * 8);
	launch_pdl(k_owner_scatter, dim3(grid), dim3(kNT), 0, s, b.stats, b.dense ? &b.stats->tmp_pairs : &b.stats->pairs, b.pair_cap,
	           out_cap, b.pairs_tmp, b.owner_off, b.owner_count, out, b.owner_shift);
	if (!b.dense) return;
	static const unsigned g_emit = dense_grid(k_dense_emit), g_test = dense_grid(k_dense_test<true>);
	launch_pdl(k_dense_emit, dim3(g_emit), dim3(kNT), 0, s, b.stats, b.cell_start, b.sorted_body, b.entry_cap, b.owner_count,
	           b.row_count, b.dense, b.dense_cap, b.owner_shift, b.masks, b.mask_cap, b.owner_off, out);
	launch_pdl(k_dense_test<true>, dim3(g_test), dim3(kNT), 0, s, b.stats, b.cell_start, b.sorted, b.entry_cap, b.owner_count,
	           b.row_count, b.dense, b.dense_cap, b.owner_shift, b.masks, b.mask_cap, b.owner_off, out);
}

void launch_segsort(uint64_t n, unsigned long long *out, const BpBuffers &b, cudaStream_t s) {
	const uint64_t nbk = owner_buckets(n, b.owner_shift);
	const KeyPack kp{b.owner_shift, b.key_bits};
	launch_pdl(kp.shift ? k_segsort<true> : k_segsort<false>, dim3(blocks_for(nbk)), dim3(kNT), 0, s, nbk, b.owner_off, out,
	           b.big_list, b.big_cap, b.stats, kp);
}

// Opts two kernels into `bytes` of dynamic shared memory (above 48 KB) on the current
// device, once for each: the attribute is the device's. done: a bit per device.
template <class K>
void opt_in_shared(std::atomic<uint64_t> &done, int bytes, K a, K b) {
	int dev = 0;
	if (cudaGetDevice(&dev) != cudaSuccess) return;  // the launch tells
	const uint64_t bit = dev < 64 ? (uint64_t)1 << dev : 0;
	if (done.load(std::memory_order_acquire) & bit) return;
	if (cudaFuncSetAttribute(a, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess &&
	    cudaFuncSetAttribute(b, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess)
		done.fetch_or(bit, std::memory_order_release);
}

void launch_segsort_mid(unsigned long long *out, const BpBuffers &b, cudaStream_t s) {
	const KeyPack kp{b.owner_shift, b.key_bits};
	if (b.dense) {  // rows of dense cells arrive as ascending runs
		constexpr int bytes = 2 * kMergeSeg * (int)sizeof(uint32_t);  // 64 KB: three blocks fit on an SM
		static std::atomic<uint64_t> done{0};
		opt_in_shared(done, bytes, k_segsort_runs<true>, k_segsort_runs<false>);
		launch_pdl(kp.shift ? k_segsort_runs<true> : k_segsort_runs<false>, dim3(kNumSMs * 3), dim3(kNT), bytes, s, b.stats,
		           b.big_cap, b.big_list, b.owner_off, out, kp);
	}
	if (kp.shift)
		launch_pdl(k_segsort_mid<true>, dim3(kNumSMs * 6), dim3(kMidNT), 0, s, b.stats, b.big_cap, b.big_list, b.owner_off,
		           out, kp);
	else
		launch_pdl(k_segsort_mid<false>, dim3(kNumSMs * 6), dim3(kMidNT), 0, s, b.stats, b.big_cap, b.big_list, b.owner_off,
		           out, kp);
}
void launch_segsort_big(unsigned long long *out, const BpBuffers &b, cudaStream_t s) {
	static std::atomic<uint64_t> done{0};
	opt_in_shared(done, kBigSeg * (int)sizeof(uint32_t), k_segsort_big<true>, k_segsort_big<false>);
	// 64 KB of shared memory a block: three blocks fit on an SM
	const KeyPack kp{b.owner_shift, b.key_bits};
	if (kp.shift)
		launch_pdl(k_segsort_big<true>, dim3(kNumSMs * 3), dim3(512), kBigSeg * sizeof(uint32_t), s, b.stats, b.big_cap,
		           b.big_list, b.owner_off, out, kp);
	else
		launch_pdl(k_segsort_big<false>, dim3(kNumSMs * 3), dim3(512), kBigSeg * sizeof(uint32_t), s, b.stats, b.big_cap,
		           b.big_list, b.owner_off, out, kp);
}

bool fused_sort_fits(uint64_t buckets) { return buckets >= 1 && buckets <= kFusedBuckets; }
bool fused_sort_enabled() {
	static const bool on = [] {
		const char *v = getenv("CC_FUSED_SORT");
		return !(v && v[0] == '0');
	}();
	return on;
}

void launch_owner_sort_fused(uint64_t n, uint64_t out_cap, unsigned long long *out, uint64_t P_hint, const BpBuffers &b,
                             uint32_t *host_stats, cudaStream_t s) {
	const uint32_t nbk = (uint32_t)owner_buckets(n, b.owner_shift);
	const size_t smem = sizeof(uint32_t) * ((size_t)nbk + 1 + kFusedSeg);
	static std::atomic<uint64_t> done{0};
	opt_in_shared(done, (int)(sizeof(uint32_t) * ((size_t)kFusedBuckets + 1 + kFusedSeg)), k_owner_sort_fused<true>,
	              k_owner_sort_fused<false>);
	// one block an SM at most: every block scans all bucket counts, and the MPR's blocks run beside these
	const uint64_t want = (std::max<uint64_t>(P_hint, nbk) + kFusedNT - 1) / kFusedNT;
	const unsigned grid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(want, kNumSMs));
	uint64_t pair_cap = b.pair_cap;
	const unsigned long long *tmp = b.pairs_tmp;
	const uint32_t *cnt = b.owner_count;
	uint32_t *cur = b.owner_cursor;
	int oshift = b.owner_shift;
	KeyPack kp{b.owner_shift, b.key_bits};
	DevStats *st = b.stats;
	void *args[] = {&st, &pair_cap, &out_cap, &tmp, &cnt, &cur, (void *)&nbk, &out, &oshift, &kp, &host_stats};
	const void *k = kp.shift ? (const void *)k_owner_sort_fused<true> : (const void *)k_owner_sort_fused<false>;
	cudaLaunchCooperativeKernel(k, dim3(grid), dim3(kFusedNT), args, smem, s);
}

void launch_ref_count(uint64_t n, const float *aabb_shifted, const DevStats *stats, uint32_t *cnt, cudaStream_t s) {
	if (n) k_ref_count<<<blocks_for(n), kNT, 0, s>>>(n, aabb_shifted, stats, cnt);
}
void launch_ref_emit(uint64_t n, const float *aabb_shifted, DevStats *stats, const unsigned long long *off,
                     unsigned long long *keys, uint64_t cap, cudaStream_t s) {
	if (n) k_ref_emit<<<blocks_for(n), kNT, 0, s>>>(n, aabb_shifted, stats, off, keys, cap);
}
void launch_ref_flags(const unsigned long long *keys, uint64_t E, uint32_t *flags, cudaStream_t s) {
	if (E) k_ref_flags<<<blocks_for(E), kNT, 0, s>>>(keys, E, flags);
}
void launch_ref_split(const unsigned long long *keys, uint64_t E, const uint32_t *run_pos, uint32_t *bin_number,
                      uint32_t *body_number, uint32_t *active_bins, uint32_t *bin_end, uint64_t cap_a,
                      cudaStream_t s) {
	if (E)
		k_ref_split<<<blocks_for(E), kNT, 0, s>>>(keys, E, run_pos, bin_number, body_number, active_bins, bin_end,
		                                          cap_a);
}

}  // namespace cc
