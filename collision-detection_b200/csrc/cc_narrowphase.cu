// Narrowphase: the reference's Narrowphase::DoNarrowphase
// (src/narrowphase/Narrowphase.cu:316-595) as sm_100a kernels.
//
// k_mpr: the MPR state machine of cc_mpr.cuh on persistent lanes fed from a
// queue of pair indices grouped by shape-type combination (k_np_classes);
// the exact mode has its own kernel and takes the pairs as they come.
// Sphere-sphere pairs take the analytic branch (:382-397); every other pair
// runs Minkowski portal refinement (CollideAndFindPoint :122-314) with the
// same branch structure, iteration caps (35 discovery, 35 refinement) and
// termination rule (delta <= 1e-20, depth <= 0).
//
// Precision (the portal arithmetic is FP64 in all three):
//  0 exact  (cc_mpr_exact.cu, -fmad=false): the reference's arithmetic in
//           double, world frame — equal to the FP64 oracle, rounded to float;
//  1 fp64   (k_mpr<double>): pair-local frame (origin = body A's position),
//           rsqrt normalization, fused multiply-add;
//  2 mixed  (k_mpr<float>): as fp64 with FP32 support maps.
//
// k_np_classes: the pairs grouped by shape-type class (counting sort), and
// k_np_compact: the stable hit-first ordering of :580-593
// (thrust::sort_by_key on the 0/1 flag) as a scan + scatter, the pair keys
// permuted the same way; each is one cooperative launch with a grid barrier.
#include <algorithm>

#include "cc_common.cuh"
#include "cc_internal.h"
#include "cc_math.cuh"
#include "cc_mpr.cuh"

namespace cc {

namespace {
constexpr int kNT = 64;  // MPR: few, long-running threads; small blocks spread them over all SMs

template <class S>
__global__ void __launch_bounds__(kNT, 6) k_mpr(uint64_t P_cap, const unsigned long long *P_dev, uint64_t n,
                                              const int32_t *__restrict__ T, const float *__restrict__ A,
                                              const float *__restrict__ B, const float *__restrict__ C,
                                              const float *__restrict__ R, const uint32_t *__restrict__ ID,
                                              uint64_t nb, const uint8_t *__restrict__ active,
                                              const float *__restrict__ pos, const float *__restrict__ rot,
                                              float envelope, const long long *__restrict__ pairs, NpScratch sc) {
	pdl_begin();
	mpr::run<S, kNT>(P_cap, P_dev, n, T, A, B, C, R, ID, nb, active, pos, rot, envelope, pairs, sc,
	                        sc.classes + 2 * kNpClasses);
}

// Pairs grouped by (type A, type B) so that the threads of a warp run the
// same support maps: a counting sort of the pair indices by class.
__device__ __forceinline__ uint32_t pair_class(uint64_t i, uint64_t n, const int32_t *T, const long long *pairs) {
	const uint64_t key = (uint64_t)pairs[i];
	const uint64_t a = key >> 32, b = key & 0xffffffffull;
	if (a >= n || b >= n) return kNpClasses - 1;
	const int ta = __ldg(T + a), tb = __ldg(T + b);
	if (ta < 0 || ta > 6 || tb < 0 || tb > 6) return kNpClasses - 1;
	return (uint32_t)(ta * 7 + tb);
}

// Relative MPR cost of a shape type: smooth surfaces refine longest.
__device__ __forceinline__ int type_cost(int t) {
	switch (t) {
	case SPHERE: return 1;
	case BOX: return 2;
	case CYLINDER: return 3;
	case ELLIPSOID: return 4;
	default: return 2;
	}
}
// Sphere-sphere pairs take the analytic path and invalid pairs do nothing:
// cost 0.
__device__ __forceinline__ int class_cost(int c) {
	if (c >= 49) return 0;
	const int ta = c / 7, tb = c % 7;
	if (ta == SPHERE && tb == SPHERE) return 0;
	return type_cost(ta) + type_cost(tb);
}

// The class grouping as one cooperative launch: every block counts the classes
// of its pairs (shared-memory histogram, one global atomic per class and
// block), a grid barrier, then every block derives the class offsets (longest
// classes first) and places its pairs, one cursor atomic per class and tile.
constexpr int kCoopNT = 256;
__global__ void __launch_bounds__(kCoopNT) k_np_classes(uint64_t P_cap, const unsigned long long *P_dev, uint64_t n,
                                                         const int32_t *__restrict__ T,
                                                         const long long *__restrict__ pairs, uint32_t *classes,
                                                         uint32_t *__restrict__ order, GridBarrier *bar,
                                                         uint32_t *err) {
	__shared__ uint32_t h[kNpClasses], off[kNpClasses], base[kNpClasses];
	__shared__ int cost[kNpClasses];
	const uint64_t P = P_dev ? min(P_cap, (uint64_t)*P_dev) : P_cap;
	if (threadIdx.x < kNpClasses) h[threadIdx.x] = 0;
	__syncthreads();
	const uint64_t step = (uint64_t)gridDim.x * kCoopNT;
	for (uint64_t i = (uint64_t)blockIdx.x * kCoopNT + threadIdx.x; i < P; i += step)
		atomicAdd(&h[pair_class(i, n, T, pairs)], 1u);
	__syncthreads();
	if (threadIdx.x < kNpClasses && h[threadIdx.x]) atomicAdd(&classes[threadIdx.x], h[threadIdx.x]);
	grid_barrier(bar, err);
	if (threadIdx.x < kNpClasses) {
		h[threadIdx.x] = __ldcg(&classes[threadIdx.x]);
		cost[threadIdx.x] = class_cost(threadIdx.x);
	}
	__syncthreads();
	if (threadIdx.x < kNpClasses) {
		const int c = threadIdx.x, k = cost[c];
		uint32_t acc = 0;
		for (int d = 0; d < kNpClasses; d++)
			if (cost[d] > k || (cost[d] == k && d < c)) acc += h[d];
		off[c] = acc;
	}
	uint32_t *cursor = classes + kNpClasses;
	for (uint64_t i0 = (uint64_t)blockIdx.x * kCoopNT; i0 < P; i0 += step) {
		__syncthreads();
		if (threadIdx.x < kNpClasses) h[threadIdx.x] = 0;
		__syncthreads();
		const uint64_t i = i0 + threadIdx.x;
		uint32_t c = 0, r = 0;
		if (i < P) {
			c = pair_class(i, n, T, pairs);
			r = atomicAdd(&h[c], 1u);
		}
		__syncthreads();
		if (threadIdx.x < kNpClasses && h[threadIdx.x]) base[threadIdx.x] = atomicAdd(&cursor[threadIdx.x], h[threadIdx.x]);
		__syncthreads();
		if (i < P) order[off[c] + base[c] + r] = (uint32_t)i;
	}
}

// ---------------------------------------------------------------- compaction
// Hit-first stable compaction in one cooperative launch: block b owns the contiguous chunk b
// of the results; it counts its hits, a barrier over the grid, then it adds the
// counts of the blocks before it and ranks its chunk's hits tile by tile. A pass's
// list is short, so all of it is latency: chains of dependent loads, the barrier,
// the launch. Where a chunk is one tile (the grids below make it so) every thread
// has its row in registers before the barrier and only writes behind it, and the
// block's sums take two block barriers. A step of 1M mixed shapes (25K pairs) 191.5
// -> 181.4 us, 130K 105 -> 97, a batch of 64 285 -> 278, 500K stepping 158 -> 150.
// (As one cluster of 16 blocks, with its cheaper barrier: up to 1.5 us less below
// 16K pairs, 9 more at 25K.)

// Sums of a and b over the block, in every thread (sm: 64 words).
__device__ __forceinline__ void block_sum2(unsigned long long &a, unsigned long long &b, unsigned long long *sm) {
	constexpr int NW = kCoopNT / 32;
	const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
	for (int d = 16; d; d >>= 1) {
		a += __shfl_xor_sync(0xffffffffu, a, d);
		b += __shfl_xor_sync(0xffffffffu, b, d);
	}
	if (l == 0) {
		sm[w] = a;
		sm[32 + w] = b;
	}
	__syncthreads();
	a = l < NW ? sm[l] : 0ull;
	b = l < NW ? sm[32 + l] : 0ull;
	for (int d = 16; d; d >>= 1) {
		a += __shfl_xor_sync(0xffffffffu, a, d);
		b += __shfl_xor_sync(0xffffffffu, b, d);
	}
	__syncthreads();
}

// Hits of the block's threads before this one, and of the block (sm: 32 words).
__device__ __forceinline__ uint32_t block_rank(bool f, uint32_t *sm, uint32_t &total) {
	constexpr int NW = kCoopNT / 32;
	const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
	const uint32_t m = __ballot_sync(0xffffffffu, f);
	if (l == 0) sm[w] = __popc(m);
	__syncthreads();
	const uint32_t v = l < NW ? sm[l] : 0u;
	total = __reduce_add_sync(0xffffffffu, v);
	const uint32_t r = __reduce_add_sync(0xffffffffu, l < w ? v : 0u) + __popc(m & ((1u << l) - 1u));
	__syncthreads();
	return r;
}

// One result row.
struct ContactRow {
	float v[10];
	int32_t ida, idb;
};
__device__ __forceinline__ ContactRow load_row(const NpScratch &sc, uint64_t t) {
	ContactRow r;
#pragma unroll
	for (int d = 0; d < 3; d++) {
		r.v[d] = sc.norm[3 * t + d];
		r.v[3 + d] = sc.pa[3 * t + d];
		r.v[6 + d] = sc.pb[3 * t + d];
	}
	r.v[9] = sc.depth[t];
	r.ida = sc.ids[2 * t];
	r.idb = sc.ids[2 * t + 1];
	return r;
}

constexpr uint32_t kNoHit = 0xffffffffu;

// Contact hash: the row of a pair's result, kNoHit where it is no contact.
__device__ __forceinline__ uint32_t hash_find(const NpScratch &sc, unsigned long long key) {
	const unsigned long long tag = key + 1ull;
	uint64_t h = contact_slot(tag);
	for (uint64_t probe = 0; probe <= sc.hmask && probe < 256; probe++, h++) {
		const unsigned long long v = __ldcg(&sc.hkeys[h & sc.hmask]);
		if (v == tag) return __ldcg(&sc.hvals[h & sc.hmask]);
		if (v == 0ull) break;
	}
	return kNoHit;
}

// kSorted: the MPR ran on the unsorted pairs (overlapped with their sort) and each
// sorted key in `pairs` finds its result through the contact hash; else results
// and sc.pairs are in pair order. tmp: receives the sorted keys.
template <bool kSorted>
__global__ void __launch_bounds__(kCoopNT) k_np_compact(uint64_t P_cap, const unsigned long long *P_dev, NpScratch sc,
                                                   long long *__restrict__ pairs, unsigned long long *__restrict__ tmp,
                                                   float *__restrict__ norm, float *__restrict__ cpta,
                                                   float *__restrict__ cptb, float *__restrict__ depth,
                                                   int32_t *__restrict__ bids, unsigned long long *contacts_out) {
	__shared__ unsigned long long sm[64];
	const uint64_t P = P_dev ? min(P_cap, (uint64_t)*P_dev) : P_cap;
	const uint64_t chunk = (P + gridDim.x - 1) / gridDim.x;
	const uint64_t c0 = min((uint64_t)blockIdx.x * chunk, P), c1 = min(c0 + chunk, P);
	const bool one = chunk <= kCoopNT;
	unsigned long long cnt = 0, unused = 0;
	unsigned long long key = 0;
	uint64_t t = kNoHit;
	ContactRow row = {};
	for (uint64_t i = c0 + threadIdx.x; i < c1; i += kCoopNT) {
		key = kSorted ? (unsigned long long)pairs[i] : sc.pairs[i];
		bool hit;
		if constexpr (kSorted) {
			t = hash_find(sc, key);
			hit = t != kNoHit;
			tmp[i] = key;  // also where the block does not read it again: a full hash has the sorted list restored from it
			if (!one) sc.order[i] = (uint32_t)t;
		} else {
			hit = sc.flag[i] != 0;
			t = hit ? i : (uint64_t)kNoHit;
		}
		if (one && hit) row = load_row(sc, t);
		cnt += hit ? 1ull : 0ull;
	}
	bool hit = kSorted ? t != kNoHit : cnt != 0;  // one tile
	block_sum2(cnt, unused, sm);
	if (threadIdx.x == 0) sc.block_sums[blockIdx.x] = cnt;
	grid_barrier(reinterpret_cast<GridBarrier *>(sc.bar_compact), sc.err);
	// hits before this block's, and all, from the per-block counts
	unsigned long long run = 0, nh = 0;
	for (uint32_t b = threadIdx.x; b < gridDim.x; b += kCoopNT) {
		const unsigned long long v = __ldcg(&sc.block_sums[b]);
		nh += v;
		if (b < blockIdx.x) run += v;
	}
	block_sum2(run, nh, sm);
	if (blockIdx.x == 0 && threadIdx.x == 0 && contacts_out) *contacts_out = nh;
	report_by_last(sc.stats, sc.host_stats);
	for (uint64_t t0 = c0; t0 < c1; t0 += kCoopNT) {
		const uint64_t i = t0 + threadIdx.x;
		if (!one && i < c1) {
			if constexpr (kSorted) {
				key = tmp[i];
				t = sc.order[i];
				hit = t != kNoHit;
			} else {
				key = sc.pairs[i];
				t = i;
				hit = sc.flag[i] != 0;
			}
			if (hit) row = load_row(sc, t);
		}
		uint32_t tile_total;
		const uint32_t r = block_rank(i < c1 && hit, reinterpret_cast<uint32_t *>(sm), tile_total);
		if (i < c1) {
			const uint64_t j = run + r;
			if (hit) {
				pairs[j] = (long long)key;
#pragma unroll
				for (int d = 0; d < 3; d++) {
					norm[3 * j + d] = row.v[d];
					cpta[3 * j + d] = row.v[3 + d];
					cptb[3 * j + d] = row.v[6 + d];
				}
				depth[j] = row.v[9];
				bids[2 * j] = row.ida;
				bids[2 * j + 1] = row.idb;
			} else {
				pairs[nh + (i - j)] = (long long)key;
			}
		}
		run += tile_total;
	}
}

// Short lists (kRankPairs expected, kRankRoom at most): with the miss bit above the
// pair, the final order is that of the keys, and a row's place is the number of
// smaller keys. Every block holds all keys in shared memory; a warp counts for
// kRankRows rows at once, 32 keys a step. P^2 compares, but no sort, no hash and no
// barrier over the grid, and the MPR has the
// chip for itself. Steps with the sort and the compaction by the hash, and with
// this, us: 16K spheres (600 pairs) 57 and 44, 1K bodies (2K pairs) 95 and 85, 130K
// bodies (3.4K pairs) 97 and 86. The counting itself takes 2, 4 and 7 us, the
// compaction it replaces 6: above kRankPairs the sort beside the MPR is faster.
constexpr int kRankNT = 256, kRankRows = 2;
__global__ void __launch_bounds__(kRankNT) k_np_rank(DevStats *stats, uint64_t pair_cap, uint64_t out_cap, NpScratch sc,
                                                     uint32_t room, long long *__restrict__ pairs, float *__restrict__ norm,
                                                     float *__restrict__ cpta, float *__restrict__ cptb,
                                                     float *__restrict__ depth, int32_t *__restrict__ bids) {
	pdl_begin();
	// the pass's counters, final once the first block has added its own, to the host
	const auto report = [&] {
		if (blockIdx.x != 0 || !sc.host_stats) return;
		__syncthreads();
		report_stats(stats, sc.host_stats);
	};
	constexpr unsigned long long kMiss = 1ull << 63;
	extern __shared__ unsigned long long rank_keys[];
	const unsigned long long P = stats->pairs;
	const bool fits = P <= pair_cap && P <= out_cap, first = blockIdx.x == 0 && threadIdx.x == 0;
	if (first) {
		stats->np_n = fits ? P : 0ull;
		if (fits && P > room) atomicOr(&stats->err, (uint32_t)kErrLongList);
		__threadfence();
	}
	if (!fits || P > room) return report();
	const uint32_t n = (uint32_t)P, padded = (n + 31u) & ~31u;
	uint32_t hits = 0;
	for (uint32_t i0 = threadIdx.x; i0 < padded; i0 += 8 * kRankNT) {  // eight keys a thread in flight
		unsigned long long key[8];
		uint32_t flag[8];
#pragma unroll
		for (int r = 0; r < 8; r++) {
			const uint32_t i = i0 + r * kRankNT;
			key[r] = i < n ? sc.pairs[i] : ~0ull;
			flag[r] = i < n ? sc.flag[i] : 0u;
		}
#pragma unroll
		for (int r = 0; r < 8; r++) {
			const uint32_t i = i0 + r * kRankNT;
			if (i < padded) rank_keys[i] = key[r] | (flag[r] ? 0ull : kMiss);
			hits += flag[r] ? 1u : 0u;
		}
	}
	hits = __reduce_add_sync(0xffffffffu, hits);
	const uint32_t lane = threadIdx.x & 31;
	if (blockIdx.x == 0 && lane == 0 && hits) {
		atomicAdd(&stats->contacts, (unsigned long long)hits);
		__threadfence();
	}
	__syncthreads();
	report();
	const uint32_t step = gridDim.x * (kRankNT / 32) * kRankRows;
	for (uint32_t i0 = (blockIdx.x * (kRankNT / 32) + (threadIdx.x >> 5)) * kRankRows; i0 < n; i0 += step) {
		unsigned long long own[kRankRows];
		uint32_t before[kRankRows];
		float v[kRankRows];
#pragma unroll
		for (int r = 0; r < kRankRows; r++) {
			const uint32_t i = i0 + r;
			own[r] = i < n ? rank_keys[i] : 0ull;
			before[r] = 0;
			v[r] = 0.f;
			if (i < n && !(own[r] & kMiss)) {
				if (lane < 3) v[r] = sc.norm[3 * i + lane];
				else if (lane < 6) v[r] = sc.pa[3 * i + lane - 3];
				else if (lane < 9) v[r] = sc.pb[3 * i + lane - 6];
				else if (lane == 9) v[r] = sc.depth[i];
				else if (lane < 12) v[r] = __int_as_float(sc.ids[2 * i + lane - 10]);
			}
		}
#pragma unroll 4
		for (uint32_t j = lane; j < padded; j += 32) {
			const unsigned long long k = rank_keys[j];
#pragma unroll
			for (int r = 0; r < kRankRows; r++) before[r] += k < own[r] ? 1u : 0u;
		}
#pragma unroll
		for (int r = 0; r < kRankRows; r++) {
			const uint64_t at = __reduce_add_sync(0xffffffffu, before[r]);
			if (i0 + r >= n) continue;
			if (lane == 12) pairs[at] = (long long)(own[r] & ~kMiss);
			if (own[r] & kMiss) continue;
			if (lane < 3) norm[3 * at + lane] = v[r];
			else if (lane < 6) cpta[3 * at + lane - 3] = v[r];
			else if (lane < 9) cptb[3 * at + lane - 6] = v[r];
			else if (lane == 9) depth[at] = v[r];
			else if (lane < 12) bids[2 * at + lane - 10] = __float_as_int(v[r]);
		}
	}
}
}  // namespace

namespace {
template <class K>
int resident(K kernel) {
	int v = 0;
	if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, kernel, kNT, 0) != cudaSuccess || v < 1) v = 1;
	return v;
}
// Blocks of a fast MPR kernel (modes 1 and 2) resident per SM.
int mpr_resident_blocks(int precision) {
	static const int b[2] = {resident(k_mpr<double>), resident(k_mpr<float>)};
	return b[precision == 2 ? 1 : 0];
}

// Largest co-resident grid of a cooperative kernel of kCoopNT threads.
template <class K>
unsigned coop_blocks(K kernel) {
	int per_sm = 0, dev = 0, sms = kNumSMs;
	if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kCoopNT, 0) != cudaSuccess || per_sm < 1)
		per_sm = 1;
	if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
	return (unsigned)(per_sm * sms);
}

template <class... A>
void launch_coop(void (*k)(A...), unsigned grid, cudaStream_t s, A... args) {
	void *ptrs[] = {(void *)&args...};
	cudaLaunchCooperativeKernel((const void *)k, dim3(grid), dim3(kCoopNT), ptrs, 0, s);
}
}  // namespace

unsigned np_coop_max_blocks() {
	static const unsigned m = std::min(std::min(coop_blocks(k_np_classes), coop_blocks(k_np_compact<false>)),
	                                   coop_blocks(k_np_compact<true>));
	return m;
}

// Up to kUngrouped pairs a warp of the fast modes' grid has one or two, and grouping
// them costs more than their divergence (steps, us, grouped and not: 16K spheres with
// 600 pairs in fp64 56 and 44, 600 mixed shapes with 540 in fp64 81 and 77, in mixed
// 81 and 72; but 130K mixed shapes with 3.4K pairs in fp64 106 and 115).
constexpr uint64_t kUngrouped = 1024;
int mpr_launches(uint64_t P_cap, int precision, uint64_t P_hint) {
	return precision == 0 || std::min<uint64_t>(P_hint ? P_hint : P_cap, P_cap) <= kUngrouped ? 1 : 2;
}

void launch_mpr(uint64_t P_cap, const unsigned long long *P_dev, uint64_t n, const int32_t *T, const float *A,
                const float *B, const float *C, const float *R, const uint32_t *ID, uint64_t nb,
                const uint8_t *active, const float *pos, const float *rot, float envelope, const long long *pairs,
                const NpScratch &sc, int precision, uint64_t P_hint, cudaStream_t s, bool beside) {
	if (!P_cap) return;
	const uint64_t Pe = std::min<uint64_t>(P_hint ? P_hint : P_cap, P_cap);
	if (precision == 0) {
		// The exact kernel's lanes share one instruction sequence whatever their
		// types, so its pairs are not grouped by class (grouped: 4 us more at
		// 1,800 pairs, the same at 27,500 and 195,000). Grid: sixteen pairs a
		// warp; below two blocks per SM the pairs spread over that many blocks
		// instead, one warp per scheduler (3,400 pairs: 46 us with two blocks per
		// SM, 60 us with six), at most what is resident (27,500 pairs: 75 us with
		// six, 82 with three; 195,000: 239 with six, 373 with three).
		if (!sc.pre_zeroed) cudaMemsetAsync(sc.queue, 0, sizeof(uint32_t), s);
		const uint64_t want = std::max<uint64_t>((Pe + kNT / 2 - 1) / (kNT / 2), 2 * kNumSMs);
		launch_mpr_exact((unsigned)std::min<uint64_t>(want, (uint64_t)kNumSMs * mpr_exact_resident_blocks()), P_cap, P_dev, n,
		                 T, A, B, C, R, ID, nb, active, pos, rot, envelope, pairs, sc, s, beside);
		return;
	}
	NpScratch scm = sc;
	if (!sc.pre_zeroed) cudaMemsetAsync(sc.classes, 0, (2 * kNpClasses + 1) * sizeof(uint32_t), s);
	if (mpr_launches(P_cap, precision, P_hint) == 1) {
		scm.order = nullptr;
	} else {  // group the pairs by shape-type combination; the last word is the work queue
		// blocks for the expected pair count (the loops stride over the device count)
		const unsigned g = (unsigned)std::max<uint64_t>(
		    1, std::min<uint64_t>((Pe + kCoopNT - 1) / kCoopNT, std::min<uint64_t>(np_coop_max_blocks(), kNpCoopBlocks)));
		launch_coop(k_np_classes, g, s, P_cap, P_dev, n, T, pairs, sc.classes, sc.order,
		            reinterpret_cast<GridBarrier *>(sc.bar_classes), sc.err);
	}
	// persistent lanes: one per pair up to the resident limit, so that every
	// pair starts at once (the kernel is latency-bound: its time is the
	// longest pair's dependency chain); beyond that the queue balances
	const uint64_t want = (Pe + kNT - 1) / kNT;
	const unsigned grid = (unsigned)std::min<uint64_t>(std::max<uint64_t>(want, 2 * kNumSMs),
	                                                   (uint64_t)kNumSMs * mpr_resident_blocks(precision));
	if (precision == 2)
		launch_pdl(k_mpr<float>, dim3(grid), dim3(kNT), 0, s, P_cap, P_dev, n, T, A, B, C, R, ID, nb, active, pos, rot, envelope, pairs,
		           scm);
	else
		launch_pdl(k_mpr<double>, dim3(grid), dim3(kNT), 0, s, P_cap, P_dev, n, T, A, B, C, R, ID, nb, active, pos, rot, envelope, pairs,
		           scm);
}

void launch_np_compact(uint64_t P_cap, const unsigned long long *P_dev, const NpScratch &sc, long long *pairs,
                       float *norm, float *cpta, float *cptb, float *depth, int32_t *bids,
                       unsigned long long *contacts_out, uint64_t P_hint, cudaStream_t s) {
	if (!P_cap) {
		if (contacts_out) cudaMemsetAsync(contacts_out, 0, sizeof(unsigned long long), s);
		return;
	}
	// one block per 256 flags of the expected count (one tile each: the scan
	// and scatter of a tile are a chain of dependent loads), within the co-resident limit
	const uint64_t Pe = std::min<uint64_t>(P_hint ? P_hint : P_cap, P_cap);
	const unsigned grid = (unsigned)std::max<uint64_t>(
	    1, std::min<uint64_t>((Pe + kCoopNT - 1) / kCoopNT, std::min<uint64_t>(np_coop_max_blocks(), kNpCoopBlocks)));
	launch_coop(k_np_compact<false>, grid, s, P_cap, P_dev, sc, pairs, (unsigned long long *)nullptr, norm,
	            cpta, cptb, depth, bids, contacts_out);
}

void launch_np_compact_sorted(uint64_t P_cap, const unsigned long long *P_dev, const NpScratch &sc,
                              long long *pairs, unsigned long long *tmp, float *norm, float *cpta, float *cptb,
                              float *depth, int32_t *bids, unsigned long long *contacts_out, uint64_t P_hint,
                              cudaStream_t s) {
	if (!P_cap) {
		if (contacts_out) cudaMemsetAsync(contacts_out, 0, sizeof(unsigned long long), s);
		return;
	}
	const uint64_t Pe = std::min<uint64_t>(P_hint ? P_hint : P_cap, P_cap);
	const unsigned grid = (unsigned)std::max<uint64_t>(
	    1, std::min<uint64_t>((Pe + kCoopNT - 1) / kCoopNT, std::min<uint64_t>(np_coop_max_blocks(), kNpCoopBlocks)));
	launch_coop(k_np_compact<true>, grid, s, P_cap, P_dev, sc, pairs, tmp, norm, cpta, cptb, depth, bids,
	            contacts_out);
}

void launch_np_rank(DevStats *stats, uint64_t pair_cap, uint64_t out_cap, const NpScratch &sc, long long *pairs,
                    float *norm, float *cpta, float *cptb, float *depth, int32_t *bids, uint64_t P_hint, cudaStream_t s) {
	// keys for twice the expected count, within the 48 KB that need no opt-in (which is per device)
	const uint32_t room = (uint32_t)std::min<uint64_t>(kRankRoom, std::max<uint64_t>(1024, 2 * P_hint));
	constexpr unsigned rows = (kRankNT / 32) * kRankRows;
	const unsigned grid = (unsigned)std::max<uint64_t>(1, (std::min(P_hint, kRankRoom) + rows - 1) / rows);
	launch_pdl(k_np_rank, dim3(grid), dim3(kRankNT), room * sizeof(unsigned long long), s, stats, pair_cap, out_cap, sc, room, pairs, norm, cpta, cptb, depth, bids);
}

}  // namespace cc
