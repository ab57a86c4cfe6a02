// Batched scenes: many independent scenes collided by one pass of the
// pipeline. The batch is laid out as one concatenated scene (shapes
// [shape_off[s], shape_off[s+1]) and bodies [body_off[s], body_off[s+1]) of
// scene s); each scene gets the bounds, reference shift and search grid that
// a separate call would give it (Broadphase.cu:368-386 per scene), and the
// scenes' grids occupy disjoint global cell ranges, so no pair crosses scenes
// and every scene's pairs, shifted boxes and contacts equal those of a
// separate call. The pass starts with k_batch_front (cc_aabb.cu: scene lookup,
// gather, boxes, per-scene bounds and plans) and ends here (per-scene counts);
// the search kernels take the SceneMap built by the front. Also here: the time-
// step updates of served scenes and small host-to-device helpers.
//
// Compiled with -fmad=false, like the other front kernels.
#include "cc_common.cuh"
#include "cc_internal.h"
#include "cc_math.cuh"
#include "cc_stats.cuh"

namespace cc {

namespace {
constexpr int kNT = 256;

// Per-scene results from the final pair list (contacts' pairs first, both parts
// sorted): the pairs and contacts before a scene's first shape, by binary search
// in either part. Each block covers kNT - 1 scenes and the first bound of the next.
__device__ __forceinline__ void count_below(const unsigned long long *pairs, uint64_t P, uint64_t C,
                                            unsigned long long key, uint64_t &hits, uint64_t &misses) {
	uint64_t lo = 0, hi = C, lo2 = C, hi2 = P;
	while (lo < hi || lo2 < hi2) {  // side by side: two loads in flight
		const uint64_t mid = (lo + hi) >> 1, mid2 = (lo2 + hi2) >> 1;
		const bool a = lo < hi, b = lo2 < hi2;
		const unsigned long long va = a ? pairs[mid] : 0ull, vb = b ? pairs[mid2] : 0ull;
		if (a) {
			if (va < key) lo = mid + 1;
			else hi = mid;
		}
		if (b) {
			if (vb < key) lo2 = mid2 + 1;
			else hi2 = mid2;
		}
	}
	hits = lo;
	misses = lo2 - C;
}
__global__ void __launch_bounds__(kNT) k_batch_offsets(uint32_t S, const unsigned long long *__restrict__ shape_off,
                                                        const unsigned long long *__restrict__ pairs,
                                                        const DevStats *stats, unsigned long long *__restrict__ scene_pairs,
                                                        unsigned long long *__restrict__ contact_off) {
	pdl_begin();
	__shared__ unsigned long long before[kNT];
	const uint64_t s = (uint64_t)blockIdx.x * (kNT - 1) + threadIdx.x;
	const uint64_t P = stats->np_n, C = min((uint64_t)stats->contacts, P);  // no list: zeros
	uint64_t h = 0, m = 0;
	if (s <= S) {
		count_below(pairs, P, C, shape_off[s] << 32, h, m);
		contact_off[s] = h;
	}
	before[threadIdx.x] = h + m;
	__syncthreads();
	if (threadIdx.x < kNT - 1 && s < S) scene_pairs[s] = before[threadIdx.x + 1] - before[threadIdx.x];
}

// Pairs of every scene counted from an unsorted list (an output too small for
// the sorted one).
__global__ void __launch_bounds__(kNT) k_batch_pair_counts(uint64_t P, const unsigned long long *__restrict__ pairs,
                                                            const uint32_t *__restrict__ scene_of,
                                                            unsigned long long *__restrict__ scene_pairs) {
	for (uint64_t i = (uint64_t)blockIdx.x * kNT + threadIdx.x; i < P; i += (uint64_t)gridDim.x * kNT)
		atomicAdd(scene_pairs + scene_of[pairs[i] >> 32], 1ull);
}

// The same from the owners' offsets (one owner per bucket).
__global__ void __launch_bounds__(kNT) k_batch_owner_counts(uint32_t S, const unsigned long long *__restrict__ shape_off,
                                                             const unsigned long long *__restrict__ owner_off,
                                                             unsigned long long *__restrict__ scene_pairs) {
	const uint32_t s = blockIdx.x * kNT + threadIdx.x;
	if (s < S) scene_pairs[s] = owner_off[shape_off[s + 1]] - owner_off[shape_off[s]];
}

// The third shape array (C) of the shapes that read it: CONE, which GenerateAABB
// bounds as a triangle (AABBGenerator.cu:103-107), and TRIANGLEMESH, whose
// third vertex the support map and centre use (Narrowphase.cu:11-17, 44-47).
// `src` is the caller's pinned host array, read through its device mapping, so
// a scene without such shapes moves none of its bytes over PCIe.
__global__ void __launch_bounds__(kNT) k_gather_c(uint64_t n, const int32_t *__restrict__ T,
                                                   const float *__restrict__ src, float *__restrict__ dst) {
	for (uint64_t i = (uint64_t)blockIdx.x * kNT + threadIdx.x; i < n; i += (uint64_t)gridDim.x * kNT) {
		const int t = __ldg(T + i);
		if (t == CONE || t == TRIANGLEMESH) {
			const float x = src[3 * i], y = src[3 * i + 1], z = src[3 * i + 2];
			dst[3 * i] = x;
			dst[3 * i + 1] = y;
			dst[3 * i + 2] = z;
		}
	}
}

// The arrays of a MoveList, through the host mapping: the link to the host is
// filled by the loads or stores of all SMs at once, where nine copies one after the
// other spend most of their time starting (60K shapes, 4.6 MB in: a step of 315 us, by
// kernel 291, with the results out by kernel too 272; 2K shapes 147, 121, 94). An array
// is cut into units of 16 bytes, or of 4 or 1 where its addresses ask for that; a
// thread has four units in flight.
struct MoveUnits {
	uint64_t end[MoveList::kMax];  // units of the arrays so far
	uint64_t bytes[MoveList::kMax];
	uint32_t size[MoveList::kMax];
};
__device__ __forceinline__ void move_bytes(const char *src, char *dst, uint64_t from, uint64_t to) {
	for (uint64_t b = from; b < to; b++) dst[b] = src[b];
}
__global__ void __launch_bounds__(kNT) k_move(MoveList m, const DevStats *stats, PassRoom room) {
	__shared__ MoveUnits u;
	if (threadIdx.x == 0) {
		uint64_t P = 0, nc = 0, end = 0;
		bool ok = true;
		if (stats) {
			P = stats->np_n;
			nc = stats->contacts;
			ok = complete_pass(*stats, room);  // a result to be redone must not reach the caller's boxes, the redo's input
		}
		for (int k = 0; k < m.count; k++) {
			const uint64_t at = reinterpret_cast<uint64_t>(m.src[k]) | reinterpret_cast<uint64_t>(m.dst[k]);
			u.size[k] = at % 16 == 0 ? 16 : at % 4 == 0 ? 4 : 1;
			u.bytes[k] = ok ? m.fixed[k] + m.per_pair[k] * P + m.per_contact[k] * nc : 0;
			end += (u.bytes[k] + u.size[k] - 1) / u.size[k];
			u.end[k] = end;
		}
	}
	__syncthreads();
	const uint64_t total = m.count ? u.end[m.count - 1] : 0, step = (uint64_t)gridDim.x * kNT;
	for (uint64_t i0 = (uint64_t)blockIdx.x * kNT + threadIdx.x; i0 < total; i0 += 4 * step) {
		uint4 v[4];
		int arr[4];
		uint64_t at[4];  // first byte of the unit
#pragma unroll
		for (int q = 0; q < 4; q++) {
			const uint64_t i = i0 + q * step;
			arr[q] = -1;
			if (i >= total) continue;
			int k = 0;
			while (i >= u.end[k]) k++;
			arr[q] = k;
			at[q] = (i - (k ? u.end[k - 1] : 0)) * u.size[k];
			if (at[q] + u.size[k] > u.bytes[k]) continue;  // the last, partial unit
			const char *src = static_cast<const char *>(m.src[k]) + at[q];
			if (u.size[k] == 16) v[q] = __ldcs(reinterpret_cast<const uint4 *>(src));
			else if (u.size[k] == 4) v[q].x = __ldcs(reinterpret_cast<const uint32_t *>(src));
			else v[q].x = *reinterpret_cast<const uint8_t *>(src);
		}
#pragma unroll
		for (int q = 0; q < 4; q++) {
			const int k = arr[q];
			if (k < 0) continue;
			char *dst = static_cast<char *>(m.dst[k]);
			if (at[q] + u.size[k] > u.bytes[k]) move_bytes(static_cast<const char *>(m.src[k]), dst, at[q], u.bytes[k]);
			else if (u.size[k] == 16) *reinterpret_cast<uint4 *>(dst + at[q]) = v[q];
			else if (u.size[k] == 4) *reinterpret_cast<uint32_t *>(dst + at[q]) = v[q].x;
			else *reinterpret_cast<uint8_t *>(dst + at[q]) = (uint8_t)v[q].x;
			if (k == 0 && m.c_src) {  // shape types: this unit's shapes with a third vertex or axis
				const uint64_t last = min(at[q] + u.size[k], u.bytes[k]) / 4;
				for (uint64_t s = at[q] / 4; s < last; s++) {
					const int t = reinterpret_cast<const int32_t *>(dst)[s];
					if (t == CONE || t == TRIANGLEMESH)
						for (int d = 0; d < 3; d++) m.c_dst[3 * s + d] = m.c_src[3 * s + d];
				}
			}
		}
	}
}

// Counter-based random numbers for the time-step update: SplitMix64's output
// function (Steele, Lea, Flood 2014) applied to seed + counter, so every body
// draws the same numbers whatever the launch shape.
__device__ __forceinline__ uint64_t mix64(uint64_t z) {
	z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
	z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
	return z ^ (z >> 31);
}
__device__ __forceinline__ float unit_open(uint64_t h) {  // (0, 1)
	return ((float)(h >> 40) + 0.5f) * (1.0f / 16777216.0f);
}
// Two standard normals by the Box-Muller transform (Box and Muller, 1958).
__device__ __forceinline__ float2 normal2(uint64_t key) {
	const float u1 = unit_open(mix64(key)), u2 = unit_open(mix64(key ^ 0x5851f42d4c957f2dull));
	const float r = sqrtf(-2.0f * logf(u1));
	float s, c;
	sincosf(6.283185307179586f * u2, &s, &c);
	return make_float2(r * c, r * s);
}

// pos += N(0, sigma^2); rot = normalize(dq * rot), dq = (cos(a/2), u sin(a/2))
// with u uniform on the sphere and a ~ U[0, max_angle]. Quaternions (w,x,y,z).
// Body i of a scene updated with `seed` (the random numbers are a function of
// (seed, i) alone).
__device__ __forceinline__ void perturb_one(float *__restrict__ pos, float *__restrict__ rot, uint64_t i,
                                            uint64_t seed, float sigma, float max_angle) {
	{
		const uint64_t key = mix64(seed) + 8 * i;
		const float2 n01 = normal2(key), n23 = normal2(key + 1), n45 = normal2(key + 2);
		pos[3 * i] += sigma * n01.x;
		pos[3 * i + 1] += sigma * n01.y;
		pos[3 * i + 2] += sigma * n23.x;
		float ux = n23.y, uy = n45.x, uz = n45.y;
		const float ul = sqrtf(ux * ux + uy * uy + uz * uz);
		if (ul > 0.f) {
			ux /= ul; uy /= ul; uz /= ul;
		} else {
			ux = 1.f; uy = 0.f; uz = 0.f;
		}
		const float h = 0.5f * max_angle * unit_open(mix64(key + 3));
		float sh, ch;
		sincosf(h, &sh, &ch);
		const float bx = ux * sh, by = uy * sh, bz = uz * sh;
		float4 q = reinterpret_cast<float4 *>(rot)[i];
		float4 r;
		r.x = ch * q.x - bx * q.y - by * q.z - bz * q.w;
		r.y = ch * q.y + bx * q.x + by * q.w - bz * q.z;
		r.z = ch * q.z - bx * q.w + by * q.x + bz * q.y;
		r.w = ch * q.w + bx * q.z - by * q.y + bz * q.x;
		const float rl = sqrtf(r.x * r.x + r.y * r.y + r.z * r.z + r.w * r.w);
		reinterpret_cast<float4 *>(rot)[i] = make_float4(r.x / rl, r.y / rl, r.z / rl, r.w / rl);
	}
}

__global__ void __launch_bounds__(kNT) k_perturb(uint64_t nb, float *__restrict__ pos, float *__restrict__ rot,
                                                  uint64_t seed, float sigma, float max_angle) {
	for (uint64_t i = (uint64_t)blockIdx.x * kNT + threadIdx.x; i < nb; i += (uint64_t)gridDim.x * kNT)
		perturb_one(pos, rot, i, seed, sigma, max_angle);
}

// Several scenes in one launch: the bodies of all scenes as one index range,
// scene k owning [d[k].first, d[k].first + d[k].nb) (found by binary search).
__global__ void __launch_bounds__(kNT) k_perturb_scenes(uint32_t count, uint64_t total,
                                                         const PerturbScene *__restrict__ d, float sigma,
                                                         float max_angle) {
	for (uint64_t g = (uint64_t)blockIdx.x * kNT + threadIdx.x; g < total; g += (uint64_t)gridDim.x * kNT) {
		uint32_t lo = 0, hi = count;  // last scene with first <= g
		while (hi - lo > 1) {
			const uint32_t mid = (lo + hi) >> 1;
			if (d[mid].first <= g) lo = mid;
			else hi = mid;
		}
		const PerturbScene sc = d[lo];
		perturb_one(sc.pos, sc.rot, g - sc.first, sc.seed, sigma, max_angle);
	}
}
}  // namespace

// Small host tables go to the device inside kernel parameters: the driver
// copies a launch's parameters with the launch, so the table needs no copy
// engine and no staging of pageable memory, and cannot queue behind bulk
// uploads running on another stream.
struct ParamChunk {
	uint32_t words[kParamChunkBytes / 4];
};
__global__ void k_param_copy(uint32_t *__restrict__ dst, uint32_t nwords, ParamChunk c) {
	for (uint32_t i = threadIdx.x; i < nwords; i += blockDim.x) dst[i] = c.words[i];
}

cudaError_t copy_small_h2d(void *dst, const void *src, size_t bytes, cudaStream_t s) {
	if (bytes > kParamCopyMax || (bytes & 3) || (reinterpret_cast<uintptr_t>(dst) & 3))
		return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s);
	const unsigned char *from = static_cast<const unsigned char *>(src);
	uint32_t *to = static_cast<uint32_t *>(dst);
	for (size_t off = 0; off < bytes; off += kParamChunkBytes) {
		const size_t n = std::min<size_t>(kParamChunkBytes, bytes - off);
		ParamChunk c;
		memcpy(c.words, from + off, n);
		k_param_copy<<<1, 256, 0, s>>>(to + off / 4, (uint32_t)(n / 4), c);
	}
	return cudaGetLastError();
}

void launch_perturb_scenes(uint32_t count, uint64_t total, const PerturbScene *d, float sigma, float max_angle,
                           cudaStream_t s) {
	if (!count || !total) return;
	const unsigned g = (unsigned)std::min<uint64_t>((total + kNT - 1) / kNT, (uint64_t)kNumSMs * 16);
	k_perturb_scenes<<<g, kNT, 0, s>>>(count, total, d, sigma, max_angle);
}

void launch_perturb(uint64_t nb, float *pos, float *rot, uint64_t seed, float sigma, float max_angle, cudaStream_t s) {
	if (!nb) return;
	const unsigned g = (unsigned)std::min<uint64_t>((nb + kNT - 1) / kNT, (uint64_t)kNumSMs * 16);
	k_perturb<<<g, kNT, 0, s>>>(nb, pos, rot, seed, sigma, max_angle);
}

void launch_gather_c(uint64_t n, const int32_t *T, const float *src, float *dst, cudaStream_t s) {
	if (!n) return;
	const unsigned g = (unsigned)std::min<uint64_t>((n + kNT - 1) / kNT, (uint64_t)kNumSMs * 8);
	k_gather_c<<<g, kNT, 0, s>>>(n, T, src, dst);
}

void launch_move(const MoveList &m, uint64_t bytes_hint, const DevStats *stats, const PassRoom &room, cudaStream_t s) {
	const unsigned g = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(bytes_hint / (16 * 4 * kNT) + 1, (uint64_t)kNumSMs * 8));
	k_move<<<g, kNT, 0, s>>>(m, stats, room);
}

void launch_batch_pair_counts(uint64_t P, const unsigned long long *pairs, const uint32_t *scene_of,
                              unsigned long long *scene_pairs, cudaStream_t s) {
	if (!P) return;
	const unsigned g = (unsigned)std::min<uint64_t>((P + kNT - 1) / kNT, (uint64_t)kNumSMs * 8);
	k_batch_pair_counts<<<g, kNT, 0, s>>>(P, pairs, scene_of, scene_pairs);
}

void launch_batch_owner_counts(uint32_t S, const unsigned long long *shape_off, const unsigned long long *owner_off,
                               unsigned long long *scene_pairs, cudaStream_t s) {
	k_batch_owner_counts<<<(S + kNT - 1) / kNT, kNT, 0, s>>>(S, shape_off, owner_off, scene_pairs);
}

void launch_batch_offsets(uint32_t S, const unsigned long long *shape_off, const unsigned long long *pairs,
                          const DevStats *stats, unsigned long long *scene_pairs, unsigned long long *contact_off,
                          cudaStream_t s) {
	launch_pdl(k_batch_offsets, dim3(S / (kNT - 1) + 1), dim3(kNT), 0, s, S, shape_off, pairs, stats, scene_pairs, contact_off);
}

}  // namespace cc
