// prt_build.cu - LBVH build of 8-wide trees on the GPU, for one scene or many at once,
// and the stages every build shares (collapse, re-layout, compression).
//
// Replaces the single-threaded binned-SAH build of portableRT (bvh.hpp:58-193).  The
// tree's shape does not affect the answers (every triangle whose own box passes the
// reference slab test is examined; see prt_traverse.cu), only how many boxes a ray
// passes: set_tris, batch builds and servers build their binary trees with binned SAH
// by default (prt_sah.cu, steps 1-5 replaced); graph-captured batch builds and the
// option build_sah = 0 use this LBVH, about 3x faster to build.  Several scenes are
// built in the same launches: scene s owns the input triangles [tri_off[s],
// tri_off[s+1]), its sort key carries the scene index above the Morton code, its binary
// nodes are the range [int_off[s], int_off[s+1]) and its 8-wide root is node s.
//   1. centroid bounds per scene  (k_centroid_bounds; warp reduce + ordered-int atomics)
//   2. 30-bit Morton codes        (k_morton; 10 bits per axis, centroids normalised)
//   3. onesweep radix sort        (prt_sort.cu; 4 digit passes, +1 or 2 for the scene)
//   4. Karras hierarchy           (k_karras; Karras 2012 within each scene's range)
//   5. bottom-up pass             (k_bottom_up: boxes and, for the collapse, the least
//                                  expected cost per ray: which subtrees become nodes and
//                                  which leaves)
//   6. collapse to 8-wide nodes   (after step 5's costs, which SAH builds compute as well;
//                                  then k_collapse, one launch per level, per-level
//                                  counters, so the host checks progress every few levels;
//                                  with each node its optional 8-bit encoding, outward-
//                                  rounded child boxes, and its leaf triangles' records,
//                                  contiguous)
// A triangle with a non-finite vertex gets the box [-FLT_MAX, FLT_MAX]^3 in the tree,
// which every finite ray passes, so the exact per-triangle test still sees it.
#include <algorithm>
#include <atomic>
#include <cfloat>
#include <cmath>
#include <cstddef>
#include <cstring>

#include "../../include/prt_b200.h"
#include "prt_build.cuh"
#include "prt_collapse.cuh"
#include "prt_launch.cuh"
#include "prt_sah.cuh"

namespace prt {

namespace {
std::atomic<int64_t> g_alloc_failure{0}; // growths left before the injected failure
} // namespace

void arm_alloc_failure(int64_t n) { g_alloc_failure.store(n > 0 ? n : 0); }

bool alloc_failure_due() {
	int64_t v = g_alloc_failure.load(std::memory_order_relaxed);
	while (v > 0)
		if (g_alloc_failure.compare_exchange_weak(v, v - 1))
			return v == 1;
	return false;
}

void BuildScratch::release() {
	DevBuf *all[] = {&keys,        &vals,     &keys2,      &vals2,    &scene_of,   &int_off,
	                 &left,        &right,    &splits,     &rfirst,   &rlast,
	                 &ibox,        &lbox,     &flags,      &items_a,  &items_b,    &counters,
	                 &sort_hist, &sort_tiles, &sort_status, &bounds,
	                 &sah,         &roots,    &cost};
	for (DevBuf *b : all)
		b->release();
	if (h_counters)
		cudaFreeHost(h_counters);
	h_counters = nullptr;
	h_sah = nullptr;
}

namespace {

struct Item {
	uint32_t ref;  // binary-tree reference (bit 31 = leaf); kNone = empty scene
	uint32_t slot; // index of the 8-wide node it becomes
};

__device__ __forceinline__ bool tri_finite(const float *t) {
	bool ok = true;
#pragma unroll
	for (int k = 0; k < 9; ++k)
		ok = ok && isfinite(t[k]);
	return ok;
}

__device__ __forceinline__ float centroid(const float *t, int k) {
	return t[k] * (1.0f / 3.0f) + t[k + 3] * (1.0f / 3.0f) + t[k + 6] * (1.0f / 3.0f);
}

__device__ __forceinline__ uint32_t scene_at(const uint32_t *scene_of, uint32_t i) {
	return scene_of ? scene_of[i] : 0u;
}

// scene_of[i] = s for every triangle of scene s (one block per scene, grid-stride).
__global__ void k_scene_of(const uint32_t *tri_off, uint32_t n_scenes, uint32_t *scene_of) {
	for (uint32_t s = blockIdx.x; s < n_scenes; s += gridDim.x)
		for (uint32_t i = tri_off[s] + threadIdx.x; i < tri_off[s + 1]; i += blockDim.x)
			scene_of[i] = s;
}

__global__ void k_clear_error(uint32_t *err, uint32_t bits) { clear_error_bits(err, bits); }

// Empty bounds, and no split after each scene's last leaf.
__global__ void k_bounds_init(uint32_t *gb, uint32_t n_scenes, const uint32_t *tri_off,
                              uint4 *splits, uint32_t *x_drop) {
	if (x_drop && blockIdx.x == 0 && threadIdx.x == 0)
		x_drop[0] = 1u;
	for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < 6 * n_scenes;
	     i += gridDim.x * blockDim.x) {
		gb[i] = (i % 6) < 3 ? 0xFFFFFFFFu : 0u;
		if (i < n_scenes && tri_off[i + 1] > tri_off[i])
			splits[tri_off[i + 1] - 1u] = PRT_NO_SPLIT;
	}
}

// Per-scene centroid bounds as ordered words: a warp whose triangles all belong to one
// scene reduces first; otherwise each lane updates its own scene.
__global__ void k_centroid_bounds(const float *__restrict__ tris, uint32_t n,
                                  const uint32_t *__restrict__ scene_of, uint32_t *gb) {
	const int lane = threadIdx.x & 31;
	if (!scene_of) {
		// One scene: each thread folds its grid-stride share, then the block reduces and
		// one thread updates the six words (so the same-address atomics stay few).
		float mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
		for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
		     i += gridDim.x * blockDim.x) {
			const float *t = tris + 9 * (size_t)i;
			if (tri_finite(t)) {
#pragma unroll
				for (int k = 0; k < 3; ++k) {
					const float c = centroid(t, k);
					mn[k] = fminf(mn[k], c);
					mx[k] = fmaxf(mx[k], c);
				}
			}
		}
		__shared__ float red[32][6];
#pragma unroll
		for (int k = 0; k < 3; ++k)
			for (int o = 16; o > 0; o >>= 1) {
				mn[k] = fminf(mn[k], __shfl_xor_sync(0xFFFFFFFFu, mn[k], o));
				mx[k] = fmaxf(mx[k], __shfl_xor_sync(0xFFFFFFFFu, mx[k], o));
			}
		const int w = threadIdx.x >> 5, nw = blockDim.x >> 5;
		if (lane == 0)
			for (int k = 0; k < 3; ++k) {
				red[w][k] = mn[k];
				red[w][3 + k] = mx[k];
			}
		__syncthreads();
		if (threadIdx.x == 0) {
			for (int v = 1; v < nw; ++v)
				for (int k = 0; k < 3; ++k) {
					mn[k] = fminf(mn[k], red[v][k]);
					mx[k] = fmaxf(mx[k], red[v][3 + k]);
				}
			if (mn[0] <= mx[0])
				for (int k = 0; k < 3; ++k) {
					atomicMin(&gb[k], f2ord(mn[k]));
					atomicMax(&gb[3 + k], f2ord(mx[k]));
				}
		}
		return;
	}
	for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += gridDim.x * blockDim.x) {
		const uint32_t i = base + threadIdx.x;
		float mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
		uint32_t s = 0;
		if (i < n) {
			const float *t = tris + 9 * (size_t)i;
			s = scene_at(scene_of, i);
			if (tri_finite(t)) {
#pragma unroll
				for (int k = 0; k < 3; ++k)
					mn[k] = mx[k] = centroid(t, k);
			}
		}
		// Lanes past the end hold empty bounds, so they never change a reduction.
		const uint32_t s0 = __shfl_sync(0xFFFFFFFFu, s, 0);
		const bool same = __all_sync(0xFFFFFFFFu, s == s0 || i >= n);
		if (same) {
#pragma unroll
			for (int k = 0; k < 3; ++k) {
				for (int o = 16; o > 0; o >>= 1) {
					mn[k] = fminf(mn[k], __shfl_xor_sync(0xFFFFFFFFu, mn[k], o));
					mx[k] = fmaxf(mx[k], __shfl_xor_sync(0xFFFFFFFFu, mx[k], o));
				}
			}
			if (lane == 0 && mn[0] <= mx[0]) {
#pragma unroll
				for (int k = 0; k < 3; ++k) {
					atomicMin(&gb[6 * s0 + k], f2ord(mn[k]));
					atomicMax(&gb[6 * s0 + 3 + k], f2ord(mx[k]));
				}
			}
		} else if (i < n && mn[0] <= mx[0]) {
#pragma unroll
			for (int k = 0; k < 3; ++k) {
				atomicMin(&gb[6 * s + k], f2ord(mn[k]));
				atomicMax(&gb[6 * s + 3 + k], f2ord(mx[k]));
			}
		}
	}
}

__device__ __forceinline__ uint32_t spread10(uint32_t x) {
	x &= 1023u;
	x = (x | (x << 16)) & 0x030000FFu;
	x = (x | (x << 8)) & 0x0300F00Fu;
	x = (x | (x << 4)) & 0x030C30C3u;
	x = (x | (x << 2)) & 0x09249249u;
	return x;
}

// Key = Morton code of the centroid in its scene's centroid box; with several scenes
// (64-bit keys) the scene index sits above it.
template <typename K>
__global__ void k_morton(const float *__restrict__ tris, uint32_t n,
                         const uint32_t *__restrict__ scene_of, const uint32_t *gb, K *keys,
                         uint32_t *vals) {
	uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n)
		return;
	const float *t = tris + 9 * (size_t)i;
	const uint32_t s = scene_at(scene_of, i);
	const uint32_t *b = gb + 6 * s;
	uint32_t code = 0;
	if (tri_finite(t) && ord2f(b[0]) <= ord2f(b[3])) {
		uint32_t q[3];
#pragma unroll
		for (int k = 0; k < 3; ++k) {
			const float lo = ord2f(b[k]), hi = ord2f(b[3 + k]);
			const float ext = hi - lo;
			const float sc = ext > 0.0f ? 1024.0f / ext : 0.0f;
			const float qf = fminf(fmaxf((centroid(t, k) - lo) * sc, 0.0f), 1023.0f);
			q[k] = (uint32_t)qf;
		}
		code = (spread10(q[0]) << 2) | (spread10(q[1]) << 1) | spread10(q[2]);
	}
	if (sizeof(K) == 8)
		keys[i] = (K)(((uint64_t)s << 32) | code);
	else
		keys[i] = (K)code;
	vals[i] = i;
}

// Common-prefix length of the Morton codes of leaves i and j of one scene, with the
// index appended to break ties between equal codes; -1 outside [0, n).
template <typename K>
__device__ __forceinline__ int kdelta(const K *__restrict__ k, int n, int i, int j) {
	if (j < 0 || j >= n)
		return -1;
	const uint32_t a = (uint32_t)k[i], b = (uint32_t)k[j];
	return (a != b) ? __clz(a ^ b) : 32 + __clz((uint32_t)i ^ (uint32_t)j);
}

// Binary node gi: find its scene (int_off is non-decreasing), then Karras's
// construction on that scene's sorted leaves.  References are global: leaf positions
// are tri_off[s] + local, binary nodes int_off[s] + local.
template <typename K>
__global__ void k_karras(const K *__restrict__ keys, uint32_t n_int, const uint32_t *tri_off,
                         const uint32_t *int_off, uint32_t n_scenes, uint32_t *left,
                         uint32_t *right, uint4 *splits, uint32_t *rfirst,
                         uint32_t *rlast) {
	const uint32_t gi = blockIdx.x * blockDim.x + threadIdx.x;
	if (gi >= n_int)
		return;
	uint32_t lo_s = 0, hi_s = n_scenes; // last s with int_off[s] <= gi
	while (hi_s - lo_s > 1) {
		const uint32_t mid = (lo_s + hi_s) >> 1;
		if (int_off[mid] <= gi)
			lo_s = mid;
		else
			hi_s = mid;
	}
	const uint32_t s = lo_s;
	const uint32_t first = tri_off[s], ibase = int_off[s];
	const int n = (int)(tri_off[s + 1] - first);
	const int i = (int)(gi - ibase);
	const K *k = keys + first;
	const int d = kdelta(k, n, i, i + 1) > kdelta(k, n, i, i - 1) ? 1 : -1;
	const int dmin = kdelta(k, n, i, i - d);
	int lmax = 2;
	while (kdelta(k, n, i, i + lmax * d) > dmin)
		lmax <<= 1;
	int l = 0;
	for (int t = lmax >> 1; t >= 1; t >>= 1)
		if (kdelta(k, n, i, i + (l + t) * d) > dmin)
			l += t;
	const int j = i + l * d;
	const int dnode = kdelta(k, n, i, j);
	int sp = 0;
	for (int div = 2;; div <<= 1) {
		const int t = (l + div - 1) / div;
		if (kdelta(k, n, i, i + (sp + t) * d) > dnode)
			sp += t;
		if (t <= 1)
			break;
	}
	const int gamma = i + sp * d + min(d, 0);
	const int lo = min(i, j), hi = max(i, j);
	const bool lleaf = lo == gamma, rleaf = hi == gamma + 1;
	const uint32_t lc = lleaf ? (kLeafBit | (first + gamma)) : (ibase + gamma);
	const uint32_t rc = rleaf ? (kLeafBit | (first + gamma + 1)) : (ibase + gamma + 1);
	left[gi] = lc;
	right[gi] = rc;
	splits[first + gamma] = make_uint4(first + lo, first + hi, gi, 0u);
	rfirst[gi] = first + lo;
	rlast[gi] = first + hi;
}

// atomicAdd(p, 1) with acquire-release ordering at device scope.
__device__ __forceinline__ uint32_t arrive_acq_rel(uint32_t *p) {
	uint32_t old;
	asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(old) : "l"(p) : "memory");
	return old;
}

__device__ __forceinline__ void child_box(uint32_t ref, const float4 *ibox, const float4 *lbox,
                                          float4 &lo, float4 &hi) {
	if (ref & kLeafBit) {
		uint32_t k = ref & ~kLeafBit;
		lo = __ldcg(&lbox[2 * k]);
		hi = __ldcg(&lbox[2 * k + 1]);
	} else {
		lo = __ldcg(&ibox[2 * ref]);
		hi = __ldcg(&ibox[2 * ref + 1]);
	}
}

// Costs of child `y` in j = 1..7 slots (cs[j]), in units of its own area; returns its
// half extents.
__device__ __forceinline__ float3 child_costs(uint32_t y, const CostNode *cost,
                                              const float4 *ibox, const float4 *lbox,
                                              float cs[8]) {
	if (y & kLeafBit) {
		const uint32_t k = y & ~kLeafBit;
		leaf_costs(cs);
		return half_extent(__ldcg(&lbox[2 * k]), __ldcg(&lbox[2 * k + 1]));
	}
	CostNode c;
	c.c1 = __ldcg(&cost[y].c1);
#pragma unroll
	for (int j = 0; j < 7; ++j)
		c.cd[j] = __ldcg(&cost[y].cd[j]);
	node_costs(c, cs);
	return half_extent(__ldcg(&ibox[2 * y]), __ldcg(&ibox[2 * y + 1]));
}

struct UpArgs {
	const float *tris;        // REFIT: the triangles, by vals
	const uint32_t *vals;
	uint32_t n, n_ids;
	const uint4 *splits;
	const uint32_t *left, *right;
	float4 *ibox, *lbox;
	uint32_t *flags;          // arrivals at nodes that several blocks' leaves reach
	CostNode *cost;
	uint32_t leaf_size;
	uint32_t *walks, *n_walks; // slots at which the blocks' parts end
	uint32_t walk_cap;
	const uint32_t *gate;     // null, or: nothing to do unless it is 0
	uint32_t *err;
};

constexpr uint32_t kUpLeaves = 256; // leaf positions per block

// What a block knows of the subtrees inside its leaf positions.  The binary node that splits
// after a leaf position has that position as its slot: every node has one, every position but
// a scene's last, and the parent of the subtree over leaves [f, l] is the node of slot l (it
// is its left child) or of slot f - 1 (its right child).
struct UpShared {
	uint32_t first[kUpLeaves], last[kUpLeaves], node[kUpLeaves]; // `splits` of the positions
	float lbox[6][kUpLeaves];  // boxes of the leaves ...
	float nbox[6][kUpLeaves];  // ... and of the nodes, by slot
	float cost[8][kUpLeaves];  // c1 and cd of the nodes done
	uint32_t count[kUpLeaves]; // children done
	uint32_t n_ready[kUpLeaves + 2]; // nodes that became ready for round k
	uint32_t escape[kUpLeaves], n_escape; // slots (global) that the block's part ends at
	uint32_t walk_at;
	uint16_t child[2][kUpLeaves]; // children done: leaf position | kUpLeaf, or slot
	uint16_t ready[2][kUpLeaves];
};
constexpr uint16_t kUpLeaf = 0x8000u;

// A subtree (leaf position or slot `ref`, global leaf range [f, l]) is done: its parent gets
// it.  Round `round` takes up the parents that are complete then.
__device__ __forceinline__ void up_deliver(const UpArgs &A, UpShared &S, uint32_t b0,
                                           uint16_t ref, uint32_t f, uint32_t l,
                                           uint32_t round) {
	const bool is_left = S.first[l - b0] == f;
	if (!is_left && f == b0) {
		if (f > 0u && __ldg(&A.splits[f - 1u]).y == l) {
			const uint32_t at = atomicAdd(&S.n_escape, 1u);
			if (at < kUpLeaves)
				S.escape[at] = f - 1u;
		}
		return; // (or a root)
	}
	const uint32_t slot = is_left ? l - b0 : f - 1u - b0;
	if (!is_left && S.last[slot] != l)
		return; // a root
	if (S.first[slot] < b0 || S.last[slot] >= b0 + kUpLeaves) {
		const uint32_t at = atomicAdd(&S.n_escape, 1u);
		if (at < kUpLeaves)
			S.escape[at] = b0 + slot;
		return;
	}
	S.child[is_left ? 0 : 1][slot] = ref;
	if (atomicAdd(&S.count[slot], 1u) == 1u) {
		const uint32_t at = atomicAdd(&S.n_ready[round], 1u);
		if (at < kUpLeaves)
			S.ready[round & 1u][at] = (uint16_t)slot;
	}
}

__device__ __forceinline__ void up_child(const UpShared &S, uint16_t ref, float4 &lo, float4 &hi,
                                         float cs[8], bool cost) {
	const bool leaf = (ref & kUpLeaf) != 0;
	const uint32_t at = ref & (kUpLeaves - 1u);
	const float(*b)[kUpLeaves] = leaf ? S.lbox : S.nbox;
	lo = make_float4(b[0][at], b[1][at], b[2][at], 0.0f);
	hi = make_float4(b[3][at], b[4][at], b[5][at], 0.0f);
	if (!cost)
		return;
	if (leaf) {
		leaf_costs(cs);
	} else {
		CostNode c;
		c.c1 = S.cost[0][at];
#pragma unroll
		for (int j = 0; j < 7; ++j)
			c.cd[j] = S.cost[1 + j][at];
		node_costs(c, cs);
	}
}

// The bottom-up pass over the binary trees.  REFIT: boxes of the leaves (from the triangles in
// sorted order) and of the nodes, whose unused w words carry the surface areas of their two
// children (-1 for a leaf child), which the collapse by area reads together with the child
// indices.  COST: the least expected costs of each node (CostNode).
//
// A block takes 256 consecutive leaves and finishes every node whose leaves are all among
// them from shared memory, round by round, full warps on the nodes that became complete in
// the round before; the subtrees it ends with go to k_walk_up.  With one thread per leaf
// walking all the way, refit and costs apart, 5 of 32 lanes were active and every step was
// an acquire-release atomic and two dependent reads through L2: leaf boxes, refit and costs
// of a batch of 4.6M triangles took 110 + 252 + 694 us, the costs of the 1,048,576-triangle
// heightfield 209; now 389 + 71 and 86 + 60 (builds: 1.73 -> 1.65 ms; 8.4M clustered
// triangles 13.4 -> 12.7 ms; the batch's graph 10.95 -> 10.38 ms).
template <bool REFIT, bool COST>
__global__ void __launch_bounds__(kUpLeaves) k_bottom_up(UpArgs A) {
	chain_enter(); // (launched as usual: only lets k_walk_up be scheduled)
	__shared__ UpShared S;
	const uint32_t b0 = blockIdx.x * kUpLeaves, t = threadIdx.x, i = b0 + t;
	if (A.gate && *A.gate)
		return;
	const bool live = i < A.n;
	S.count[t] = 0;
	const uint4 sp = live ? A.splits[i] : PRT_NO_SPLIT;
	S.first[t] = sp.x;
	S.last[t] = sp.y;
	S.node[t] = sp.z;
	if (!REFIT && sp.z != kNone && sp.x >= b0 && sp.y < b0 + kUpLeaves) {
		if (sp.z >= A.n_ids) {
			set_error_bits(A.err, kErrCollapse);
			S.node[t] = 0u;
		} else {
			const float4 lo = A.ibox[2 * (size_t)sp.z], hi = A.ibox[2 * (size_t)sp.z + 1];
			S.nbox[0][t] = lo.x;
			S.nbox[1][t] = lo.y;
			S.nbox[2][t] = lo.z;
			S.nbox[3][t] = hi.x;
			S.nbox[4][t] = hi.y;
			S.nbox[5][t] = hi.z;
		}
	}
	for (uint32_t k = t; k < kUpLeaves + 2u; k += kUpLeaves)
		S.n_ready[k] = 0;
	if (t == 0)
		S.n_escape = 0;
	if (live) {
		float4 lo, hi;
		if (REFIT) {
			const float *v = A.tris + 9 * (size_t)A.vals[i];
			if (tri_finite(v)) {
				lo = make_float4(fminf(v[0], fminf(v[3], v[6])), fminf(v[1], fminf(v[4], v[7])),
				                 fminf(v[2], fminf(v[5], v[8])), 0.0f);
				hi = make_float4(fmaxf(v[0], fmaxf(v[3], v[6])), fmaxf(v[1], fmaxf(v[4], v[7])),
				                 fmaxf(v[2], fmaxf(v[5], v[8])), 0.0f);
			} else {
				lo = make_float4(-FLT_MAX, -FLT_MAX, -FLT_MAX, 0.0f);
				hi = make_float4(FLT_MAX, FLT_MAX, FLT_MAX, 0.0f);
			}
			__stcg(&A.lbox[2 * (size_t)i], lo);
			__stcg(&A.lbox[2 * (size_t)i + 1], hi);
		} else {
			lo = A.lbox[2 * (size_t)i];
			hi = A.lbox[2 * (size_t)i + 1];
		}
		S.lbox[0][t] = lo.x;
		S.lbox[1][t] = lo.y;
		S.lbox[2][t] = lo.z;
		S.lbox[3][t] = hi.x;
		S.lbox[4][t] = hi.y;
		S.lbox[5][t] = hi.z;
	}
	__syncthreads();
	if (live)
		up_deliver(A, S, b0, (uint16_t)(t | kUpLeaf), i, i, 0u);
	for (uint32_t round = 0;; ++round) { // at most kUpLeaves: each round finishes a node
		__syncthreads();
		const uint32_t m = min(S.n_ready[round], kUpLeaves);
		if (m == 0u || round > kUpLeaves)
			break;
		if (t < m) {
			const uint32_t slot = S.ready[round & 1u][t];
			const uint32_t p = min(S.node[slot], A.n_ids - 1u);
			const uint32_t f = S.first[slot], l = S.last[slot];
			const uint16_t cl16 = S.child[0][slot], cr16 = S.child[1][slot];
			float4 llo, lhi, rlo, rhi, lo, hi;
			float cl[8], cr[8];
			up_child(S, cl16, llo, lhi, cl, COST);
			up_child(S, cr16, rlo, rhi, cr, COST);
			if (REFIT) {
				lo = make_float4(fminf(llo.x, rlo.x), fminf(llo.y, rlo.y), fminf(llo.z, rlo.z),
				                 (cl16 & kUpLeaf) ? -1.0f : half_area(llo, lhi));
				hi = make_float4(fmaxf(lhi.x, rhi.x), fmaxf(lhi.y, rhi.y), fmaxf(lhi.z, rhi.z),
				                 (cr16 & kUpLeaf) ? -1.0f : half_area(rlo, rhi));
				__stcg(&A.ibox[2 * (size_t)p], lo);
				__stcg(&A.ibox[2 * (size_t)p + 1], hi);
				S.nbox[0][slot] = lo.x;
				S.nbox[1][slot] = lo.y;
				S.nbox[2][slot] = lo.z;
				S.nbox[3][slot] = hi.x;
				S.nbox[4][slot] = hi.y;
				S.nbox[5][slot] = hi.z;
			} else {
				lo = make_float4(S.nbox[0][slot], S.nbox[1][slot], S.nbox[2][slot], 0.0f);
				hi = make_float4(S.nbox[3][slot], S.nbox[4][slot], S.nbox[5][slot], 0.0f);
			}
			if (COST) {
				const CostNode c =
				    merge_costs(cl, cr, half_extent(llo, lhi), half_extent(rlo, rhi),
				                half_extent(lo, hi), l - f + 1u, A.leaf_size);
				S.cost[0][slot] = c.c1;
				__stcg(&A.cost[p].c1, c.c1);
#pragma unroll
				for (int k = 0; k < 7; ++k) {
					S.cost[1 + k][slot] = c.cd[k];
					__stcg(&A.cost[p].cd[k], c.cd[k]);
				}
				__stcg(&A.cost[p].bits, c.bits);
			}
			up_deliver(A, S, b0, (uint16_t)slot, f, l, round + 1u);
		}
	}
	const uint32_t n_out = min(S.n_escape, kUpLeaves);
	if (t == 0 && n_out)
		S.walk_at = atomicAdd(A.n_walks, n_out);
	__syncthreads();
	if (t < n_out) {
		if (S.walk_at + t < A.walk_cap)
			A.walks[S.walk_at + t] = S.escape[t];
		else
			set_error_bits(A.err, kErrCollapse);
	}
}

// The rest of the bottom-up pass: one thread per subtree that a block ended with walks
// towards the root; at each node the first to arrive stops and the second, which sees both
// children, goes on (nobody waits).  What does not depend on the sibling is read before the
// arrival: a step is bound by its atomic and the reads after it.  A launch of its own,
// because a block of k_bottom_up kept its place for the longest of its walks.
template <bool REFIT, bool COST>
__global__ void __launch_bounds__(128) k_walk_up(UpArgs A) {
	chain_enter();
	const uint32_t n = min(*A.n_walks, A.walk_cap);
	for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
		uint4 at = A.splits[A.walks[k]];
		// A path to the root passes each binary node once; a longer walk (or an index out of
		// range) means corrupt splits, reported instead of followed.
		for (uint32_t steps = 0;; ++steps) {
			const uint32_t p = at.z;
			if (p >= A.n_ids || steps >= A.n_ids || at.y >= A.n) {
				set_error_bits(A.err, kErrCollapse);
				break;
			}
			const uint32_t l = A.left[p], r = A.right[p];
			const uint4 as_left = A.splits[at.y]; // the parent, if p is its left child ...
			const uint4 as_right = at.x > 0u ? A.splits[at.x - 1u] : PRT_NO_SPLIT; // ... or right
			float4 lo, hi;
			if (!REFIT) {
				lo = A.ibox[2 * (size_t)p];
				hi = A.ibox[2 * (size_t)p + 1];
			}
			// Release: what was written below is visible before this arrival counts.
			// Acquire: the sibling's results are read after its arrival.
			if (arrive_acq_rel(&A.flags[p]) == 0u)
				break;
			if (REFIT) {
				float4 llo, lhi, rlo, rhi;
				child_box(l, A.ibox, A.lbox, llo, lhi);
				child_box(r, A.ibox, A.lbox, rlo, rhi);
				lo = make_float4(fminf(llo.x, rlo.x), fminf(llo.y, rlo.y), fminf(llo.z, rlo.z),
				                 (l & kLeafBit) ? -1.0f : half_area(llo, lhi));
				hi = make_float4(fmaxf(lhi.x, rhi.x), fmaxf(lhi.y, rhi.y), fmaxf(lhi.z, rhi.z),
				                 (r & kLeafBit) ? -1.0f : half_area(rlo, rhi));
				__stcg(&A.ibox[2 * (size_t)p], lo);
				__stcg(&A.ibox[2 * (size_t)p + 1], hi);
			}
			if (COST) {
				float cl[8], cr[8];
				const float3 el = child_costs(l, A.cost, A.ibox, A.lbox, cl);
				const float3 er = child_costs(r, A.cost, A.ibox, A.lbox, cr);
				const CostNode c = merge_costs(cl, cr, el, er, half_extent(lo, hi),
				                               at.y - at.x + 1u, A.leaf_size);
				__stcg(&A.cost[p].c1, c.c1);
#pragma unroll
				for (int j = 0; j < 7; ++j)
					__stcg(&A.cost[p].cd[j], c.cd[j]);
				__stcg(&A.cost[p].bits, c.bits);
			}
			if (as_left.x == at.x)
				at = as_left;
			else if (as_right.y == at.y)
				at = as_right;
			else
				break; // a root
		}
	}
}

// Child slot `r` of an 8-wide node becomes an 8-wide node of its own (else a leaf).
__device__ __forceinline__ bool is_inner(uint32_t r, uint32_t count, uint32_t leaf_size,
                                         const CostNode *cost) {
	if (r & kLeafBit)
		return false;
	if (count > leaf_size)
		return true;
	return cost ? (cost[r].bits >> 31) == 0u : false;
}

// Level-0 frontier: the root of every scene becomes 8-wide node s; the node counter
// starts after the roots.
__global__ void k_collapse_roots(const uint32_t *tri_off, const uint32_t *int_off,
                                 uint32_t n_scenes, Item *items, uint32_t *ctr,
                                 const uint32_t *gb, float4 *far) {
	chain_enter();
	const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
	if (s == 0) {
		ctr[0] = ctr[kCtrGate] ? 0u : n_scenes; // (incomplete trees: no items, no levels)
		ctr[kCtrNodes] = n_scenes;
	}
	if (s >= n_scenes)
		return;
	const uint32_t n = tri_off[s + 1] - tri_off[s];
	const uint32_t ref = n == 0 ? kNone : (n == 1 ? (kLeafBit | tri_off[s]) : int_off[s]);
	items[s] = Item{ref, s};
	const float lo[3] = {ord2f(gb[6 * s]), ord2f(gb[6 * s + 1]), ord2f(gb[6 * s + 2])};
	const float hi[3] = {ord2f(gb[6 * s + 3]), ord2f(gb[6 * s + 4]), ord2f(gb[6 * s + 5])};
	far[s] = far_scene(lo, hi, n);
}

__device__ __forceinline__ float open_area(uint32_t r, const float4 *ibox) {
	return (r & kLeafBit) ? -1.0f : half_area(ibox[2 * r], ibox[2 * r + 1]);
}

__device__ __forceinline__ float cdec(float o, uint32_t q, float s) { return cdec_f(o, (float)q, s); }

// Largest q in [0, 255] whose decoded value is <= v (decoding is monotone in q and
// q = 0 decodes to the origin, which is <= every child bound).  The estimate comes from
// a directed-rounding FP32 quotient; the loops make the answer exact, so it does not
// depend on the estimate.
__device__ uint32_t quant_lo(float o, float s, float v) {
	const float g = floorf(__fdiv_rd(__fsub_rd(v, o), s));
	uint32_t q = (uint32_t)fminf(fmaxf(g, 0.0f), 255.0f);
	while (q > 0 && cdec(o, q, s) > v)
		--q;
	while (q < 255 && cdec(o, q + 1, s) <= v)
		++q;
	return q;
}

// Smallest q in [0, 255] whose decoded value is >= v (the exponent was chosen so that
// q = 255 qualifies).
__device__ uint32_t quant_hi(float o, float s, float v) {
	const float g = ceilf(__fdiv_ru(__fsub_ru(v, o), s));
	uint32_t q = (uint32_t)fminf(fmaxf(g, 0.0f), 255.0f);
	while (q < 255 && cdec(o, q, s) < v)
		++q;
	while (q > 0 && cdec(o, q - 1, s) >= v)
		--q;
	return q;
}

// Smallest biased exponent e in [1, 254] with o + 255 * 2^(e-127) >= mx in FP32 (254
// when none is; the traversal then still tests the children exactly at the leaves).
// The start is at most the answer: the FP32 range rounded up, over 255 rounded up, has
// an exponent at least that of the answer's scale less two.
__device__ uint32_t scale_exponent(float mn, float mx) {
	const float r = __fdiv_ru(__fsub_ru(mx, mn), 255.0f);
	int e = 254;
	if (isfinite(r)) {
		const uint32_t bits = __float_as_uint(r);
		const int e0 = (int)((bits >> 23) & 0xFFu) + ((bits & 0x7FFFFFu) ? 1 : 0);
		e = max(1, min(254, e0 - 2));
	}
	while (e < 254 && cdec(mn, 255u, cscale((uint8_t)e)) < mx)
		++e;
	return (uint32_t)e;
}

// One compressed node from its eight children, lane k of a group of 8 lanes (gmask) on child
// k: its reference r (kNone: an unused slot) and box.  Every lane of the warp calls this;
// groups with live == false write nothing.
__device__ __forceinline__ void write_cnode(CNode8 *cn, uint32_t i, bool live, unsigned gmask,
                                            uint32_t k, uint32_t r, const float lo[3],
                                            const float hi[3]) {
	const bool used = r != kNone;
	const bool leaf = used && (r & kLeafBit);
	uint32_t cb = (used && !leaf) ? r : kNone;
	uint32_t tb = leaf ? leaf_first(r) : kNone;
	float mn[3], mx[3];
	for (int a = 0; a < 3; ++a) {
		mn[a] = used ? lo[a] : INFINITY;
		mx[a] = used ? hi[a] : -INFINITY;
	}
	for (int o = 4; o > 0; o >>= 1) {
		cb = min(cb, __shfl_xor_sync(gmask, cb, o, 8));
		tb = min(tb, __shfl_xor_sync(gmask, tb, o, 8));
		for (int a = 0; a < 3; ++a) {
			mn[a] = fminf(mn[a], __shfl_xor_sync(gmask, mn[a], o, 8));
			mx[a] = fmaxf(mx[a], __shfl_xor_sync(gmask, mx[a], o, 8));
		}
	}
	const uint32_t imask = (__ballot_sync(gmask, used && !leaf) >> (threadIdx.x & 24u)) & 0xFFu;
	if (!live)
		return;
	float org[3];
	uint32_t ex[3];
	for (int a = 0; a < 3; ++a) {
		if (!(mn[a] <= mx[a])) { // no children: an empty frame at the origin
			mn[a] = 0.0f;
			mx[a] = 0.0f;
		}
		org[a] = mn[a];
		ex[a] = scale_exponent(mn[a], mx[a]);
	}
	const uint32_t tri_base = tb == kNone ? 0u : tb;
	CChild8 c;
	c.qlo_x = c.qhi_x = c.qlo_y = c.qhi_y = c.qlo_z = c.qhi_z = 0;
	c.count = 0;
	c.first = 0;
	if (used) {
		uint8_t q[6];
		for (int a = 0; a < 3; ++a) {
			const float sc = cscale((uint8_t)ex[a]);
			q[2 * a] = (uint8_t)quant_lo(org[a], sc, lo[a]);
			q[2 * a + 1] = (uint8_t)quant_hi(org[a], sc, hi[a]);
		}
		c.qlo_x = q[0];
		c.qhi_x = q[1];
		c.qlo_y = q[2];
		c.qhi_y = q[3];
		c.qlo_z = q[4];
		c.qhi_z = q[5];
		if (leaf) {
			c.count = (uint8_t)leaf_count(r);
			c.first = (uint8_t)(leaf_first(r) - tri_base);
		}
	}
	cn[i].c[k] = c;
	if (k == 0) { // the 32-byte header as two 16-byte stores (ex, ey, ez, imask: bytes 12-15)
		uint4 *h = reinterpret_cast<uint4 *>(&cn[i]);
		h[0] = make_uint4(__float_as_uint(org[0]), __float_as_uint(org[1]),
		                  __float_as_uint(org[2]),
		                  ex[0] | (ex[1] << 8) | (ex[2] << 16) | (imask << 24));
		h[1] = make_uint4(cb == kNone ? 0u : cb, tri_base, 0u, 0u);
	}
}
static_assert(offsetof(CNode8, ex) == 12 && offsetof(CNode8, imask) == 15 &&
                  offsetof(CNode8, child_base) == 16 && offsetof(CNode8, tri_base) == 20 &&
                  offsetof(CNode8, c) == 32,
              "CNode8 header layout");


// The compressed nodes of a tree whose Node8 array is built (the one-block build; the
// level-by-level collapse writes them itself).  n_nodes_dev holds the node count on the
// device: the launch covers the node capacity.
__global__ void __launch_bounds__(256)
    k_compress(const Node8 *__restrict__ nodes, const uint32_t *n_nodes_dev, CNode8 *cn) {
	const uint32_t k = threadIdx.x & 7u;
	const uint32_t i = blockIdx.x * (blockDim.x / 8u) + threadIdx.x / 8u;
	const bool live = i < *n_nodes_dev;
	uint32_t r = kNone;
	float lo[3] = {0.0f, 0.0f, 0.0f}, hi[3] = {0.0f, 0.0f, 0.0f};
	if (live) {
		const float4 *src = reinterpret_cast<const float4 *>(&nodes[i].c[k]);
		const float4 a = __ldg(src), b = __ldg(src + 1);
		lo[0] = child_lo(a.x, a.z);
		hi[0] = child_hi(a.x, a.z);
		lo[1] = child_lo(a.y, a.w);
		hi[1] = child_hi(a.y, a.w);
		lo[2] = child_lo(b.x, b.y);
		hi[2] = child_hi(b.x, b.y);
		r = __float_as_uint(b.z);
	}
	write_cnode(cn, i, live, 0xFFu << (threadIdx.x & 24u), k, r, lo, hi);
}


struct CollapseArgs {
	const float *tris;
	const uint32_t *vals;     // position -> input triangle
	const uint32_t *scene_of; // scene of each input triangle (null: one scene)
	const uint32_t *tri_off;
	const uint32_t *left, *right, *rfirst, *rlast;
	const float4 *ibox, *lbox;
	const CostNode *cost;     // null: open the largest child first
	uint32_t leaf_size, n, node_cap;
	uint32_t *node_counter, *tri_counter;
	Node8 *nodes;
	CNode8 *cnodes;           // null: not built
	float4 *tri4;
	uint32_t *inv;
	uint32_t *err;
};

constexpr uint32_t kCollapseItems = 32; // frontier items per block (8 lanes each)

// One level: each frontier item becomes an 8-wide node, with its compressed form and the
// records of its leaf triangles (tri4.w holds the per-scene primitive id, inv maps an
// input triangle to its position).  Eight lanes per item; the node slots, triangle ranges
// and next-level items of a block's 32 items are reserved with one atomic per counter.
//
// A level is a chain of dependent loads, which bounds the small levels, and scattered
// reads of the binary tree.  With one thread per item, opening up to seven subtrees one
// after another, a level took 14 to 53 us even for a few hundred items; here every subtree
// of an item opens at once (at most 7 rounds, mostly 3 or 4) and a node's children, 256 B,
// its compressed form and its triangles are written by neighbouring lanes.  Compression
// and triangle records were passes of their own over all nodes and triangles (46 and 23 us
// on the 1,048,576-triangle heightfield, 278 and 138 us on a batch of 4.6M triangles).
// Builds: 65,790-triangle heightfield 0.89 -> 0.80 ms, 1,048,576 triangles 2.32 -> 2.17 ms; the
// batch's collapse, compression and records 926 -> 702 us.
__global__ void __launch_bounds__(8 * kCollapseItems)
    k_collapse(CollapseArgs A, const Item *in, const uint32_t *in_count, Item *out,
               uint32_t *out_count) {
	chain_enter();
	__shared__ uint32_t xch[8 * kCollapseItems]; // per item: what each child slot receives
	__shared__ uint32_t need[kCollapseItems];    // per item: inner children | triangles << 16
	__shared__ uint32_t got[3];                  // the block's nodes, triangles, items
	const uint32_t n_in = *in_count;
	const uint32_t lane = threadIdx.x & 31u, c8 = lane & 7u, gsh = lane & 24u;
	const unsigned gmask = 0xFFu << gsh;
	uint32_t *x = xch + (threadIdx.x & ~7u);
	for (uint32_t base = blockIdx.x * kCollapseItems; base < n_in;
	     base += gridDim.x * kCollapseItems) {
		const uint32_t w = base + threadIdx.x / 8u;
		const bool live = w < n_in;
		const Item it = live ? in[w] : Item{kNone, 0u};
		const bool full = live && it.ref != kNone; // (an empty scene: a node without children)
		// The item's children: lane c8 ends with child c8 in order of first leaf.
		uint32_t y = kNone;
		if (A.cost) {
			// Slot ranges: lane c8 holds the subtree covering slots [c8, c8 + span).  A
			// subtree opened into its span (the item itself always; another when its cost in
			// `span` slots is below its cost in one) splits it: the left child keeps the first
			// split_of(span) slots, the right child goes to the lane after them.  The ranges
			// end in depth-first order, left subtrees first: by first leaf.
			uint32_t span = (full && c8 == 0u) ? 8u : 0u;
			y = it.ref;
			for (int round = 0; round < 8; ++round) {
				uint32_t give = kNone, a = 0;
				if (span > 1u && !(y & kLeafBit)) {
					const CostNode *cn = A.cost + y;
					const uint32_t bits = cn->bits, l = A.left[y], r = A.right[y];
					const float one = cn->c1, open = cn->cd[span - 2u];
					if (round == 0 || open < one) {
						a = split_of(bits, span);
						give = r;
						y = l;
					}
				}
				if (!__any_sync(0xFFFFFFFFu, give != kNone))
					break;
				// The right child's lane is inside the giver's range: no other holder is there.
				const uint32_t given = give != kNone ? span - a : 0u;
				x[c8] = kNone;
				__syncwarp();
				if (give != kNone)
					x[c8 + a] = (c8 << 8) | given;
				__syncwarp();
				const uint32_t from = x[c8];
				const uint32_t moved = __shfl_sync(0xFFFFFFFFu, give, (int)(gsh | ((from >> 8) & 7u)));
				if (from != kNone) {
					y = moved;
					span = from & 0xFFu;
				} else if (give != kNone) {
					span = a;
				}
			}
			const bool has = span > 0u;
			const uint32_t held = (__ballot_sync(0xFFFFFFFFu, has) >> gsh) & 0xFFu;
			x[c8] = kNone;
			__syncwarp();
			if (has)
				x[__popc(held & ((1u << c8) - 1u))] = y;
			__syncwarp();
			y = x[c8];
		} else {
			// Open the binary child of largest surface area until 8 children: any binary
			// node can be opened, so nodes fill up and small subtrees end as single
			// triangles.  Ties go to the child created first.
			uint32_t nc = full ? 1u : 0u;
			y = (full && c8 == 0u) ? it.ref : kNone;
			float area = y != kNone ? open_area(y, A.ibox) : -1.0f;
			for (int round = 0; round < 7; ++round) {
				float m = area;
				uint32_t at = c8;
#pragma unroll
				for (int o = 4; o > 0; o >>= 1) {
					const float mo = __shfl_xor_sync(0xFFFFFFFFu, m, o, 8);
					const uint32_t ao = __shfl_xor_sync(0xFFFFFFFFu, at, o, 8);
					if (mo > m || (mo == m && ao < at)) {
						m = mo;
						at = ao;
					}
				}
				const bool go = nc > 0u && m > -1.0f;
				if (!__any_sync(0xFFFFFFFFu, go))
					break;
				const uint32_t b = __shfl_sync(0xFFFFFFFFu, y, (int)at, 8);
				if (go) {
					// Children and their areas (stored by the build) in one round of loads.
					if (c8 == at) {
						y = A.left[b];
						area = A.ibox[2 * (size_t)b].w;
					} else if (c8 == nc) {
						y = A.right[b];
						area = A.ibox[2 * (size_t)b + 1].w;
					}
					++nc;
				}
			}
			// By first leaf (first leaves of distinct children differ).
			const uint32_t first =
			    y == kNone ? 0xFFFFFFFFu : ((y & kLeafBit) ? (y & ~kLeafBit) : A.rfirst[y]);
			uint32_t rank = 0;
#pragma unroll
			for (int o = 1; o < 8; ++o) {
				const uint32_t fo = __shfl_sync(0xFFFFFFFFu, first, (int)((c8 + o) & 7u), 8);
				rank += fo < first;
			}
			x[c8] = kNone;
			__syncwarp();
			if (y != kNone)
				x[rank] = y;
			__syncwarp();
			y = x[c8];
		}
		// This lane's child: its box, first leaf and triangle count, and whether it becomes a
		// node.  A leaf's first triangle is read now, so that its wait overlaps the scan.
		const bool has = y != kNone;
		float lo[3] = {0.0f, 0.0f, 0.0f}, hi[3] = {0.0f, 0.0f, 0.0f};
		uint32_t first = 0, cnt = 0;
		bool inner = false;
		if (has) {
			const bool single = (y & kLeafBit) != 0u;
			const uint32_t id = y & ~kLeafBit;
			const float4 *src = single ? A.lbox + 2 * (size_t)id : A.ibox + 2 * (size_t)id;
			const float4 l = *src, h = src[1];
			lo[0] = l.x;
			lo[1] = l.y;
			lo[2] = l.z;
			hi[0] = h.x;
			hi[1] = h.y;
			hi[2] = h.z;
			first = single ? id : A.rfirst[id];
			cnt = single ? 1u : A.rlast[id] - first + 1u;
			inner = is_inner(y, cnt, A.leaf_size, A.cost);
		}
		const bool leaf = has && !inner;
		const uint32_t g0 = leaf ? A.vals[first] : 0u;
		const uint32_t inners = (__ballot_sync(0xFFFFFFFFu, inner) >> gsh) & 0xFFu;
		const uint32_t my_tris = leaf ? cnt : 0u;
		uint32_t sum = my_tris;
#pragma unroll
		for (uint32_t o = 1; o < 8u; o <<= 1) {
			const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, sum, o, 8);
			if (c8 >= o)
				sum += v;
		}
		const uint32_t group = __popc(inners) | (__shfl_sync(0xFFFFFFFFu, sum, 7, 8) << 16);
		if (c8 == 0u)
			need[threadIdx.x / 8u] = group;
		__syncthreads();
		if (threadIdx.x < 32u) {
			uint32_t v = need[lane];
			const uint32_t own = v;
#pragma unroll
			for (uint32_t o = 1; o < 32u; o <<= 1) {
				const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, v, o);
				if (lane >= o)
					v += u;
			}
			need[lane] = v - own; // exclusive
			const uint32_t total = __shfl_sync(0xFFFFFFFFu, v, 31);
			const uint32_t nodes = total & 0xFFFFu, tris = total >> 16;
			if (lane == 0)
				got[0] = nodes ? atomicAdd(A.node_counter, nodes) : 0u;
			if (lane == 1)
				got[1] = tris ? atomicAdd(A.tri_counter, tris) : 0u;
			if (lane == 2)
				got[2] = nodes ? atomicAdd(out_count, nodes) : 0u;
			__syncwarp();
			if (lane == 0 && (got[0] + nodes > A.node_cap || got[1] + tris > A.n ||
			                  got[2] + nodes > A.node_cap)) {
				set_error_bits(A.err, kErrCollapse);
				got[0] = kNone; // nothing of the block's items is written
			}
		}
		__syncthreads();
		const uint32_t before = need[threadIdx.x / 8u];
		if (got[0] != kNone) {
			const uint32_t k = __popc(inners & ((1u << c8) - 1u)) + (before & 0xFFFFu);
			uint32_t dst = got[1] + (before >> 16) + sum - my_tris;
			uint32_t ref = kNone;
			if (inner) {
				ref = got[0] + k;
				out[got[2] + k] = Item{y, ref};
			} else if (leaf) {
				ref = make_leaf(dst, cnt);
			}
			if (live)
				A.nodes[it.slot].c[c8] =
				    encode_child(make_float4(lo[0], lo[1], lo[2], 0.0f),
				                 make_float4(hi[0], hi[1], hi[2], 0.0f), ref);
			if (A.cnodes)
				write_cnode(A.cnodes, it.slot, live, gmask, c8, ref, lo, hi);
			if (leaf)
				for (uint32_t j = 0; j < cnt; ++j, ++dst) {
					const uint32_t g = j == 0 ? g0 : A.vals[first + j];
					const uint32_t pid = A.scene_of ? g - A.tri_off[A.scene_of[g]] : g;
					const float *t = A.tris + 9 * (size_t)g;
					A.inv[g] = dst;
					float4 *to = A.tri4 + 3 * (size_t)dst;
					to[0] = make_float4(t[0], t[1], t[2], __uint_as_float(pid));
					to[1] = make_float4(t[3], t[4], t[5], tri_finite(t) ? 0.0f : 1.0f);
					to[2] = make_float4(t[6], t[7], t[8], 0.0f);
				}
		}
		__syncthreads(); // got and need are read before the next items overwrite them
	}
}

#define BUILD_TRY(call)                                                                        \
	do {                                                                                       \
		cudaError_t e_ = (call);                                                               \
		if (e_ != cudaSuccess) {                                                               \
			msg = std::string("CUDA error in build: ") + cudaGetErrorString(e_) + " (" #call ")"; \
			return e_ == cudaErrorMemoryAllocation ? PRT_ERR_OOM : PRT_ERR_CUDA;              \
		}                                                                                      \
	} while (0)

inline unsigned blocks_for(uint64_t n, unsigned t) { return (unsigned)((n + t - 1) / t); }

// log2 of the bits of XFaces for n triangles.
inline uint32_t x_faces_log(uint64_t n) {
	uint32_t log = 10;
	while ((1ull << log) < 8ull * n)
		++log;
	return log;
}

} // namespace

int build_plan(const uint64_t *tri_off64, uint32_t S, int leaf_size, bool compressed,
               SceneGPU &sc, BuildScratch &ws, cudaStream_t st, BuildPlan &plan,
               std::string &msg, bool sah, bool collapse_cost, bool one_block) {
	if (leaf_size < 1 || leaf_size > kMaxLeaf) {
		msg = "leaf_size must be in [1, 8]";
		return PRT_ERR_ARG;
	}
	if (S == 0 || !tri_off64 || tri_off64[0] != 0) {
		msg = "build: at least one scene, offsets starting at 0";
		return PRT_ERR_ARG;
	}
	for (uint32_t s = 0; s < S; ++s) {
		if (tri_off64[s + 1] < tri_off64[s]) {
			msg = "build: triangle offsets must not decrease";
			return PRT_ERR_ARG;
		}
	}
	const uint64_t n64 = tri_off64[S];
	if (n64 > kMaxTris) {
		msg = "set_tris: at most 134217727 triangles per scene";
		return PRT_ERR_LIMIT;
	}
	plan.S = S;
	plan.n = (uint32_t)n64;
	plan.leaf_size = leaf_size;
	plan.compressed = compressed;
	plan.multi = S > 1;
	plan.sah = sah;
	plan.collapse_cost = collapse_cost;
	plan.small = one_block && sah && S == 1 && n64 >= 1 && n64 <= small_build_max();
	plan.toff.resize(S + 1);
	plan.ioff.resize(S + 1);
	for (uint32_t s = 0; s <= S; ++s)
		plan.toff[s] = (uint32_t)tri_off64[s];
	plan.n_int = 0;
	for (uint32_t s = 0; s <= S; ++s) {
		plan.ioff[s] = plan.n_int;
		if (s < S) {
			const uint32_t ns = plan.toff[s + 1] - plan.toff[s];
			plan.n_int += ns > 1 ? ns - 1 : 0;
		}
	}
	if (plan.n_int >= std::max<uint32_t>(plan.toff[S], 1u)) {
		msg = "build: inconsistent scene offsets";
		return PRT_ERR_ARG;
	}
	plan.scene_digits = 0;
	for (uint32_t v = S - 1; v; v >>= 8)
		++plan.scene_digits;
	const uint32_t n = plan.n;
	plan.node_cap = n + S;

	sc.n_scenes = S;
	sc.n_tris = n;
	sc.leaf_size = leaf_size;
	sc.n_nodes = 0;
	sc.depth = 0;
	sc.has_cnodes = false;
	sc.built_small = false;
	sc.x_log = 0;
	sc.h_tri_off.assign(tri_off64, tri_off64 + S + 1);

	const size_t key_bytes = plan.multi ? 8 : 4;
	// SAH node ids run up to n_int + S (scene s's root is node s).
	const size_t ni = std::max<size_t>((size_t)plan.n_int + (sah ? S : 0u), 1);
	const size_t nn = std::max<uint32_t>(n, 1);
	BUILD_TRY(sc.tri_off.reserve(4ull * (S + 1)));
	BUILD_TRY(ws.keys.reserve(key_bytes * nn));
	BUILD_TRY(ws.keys2.reserve(key_bytes * nn));
	BUILD_TRY(ws.vals.reserve(4 * nn));
	BUILD_TRY(ws.vals2.reserve(4 * nn));
	if (plan.multi)
		BUILD_TRY(ws.scene_of.reserve(4 * nn));
	BUILD_TRY(ws.int_off.reserve(4ull * (S + 1)));
	BUILD_TRY(ws.left.reserve(4 * ni));
	BUILD_TRY(ws.right.reserve(4 * ni));
	BUILD_TRY(ws.splits.reserve(16 * nn));
	BUILD_TRY(ws.rfirst.reserve(4 * ni));
	BUILD_TRY(ws.rlast.reserve(4 * ni));
	BUILD_TRY(ws.flags.reserve(4 * ni));
	BUILD_TRY(ws.ibox.reserve(32 * ni));
	BUILD_TRY(ws.lbox.reserve(32 * nn));
	BUILD_TRY(ws.items_a.reserve(8ull * plan.node_cap));
	BUILD_TRY(ws.items_b.reserve(8ull * plan.node_cap));
	BUILD_TRY(ws.counters.reserve(4 * kCtrWords));
	BUILD_TRY(ws.sort_hist.reserve(8 * 256 * 4));
	BUILD_TRY(ws.sort_tiles.reserve(8 * 4));
	BUILD_TRY(ws.sort_status.reserve(4 * sort_status_words(n)));
	BUILD_TRY(ws.bounds.reserve(24ull * S));
	if (sah && !plan.small) {
		BUILD_TRY(ws.sah.reserve(sah_scratch_bytes(n, S)));
		BUILD_TRY(ws.roots.reserve(4ull * S));
	}
	if (collapse_cost)
		BUILD_TRY(ws.cost.reserve(sizeof(CostNode) * ni));
	BUILD_TRY(sc.tri4.reserve(48 * nn));
	BUILD_TRY(sc.inv.reserve(4 * nn));
	// One node past the capacity: the empty node the traversal pads partial steps with; after
	// it what tells far rays, per scene (far_scenes).
	// As large as the triangle records' buffer may need: it moves only when that does, so that a
	// captured query that still finds the one finds the other.
	plan.x_log = 0;
	if (sah && !plan.small && !plan.multi && n) {
		BUILD_TRY(sc.x_faces.reserve(4ull * (kXHead + (1ull << (x_faces_log(sc.tri4.bytes / 48) - 5u)))));
		plan.x_log = x_faces_log(n);
	}
	plan.x_drop = plan.x_log ? nullptr : sc.x_faces.as<uint32_t>();
	BUILD_TRY(sc.nodes.reserve(sizeof(Node8) * ((size_t)plan.node_cap + 1) + sizeof(float4) * S));
	if (compressed)
		BUILD_TRY(sc.cnodes.reserve(sizeof(CNode8) * ((size_t)plan.node_cap + 1)));
	// Work items hold 27-bit node indices; a tree's nodes stay below n - 1 < 2^27 - 1.
	sc.dead = std::min<uint32_t>(plan.node_cap, kIndexMask);
	if (!ws.h_counters)
		BUILD_TRY(cudaMallocHost(&ws.h_counters, 4 * (kCtrWords + kHostSahWords)));
	ws.h_sah = ws.h_counters + kCtrWords;
	if (plan.small)
		return PRT_OK; // the one-block build reads no offset table
	BUILD_TRY(cudaMemcpyAsync(sc.tri_off.p, plan.toff.data(), 4ull * (S + 1),
	                          cudaMemcpyHostToDevice, st));
	BUILD_TRY(cudaMemcpyAsync(ws.int_off.p, plan.ioff.data(), 4ull * (S + 1),
	                          cudaMemcpyHostToDevice, st));
	return PRT_OK;
}

// Morton codes, radix sort, Karras hierarchy and refit: the binary trees of the LBVH
// path, with svals set to the sorted triangle order.
static int lbvh_enqueue(const float *d_tris, const BuildPlan &plan, BuildScratch &ws,
                        const uint32_t *d_toff, const uint32_t *d_ioff, const uint32_t *scene_of,
                        cudaStream_t st, uint32_t *d_err, const uint32_t *&svals, std::string &msg) {
	const uint32_t S = plan.S, n = plan.n, n_int = plan.n_int;
	const size_t ni = std::max<uint32_t>(n_int, 1);
	const size_t nn = std::max<uint32_t>(n, 1);
	uint32_t *gb = ws.bounds.as<uint32_t>();
	svals = ws.vals.as<uint32_t>();
	k_bounds_init<<<blocks_for(6ull * S, 256), 256, 0, st>>>(gb, S, d_toff,
	                                                         ws.splits.as<uint4>(), plan.x_drop);
	if (n)
		k_centroid_bounds<<<std::min(blocks_for(n, 256), 2048u), 256, 0, st>>>(d_tris, n, scene_of,
		                                                                        gb);
	SortScratch ss{ws.sort_hist.as<uint32_t>(), ws.sort_tiles.as<uint32_t>(),
	               ws.sort_status.as<uint32_t>()};
	const void *skeys = ws.keys.p;
	if (n && !plan.multi) {
		k_morton<uint32_t><<<blocks_for(n, 256), 256, 0, st>>>(d_tris, n, nullptr, gb,
		                                                       ws.keys.as<uint32_t>(),
		                                                       ws.vals.as<uint32_t>());
		int where = sort_pairs_u32(ws.keys.as<uint32_t>(), ws.vals.as<uint32_t>(),
		                           ws.keys2.as<uint32_t>(), ws.vals2.as<uint32_t>(), n, 4, ss, st,
		                           d_err);
		skeys = where ? ws.keys2.p : ws.keys.p;
		svals = where ? ws.vals2.as<uint32_t>() : ws.vals.as<uint32_t>();
	} else if (n) {
		k_morton<uint64_t><<<blocks_for(n, 256), 256, 0, st>>>(d_tris, n, scene_of, gb,
		                                                       ws.keys.as<uint64_t>(),
		                                                       ws.vals.as<uint32_t>());
		int where = sort_pairs_u64(ws.keys.as<uint64_t>(), ws.vals.as<uint32_t>(),
		                           ws.keys2.as<uint64_t>(), ws.vals2.as<uint32_t>(), n,
		                           4 + plan.scene_digits, ss, st, d_err);
		skeys = where ? ws.keys2.p : ws.keys.p;
		svals = where ? ws.vals2.as<uint32_t>() : ws.vals.as<uint32_t>();
	}

	if (n_int) {
		if (plan.multi)
			k_karras<uint64_t><<<blocks_for(n_int, 256), 256, 0, st>>>(
			    static_cast<const uint64_t *>(skeys), n_int, d_toff, d_ioff, S,
			    ws.left.as<uint32_t>(), ws.right.as<uint32_t>(), ws.splits.as<uint4>(),
			    ws.rfirst.as<uint32_t>(), ws.rlast.as<uint32_t>());
		else
			k_karras<uint32_t><<<blocks_for(n_int, 256), 256, 0, st>>>(
			    static_cast<const uint32_t *>(skeys), n_int, d_toff, d_ioff, S,
			    ws.left.as<uint32_t>(), ws.right.as<uint32_t>(), ws.splits.as<uint4>(),
			    ws.rfirst.as<uint32_t>(), ws.rlast.as<uint32_t>());
	}
	return PRT_OK;
}

// The empty node at index sc.dead (node_cap, past every built node): eight NaN boxes with no reference (no slab test
// passes them, and the general test skips a child without reference); compressed, a
// node with no inner mask and no leaf counts.  Queued on the build's stream, so a batch
// graph captures it with the build.
static cudaError_t write_dead_node(const BuildPlan &plan, SceneGPU &sc, cudaStream_t st) {
	cudaError_t e = cudaMemsetAsync(static_cast<char *>(sc.nodes.p) +
	                                    sizeof(Node8) * (size_t)sc.dead,
	                                0xFF, sizeof(Node8), st);
	if (e == cudaSuccess && plan.compressed)
		e = cudaMemsetAsync(static_cast<char *>(sc.cnodes.p) + sizeof(CNode8) * (size_t)sc.dead,
		                    0, sizeof(CNode8), st);
	return e;
}

// From the binary trees to the 8-wide ones: the bottom-up pass and the collapse.  With host
// checks it waits, and the counters (kCtrGate among them) are in ws.h_counters.
static int collapse_enqueue(const float *d_tris, const BuildPlan &plan, SceneGPU &sc,
                            BuildScratch &ws, const uint32_t *svals, const uint32_t *roots,
                            cudaStream_t st, uint32_t *d_err, bool host_checks,
                            std::string &msg) {
	const uint32_t S = plan.S, n = plan.n, n_int = plan.n_int;
	uint32_t *d_toff = sc.tri_off.as<uint32_t>();
	uint32_t *scene_of = plan.multi ? ws.scene_of.as<uint32_t>() : nullptr;
	uint32_t *ctr = ws.counters.as<uint32_t>();
	// Binary node ids run up to n_int (LBVH) or n_int + S (SAH: scene s's root is s).
	const uint32_t n_ids = n_int + (plan.sah ? S : 0u);
	const bool use_cost = plan.collapse_cost && n_int;
	if (n && (!plan.sah || use_cost)) {
		UpArgs U;
		U.tris = d_tris;
		U.vals = svals;
		U.n = n;
		U.n_ids = n_ids;
		U.splits = ws.splits.as<uint4>();
		U.left = ws.left.as<uint32_t>();
		U.right = ws.right.as<uint32_t>();
		U.ibox = ws.ibox.as<float4>();
		U.lbox = ws.lbox.as<float4>();
		U.flags = ws.flags.as<uint32_t>();
		U.cost = ws.cost.as<CostNode>();
		U.leaf_size = (uint32_t)plan.leaf_size;
		U.gate = plan.sah ? ctr + kCtrGate : nullptr;
		U.err = d_err;
		BUILD_TRY(cudaMemsetAsync(ws.flags.p, 0, 4ull * std::max<uint32_t>(n_ids, 1u), st));
		// (items_a is free until the collapse, which starts after the walks.)
		U.walks = ws.items_a.as<uint32_t>();
		U.walk_cap = 2u * plan.node_cap;
		U.n_walks = ctr + kCtrWalks;
		const unsigned grid = blocks_for(n, kUpLeaves);
		const unsigned g_walk = std::min(1216u, blocks_for(n, 128));
		if (plan.sah) {
			k_bottom_up<false, true><<<grid, kUpLeaves, 0, st>>>(U);
			launch_after(host_checks, k_walk_up<false, true>, g_walk, 128, st, U);
		} else if (use_cost) {
			k_bottom_up<true, true><<<grid, kUpLeaves, 0, st>>>(U);
			launch_after(host_checks, k_walk_up<true, true>, g_walk, 128, st, U);
		} else {
			k_bottom_up<true, false><<<grid, kUpLeaves, 0, st>>>(U);
			launch_after(host_checks, k_walk_up<true, false>, g_walk, 128, st, U);
		}
	}
	const CostNode *cost = use_cost ? ws.cost.as<CostNode>() : nullptr;

	Item *items_of[2] = {ws.items_a.as<Item>(), ws.items_b.as<Item>()};
	launch_after(host_checks, k_collapse_roots, blocks_for(S, 128), 128, st, d_toff, roots, S,
	             items_of[0], ctr, ws.bounds.as<uint32_t>(), far_scenes(sc.nodes.p, sc.dead));
	CollapseArgs A;
	A.tris = d_tris;
	A.vals = svals;
	A.scene_of = scene_of;
	A.tri_off = d_toff;
	A.left = ws.left.as<uint32_t>();
	A.right = ws.right.as<uint32_t>();
	A.rfirst = ws.rfirst.as<uint32_t>();
	A.rlast = ws.rlast.as<uint32_t>();
	A.ibox = ws.ibox.as<float4>();
	A.lbox = ws.lbox.as<float4>();
	A.cost = cost;
	A.leaf_size = (uint32_t)plan.leaf_size;
	A.n = n;
	A.node_cap = plan.node_cap;
	A.node_counter = ctr + kCtrNodes;
	A.tri_counter = ctr + kCtrTris;
	A.nodes = sc.nodes.as<Node8>();
	A.cnodes = plan.compressed ? sc.cnodes.as<CNode8>() : nullptr;
	A.tri4 = sc.tri4.as<float4>();
	A.inv = sc.inv.as<uint32_t>();
	A.err = d_err;
	// Levels before the first look at the counters (a host wait each, about 10 us; an empty
	// level costs 2): two more than a full 8-wide tree of the largest scene needs.
	int ahead = kMaxLevels;
	if (host_checks) {
		uint32_t biggest = 1;
		for (uint32_t s = 0; s < S; ++s)
			biggest = std::max(biggest, plan.toff[s + 1] - plan.toff[s]);
		ahead = 2;
		for (uint64_t c = 1; c < biggest; c *= 8)
			++ahead;
	}
	int level = 0;
	for (;;) {
		for (int k = 0; k < ahead && level < kMaxLevels; ++k, ++level) {
			// No more blocks than the level can have items for.
			const uint64_t items =
			    std::min<uint64_t>((uint64_t)S << std::min(3 * level, 30), plan.node_cap);
			const unsigned grid = (unsigned)std::min<uint64_t>(
			    1216, (items + kCollapseItems - 1) / kCollapseItems);
			launch_after(host_checks, k_collapse, grid, 8 * kCollapseItems, st, A,
			             items_of[level & 1], ctr + level, items_of[(level + 1) & 1],
			             ctr + level + 1);
		}
		if (!host_checks)
			break;
		BUILD_TRY(cudaMemcpyAsync(ws.h_counters, ctr, 4 * kCtrWords, cudaMemcpyDeviceToHost, st));
		BUILD_TRY(cudaStreamSynchronize(st));
		if (ws.h_counters[level] == 0 || ws.h_counters[kCtrGate] != 0)
			break;
		if (level >= kMaxLevels) {
			msg = "tree deeper than " + std::to_string(kMaxLevels) + " levels";
			return PRT_ERR_LIMIT;
		}
		ahead = kLevelsPerCheck;
	}
	BUILD_TRY(cudaGetLastError());
	return PRT_OK;
}

int build_enqueue(const float *d_tris, const BuildPlan &plan, SceneGPU &sc, BuildScratch &ws,
                  cudaStream_t st, uint32_t *d_err, bool host_checks, std::string &msg) {
	const uint32_t S = plan.S, n = plan.n;
	if (plan.sah && !host_checks) {
		msg = "the SAH build needs a look at its gate on the host";
		return PRT_ERR_ARG;
	}
	if (plan.small) {
		// One block: PLOC, collapse and re-layout in one launch, which also zeroes the
		// counters, writes the empty node and leaves the counters in the pinned host
		// buffer; the compression reads the node count on the device, so the host only
		// waits, once, at the end.
		uint32_t *ctr = ws.counters.as<uint32_t>();
		BUILD_TRY(launch_build_small(d_tris, n, (uint32_t)plan.leaf_size, plan.collapse_cost,
		                             plan.compressed, ws, sc, plan.node_cap, ctr, ws.h_counters,
		                             plan.x_drop, d_err, st));
		sc.built_small = true;
		if (plan.compressed) {
			k_compress<<<blocks_for(8ull * plan.node_cap, 256), 256, 0, st>>>(
			    sc.nodes.as<Node8>(), ctr + kCtrNodes, sc.cnodes.as<CNode8>());
			sc.has_cnodes = true;
		}
		BUILD_TRY(cudaGetLastError());
		return host_checks ? build_finish(sc, ws, st, msg, true) : PRT_OK;
	}
	BUILD_TRY(write_dead_node(plan, sc, st));
	uint32_t *d_toff = sc.tri_off.as<uint32_t>();
	uint32_t *d_ioff = ws.int_off.as<uint32_t>();
	uint32_t *scene_of = plan.multi ? ws.scene_of.as<uint32_t>() : nullptr;
	if (plan.multi)
		k_scene_of<<<std::min(S, 4096u), 256, 0, st>>>(d_toff, S, scene_of);
	const uint32_t *svals = ws.vals.as<uint32_t>();
	const uint32_t *roots = d_ioff;
	uint32_t *ctr = ws.counters.as<uint32_t>();
	int sah_level = 0; // large levels of the SAH build queued so far
	BUILD_TRY(cudaMemsetAsync(ctr, 0, 4 * kCtrWords, st));
	if (plan.sah) {
		const XFaces x_faces{sc.x_faces.as<uint32_t>(), plan.x_log};
		int rc = sah_build_enqueue(d_tris, plan, ws, d_toff, scene_of, x_faces, st, d_err,
		                           ctr + kCtrGate, sah_level, msg);
		if (rc != PRT_OK)
			return rc;
		roots = ws.roots.as<uint32_t>();
	} else {
		int rc = lbvh_enqueue(d_tris, plan, ws, d_toff, d_ioff, scene_of, st, d_err, svals, msg);
		if (rc != PRT_OK)
			return rc;
	}
	int rc = collapse_enqueue(d_tris, plan, sc, ws, svals, roots, st, d_err, host_checks, msg);
	while (rc == PRT_OK && plan.sah && ws.h_counters[kCtrGate] != 0) {
		if (ws.h_counters[kCtrGate] != kGateLevels) {
			k_clear_error<<<1, 1, 0, st>>>(d_err, kErrSah); // (reported here)
			BUILD_TRY(cudaStreamSynchronize(st));
			msg = "sah build: internal check failed";
			return PRT_ERR_DEVICE;
		}
		// Splits more uneven than the levels queued ahead allow for: the rest of them.
		BUILD_TRY(cudaMemsetAsync(ctr, 0, 4 * kCtrWords, st));
		rc = sah_build_more(plan, ws, st, d_err, ctr + kCtrGate, sah_level, msg);
		if (rc == PRT_OK)
			rc = collapse_enqueue(d_tris, plan, sc, ws, svals, roots, st, d_err, host_checks, msg);
	}
	if (rc != PRT_OK)
		return rc;
	sc.has_cnodes = plan.compressed;
	sc.x_log = plan.x_log;
	return host_checks ? build_finish(sc, ws, st, msg, true) : PRT_OK;
}

int build_finish(SceneGPU &sc, BuildScratch &ws, cudaStream_t st, std::string &msg,
                 bool on_host) {
	if (!on_host)
		BUILD_TRY(cudaMemcpyAsync(ws.h_counters, ws.counters.p, 4 * kCtrWords,
		                          cudaMemcpyDeviceToHost, st));
	BUILD_TRY(cudaStreamSynchronize(st));
	uint32_t depth = 0;
	while (depth < (uint32_t)kMaxLevels && ws.h_counters[depth])
		++depth;
	if (depth == (uint32_t)kMaxLevels && ws.h_counters[kMaxLevels]) {
		msg = "tree deeper than " + std::to_string(kMaxLevels) + " levels";
		return PRT_ERR_LIMIT;
	}
	sc.n_nodes = ws.h_counters[kCtrNodes];
	sc.depth = depth;
	if (ws.h_counters[kCtrTris] != sc.n_tris) {
		msg = "collapse placed " + std::to_string(ws.h_counters[kCtrTris]) + " of " +
		      std::to_string(sc.n_tris) + " triangles";
		return PRT_ERR_DEVICE;
	}
	return PRT_OK;
}

int build_scenes(const float *d_tris, const uint64_t *tri_off, uint32_t n_scenes, int leaf_size,
                 bool compressed, SceneGPU &sc, BuildScratch &ws, cudaStream_t st,
                 uint32_t *d_err, std::string &msg, bool sah, bool collapse_cost,
                 bool one_block) {
	BuildPlan plan;
	int rc = build_plan(tri_off, n_scenes, leaf_size, compressed, sc, ws, st, plan, msg, sah,
	                    collapse_cost, one_block);
	if (rc != PRT_OK)
		return rc;
	return build_enqueue(d_tris, plan, sc, ws, st, d_err, true, msg);
}

int build_scene(const float *d_tris, uint64_t n, int leaf_size, bool compressed, SceneGPU &sc,
                BuildScratch &ws, cudaStream_t st, uint32_t *d_err, std::string &msg, bool sah,
                bool collapse_cost, bool one_block) {
	const uint64_t off[2] = {0, n};
	return build_scenes(d_tris, off, 1, leaf_size, compressed, sc, ws, st, d_err, msg, sah,
	                    collapse_cost, one_block);
}

} // namespace prt
