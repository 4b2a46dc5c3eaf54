// prt_sah.cu - binned-SAH construction of the binary tree, the alternative to the
// Morton/Karras hierarchy of prt_build.cu for a scene that is built once and queried
// many times.
//
// portableRT's own build (bvh.hpp:58-193) splits each node top-down at the best of a
// few binned surface-area-heuristic planes; this is the same kind of tree, built
// breadth-first on the GPU.  Every node is a contiguous range of a permutation of the
// scene's triangles, so the outputs are exactly what the LBVH path hands the collapse:
// the final order (vals), leaf boxes in that order, children, leaf ranges and node
// boxes with the children's surface areas in the w slots.  The answers do not depend on
// the tree (the traversal examines every triangle whose box the ray passes); only the
// number of boxes a ray passes does, which is what the heuristic minimises.
//
// Tasks are ranges still to be split, in three tiers by size:
//   large (> 512 triangles): level by level, one warp per task picks the plane from the
//         task's 3 x 32 global bins (k_sah_split) and blocks scatter chunks of 256 to 1,024
//         triangles to the other buffer, adding each to the bins of the child it goes to
//         (k_sah_part; k_sah_bin fills the roots' bins);
//   mid   (33-512): one block per task, all its levels in shared memory (k_sah_mid);
//   small (<= 32): one warp builds the whole subtree, one triangle per lane, with an
//         exact sweep over the sorted centres of each axis (k_sah_small).
// Binning uses box centres; a task deeper than 48 levels, or one whose centres all fall
// into one bin on every axis, is split into halves instead.  All positions, node ids and
// list slots are checked before they are written; a failed check sets kErrSah.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>

#include "../../include/prt_b200.h"
#include "prt_build.cuh"
#include "prt_launch.cuh"
#include "prt_sah.cuh"

namespace prt {
namespace {

constexpr int kBins = 32;
constexpr uint32_t kLarge = 512;    // larger tasks are binned by many blocks (512 / 1,024
                                    // / 4,096: heightfield build 3.05 / 3.16 / 3.83 ms)
constexpr uint32_t kSmall = 32;     // tasks up to this size go to one warp each
// Triangles per thread of a binning / partition block (256 threads): chunks of 1,024, or of 512
// or 256 where fewer than kSpread chunks, the partition blocks the chip holds, would leave
// SMs without one.  Builds with 256 / 512 / 1,024, us: 16,384 triangles 396 / 411 / 429,
// 65,790 465 / 482 / 505, 131,072 532 / 553 / 565, 262,144 843 / 817 / 856, 524,288 1126 /
// 1079 / 1057, 1,048,576 - / 1629 / 1571.
constexpr uint32_t kMaxPer = 4;
constexpr uint32_t kSpread = 4 * 152;
inline uint32_t tris_per_thread(uint32_t n) {
	return n <= 256u * kSpread ? 1u : n <= 512u * kSpread ? 2u : kMaxPer;
}
constexpr uint32_t kDepthGuard = 48;
constexpr int kMaxLevels = 96;
constexpr int kLevelsPerCheck = 4;
constexpr int kBinWords = 3 * kBins * 7; // per axis and bin: lo xyz, hi xyz (ordered), count
constexpr uint32_t kOrdPosInf = 0xFF800000u; // f2ord(+inf)
constexpr uint32_t kOrdNegInf = 0x007FFFFFu; // f2ord(-inf)
constexpr uint32_t kHalves = 3;              // split "axis" meaning: first half / second half

// Counter words: list sizes and node ids, then the large tasks and the chunks of each
// level.
enum : int {
	kCtrSmall = 0,
	kCtrMid = 1,
	kCtrNodesSah = 2,
	kCtrLarge = 4,
	kCtrChunks = kCtrLarge + kMaxLevels + 2,
	kCtrWordsSah = kCtrChunks + kMaxLevels + 2
};

struct alignas(16) SahTask {
	uint32_t begin, count, node, parent; // parent = (node << 1 | side), kNone at a root;
	                                     // a split large task keeps here the list slots
	                                     // of its left and right child (kNone: not large)
	uint32_t meta;                       // bit 0: buffer holding the range; bits 8-15: depth
	uint32_t axis, split, n_left;        // the split chosen (large tasks)
	float lo[3];
	uint32_t cur_l;                      // partition cursors (large tasks)
	float scale[3];
	uint32_t cur_r;
};
static_assert(sizeof(SahTask) == 64, "task layout");

struct SmallTask {
	uint32_t begin, meta, node, parent;  // meta: count | buffer << 8 | depth << 16
	uint32_t base;                       // first id for the nodes below (kNone: to be drawn)
};

struct SahArgs {
	float4 *rec[2];         // (lo, id) (hi, 0) per triangle, two buffers
	SahTask *large[2];      // (these three by level % 2)
	uint32_t *bins[2];      // kBinWords per large task
	uint2 *chunk[2];        // per chunk of the level: large task, first triangle
	SahTask *mid;
	SmallTask *small;
	uint32_t *ctr;
	uint32_t *vals;         // out: position -> triangle index
	float4 *lbox;           // out: leaf boxes by position
	uint32_t *left, *right, *rfirst, *rlast;
	float4 *ibox;
	uint4 *splits;          // out: by leaf position, for the bottom-up cost pass
	uint32_t node_cap, max_large, max_mid, max_small, max_chunks;
	uint32_t n;             // triangles (records per buffer)
	uint32_t chunk_log;     // log2 of the triangles per chunk, 256 * tris_per_thread
	uint32_t *err;
};

__device__ __forceinline__ uint32_t chunks_of(const SahArgs &A, uint32_t count) {
	return (count + (1u << A.chunk_log) - 1u) >> A.chunk_log;
}

// Counts clamped to the list capacities (a list that overflowed was flagged).
__device__ __forceinline__ uint32_t n_large(const SahArgs &A, int level) {
	return min(A.ctr[kCtrLarge + level], A.max_large);
}
__device__ __forceinline__ uint32_t n_chunks(const SahArgs &A, int level) {
	return min(A.ctr[kCtrChunks + level], A.max_chunks);
}

__device__ __forceinline__ bool range_ok(const SahArgs &A, uint32_t begin, uint32_t count) {
	return begin <= A.n && count <= A.n - begin && count >= 2;
}

__device__ __forceinline__ float centre(float lo, float hi) {
	return __fadd_rn(__fmul_rn(lo, 0.5f), __fmul_rn(hi, 0.5f));
}

__device__ __forceinline__ int bin_of(float c, float lo, float scale) {
	const float t = __fmul_rn(__fsub_rn(c, lo), scale);
	return (int)fminf(fmaxf(t, 0.0f), (float)(kBins - 1)); // NaN -> 0
}

__device__ __forceinline__ float frame_scale(float lo, float hi) {
	const float e = hi - lo;
	return (e > 0.0f && isfinite(e)) ? (float)kBins / e : 0.0f;
}

__device__ __forceinline__ float area3(float lx, float ly, float lz, float hx, float hy,
                                       float hz) {
	const float dx = hx - lx, dy = hy - ly, dz = hz - lz;
	const float a = dx * dy + dx * dz + dy * dz;
	return isfinite(a) ? a : FLT_MAX;
}

__device__ __forceinline__ float rec_c(const float4 &lo, const float4 &hi, int k) {
	return k == 0 ? centre(lo.x, hi.x) : (k == 1 ? centre(lo.y, hi.y) : centre(lo.z, hi.z));
}

__device__ __forceinline__ void flag(uint32_t *err) { set_error_bits(err, kErrSah); }

__device__ __forceinline__ void bins_init(uint32_t *b, int at, int step, int words = kBinWords) {
	for (int k = at; k < words; k += step) {
		const int w = k % 7;
		b[k] = w < 3 ? kOrdPosInf : (w < 6 ? kOrdNegInf : 0u);
	}
}

// Adds each valid lane's triangle to the bins of all three axes; `set` selects one of two
// sets of kBinWords words (with the lane's own frame).  Where the warp's triangles fall into
// few bins (meshes list neighbours together), each group of lanes with the same bin reduces
// first and one lane updates the bin; lanes of many bins update them one by one, bounds only
// when they improve what is there.
// 0 / 1 / 2 / 4 / 8: heightfield build 1.89 / 1.86 / 1.80 / 1.85 / 2.07 ms; the clusters, in
// random order, 13.6 ms with 0 and 14.3 with 2: set for meshes, whose files list neighbours
// together.
constexpr int kBinGroups = 2;

__device__ __forceinline__ void bins_add(uint32_t *b, bool valid, uint32_t set, const float4 &lo,
                                         const float4 &hi, const float *flo, const float *fsc,
                                         int lane) {
	const uint32_t v[6] = {f2ord(lo.x), f2ord(lo.y), f2ord(lo.z),
	                       f2ord(hi.x), f2ord(hi.y), f2ord(hi.z)};
	int bins[3] = {-1, -1, -1};
	if (valid)
#pragma unroll
		for (int a = 0; a < 3; ++a)
			bins[a] = ((int)set * 3 + a) * kBins + bin_of(rec_c(lo, hi, a), flo[a], fsc[a]);
#pragma unroll
	for (int a = 0; a < 3; ++a) {
		const int bin = bins[a];
		const uint32_t g = __match_any_sync(0xFFFFFFFFu, bin);
		const bool lead = valid && lane == __ffs(g) - 1;
		uint32_t leads = __ballot_sync(0xFFFFFFFFu, lead);
		uint32_t *w = b + bin * 7;
		if (__popc(leads) <= kBinGroups) {
			while (leads) { // one group of lanes at a time
				const uint32_t m = __shfl_sync(0xFFFFFFFFu, g, __ffs(leads) - 1);
				leads &= leads - 1u;
				if ((m >> lane) & 1u) {
					uint32_t x[6];
#pragma unroll
					for (int k = 0; k < 3; ++k)
						x[k] = __reduce_min_sync(m, v[k]);
#pragma unroll
					for (int k = 3; k < 6; ++k)
						x[k] = __reduce_max_sync(m, v[k]);
					if (lead) {
						atomicAdd(&w[6], (uint32_t)__popc(m));
#pragma unroll
						for (int k = 0; k < 3; ++k)
							atomicMin(&w[k], x[k]);
#pragma unroll
						for (int k = 3; k < 6; ++k)
							atomicMax(&w[k], x[k]);
					}
				}
				__syncwarp();
			}
		} else if (valid) {
			if (lead)
				atomicAdd(&w[6], (uint32_t)__popc(g));
#pragma unroll
			for (int k = 0; k < 3; ++k)
				if (v[k] < *(volatile uint32_t *)&w[k])
					atomicMin(&w[k], v[k]);
#pragma unroll
			for (int k = 3; k < 6; ++k)
				if (v[k] > *(volatile uint32_t *)&w[k])
					atomicMax(&w[k], v[k]);
		}
	}
}

// Folds a block's bins of one task into the task's global bins.
__device__ __forceinline__ void bins_merge(const uint32_t *sb, uint32_t *gbins) {
	for (int k = threadIdx.x; k < kBinWords; k += blockDim.x) {
		const int w = k % 7;
		const uint32_t cnt = sb[k - w + 6];
		if (cnt == 0)
			continue;
		if (w < 3)
			atomicMin(&gbins[k], sb[k]);
		else if (w < 6)
			atomicMax(&gbins[k], sb[k]);
		else
			atomicAdd(&gbins[k], cnt);
	}
}

struct Box6 {
	float lx, ly, lz, hx, hy, hz;
};

__device__ __forceinline__ Box6 box_union(const Box6 &a, const Box6 &b) {
	return Box6{fminf(a.lx, b.lx), fminf(a.ly, b.ly), fminf(a.lz, b.lz),
	            fmaxf(a.hx, b.hx), fmaxf(a.hy, b.hy), fmaxf(a.hz, b.hz)};
}

__device__ __forceinline__ Box6 shfl_box(const Box6 &b, int src) {
	return Box6{__shfl_sync(0xFFFFFFFFu, b.lx, src), __shfl_sync(0xFFFFFFFFu, b.ly, src),
	            __shfl_sync(0xFFFFFFFFu, b.lz, src), __shfl_sync(0xFFFFFFFFu, b.hx, src),
	            __shfl_sync(0xFFFFFFFFu, b.hy, src), __shfl_sync(0xFFFFFFFFu, b.hz, src)};
}

__device__ __forceinline__ Box6 empty_box() {
	return Box6{INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
}

__device__ __forceinline__ float box_area(const Box6 &b) {
	return area3(b.lx, b.ly, b.lz, b.hx, b.hy, b.hz);
}

// Union over the lanes in [a, b) of the warp (every lane calls).
__device__ __forceinline__ Box6 range_box(const Box6 &mine, int lane, int a, int b) {
	Box6 x = (lane >= a && lane < b) ? mine : empty_box();
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) {
		Box6 y{__shfl_xor_sync(0xFFFFFFFFu, x.lx, o), __shfl_xor_sync(0xFFFFFFFFu, x.ly, o),
		       __shfl_xor_sync(0xFFFFFFFFu, x.lz, o), __shfl_xor_sync(0xFFFFFFFFu, x.hx, o),
		       __shfl_xor_sync(0xFFFFFFFFu, x.hy, o), __shfl_xor_sync(0xFFFFFFFFu, x.hz, o)};
		x = box_union(x, y);
	}
	return x;
}

struct Split {
	uint32_t axis, bin, n_left; // axis kHalves: no plane
	Box6 node, left, right;     // left / right valid for a binned split
};

// The best plane over the three axes' bins (word(a, k): word k of bin `lane` on axis a).  Ties
// go to the lower axis, then the lower bin.  Every lane returns the same result.
template <class Word>
__device__ __forceinline__ Split choose_split(Word word, const float *fsc, uint32_t count,
                                              int lane) {
	Split s;
	s.axis = kHalves;
	s.bin = 0;
	s.n_left = count / 2;
	uint64_t best = ~0ull;
#pragma unroll
	for (int a = 0; a < 3; ++a) {
		uint32_t w[7];
#pragma unroll
		for (int k = 0; k < 7; ++k)
			w[k] = word(a, k);
		Box6 p{ord2f(w[0]), ord2f(w[1]), ord2f(w[2]), ord2f(w[3]), ord2f(w[4]), ord2f(w[5])};
		uint32_t pc = w[6];
		Box6 q = p;
		uint32_t qc = pc;
#pragma unroll
		for (int o = 1; o < 32; o <<= 1) {
			const Box6 pu = shfl_box(p, max(lane - o, 0));
			const uint32_t pcu = __shfl_up_sync(0xFFFFFFFFu, pc, o);
			const Box6 qd = shfl_box(q, min(lane + o, 31));
			const uint32_t qcd = __shfl_down_sync(0xFFFFFFFFu, qc, o);
			if (lane >= o) {
				p = box_union(p, pu);
				pc += pcu;
			}
			if (lane + o < 32) {
				q = box_union(q, qd);
				qc += qcd;
			}
		}
		if (a == 0)
			s.node = shfl_box(p, 31);
		const Box6 r = shfl_box(q, min(lane + 1, 31));
		const uint32_t rc = __shfl_down_sync(0xFFFFFFFFu, qc, 1);
		// The least cost on this axis, then the lowest plane with it (two redux.sync
		// minima).
		uint32_t c32 = 0xFFFFFFFFu;
		if (fsc[a] > 0.0f && lane < 31 && pc > 0 && rc > 0)
			c32 = f2ord(box_area(p) * (float)pc + box_area(r) * (float)rc);
		const uint32_t cmin = __reduce_min_sync(0xFFFFFFFFu, c32);
		const uint32_t plane = __reduce_min_sync(
		    0xFFFFFFFFu, (c32 == cmin && c32 != 0xFFFFFFFFu) ? (uint32_t)lane : 0xFFu);
		const uint64_t key =
		    cmin == 0xFFFFFFFFu ? ~0ull : (((uint64_t)cmin << 32) | ((uint32_t)a << 8) | plane);
		if (key < best) {
			best = key;
			const int src = (int)(key & 0xFF);
			s.axis = (uint32_t)a;
			s.bin = (uint32_t)src;
			s.n_left = __shfl_sync(0xFFFFFFFFu, pc, src);
			s.left = shfl_box(p, src);
			s.right = shfl_box(r, src);
		}
	}
	return s;
}

__device__ __forceinline__ void write_node_box(const SahArgs &A, uint32_t node, const Box6 &b,
                                               float wl, float wr) {
	A.ibox[2 * (size_t)node] = make_float4(b.lx, b.ly, b.lz, wl);
	A.ibox[2 * (size_t)node + 1] = make_float4(b.hx, b.hy, b.hz, wr);
}

__device__ __forceinline__ void write_parent_area(const SahArgs &A, uint32_t parent, float a) {
	if (parent != kNone)
		reinterpret_cast<float *>(&A.ibox[2 * (size_t)(parent >> 1) + (parent & 1u)])[3] = a;
}

__device__ __forceinline__ uint32_t new_node(const SahArgs &A, uint32_t k) {
	const uint32_t id = atomicAdd(&A.ctr[kCtrNodesSah], k);
	if (id + k > A.node_cap) {
		flag(A.err);
		return kNone;
	}
	return id;
}

// A place in the list of the tier that a range of `count` triangles belongs to (large tasks by
// level); kNone, flagged, when the list is full.
__device__ __forceinline__ uint32_t list_slot(const SahArgs &A, int level, uint32_t count) {
	const bool large = count > kLarge, mid = !large && count > kSmall;
	const uint32_t word = large ? kCtrLarge + level : (mid ? kCtrMid : kCtrSmall);
	const uint32_t cap = large ? A.max_large : (mid ? A.max_mid : A.max_small);
	const uint32_t i = atomicAdd(&A.ctr[word], 1u);
	if (i < cap)
		return i;
	flag(A.err);
	return kNone;
}

// Writes a child range as a task into place `i` of its tier's list.  `frame` gives the binning
// frame of a large child (null: its parent's).
__device__ __forceinline__ void put_child(const SahArgs &A, int level, uint32_t i, uint32_t begin,
                                          uint32_t count, uint32_t node, uint32_t parent,
                                          uint32_t buf, uint32_t depth, const Box6 *frame,
                                          const float *pflo, const float *pfsc) {
	if (count <= kSmall) {
		A.small[i] = SmallTask{begin, count | (buf << 8) | (depth << 16), node, parent, kNone};
		return;
	}
	SahTask t;
	memset(&t, 0, sizeof(t));
	t.begin = begin;
	t.count = count;
	t.node = node;
	t.parent = parent;
	t.meta = buf | (depth << 8);
	if (count > kLarge) {
		t.axis = kHalves;
		if (frame) {
			t.lo[0] = frame->lx;
			t.lo[1] = frame->ly;
			t.lo[2] = frame->lz;
			t.scale[0] = frame_scale(frame->lx, frame->hx);
			t.scale[1] = frame_scale(frame->ly, frame->hy);
			t.scale[2] = frame_scale(frame->lz, frame->hz);
		} else {
			for (int k = 0; k < 3; ++k) {
				t.lo[k] = pflo[k];
				t.scale[k] = pfsc[k];
			}
		}
		A.large[level & 1][i] = t;
	} else {
		A.mid[i] = t;
	}
}

// Makes a large task that lane `from` filed (its slot and first chunk place) ready for its
// level: the whole warp clears its bins (a single lane clearing the 672 words of two children
// took most of k_sah_split's time) and lists its chunks.
__device__ __forceinline__ void open_large(const SahArgs &A, int level, uint32_t slot, uint32_t at,
                                           uint32_t begin, uint32_t count, int from, int lane) {
	slot = __shfl_sync(0xFFFFFFFFu, slot, from);
	at = __shfl_sync(0xFFFFFFFFu, at, from);
	if (slot == kNone)
		return;
	bins_init(A.bins[level & 1] + (size_t)slot * kBinWords, lane, 32);
	const uint32_t n = chunks_of(A, count);
	if (at + n > A.max_chunks) {
		if (lane == 0)
			flag(A.err);
		return;
	}
	for (uint32_t c = lane; c < n; c += 32)
		A.chunk[level & 1][at + c] = make_uint2(slot, begin + (c << A.chunk_log));
}

// Writes node `t.node` (box, children, range) for split `s` of a large task and files its
// children, lane 0 the left one and lane 1 the right one; children whose range holds one
// triangle are leaves.  Lanes 0 and 1 return the list slot of a child filed as a large task
// (else kNone).
__device__ __forceinline__ uint32_t file_children(const SahArgs &A, const SahTask &t,
                                                  const Split &s, int level, int lane) {
	const uint32_t buf = (t.meta & 1u) ^ 1u, depth = ((t.meta >> 8) & 0xFFu) + 1u;
	const uint32_t nl = s.n_left, nr = t.count - nl;
	const bool binned = s.axis != kHalves;
	const bool right = lane == 1, mine = lane < 2;
	const uint32_t begin = right ? t.begin + nl : t.begin, count = right ? nr : nl;
	const uint32_t n_ids = (nl > 1) + (nr > 1);
	// Every atomic of the task before any of their results is needed.
	uint32_t id = 0, slot = kNone, at = 0;
	if (lane == 2 && n_ids)
		id = new_node(A, n_ids);
	if (mine && count > kLarge)
		at = atomicAdd(&A.ctr[kCtrChunks + level], chunks_of(A, count));
	if (mine)
		slot = list_slot(A, level, count);
	id = __shfl_sync(0xFFFFFFFFu, id, 2);
	if (id == kNone || !__all_sync(0xFFFFFFFFu, !mine || slot != kNone))
		return kNone; // (flagged)
	const uint32_t id_l = id, id_r = id + (nl > 1 ? 1u : 0u);
	if (mine) {
		const uint32_t node = count > 1 ? (right ? id_r : id_l) : kNone;
		// Children's areas: known now for a binned split (leaves keep -1); after halves each
		// child writes its own when it is split.
		const uint32_t parent = binned ? kNone : ((t.node << 1) | (right ? 1u : 0u));
		Box6 frame{t.lo[0], t.lo[1], t.lo[2], 0.0f, 0.0f, 0.0f};
		if (binned)
			frame = right ? s.right : s.left;
		put_child(A, level, slot, begin, count, node, parent, buf, depth, binned ? &frame : nullptr,
		          t.lo, t.scale);
		if (!right) {
			A.left[t.node] = nl > 1 ? id_l : (kLeafBit | t.begin);
			A.right[t.node] = nr > 1 ? id_r : (kLeafBit | (t.begin + nl));
			A.rfirst[t.node] = t.begin;
			A.rlast[t.node] = t.begin + t.count - 1u;
			A.splits[t.begin + nl - 1u] = make_uint4(t.begin, t.begin + t.count - 1u, t.node, 0u);
			write_node_box(A, t.node, s.node, (binned && nl > 1) ? box_area(s.left) : -1.0f,
			               (binned && nr > 1) ? box_area(s.right) : -1.0f);
		}
	}
	if (count <= kLarge)
		slot = kNone;
	open_large(A, level, slot, at, t.begin, nl, 0, lane);
	open_large(A, level, slot, at, t.begin + nl, nr, 1, lane);
	return slot;
}

// ---------------------------------------------------------------------------------------
// Set-up: records, per-scene centre bounds, root tasks.

__global__ void k_sah_records(const float *__restrict__ tris, uint32_t n,
                              const uint32_t *scene_of, float4 *rec, uint32_t *gb,
                              XFaces x_faces) {
	chain_enter();
	const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
	const int lane = threadIdx.x & 31;
	const bool live = i < n;
	float4 lo = make_float4(0, 0, 0, 0), hi = lo;
	uint32_t s = 0;
	if (live) {
		const float *t = tris + 9 * (size_t)i;
		bool fin = true;
#pragma unroll
		for (int k = 0; k < 9; ++k)
			fin = fin && isfinite(t[k]);
		if (fin) {
			lo = make_float4(fminf(t[0], fminf(t[3], t[6])), fminf(t[1], fminf(t[4], t[7])),
			                 fminf(t[2], fminf(t[5], t[8])), __uint_as_float(i));
			hi = make_float4(fmaxf(t[0], fmaxf(t[3], t[6])), fmaxf(t[1], fmaxf(t[4], t[7])),
			                 fmaxf(t[2], fmaxf(t[5], t[8])), 0.0f);
		} else {
			lo = make_float4(-FLT_MAX, -FLT_MAX, -FLT_MAX, __uint_as_float(i));
			hi = make_float4(FLT_MAX, FLT_MAX, FLT_MAX, 0.0f);
		}
		if (x_faces.log) {
			if (fin)
				x_face_add(x_faces, lo.x);
			else
				x_faces.words[0] = 1u;
		}
		rec[2 * (size_t)i] = lo;
		rec[2 * (size_t)i + 1] = hi;
		s = scene_of ? scene_of[i] : 0u;
	}
	float mn[3], mx[3];
#pragma unroll
	for (int k = 0; k < 3; ++k) {
		const float c = rec_c(lo, hi, k);
		mn[k] = live ? c : INFINITY;
		mx[k] = live ? c : -INFINITY;
	}
	if (!scene_of) {
		// One scene: warps reduce, then the block, and one thread updates the six words
		// (one set of same-address atomics per block instead of per warp: with 32k warps
		// on a 1M-triangle scene those atomics were most of this kernel's time).
		__shared__ float red[32][6];
#pragma unroll
		for (int k = 0; k < 3; ++k)
			for (int o = 16; o > 0; o >>= 1) {
				mn[k] = fminf(mn[k], __shfl_xor_sync(0xFFFFFFFFu, mn[k], o));
				mx[k] = fmaxf(mx[k], __shfl_xor_sync(0xFFFFFFFFu, mx[k], o));
			}
		const int w = threadIdx.x >> 5;
		if (lane == 0)
			for (int k = 0; k < 3; ++k) {
				red[w][k] = mn[k];
				red[w][3 + k] = mx[k];
			}
		__syncthreads();
		if (threadIdx.x < 6) {
			const int k = threadIdx.x;
			float v = red[0][k];
			for (int j = 1; j < (int)(blockDim.x >> 5); ++j)
				v = k < 3 ? fminf(v, red[j][k]) : fmaxf(v, red[j][k]);
			if (k < 3 && v != INFINITY)
				atomicMin(&gb[k], f2ord(v));
			else if (k >= 3 && v != -INFINITY)
				atomicMax(&gb[k], f2ord(v));
		}
		return;
	}
	const uint32_t s0 = __shfl_sync(0xFFFFFFFFu, s, 0);
	if (__all_sync(0xFFFFFFFFu, !live || s == s0)) {
#pragma unroll
		for (int k = 0; k < 3; ++k)
			for (int o = 16; o > 0; o >>= 1) {
				mn[k] = fminf(mn[k], __shfl_xor_sync(0xFFFFFFFFu, mn[k], o));
				mx[k] = fmaxf(mx[k], __shfl_xor_sync(0xFFFFFFFFu, mx[k], o));
			}
		if (lane == 0 && mn[0] <= mx[0])
			for (int k = 0; k < 3; ++k) {
				atomicMin(&gb[6 * s0 + k], f2ord(mn[k]));
				atomicMax(&gb[6 * s0 + 3 + k], f2ord(mx[k]));
			}
	} else if (live) {
		for (int k = 0; k < 3; ++k) {
			atomicMin(&gb[6 * s + k], f2ord(mn[k]));
			atomicMax(&gb[6 * s + 3 + k], f2ord(mx[k]));
		}
	}
}

__global__ void k_sah_first_id(uint32_t *ctr, uint32_t S) {
	chain_enter();
	ctr[kCtrNodesSah] = S;
}

// One warp per scene: lane 0 files the root task, the warp clears a large root's bins.
__global__ void k_sah_roots(SahArgs A, const uint32_t *tri_off, uint32_t n_scenes,
                            const uint32_t *gb, uint32_t *roots) {
	chain_enter();
	const uint32_t s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
	const int lane = threadIdx.x & 31;
	if (s >= n_scenes)
		return;
	const uint32_t b = tri_off[s], n = tri_off[s + 1] - b;
	uint32_t slot = kNone, at = 0;
	if (lane == 0) {
		roots[s] = s;
		if (n) {
			A.splits[b + n - 1u] = PRT_NO_SPLIT;
			float flo[3], fsc[3];
			for (int k = 0; k < 3; ++k) {
				flo[k] = ord2f(gb[6 * s + k]);
				fsc[k] = frame_scale(flo[k], ord2f(gb[6 * s + 3 + k]));
			}
			if (n > kLarge)
				at = atomicAdd(&A.ctr[kCtrChunks], chunks_of(A, n));
			slot = list_slot(A, 0, n);
			if (slot != kNone)
				put_child(A, 0, slot, b, n, n > 1 ? s : kNone, kNone, 0u, 0u, nullptr, flo, fsc);
		}
	}
	open_large(A, 0, n > kLarge ? slot : kNone, at, b, n, 0, lane);
}

// ---------------------------------------------------------------------------------------
// Large tasks.

// The roots' bins (the bins of later levels are filled by the partition above them).
template <uint32_t kPer>
__global__ void __launch_bounds__(256) k_sah_bin(SahArgs A) {
	chain_enter();
	__shared__ uint32_t sb[kBinWords];
	const uint32_t n = n_chunks(A, 0);
	const int lane = threadIdx.x & 31;
	for (uint32_t c = blockIdx.x; c < n; c += gridDim.x) {
		const uint2 ch = A.chunk[0][c];
		const SahTask &t = A.large[0][ch.x];
		const uint32_t end = min(ch.y + 256u * kPer, t.begin + t.count);
		const float4 *src = A.rec[0];
		float4 lo[kPer], hi[kPer];
#pragma unroll
		for (uint32_t j = 0; j < kPer; ++j) {
			const uint32_t i = ch.y + j * 256u + threadIdx.x;
			lo[j] = hi[j] = make_float4(0, 0, 0, 0);
			if (i < end) {
				lo[j] = src[2 * (size_t)i];
				hi[j] = src[2 * (size_t)i + 1];
			}
		}
		bins_init(sb, threadIdx.x, 256);
		__syncthreads();
#pragma unroll
		for (uint32_t j = 0; j < kPer; ++j)
			bins_add(sb, ch.y + j * 256u + threadIdx.x < end, 0u, lo[j], hi[j], t.lo, t.scale, lane);
		__syncthreads();
		bins_merge(sb, A.bins[0] + (size_t)ch.x * kBinWords);
		__syncthreads();
	}
}

// One warp per large task: the plane, the node and the child tasks.  A level has few tasks, so
// the launch takes as long as one warp's chain of dependent reads and atomics: the bins of
// all axes are read at once, and lanes 0 and 1 file one child each while lane 2 draws the
// node ids (10 -> 7.5 us per level).
__global__ void __launch_bounds__(128) k_sah_split(SahArgs A, int level) {
	chain_enter();
	const uint32_t n_tasks = n_large(A, level);
	const int lane = threadIdx.x & 31;
	for (uint32_t ti = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; ti < n_tasks;
	     ti += (gridDim.x * blockDim.x) >> 5) {
		SahTask &tr = A.large[level & 1][ti];
		const uint32_t *b = A.bins[level & 1] + (size_t)ti * kBinWords;
		uint32_t w[3][7];
#pragma unroll
		for (int a = 0; a < 3; ++a)
#pragma unroll
			for (int k = 0; k < 7; ++k)
				w[a][k] = b[(a * kBins + lane) * 7 + k];
		const SahTask t = tr;
		if (!range_ok(A, t.begin, t.count)) {
			if (lane == 0)
				flag(A.err);
			continue;
		}
		Split s = choose_split([&](int a, int k) { return w[a][k]; }, t.scale, t.count, lane);
		const uint32_t total = __reduce_add_sync(0xFFFFFFFFu, w[0][6]); // every triangle once
		if (((t.meta >> 8) & 0xFFu) >= kDepthGuard) {
			s.axis = kHalves;
			s.n_left = t.count / 2;
		}
		uint32_t slot = kNone; // lanes 0, 1: the child's list slot when it is a large task
		if (total != t.count || s.n_left == 0 || s.n_left >= t.count || t.node >= A.node_cap) {
			// Nothing placed: the partition then writes no triangle of this task.
			if (lane == 0) {
				flag(A.err);
				tr.axis = kHalves;
				tr.n_left = 0;
				tr.cur_l = tr.cur_r = A.n;
			}
		} else {
			slot = file_children(A, t, s, level + 1, lane);
			if (lane == 0) {
				write_parent_area(A, t.parent, box_area(s.node));
				tr.axis = s.axis;
				tr.split = s.bin;
				tr.n_left = s.n_left;
				tr.cur_l = t.begin;
				tr.cur_r = t.begin + s.n_left;
			}
		}
		if (lane == 0)
			tr.node = slot;
		if (lane == 1)
			tr.parent = slot;
	}
}

// Scatters the triangles of the large tasks to the other buffer, left side first, and adds
// each to the bins of the child it goes to (when that is a large task).  A thread reads its
// triangles (up to four) at once and the block reserves its places with one atomic per side: the
// level is bound by the latency of its few dependent steps and by the shared-memory bins.
// As two kernels, each reading every record, with a pair of atomics per 32 triangles and a
// chunk table built by a third, a level of the 1,048,576-triangle heightfield took 60 to 90
// us; now 33 to 64.  (The split of the children in a task's last block, without a launch of
// its own: 53 us per level against 38 + 10, with its fences and 80 registers.)
// (Four blocks per SM: 64 registers; with 76, three blocks, a heightfield build took 1.72 ms
// where it takes 1.62.)
template <uint32_t kPer>
__global__ void __launch_bounds__(256, 4) k_sah_part(SahArgs A, int level) {
	chain_enter();
	__shared__ uint32_t sb[2 * kBinWords];
	__shared__ uint32_t cnt_l[8 * kPer], cnt_r[8 * kPer]; // per warp and j; then exclusive sums
	__shared__ uint32_t base[2];
	static_assert(8 * kPer <= 32, "one warp scans the block's counts");
	const uint32_t n = n_chunks(A, level);
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	const uint32_t lt = (1u << lane) - 1u;
	for (uint32_t c = blockIdx.x; c < n; c += gridDim.x) {
		const uint2 ch = A.chunk[level & 1][c];
		SahTask &t = A.large[level & 1][ch.x];
		const uint32_t begin = t.begin, count = t.count, nl = t.n_left, axis = t.axis,
		               split = t.split, buf = t.meta & 1u;
		const uint32_t end = min(ch.y + 256u * kPer, begin + count);
		const uint32_t slot[2] = {t.node, t.parent};
		const float4 *src = A.rec[buf];
		float4 *dst = A.rec[buf ^ 1u];
		const float flo = axis < 3 ? t.lo[axis] : 0.0f, fsc = axis < 3 ? t.scale[axis] : 0.0f;
		float4 lo[kPer], hi[kPer];
		uint32_t side = 0; // bit j: triangle j goes right
		uint32_t ml[kPer], mr[kPer];
#pragma unroll
		for (uint32_t j = 0; j < kPer; ++j) {
			const uint32_t i = ch.y + j * 256u + threadIdx.x;
			lo[j] = hi[j] = make_float4(0, 0, 0, 0);
			if (i < end) {
				lo[j] = src[2 * (size_t)i];
				hi[j] = src[2 * (size_t)i + 1];
			}
		}
		bins_init(sb, threadIdx.x, 256, 2 * kBinWords);
#pragma unroll
		for (uint32_t j = 0; j < kPer; ++j) {
			const uint32_t i = ch.y + j * 256u + threadIdx.x;
			const bool v = i < end;
			const bool right =
			    axis == kHalves ? (i - begin >= nl)
			                    : (bin_of(rec_c(lo[j], hi[j], (int)axis), flo, fsc) > (int)split);
			side |= (uint32_t)right << j;
			ml[j] = __ballot_sync(0xFFFFFFFFu, v && !right);
			mr[j] = __ballot_sync(0xFFFFFFFFu, v && right);
			if (lane == 0) {
				cnt_l[warp * kPer + j] = __popc(ml[j]);
				cnt_r[warp * kPer + j] = __popc(mr[j]);
			}
		}
		__syncthreads();
		if (warp < 2) { // warp 0 the left side, warp 1 the right
			uint32_t *cnt = warp ? cnt_r : cnt_l;
			const bool in = lane < 8 * (int)kPer;
			const uint32_t own = in ? cnt[lane] : 0u;
			uint32_t x = own;
#pragma unroll
			for (int o = 1; o < 32; o <<= 1) {
				const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
				if (lane >= o)
					x += y;
			}
			if (in)
				cnt[lane] = x - own;
			if (lane == 31)
				base[warp] = x ? atomicAdd(warp ? &t.cur_r : &t.cur_l, x) : 0u;
		}
		__syncthreads();
		float clo[2][3], csc[2][3]; // the children's binning frames
#pragma unroll
		for (int k = 0; k < 2; ++k) {
			const SahTask &ct = A.large[(level + 1) & 1][slot[k] == kNone ? 0u : slot[k]];
#pragma unroll
			for (int q = 0; q < 3; ++q) {
				clo[k][q] = slot[k] == kNone ? 0.0f : ct.lo[q];
				csc[k][q] = slot[k] == kNone ? 0.0f : ct.scale[q];
			}
		}
#pragma unroll
		for (uint32_t j = 0; j < kPer; ++j) {
			const bool v = ch.y + j * 256u + threadIdx.x < end;
			const uint32_t right = (side >> j) & 1u;
			if (v) {
				const uint32_t pos = right ? base[1] + cnt_r[warp * kPer + j] + __popc(mr[j] & lt)
				                           : base[0] + cnt_l[warp * kPer + j] + __popc(ml[j] & lt);
				const bool ok = right ? (pos >= begin + nl && pos < begin + count)
				                      : (pos >= begin && pos < begin + nl);
				if (ok) {
					dst[2 * (size_t)pos] = lo[j];
					dst[2 * (size_t)pos + 1] = hi[j];
				} else {
					flag(A.err);
				}
			}
			if (slot[0] != kNone || slot[1] != kNone) {
				float f[3], g[3];
#pragma unroll
				for (int q = 0; q < 3; ++q) {
					f[q] = right ? clo[1][q] : clo[0][q];
					g[q] = right ? csc[1][q] : csc[0][q];
				}
				bins_add(sb, v && (right ? slot[1] : slot[0]) != kNone, right, lo[j], hi[j], f, g,
				         lane);
			}
		}
		__syncthreads();
#pragma unroll
		for (int k = 0; k < 2; ++k)
			if (slot[k] != kNone)
				bins_merge(sb + k * kBinWords,
				           A.bins[(level + 1) & 1] + (size_t)slot[k] * kBinWords);
		__syncthreads();
	}
}

// ---------------------------------------------------------------------------------------
// Mid tasks: one block each.  The task's records stay in shared memory while a permutation
// of them is split level by level, one warp per range, down to ranges of at most 32, whose
// records then go to the other buffer in order as small tasks.  The first range is split by
// all four warps and the next two by two each: with one warp each, three waited 42 % of the
// kernel's time for the others (8.4M clustered triangles 14.3 -> 13.4 ms).  (One launch per level, each
// reading and writing every record, took 0.41 of the 2.17 ms build of the 1,048,576-triangle
// heightfield, most of it waiting: 20 launches of 3 to 80 us.)  With the large tier's levels
// halved as well, heightfield builds went from 0.80 to 0.53 ms (65,790 triangles) and 2.17 to
// 1.81 ms (1,048,576), 8.4M clustered triangles from 15.2 to 14.3 ms, with the same trees.

struct MidRange {
	uint32_t begin, count; // within the task
	uint32_t node, base;   // its node, and the first id for the nodes below it (count - 2)
	uint32_t parent, depth;
};

constexpr int kMidWarps = 4; // (teams of 4, 2 and 1 warps)
constexpr uint32_t kMidRanges = kLarge / (kSmall + 1) + 1;

struct MidShared {
	float4 rec[2 * kLarge];
	uint32_t bins[kMidWarps][kBinWords];
	MidRange range[2][kMidRanges];
	uint32_t n_range[2];
	float bound[kMidWarps][6];
	uint32_t choice[kMidWarps][3], left_of[kMidWarps], total[kMidWarps];
	uint16_t perm[2][kLarge];
};

// A barrier of the `team` warps that split one range (the block's warps in order, so teams
// of equal size are numbered by their first warp).
__device__ __forceinline__ void team_sync(int team, int warp) {
	if (team == 1)
		__syncwarp();
	else
		asm volatile("bar.sync %0, %1;" ::"r"(1 + warp / team), "r"(32 * team) : "memory");
}

// Splits one range with a team of 1, 2 or 4 warps: writes its node and files or queues its
// two parts.  Each warp takes a slice of the range; the first chooses the split.
__device__ __forceinline__ void split_range(const SahArgs &A, MidShared &S, const MidRange &r,
                                            int in, uint32_t task_begin, float4 *dst,
                                            uint32_t dst_buf, int team, int warp, int lane) {
	const uint32_t lt = (1u << lane) - 1u;
	const int lead = warp - warp % team;
	const uint16_t *perm = S.perm[in] + r.begin;
	uint16_t *out = S.perm[in ^ 1] + r.begin;
	uint32_t *sb = S.bins[lead];
	const uint32_t slice = (r.count + 32u * team - 1u) / (32u * team) * 32u;
	const uint32_t i_lo = min(slice * (uint32_t)(warp - lead), r.count);
	const uint32_t i_hi = min(i_lo + slice, r.count);
	// Exact centre bounds of the range: the binning frame.
	float mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
	for (uint32_t i = i_lo + lane; i < i_hi; i += 32) {
		const uint32_t p = perm[i];
		const float4 lo = S.rec[p], hi = S.rec[kLarge + p];
#pragma unroll
		for (int k = 0; k < 3; ++k) {
			const float c = rec_c(lo, hi, k);
			mn[k] = fminf(mn[k], c);
			mx[k] = fmaxf(mx[k], c);
		}
	}
	float flo[3], fsc[3];
#pragma unroll
	for (int k = 0; k < 3; ++k)
		for (int o = 16; o > 0; o >>= 1) {
			mn[k] = fminf(mn[k], __shfl_xor_sync(0xFFFFFFFFu, mn[k], o));
			mx[k] = fmaxf(mx[k], __shfl_xor_sync(0xFFFFFFFFu, mx[k], o));
		}
	bins_init(sb, 32 * (warp - lead) + lane, 32 * team);
	if (team > 1) {
		if (lane == 0)
			for (int k = 0; k < 3; ++k) {
				S.bound[warp][k] = mn[k];
				S.bound[warp][3 + k] = mx[k];
			}
		team_sync(team, warp);
		for (int w = lead; w < lead + team; ++w)
#pragma unroll
			for (int k = 0; k < 3; ++k) {
				mn[k] = fminf(mn[k], S.bound[w][k]);
				mx[k] = fmaxf(mx[k], S.bound[w][3 + k]);
			}
	}
#pragma unroll
	for (int k = 0; k < 3; ++k) {
		flo[k] = mn[k];
		fsc[k] = frame_scale(mn[k], mx[k]);
	}
	__syncwarp();
	for (uint32_t i0 = i_lo; i0 < i_hi; i0 += 32) {
		const bool v = i0 + lane < i_hi;
		float4 lo = make_float4(0, 0, 0, 0), hi = lo;
		if (v) {
			const uint32_t p = perm[i0 + lane];
			lo = S.rec[p];
			hi = S.rec[kLarge + p];
		}
		bins_add(sb, v, 0u, lo, hi, flo, fsc, lane);
	}
	team_sync(team, warp);
	Split s;
	if (warp == lead) {
		s = choose_split([&](int a, int k) { return sb[(a * kBins + lane) * 7 + k]; }, fsc, r.count,
		                 lane);
		if (r.depth >= kDepthGuard) {
			s.axis = kHalves;
			s.n_left = r.count / 2;
		}
		if (team > 1 && lane == 0) {
			S.choice[lead][0] = s.axis;
			S.choice[lead][1] = s.bin;
			S.choice[lead][2] = s.n_left;
		}
	}
	if (team > 1) {
		team_sync(team, warp);
		if (warp != lead) {
			s.axis = S.choice[lead][0];
			s.bin = S.choice[lead][1];
			s.n_left = S.choice[lead][2];
		}
	}
	// Stable partition of the permutation: each warp counts its slice's left part first when
	// the slices have to be placed after one another.
	auto goes_right = [&](uint32_t i, uint32_t p) {
		return s.axis == kHalves
		           ? (i >= s.n_left)
		           : (bin_of(rec_c(S.rec[p], S.rec[kLarge + p], (int)s.axis),
		                     s.axis == 0 ? flo[0] : (s.axis == 1 ? flo[1] : flo[2]),
		                     s.axis == 0 ? fsc[0] : (s.axis == 1 ? fsc[1] : fsc[2])) > (int)s.bin);
	};
	uint32_t nl_seen = 0, nr_seen = 0;
	if (team > 1) {
		uint32_t mine = 0;
		for (uint32_t i0 = i_lo; i0 < i_hi; i0 += 32) {
			const uint32_t i = i0 + lane;
			mine += __popc(__ballot_sync(0xFFFFFFFFu, i < i_hi && !goes_right(i, perm[min(i, i_hi - 1u)])));
		}
		if (lane == 0)
			S.left_of[warp] = mine;
		team_sync(team, warp);
		for (int w = lead; w < warp; ++w)
			nl_seen += S.left_of[w];
		nr_seen = i_lo - nl_seen;
	}
	for (uint32_t i0 = i_lo; i0 < i_hi; i0 += 32) {
		const uint32_t i = i0 + lane;
		const bool v = i < i_hi;
		const uint32_t p = perm[min(i, i_hi - 1u)];
		const bool right = goes_right(i, p);
		const uint32_t bl = __ballot_sync(0xFFFFFFFFu, v && !right);
		const uint32_t br = __ballot_sync(0xFFFFFFFFu, v && right);
		if (v) {
			const uint32_t pos = right ? s.n_left + nr_seen + __popc(br & lt)
			                           : nl_seen + __popc(bl & lt);
			if (pos < r.count)
				out[pos] = (uint16_t)p;
		}
		nl_seen += __popc(bl);
		nr_seen += __popc(br);
	}
	if (team > 1) {
		if (warp == lead + team - 1 && lane == 0)
			S.total[lead] = nl_seen; // (its own word: left_of may still be read)
		team_sync(team, warp);
		if (warp != lead)
			return;
		nl_seen = S.total[lead];
	}
	__syncwarp();
	const uint32_t nl = s.n_left, nr = r.count - nl;
	if (nl_seen != nl || nl == 0 || nl >= r.count || r.node >= A.node_cap ||
	    r.base + r.count - 2u > A.node_cap) {
		if (lane == 0)
			flag(A.err);
		return;
	}
	const bool binned = s.axis != kHalves;
	// Ids below the node in order: the left child, its nodes, the right child, its nodes.
	const uint32_t id_l = r.base, id_r = r.base + nl - 1u;
	const uint32_t pos_l = task_begin + r.begin, pos_r = pos_l + nl;
	if (lane == 0) {
		A.left[r.node] = nl > 1 ? id_l : (kLeafBit | pos_l);
		A.right[r.node] = nr > 1 ? id_r : (kLeafBit | pos_r);
		A.rfirst[r.node] = pos_l;
		A.rlast[r.node] = pos_l + r.count - 1u;
		A.splits[pos_r - 1u] = make_uint4(pos_l, pos_l + r.count - 1u, r.node, 0u);
		// Children's areas: known now for a binned split (leaves keep -1); after halves each
		// child writes its own when it is split.
		write_node_box(A, r.node, s.node, (binned && nl > 1) ? box_area(s.left) : -1.0f,
		               (binned && nr > 1) ? box_area(s.right) : -1.0f);
		write_parent_area(A, r.parent, box_area(s.node));
	}
#pragma unroll
	for (int k = 0; k < 2; ++k) {
		const uint32_t begin = r.begin + (k ? nl : 0u), count = k ? nr : nl;
		const uint32_t node = count > 1 ? (k ? id_r : id_l) : kNone;
		const uint32_t parent = binned ? kNone : ((r.node << 1) | (uint32_t)k);
		if (count > kSmall) {
			uint32_t at = 0;
			if (lane == 0)
				at = atomicAdd(&S.n_range[in ^ 1], 1u);
			if (lane == 0 && at < kMidRanges)
				S.range[in ^ 1][at] = MidRange{begin, count, node, node + 1u, parent, r.depth + 1u};
		} else {
			if ((uint32_t)lane < count) {
				const uint32_t p = S.perm[in ^ 1][begin + lane];
				dst[2 * (size_t)(task_begin + begin + lane)] = S.rec[p];
				dst[2 * (size_t)(task_begin + begin + lane) + 1] = S.rec[kLarge + p];
			}
			if (lane == 0) {
				const uint32_t i = atomicAdd(&A.ctr[kCtrSmall], 1u);
				if (i < A.max_small)
					A.small[i] = SmallTask{task_begin + begin,
					                       count | (dst_buf << 8) | ((r.depth + 1u) << 16), node,
					                       parent, count > 2 ? node + 1u : kNone};
				else
					flag(A.err);
			}
		}
	}
}

// (level: the first that was not launched; large tasks left there mean that the trees are not
// ready for this tier yet.)
__global__ void __launch_bounds__(32 * kMidWarps) k_sah_mid(SahArgs A, int level) {
	chain_enter();
	__shared__ MidShared S;
	if (n_large(A, level))
		return;
	const uint32_t n_tasks = min(A.ctr[kCtrMid], A.max_mid);
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	for (uint32_t ti = blockIdx.x; ti < n_tasks; ti += gridDim.x) {
		const SahTask t = A.mid[ti];
		if (!range_ok(A, t.begin, t.count) || t.count > kLarge || t.count <= kSmall) {
			if (threadIdx.x == 0)
				flag(A.err);
			continue;
		}
		const uint32_t buf = t.meta & 1u;
		const float4 *src = A.rec[buf];
		for (uint32_t i = threadIdx.x; i < t.count; i += 32 * kMidWarps) {
			S.rec[i] = src[2 * (size_t)(t.begin + i)];
			S.rec[kLarge + i] = src[2 * (size_t)(t.begin + i) + 1];
			S.perm[0][i] = (uint16_t)i;
		}
		if (threadIdx.x == 0) {
			const uint32_t base = new_node(A, t.count - 2u);
			S.range[0][0] = MidRange{0u, t.count, t.node, base, t.parent, (t.meta >> 8) & 0xFFu};
			S.n_range[0] = base == kNone ? 0u : 1u;
			S.n_range[1] = 0u;
		}
		__syncthreads();
		for (int level = 0;; ++level) {
			const int in = level & 1;
			const uint32_t n = min(S.n_range[in], kMidRanges);
			if (n == 0u)
				break;
			// One range: all four warps split it; two: two each; more: one warp each.
			const int team = n == 1u ? 4 : (n == 2u ? 2 : 1);
			for (uint32_t k = warp / team; k < n; k += kMidWarps / team) {
				const MidRange r = S.range[in][k];
				split_range(A, S, r, in, t.begin, A.rec[buf ^ 1u], buf ^ 1u, team, warp, lane);
				__syncwarp();
			}
			__syncthreads();
			if (threadIdx.x == 0)
				S.n_range[in] = 0u;
			__syncthreads();
		}
		__syncthreads(); // the ranges are read before the next task's overwrite them
	}
}

// ---------------------------------------------------------------------------------------
// Small tasks: one warp builds the subtree of up to 32 triangles, one per lane.  The
// triangles are ranked once per axis by (centre, index); each node orders its lanes on
// each axis from those ranks (one OR of rank bits and a population count), sweeps prefix
// and suffix boxes and reorders its lanes by the best axis; the children are the two
// parts.
//
// The kernel is bound by instruction issue, and half of a task's nodes are pairs and most
// others have at most 10 triangles (a task of 20 has about 19 nodes: 10 pairs, 7 of 3 to
// 10).  So nodes of 3 to kTrio triangles sweep all three axes at once, in three groups of
// kTrio lanes, pairs are written together after the task's last split (they have nothing to
// choose), and the lane that holds the best split writes the node.  With the same tree, the
// 1,048,576-triangle heightfield builds in 2.32 instead of 2.75 ms, 8.4M clustered triangles
// in 15.4 instead of 18.8 ms.

constexpr int kTrio = 10; // triangles of a node whose three axes share one sweep

struct SmallSplit {
	Box6 lb, rb;  // in lane `src`: the boxes of the two parts
	int src;      // the lane that holds the split (-1: none found)
	int axis, k;  // axis and last position of the left part
};

// Inclusive prefix (p) and the box after it (r) of the `cnt` boxes in positions i = 0.. of
// each segment of lanes; `in`: the lane holds one of them.
__device__ __forceinline__ void sweep(const Box6 &b, bool in, int i, int cnt, int lane, Box6 &p,
                                      Box6 &r) {
	Box6 q = b;
	p = b;
	for (int o = 1; o < cnt; o <<= 1) {
		const Box6 pu = shfl_box(p, max(lane - o, 0));
		const Box6 qd = shfl_box(q, min(lane + o, 31));
		if (in && i >= o)
			p = box_union(p, pu);
		if (in && i + o < cnt)
			q = box_union(q, qd);
	}
	r = shfl_box(q, min(lane + 1, 31));
}

__device__ __forceinline__ Box6 staged_box(const float4 *stage, uint32_t at) {
	const float4 l = stage[at], h = stage[32 + at];
	return Box6{l.x, l.y, l.z, h.x, h.y, h.z};
}

// The node's box, children and range (called by one lane).
__device__ __forceinline__ void write_small_node(const SahArgs &A, uint32_t node, uint32_t first,
                                                 uint32_t nl, uint32_t nr, uint32_t id_l,
                                                 uint32_t id_r, const Box6 &lb, const Box6 &rb) {
	A.left[node] = nl > 1 ? id_l : (kLeafBit | first);
	A.right[node] = nr > 1 ? id_r : (kLeafBit | (first + nl));
	A.rfirst[node] = first;
	A.rlast[node] = first + nl + nr - 1u;
	A.splits[first + nl - 1u] = make_uint4(first, first + nl + nr - 1u, node, 0u);
	write_node_box(A, node, box_union(lb, rb), nl > 1 ? box_area(lb) : -1.0f,
	               nr > 1 ? box_area(rb) : -1.0f);
}

__global__ void __launch_bounds__(128) k_sah_small(SahArgs A, int level) {
	chain_enter();
	if (n_large(A, level))
		return;
	__shared__ float4 stage_all[4][2 * 32]; // the task's boxes, by lane
	__shared__ uint8_t order_all[4][32];    // a sweep's order: the lane of each position
	const uint32_t n_tasks = min(A.ctr[kCtrSmall], A.max_small);
	const int lane = threadIdx.x & 31;
	const int trio_a = lane / kTrio, trio_i = lane - trio_a * kTrio;
	float4 *stage = stage_all[threadIdx.x >> 5];
	uint8_t *order = order_all[threadIdx.x >> 5];
	for (uint32_t ti = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; ti < n_tasks;
	     ti += (gridDim.x * blockDim.x) >> 5) {
		const SmallTask st = A.small[ti];
		const uint32_t m = st.meta & 0xFFu, buf = (st.meta >> 8) & 1u, depth0 = st.meta >> 16;
		if (m == 0 || m > kSmall || st.begin > A.n || m > A.n - st.begin) {
			if (lane == 0)
				flag(A.err);
			continue;
		}
		const float4 *src = A.rec[buf];
		float4 lo = make_float4(0, 0, 0, 0), hi = lo;
		if ((uint32_t)lane < m) {
			lo = src[2 * (size_t)(st.begin + lane)];
			hi = src[2 * (size_t)(st.begin + lane) + 1];
		}
		if (m >= 3) {
			// Each triangle's rank among the task's on each axis, by (centre, index),
			// packed 5 bits per axis into the unused w of its box (it moves with the
			// triangle when lanes are reordered).  A node's own order on an axis is then
			// one OR over its lanes' rank bits and a population count.
			uint32_t gr = 0;
#pragma unroll
			for (int a = 0; a < 3; ++a) {
				const uint64_t key = (uint32_t)lane < m
				                         ? (((uint64_t)f2ord(rec_c(lo, hi, a)) << 32) |
				                            __float_as_uint(lo.w))
				                         : ~0ull;
				uint32_t rank = 0;
				for (uint32_t j = 0; j < m; ++j)
					rank += __shfl_sync(0xFFFFFFFFu, key, (int)j) < key;
				gr |= min(rank, 31u) << (5 * a);
			}
			hi.w = __uint_as_float(gr);
			stage[lane] = lo;
			stage[32 + lane] = hi;
			__syncwarp();
		}
		if (m >= 2) {
			uint32_t base = m > 2 ? st.base : 0u;
			if (m > 2 && base == kNone) {
				if (lane == 0)
					base = new_node(A, m - 2);
				base = __shfl_sync(0xFFFFFFFFu, base, 0);
			}
			if (base == kNone || st.node == kNone || st.node >= A.node_cap) {
				if (lane == 0 && base != kNone)
					flag(A.err);
				continue;
			}
			uint32_t next = 0;
			// The node of the pair that starts at this lane (written after the splits).
			uint32_t pair = (m == 2 && lane == 0) ? st.node : kNone;
			// Warp-distributed stack of nodes of at least 3: lane j holds entry j (first |
			// count << 8 | depth << 16, node).
			uint32_t stk_a = 0, stk_n = 0;
			int top = 0;
			if (m > 2) {
				if (lane == 0) {
					stk_a = 0u | (m << 8) | (depth0 << 16);
					stk_n = st.node;
				}
				top = 1;
			}
			while (top > 0) {
				--top;
				const uint32_t ea = __shfl_sync(0xFFFFFFFFu, stk_a, top);
				const uint32_t node = __shfl_sync(0xFFFFFFFFu, stk_n, top);
				const int f = (int)(ea & 0xFFu), cnt = (int)((ea >> 8) & 0xFFu);
				const uint32_t dep = ea >> 16;
				if (cnt < 3 || f + cnt > (int)m || node >= A.node_cap || top >= 30) {
					if (lane == 0)
						flag(A.err);
					break;
				}
				const bool in = lane >= f && lane < f + cnt;
				const uint32_t ranks = __float_as_uint(hi.w);
				SmallSplit s;
				s.src = -1;
				s.axis = -1;
				s.k = cnt / 2 - 1;
				uint32_t rank_best = 0;
				if (dep < kDepthGuard && cnt <= kTrio) {
					uint32_t rank[3];
#pragma unroll
					for (int a = 0; a < 3; ++a) {
						const uint32_t bit = 1u << ((ranks >> (5 * a)) & 31u);
						const uint32_t members = __reduce_or_sync(0xFFFFFFFFu, in ? bit : 0u);
						rank[a] = __popc(members & (bit - 1u));
						if (in)
							order[a * kTrio + rank[a]] = (uint8_t)lane;
					}
					__syncwarp();
					const bool on = trio_a < 3 && trio_i < cnt;
					const Box6 b = staged_box(stage, on ? order[lane] : (uint32_t)f);
					Box6 p, r;
					sweep(b, on, trio_i, cnt, lane, p, r);
					uint32_t c32 = 0xFFFFFFFFu;
					if (on && trio_i < cnt - 1)
						c32 = f2ord(box_area(p) * (float)(trio_i + 1) +
						            box_area(r) * (float)(cnt - 1 - trio_i));
					// The least cost; ties to the lower axis, then the lower position, as
					// the lanes are ordered.
					const uint32_t cmin = __reduce_min_sync(0xFFFFFFFFu, c32);
					if (cmin != 0xFFFFFFFFu) {
						s.src = __ffs(__ballot_sync(0xFFFFFFFFu, c32 == cmin)) - 1;
						s.axis = s.src / kTrio;
						s.k = s.src - s.axis * kTrio;
						s.lb = p;
						s.rb = r;
						rank_best = s.axis == 0 ? rank[0] : (s.axis == 1 ? rank[1] : rank[2]);
					}
				} else if (dep < kDepthGuard) {
					uint32_t best = 0xFFFFFFFFu;
					for (int a = 0; a < 3; ++a) {
						const uint32_t bit = 1u << ((ranks >> (5 * a)) & 31u);
						const uint32_t members = __reduce_or_sync(0xFFFFFFFFu, in ? bit : 0u);
						const uint32_t rank = __popc(members & (bit - 1u));
						if (in)
							order[f + rank] = (uint8_t)lane;
						__syncwarp();
						const Box6 b = staged_box(stage, in ? order[lane] : (uint32_t)f);
						__syncwarp();
						Box6 p, r;
						sweep(b, in, lane - f, cnt, lane, p, r);
						uint32_t c32 = 0xFFFFFFFFu;
						if (in && lane < f + cnt - 1) {
							const int nl = lane - f + 1, nr = cnt - nl;
							c32 = f2ord(box_area(p) * (float)nl + box_area(r) * (float)nr);
						}
						const uint32_t cmin = __reduce_min_sync(0xFFFFFFFFu, c32);
						if (cmin < best) {
							best = cmin;
							s.src = __ffs(__ballot_sync(0xFFFFFFFFu, c32 == cmin)) - 1;
							s.axis = a;
							s.k = s.src - f;
							s.lb = p;
							s.rb = r;
							rank_best = rank;
						}
					}
				}
				__syncwarp(); // the boxes are read before they are reordered
				if (s.src >= 0) {
					// Reorder the node's lanes by the best axis.
					if (in) {
						stage[f + rank_best] = lo;
						stage[32 + f + rank_best] = hi;
					}
					__syncwarp();
					if (in) {
						lo = stage[lane];
						hi = stage[32 + lane];
					}
				} else {
					const Box6 me{lo.x, lo.y, lo.z, hi.x, hi.y, hi.z};
					s.lb = range_box(me, lane, f, f + s.k + 1);
					s.rb = range_box(me, lane, f + s.k + 1, f + cnt);
					s.src = 0;
				}
				const int nl = s.k + 1, nr = cnt - nl;
				// Node ids of the children (warp-uniform: nl, nr and next are).
				uint32_t ids[2] = {kNone, kNone};
				if (nl > 1)
					ids[0] = base + next++;
				if (nr > 1)
					ids[1] = base + next++;
				if (lane == s.src) {
					write_small_node(A, node, st.begin + f, (uint32_t)nl, (uint32_t)nr, ids[0], ids[1],
					                 s.lb, s.rb);
					if (node == st.node)
						write_parent_area(A, st.parent, box_area(box_union(s.lb, s.rb)));
				}
				// Push the children (right first, so the left is taken next).
				if (nr == 2 && lane == f + nl)
					pair = ids[1];
				if (nl == 2 && lane == f)
					pair = ids[0];
				if (nr > 2) {
					if (lane == top) {
						stk_a = (uint32_t)(f + nl) | ((uint32_t)nr << 8) | ((dep + 1u) << 16);
						stk_n = ids[1];
					}
					++top;
				}
				if (nl > 2) {
					if (lane == top) {
						stk_a = (uint32_t)f | ((uint32_t)nl << 8) | ((dep + 1u) << 16);
						stk_n = ids[0];
					}
					++top;
				}
			}
			const Box6 me{lo.x, lo.y, lo.z, hi.x, hi.y, hi.z};
			const Box6 after = shfl_box(me, min(lane + 1, 31));
			if (pair != kNone) {
				if (pair < A.node_cap && (uint32_t)lane + 1u < m) {
					write_small_node(A, pair, st.begin + lane, 1u, 1u, kNone, kNone, me, after);
					if (pair == st.node)
						write_parent_area(A, st.parent, box_area(box_union(me, after)));
				} else {
					flag(A.err);
				}
			}
		}
		if ((uint32_t)lane < m) {
			const uint32_t pos = st.begin + lane;
			A.vals[pos] = __float_as_uint(lo.w);
			A.lbox[2 * (size_t)pos] = make_float4(lo.x, lo.y, lo.z, 0.0f);
			A.lbox[2 * (size_t)pos + 1] = make_float4(hi.x, hi.y, hi.z, 0.0f);
		}
		__syncwarp(); // the stage is read before the next task's boxes overwrite it
	}
}

// What the stages after the binary trees may rely on: every node id handed out was written
// (the collapse follows the children) and no check failed; else they do nothing.
__global__ void k_sah_gate(SahArgs A, int level, uint32_t want, uint32_t *gate) {
	chain_enter();
	*gate = n_large(A, level)                                            ? kGateLevels
	        : ((*A.err & kErrSah) || A.ctr[kCtrNodesSah] != want) ? kGateError
	                                                              : 0u;
}

__global__ void k_sah_bounds_init(uint32_t *gb, uint32_t n_scenes, XFaces x_faces) {
	if (x_faces.log) {
		const uint32_t quads = (kXHead + (1u << (x_faces.log - 5u))) / 4u;
		for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < quads;
		     i += gridDim.x * blockDim.x)
			reinterpret_cast<uint4 *>(x_faces.words)[i] = make_uint4(0u, i ? 0u : x_faces.log, 0u, 0u);
	}
	for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < 6 * n_scenes;
	     i += gridDim.x * blockDim.x)
		gb[i] = (i % 6) < 3 ? 0xFFFFFFFFu : 0u;
}

inline unsigned blocks_for(uint64_t n, unsigned t) { return (unsigned)((n + t - 1) / t); }

struct Layout {
	size_t max_large, max_mid, max_small, max_chunks;
	size_t off[11];
	size_t total;
};

// Regions of the scratch, 256-byte aligned: records, bins, large tasks and chunks (two each),
// then mid tasks, small tasks and counters.
Layout layout(uint32_t n, uint32_t S) {
	Layout L;
	L.max_large = n / (kLarge + 1) + S + 1;
	L.max_mid = n / (kSmall + 1) + S + 1;
	L.max_small = (size_t)n + S + 1;
	// (As many for n as for any smaller n: scratch reserved for a size serves those below.)
	L.max_chunks = std::max(n / (256 * kMaxPer), std::min(n / 256, kSpread)) + L.max_large;
	const size_t bins = 4ull * kBinWords * L.max_large, large = sizeof(SahTask) * L.max_large,
	             chunks = 8 * L.max_chunks;
	const size_t sz[11] = {32ull * n, 32ull * n, bins,   bins, large, large, chunks, chunks,
	                       sizeof(SahTask) * L.max_mid, sizeof(SmallTask) * L.max_small,
	                       4 * kCtrWordsSah};
	size_t at = 0;
	for (int k = 0; k < 11; ++k) {
		L.off[k] = at;
		at += (sz[k] + 255) & ~size_t(255);
	}
	L.total = at;
	return L;
}

} // namespace

size_t sah_scratch_bytes(uint32_t n, uint32_t S) { return layout(n, S).total; }

namespace {

// The kernels' arguments over the reserved scratch; false when it is too small.
bool sah_args(const BuildPlan &plan, BuildScratch &ws, uint32_t *d_err, Layout &L, SahArgs &A) {
	const uint32_t n = plan.n, S = plan.S;
	L = layout(n, S);
	if (ws.sah.bytes < L.total || ws.roots.bytes < 4ull * S)
		return false;
	char *p = ws.sah.as<char>();
	A.rec[0] = reinterpret_cast<float4 *>(p + L.off[0]);
	A.rec[1] = reinterpret_cast<float4 *>(p + L.off[1]);
	for (int k = 0; k < 2; ++k) {
		A.bins[k] = reinterpret_cast<uint32_t *>(p + L.off[2 + k]);
		A.large[k] = reinterpret_cast<SahTask *>(p + L.off[4 + k]);
		A.chunk[k] = reinterpret_cast<uint2 *>(p + L.off[6 + k]);
	}
	A.mid = reinterpret_cast<SahTask *>(p + L.off[8]);
	A.small = reinterpret_cast<SmallTask *>(p + L.off[9]);
	A.ctr = reinterpret_cast<uint32_t *>(p + L.off[10]);
	A.vals = ws.vals.as<uint32_t>();
	A.lbox = ws.lbox.as<float4>();
	A.left = ws.left.as<uint32_t>();
	A.right = ws.right.as<uint32_t>();
	A.rfirst = ws.rfirst.as<uint32_t>();
	A.rlast = ws.rlast.as<uint32_t>();
	A.ibox = ws.ibox.as<float4>();
	A.splits = ws.splits.as<uint4>();
	A.node_cap = plan.n_int + S;
	A.max_large = (uint32_t)L.max_large;
	A.max_mid = (uint32_t)L.max_mid;
	A.max_small = (uint32_t)L.max_small;
	A.max_chunks = (uint32_t)L.max_chunks;
	A.n = n;
	const uint32_t per = tris_per_thread(n);
	A.chunk_log = per == 1u ? 8u : per == 2u ? 9u : 10u;
	A.err = d_err;
	return true;
}

void launch_levels(const SahArgs &A, const BuildPlan &plan, const Layout &L, int &level, int count,
                   cudaStream_t st) {
	for (int k = 0; k < count && level < kMaxLevels; ++k, ++level) {
		// Grids no larger than the work the level can hold: each task has at most two
		// children, so level L has at most S * 2^L tasks (a small scene's levels are then a
		// few blocks each instead of 1216 idle ones).
		const uint64_t tasks =
		    std::min<uint64_t>((uint64_t)plan.S << std::min(level, 30), L.max_large);
		const unsigned grid = (unsigned)std::min<uint64_t>(1216, (plan.n >> A.chunk_log) + tasks);
		const unsigned splits = (unsigned)std::min<uint64_t>(304, (tasks + 3) / 4);
		launch_after(true, k_sah_split, splits, 128, st, A, level);
		launch_after(true,
		             A.chunk_log == 8   ? k_sah_part<1>
		             : A.chunk_log == 9 ? k_sah_part<2>
		                                : k_sah_part<kMaxPer>,
		             grid, 256, st, A, level);
	}
}

// The mid and small tiers and the gate, after large levels 0 .. level - 1.
void launch_tail(const SahArgs &A, const BuildPlan &plan, const Layout &L, int level,
                 uint32_t *gate, cudaStream_t st) {
	const unsigned mids = (unsigned)std::min<size_t>(1216, L.max_mid);
	launch_after(true, k_sah_mid, mids, 32 * kMidWarps, st, A, level);
	launch_after(true, k_sah_small, 2432, 128, st, A, level);
	uint64_t want = plan.S;
	for (uint32_t s = 0; s < plan.S; ++s) {
		const uint32_t ns = plan.toff[s + 1] - plan.toff[s];
		want += ns >= 2 ? ns - 2 : 0;
	}
	launch_after(true, k_sah_gate, 1, 1, st, A, level, (uint32_t)want, gate);
}

} // namespace

int sah_build_enqueue(const float *d_tris, const BuildPlan &plan, BuildScratch &ws,
                      const uint32_t *d_toff, const uint32_t *scene_of, XFaces x_faces,
                      cudaStream_t st, uint32_t *d_err, uint32_t *gate, int &level,
                      std::string &msg) {
	const uint32_t n = plan.n, S = plan.S;
	Layout L;
	SahArgs A;
	if (!sah_args(plan, ws, d_err, L, A)) {
		msg = "sah build: scratch not reserved";
		return PRT_ERR_DEVICE;
	}
	uint32_t *gb = ws.bounds.as<uint32_t>();
	cudaMemsetAsync(A.ctr, 0, 4 * kCtrWordsSah, st);
	const uint64_t clear = x_faces.log ? 1ull << (x_faces.log - 5u) : 0u; // words
	k_sah_bounds_init<<<std::max(blocks_for(6ull * S, 256),
	                             std::min(blocks_for(clear / 4u, 256), 608u)),
	                    256, 0, st>>>(gb, S, x_faces);
	if (n)
		launch_after(true, k_sah_records, blocks_for(n, 256), 256, st, d_tris, n, scene_of,
		             A.rec[0], gb, x_faces);
	launch_after(true, k_sah_first_id, 1, 1, st, A.ctr, S);
	launch_after(true, k_sah_roots, blocks_for(32ull * S, 128), 128, st, A, d_toff, S, gb,
	             ws.roots.as<uint32_t>());
	// As many levels as halving splits need to bring the largest scene under the large-task
	// size, and two more, since splits are uneven (an empty level costs about 2 us, a look at
	// the counters a host wait of about 10); sah_build_more takes up what is left.
	uint32_t biggest = 0;
	for (uint32_t sc = 0; sc < S; ++sc)
		biggest = std::max(biggest, plan.toff[sc + 1] - plan.toff[sc]);
	int ahead = 0;
	for (uint64_t c = biggest; c > kLarge; c = (c + 1) / 2)
		++ahead;
	level = 0;
	if (ahead) {
		const unsigned bins = (unsigned)std::min<size_t>(1216, L.max_chunks);
		launch_after(true,
		             A.chunk_log == 8   ? k_sah_bin<1>
		             : A.chunk_log == 9 ? k_sah_bin<2>
		                                : k_sah_bin<kMaxPer>,
		             bins, 256, st, A);
		launch_levels(A, plan, L, level, ahead + 2, st);
	}
	launch_tail(A, plan, L, level, gate, st);
	return PRT_OK;
}

int sah_build_more(const BuildPlan &plan, BuildScratch &ws, cudaStream_t st, uint32_t *d_err,
                   uint32_t *gate, int &level, std::string &msg) {
	Layout L;
	SahArgs A;
	if (!sah_args(plan, ws, d_err, L, A)) {
		msg = "sah build: scratch not reserved";
		return PRT_ERR_DEVICE;
	}
	for (;;) {
		if (level >= kMaxLevels) {
			msg = "sah build: more than " + std::to_string(kMaxLevels) + " levels";
			return PRT_ERR_LIMIT;
		}
		launch_levels(A, plan, L, level, kLevelsPerCheck, st);
		cudaError_t e =
		    cudaMemcpyAsync(ws.h_sah, A.ctr + kCtrLarge + level, 4, cudaMemcpyDeviceToHost, st);
		if (e == cudaSuccess)
			e = cudaStreamSynchronize(st);
		if (e != cudaSuccess) {
			msg = std::string("sah build: ") + cudaGetErrorString(e);
			return PRT_ERR_CUDA;
		}
		if (ws.h_sah[0] == 0)
			break;
	}
	launch_tail(A, plan, L, level, gate, st);
	return PRT_OK;
}

} // namespace prt
