// prt_internal.cuh - shared definitions of the GB300 ray-query backend.
//
// Data layout in HBM for one scene (n triangles):
//   tri4   float4[3n]  triangle records in leaf order: (v0.xyz, primitive id bits),
//                      (v1.xyz, 0), (v2.xyz, 0); 48 B per triangle.
//   nodes  Node8[]     8-wide nodes, 256 B each (eight 32-B child records: box and
//                      reference), root at index 0.
//   cnodes CNode8[]    the same tree with 8-bit child boxes, 96 B each (optional).
//
// A child reference is 32 bits: 0xFFFFFFFF = empty slot; bit 31 clear = index of a
// child node; bit 31 set = leaf holding triangles [first, first + count) of tri4 with
// first in bits 0..27 and count - 1 in bits 28..30.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "prt_errword.h"

namespace prt {

constexpr uint32_t kNone = 0xFFFFFFFFu;
constexpr uint32_t kLeafBit = 0x80000000u;
constexpr uint32_t kFirstMask = 0x0FFFFFFFu;
constexpr int kMaxLeaf = 8;
// Triangles per scene: the traversal packs (ray slot, node or triangle index) into 32
// bits with 27 bits for the index.
constexpr uint64_t kMaxTris = (1ull << 27) - 1;
constexpr uint32_t kIndexBits = 27;
constexpr uint32_t kIndexMask = (1u << kIndexBits) - 1u;

// Bits of an error word (prt_errword.h).
enum : uint32_t {
	kErrStack = 1u,    // traversal stack overflow (ray abandoned)
	kErrLookback = 2u, // radix-sort look-back gave up waiting
	kErrCollapse = 4u, // 8-wide collapse ran out of node slots
	kErrSah = 8u,      // SAH build: a range, node id or task list check failed
};

// One child of an 8-wide FP32 node: its box as centre and half extent and its reference,
// 32 B, so the lane that tests child c reads it with one 32-byte load and a node's 8
// children are 256 contiguous bytes.  x and y sit in aligned pairs for the packed FP32
// arithmetic of the slab test.  encode_child makes the record, child_lo / child_hi bound
// the box from outside.
struct alignas(16) Child8 {
	float cx, cy, ex, ey, cz, ez;
	uint32_t ref;
	uint32_t x16; // the box's x bounds in 16 bits each (x_bounds16)
};
struct alignas(16) Node8 {
	Child8 c[8];
};
static_assert(sizeof(Node8) == 256, "Node8 layout");

// A decoded compressed bound, origin + q * scale with one rounding (a fused multiply-add:
// q <= 255 times a power of two is exact, so this is o + q * s correctly rounded, even
// where q * s alone would overflow).  The builder verifies every bound with this
// function and the traversal decodes with it, so the two agree bit for bit.
__device__ __forceinline__ float cdec_f(float o, float q, float s) { return __fmaf_rn(q, s, o); }

// Compressed 8-wide node (96 B = 37.5 % of Node8), the same tree as Node8.  Child box
// k, per axis a: lo = origin_a + q_lo * 2^(e_a - 127), hi = origin_a + q_hi * 2^(e_a - 127),
// evaluated in FP32 exactly as the traversal does (cdec_f); the builder chooses each q so
// that the decoded box contains the child's FP32 box (rounded outward), which keeps
// every box test conservative.  Child k is an inner node when bit k of imask is set, at
// index child_base + (number of inner children before k); otherwise, when count > 0,
// a leaf of `count` triangles starting at tri_base + first.
struct alignas(8) CChild8 {
	uint8_t qlo_x, qhi_x, qlo_y, qhi_y, qlo_z, qhi_z;
	uint8_t count; // leaf triangles (0 = inner child or empty slot)
	uint8_t first; // leaf: first triangle relative to tri_base
};
struct alignas(16) CNode8 {
	float ox, oy, oz;       // frame origin (the node's lower corner)
	uint8_t ex, ey, ez;     // scale exponents, IEEE-biased
	uint8_t imask;          // inner-node children
	uint32_t child_base;    // first inner child
	uint32_t tri_base;      // first triangle of the node's leaf children
	uint32_t pad[2];
	CChild8 c[8];
};
static_assert(sizeof(CChild8) == 8, "CChild8 layout");
static_assert(sizeof(CNode8) == 96, "CNode8 layout");

// Decodes one quantised bound.  2^(e-127) * q is exact (q < 256, e in [1, 254]); the
// sum is rounded once, and the builder verified the rounded value, so this exact
// expression must be used on both sides.
__host__ __device__ inline float cscale(uint8_t e) {
	union { uint32_t u; float f; } s;
	s.u = (uint32_t)e << 23;
	return s.f;
}

__host__ __device__ inline uint32_t make_leaf(uint32_t first, uint32_t count) {
	return kLeafBit | ((count - 1u) << 28) | first;
}
__host__ __device__ inline bool ref_is_leaf(uint32_t r) { return (r & kLeafBit) != 0; }
__host__ __device__ inline uint32_t leaf_first(uint32_t r) { return r & kFirstMask; }
__host__ __device__ inline uint32_t leaf_count(uint32_t r) { return ((r >> 28) & 7u) + 1u; }

// std::min / std::max as portableRT calls them: select on operator<, so a NaN in the
// first argument survives and a NaN in the second is dropped.
__device__ __forceinline__ float rmin(float a, float b) { return (b < a) ? b : a; }
__device__ __forceinline__ float rmax(float a, float b) { return (a < b) ? b : a; }

// Order-preserving float <-> uint32 map for atomicMin / atomicMax on floats.
__device__ __forceinline__ uint32_t f2ord(float f) {
	uint32_t u = __float_as_uint(f);
	return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float ord2f(uint32_t u) {
	return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
}

// Per-ray constants.  `kind` selects the box test used on inner nodes (prt_traverse.cu):
//   0 regular: finite, every origin component within 2^67 and every direction component at
//              least 2^-58 in magnitude: the slab test on centres and half extents (SlabRay)
//              neither overflows nor meets a NaN.
//   1 far:     like 0, but so far from the scene that the margin of that test would pass
//              many boxes that the ray misses (far_scene; FP32 nodes): the slab test on
//              bounds (AxisRay).
//   2 all:     a non-finite component or all reciprocals infinite: every inner box passes
//              and only the exact per-triangle test decides.
//   3 other:   any other ray, for instance with a zero direction component (infinite
//              reciprocal): the slab test on bounds (AxisRay).
//   4 x:       like 3 with an infinite reciprocal on the x axis, where some triangle's box
//              may have its lower x face at the origin's x (XFaces): a box around it
//              passes outright.
struct RayC {
	float ox, oy, oz, dx, dy, dz, fx, fy, fz;
	int kind;
};

// (2^67 + 2^67) * 2^58 stays below FLT_MAX; 2^67 is about 1.5e20, 2^-58 about 3.5e-18.
constexpr float kCoordMax = 0x1p67f, kDirMin = 0x1p-58f, kFltMax = 0x1.fffffep127f;

__device__ __forceinline__ bool dir_regular(float d) {
	return fabsf(d) <= kFltMax && fabsf(d) >= kDirMin;
}

__device__ __forceinline__ RayC make_ray(float ox, float oy, float oz, float dx, float dy,
                                         float dz) {
	RayC r;
	r.ox = ox; r.oy = oy; r.oz = oz;
	r.dx = dx; r.dy = dy; r.dz = dz;
	// IEEE reciprocal, identical to portableRT's 1.0f / direction (bvh.hpp:199-201).
	r.fx = __frcp_rn(dx);
	r.fy = __frcp_rn(dy);
	r.fz = __frcp_rn(dz);
	// (A NaN component fails its comparison, so it is never regular.)
	const bool regular = fabsf(ox) <= kCoordMax && fabsf(oy) <= kCoordMax &&
	                     fabsf(oz) <= kCoordMax && dir_regular(dx) && dir_regular(dy) &&
	                     dir_regular(dz);
	r.kind = 0;
	if (!regular) {
		const bool fin = isfinite(ox) && isfinite(oy) && isfinite(oz) && isfinite(dx) &&
		                 isfinite(dy) && isfinite(dz);
		const bool ix = isinf(r.fx), iy = isinf(r.fy), iz = isinf(r.fz);
		r.kind = !fin || (ix && iy && iz) ? 2 : ix ? 4 : 3;
	}
	return r;
}

// What tells rays far from a scene: its centre and the distance past which they are.  The
// margin, 2^-20 of the distance, widens a box as a ray sees it, and boxes around a triangle of a
// surface are about its extent / sqrt(n) wide; twice that distance is where the test on bounds,
// which takes 1.4 times as long, becomes the faster one.  600,000 rays at targets on the
// heightfields, from 10,000 / 100,000 times the extent, us (with bounds stored in the nodes
// 186 / 224 and 252 / 470): 65,790 triangles 277 / 2,660 -> 275 / 292, 1,048,576 triangles
// 890 / 31,300 -> 345 / 761.
// From the bounds of the triangles' centroids; kept after the empty node, scene by scene.
__device__ __forceinline__ float4 far_scene(const float lo[3], const float hi[3], uint32_t n) {
	float4 f = make_float4(0.5f * lo[0] + 0.5f * hi[0], 0.5f * lo[1] + 0.5f * hi[1],
	                       0.5f * lo[2] + 0.5f * hi[2], INFINITY);
	const float e = fmaxf(hi[0] - lo[0], fmaxf(hi[1] - lo[1], hi[2] - lo[2]));
	if (n > 0u && e > 0.0f && e < kFltMax)
		f.w = e * 0x1p21f * rsqrtf((float)n);
	return f;
}
__host__ __device__ __forceinline__ float4 *far_scenes(void *nodes, uint32_t dead) {
	return reinterpret_cast<float4 *>(static_cast<Node8 *>(nodes) + dead + 1u);
}

// One axis of a child record: centre c and half extent e with [lo, hi] inside
// [c - e, c + e] and e wider than that needs by a factor 1 + 2^-21 (the margin that the
// test's rounding uses up).  A bound beyond 2^67 makes the axis [-FLT_MAX, FLT_MAX].
__device__ __forceinline__ void encode_axis(float lo, float hi, float &c, float &e) {
	if (!(lo >= -kCoordMax && hi <= kCoordMax)) {
		c = 0.0f;
		e = kFltMax;
		return;
	}
	c = __fadd_rn(__fmul_rn(lo, 0.5f), __fmul_rn(hi, 0.5f));
	e = __fmul_ru(fmaxf(__fsub_ru(hi, c), __fsub_ru(c, lo)), 1.0f + 0x1p-21f);
}

// Lower (low half) and upper bound as the top 16 bits of a float, rounded outwards.  A
// centre and half extent lose on which side of 0 a face near 0 lies, so both boxes beside a
// mesh's symmetry plane would count as around it: a ray in that plane (a camera's middle
// column) passes every box around its x, and twice as many of them made the longest chain of
// a small image (65,536 triangles, 320 x 200: 116 -> 154 us).
__device__ __forceinline__ uint32_t x_bounds16(float lo, float hi) {
	uint32_t l = __float_as_uint(lo), h = __float_as_uint(hi);
	if (lo < 0.0f)
		l += 0xFFFFu;
	if (hi > 0.0f)
		h += 0xFFFFu;
	return (l >> 16) | (h & 0xFFFF0000u);
}

// The record of a child box; ref == kNone: an unused slot (a NaN box, which no regular
// ray's test passes).
__device__ __forceinline__ Child8 encode_child(const float4 &lo, const float4 &hi, uint32_t ref) {
	Child8 ch;
	if (ref == kNone) {
		ch.cx = ch.cy = ch.cz = ch.ex = ch.ey = ch.ez = __int_as_float(0x7FC00000);
	} else {
		encode_axis(lo.x, hi.x, ch.cx, ch.ex);
		encode_axis(lo.y, hi.y, ch.cy, ch.ey);
		encode_axis(lo.z, hi.z, ch.cz, ch.ez);
	}
	ch.ref = ref;
	ch.x16 = x_bounds16(lo.x, hi.x);
	return ch;
}

// Bounds that contain the box a record was made from.
__device__ __forceinline__ float child_lo(float c, float e) { return __fsub_rd(c, e); }
__device__ __forceinline__ float child_hi(float c, float e) { return __fadd_ru(c, e); }

// Set of the x coordinates at which some triangle's box of a scene has its lower face: a
// hash set of 2^log bits (8 to 16 per triangle) after kXHead words, of which the first is
// set when every x may be one (a triangle is not finite, or a later build made no set) and the
// second holds log: a query captured in a graph reads both when it runs, whatever has been
// built into the scene's buffers since.  Builders take log 0 for no set.
// A ray with a zero x component passed every box around its x, thousands of nodes that were
// the tail of the launch; off the faces y and z now prune (16,000 camera and secondary rays on
// a 65,790-triangle heightfield 39 -> 23 us, 6,000 through the host call 63 -> 48; the build
// of those triangles takes 2 to 6 us of 470 more).
constexpr uint32_t kXHead = 4;
struct XFaces {
	uint32_t *words;
	uint32_t log;
};
__device__ __forceinline__ uint32_t x_face_bit(float x, uint32_t log) {
	return (__float_as_uint(__fadd_rn(x, 0.0f)) * 2654435761u) >> (32u - log); // (-0 as 0)
}
__device__ __forceinline__ void x_face_add(const XFaces &f, float x) {
	const uint32_t k = x_face_bit(x, f.log), bit = 1u << (k & 31u);
	atomicOr(f.words + kXHead + (k >> 5), bit);
}
// Whether no triangle's lower x face is at x.
__device__ __forceinline__ bool x_face_free(const uint32_t *words, float x) {
	const uint2 head = __ldg(reinterpret_cast<const uint2 *>(words));
	if (head.x)
		return false;
	const uint32_t k = x_face_bit(x, head.y);
	return !((__ldg(words + kXHead + (k >> 5)) >> (k & 31u)) & 1u);
}

// Slab test of portableRT's ray_box_intersect (bvh.hpp:195-222), bit for bit: each
// t is (bound - origin) * reciprocal in round-to-nearest, combined with the select
// min/max in the reference's nesting.  Used on every triangle's own bounding box.
__device__ __forceinline__ bool ref_slab(const RayC &r, float lx, float ly, float lz, float hx,
                                         float hy, float hz) {
	float t1 = __fmul_rn(__fsub_rn(lx, r.ox), r.fx);
	float t2 = __fmul_rn(__fsub_rn(hx, r.ox), r.fx);
	float t3 = __fmul_rn(__fsub_rn(ly, r.oy), r.fy);
	float t4 = __fmul_rn(__fsub_rn(hy, r.oy), r.fy);
	float t5 = __fmul_rn(__fsub_rn(lz, r.oz), r.fz);
	float t6 = __fmul_rn(__fsub_rn(hz, r.oz), r.fz);
	float tmin = rmax(rmax(rmin(t1, t2), rmin(t3, t4)), rmin(t5, t6));
	float tmax = rmin(rmin(rmax(t1, t2), rmax(t3, t4)), rmax(t5, t6));
	if (tmax < 0.0f)
		return false;
	if (tmin > tmax)
		return false;
	return true;
}

// Inner-node test for regular rays.  Same (bound - origin) * reciprocal rounding as
// ref_slab; an inner box contains every triangle box below it and that expression is
// monotone in the bound, so whatever ref_slab accepts below, this accepts here.  No
// NaN can arise (finite bounds or +-inf, finite non-zero reciprocal).
__device__ __forceinline__ bool regular_box(const RayC &r, float lx, float hx, float ly, float hy,
                                            float lz, float hz) {
	float t1 = (lx - r.ox) * r.fx, t2 = (hx - r.ox) * r.fx;
	float t3 = (ly - r.oy) * r.fy, t4 = (hy - r.oy) * r.fy;
	float t5 = (lz - r.oz) * r.fz, t6 = (hz - r.oz) * r.fz;
	float tmin = fmaxf(fmaxf(fminf(t1, t2), fminf(t3, t4)), fminf(t5, t6));
	float tmax = fminf(fminf(fmaxf(t1, t2), fmaxf(t3, t4)), fmaxf(t5, t6));
	return tmax >= 0.0f && tmin <= tmax;
}

// Moller-Trumbore in portableRT's operation order (core.hpp:27-65): every product and
// sum rounded separately (no FMA), sums left to right, IEEE reciprocal of det.
__device__ __forceinline__ bool ref_mt(const RayC &r, float v0x, float v0y, float v0z, float v1x,
                                       float v1y, float v1z, float v2x, float v2y, float v2z,
                                       float &t, float &u, float &v) {
	float e1x = __fsub_rn(v1x, v0x), e1y = __fsub_rn(v1y, v0y), e1z = __fsub_rn(v1z, v0z);
	float e2x = __fsub_rn(v2x, v0x), e2y = __fsub_rn(v2y, v0y), e2z = __fsub_rn(v2z, v0z);
	float px = __fsub_rn(__fmul_rn(r.dy, e2z), __fmul_rn(r.dz, e2y));
	float py = __fsub_rn(__fmul_rn(r.dz, e2x), __fmul_rn(r.dx, e2z));
	float pz = __fsub_rn(__fmul_rn(r.dx, e2y), __fmul_rn(r.dy, e2x));
	float det = __fadd_rn(__fadd_rn(__fmul_rn(e1x, px), __fmul_rn(e1y, py)), __fmul_rn(e1z, pz));
	if (det == 0.0f)
		return false;
	float inv = __frcp_rn(det);
	float tx = __fsub_rn(r.ox, v0x), ty = __fsub_rn(r.oy, v0y), tz = __fsub_rn(r.oz, v0z);
	u = __fmul_rn(__fadd_rn(__fadd_rn(__fmul_rn(tx, px), __fmul_rn(ty, py)), __fmul_rn(tz, pz)),
	              inv);
	if (u < 0.0f || u > 1.0f)
		return false;
	float qx = __fsub_rn(__fmul_rn(ty, e1z), __fmul_rn(tz, e1y));
	float qy = __fsub_rn(__fmul_rn(tz, e1x), __fmul_rn(tx, e1z));
	float qz = __fsub_rn(__fmul_rn(tx, e1y), __fmul_rn(ty, e1x));
	v = __fmul_rn(
	    __fadd_rn(__fadd_rn(__fmul_rn(r.dx, qx), __fmul_rn(r.dy, qy)), __fmul_rn(r.dz, qz)), inv);
	if (v < 0.0f || __fadd_rn(u, v) > 1.0f)
		return false;
	t = __fmul_rn(
	    __fadd_rn(__fadd_rn(__fmul_rn(e2x, qx), __fmul_rn(e2y, qy)), __fmul_rn(e2z, qz)), inv);
	return true;
}

// The closest hit so far.  Ties in t go to the smaller primitive id, so the answer
// does not depend on traversal order; a t of +inf or NaN is never recorded (the
// reference keeps a hit only when t < t_near, t_near starting at +inf).
struct Best {
	float t, u, v;
	uint32_t pid;
};

__device__ __forceinline__ void best_init(Best &b) {
	b.t = INFINITY;
	b.u = 0.0f;
	b.v = 0.0f;
	b.pid = kNone;
}

// The box half of tri_test for a ray with finite origin, direction and reciprocals (kinds
// 0, 1) and a triangle whose nine coordinates are finite (its record's flag word is 0):
// then no value is NaN, the select min/max of the reference agree with fminf / fmaxf
// (three-input where they nest; a zero's sign can differ, and no comparison sees it),
// and the answer is ref_slab's with fewer instructions.
__device__ __forceinline__ bool tri_box_finite(const RayC &r, const float4 a, const float4 b,
                                               const float4 c) {
	const float lx = fminf(a.x, fminf(b.x, c.x)), ly = fminf(a.y, fminf(b.y, c.y)),
	            lz = fminf(a.z, fminf(b.z, c.z));
	const float hx = fmaxf(a.x, fmaxf(b.x, c.x)), hy = fmaxf(a.y, fmaxf(b.y, c.y)),
	            hz = fmaxf(a.z, fmaxf(b.z, c.z));
	return regular_box(r, lx, hx, ly, hy, lz, hz);
}

// A triangle record's flag word (the second float4's w): 0 when every coordinate is
// finite, 1 otherwise.
__device__ __forceinline__ bool tri_record_finite(const float4 &b) { return b.w == 0.0f; }

// Exact per-triangle test: the reference slab test on the triangle's own bounding
// box (make_aabb, bvh.hpp:28-37, select semantics) and then Moller-Trumbore.  True
// when the reference would accept the triangle (its t may still be +inf or NaN, which
// the reference never records).
// finite: the ray is of kind 0 or 1 and the triangle's record flags no non-finite coordinate
// (tri_box_finite then decides the box test, with the same answer).
__device__ __forceinline__ bool tri_test(const RayC &r, const float4 a, const float4 b,
                                         const float4 c, float &t, float &u, float &v,
                                         bool finite = false) {
	bool pass;
	if (finite) {
		pass = tri_box_finite(r, a, b, c);
	} else {
		float lx = rmin(a.x, rmin(b.x, c.x)), ly = rmin(a.y, rmin(b.y, c.y)),
		      lz = rmin(a.z, rmin(b.z, c.z));
		float hx = rmax(a.x, rmax(b.x, c.x)), hy = rmax(a.y, rmax(b.y, c.y)),
		      hz = rmax(a.z, rmax(b.z, c.z));
		pass = ref_slab(r, lx, ly, lz, hx, hy, hz);
	}
	if (!pass)
		return false;
	return ref_mt(r, a.x, a.y, a.z, b.x, b.y, b.z, c.x, c.y, c.z, t, u, v);
}

// The closest hit as one 64-bit key: order-preserving bits of t above the primitive
// id, so the minimum key is the smallest t and, among equal t, the smallest id (ties in
// t go to the smaller id).  -0 and +0 compare equal as floats, so both map to +0's key
// (the traversal keeps the winner's own zero sign, u and v beside the key, or tests the
// winner again).  kNoHit: nothing recorded.
constexpr unsigned long long kNoHit = ~0ull;

__device__ __forceinline__ unsigned long long hit_key(float t, uint32_t pid) {
	float tc = (t == 0.0f) ? 0.0f : t;
	return ((unsigned long long)f2ord(tc) << 32) | pid;
}

} // namespace prt
