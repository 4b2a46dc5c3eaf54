// prt_traverse.cu - persistent nearest-hit traversal of the 8-wide tree.
//
// Replaces BVH2::nearest_tri (portableRT bvh.hpp:224-265) and the std::thread loop of
// CPUBackend::nearest_hits (intersect_cpu.hpp:20-43).
//
// Answer (identical to the reference's on finite inputs): the smallest t over the
// triangles whose own bounding box passes the reference slab test and which
// Moller-Trumbore accepts; t may be negative, there is no t-min and no culling by t,
// exactly as in the reference.  Inner nodes only prune with tests that are
// conservative for that set (prt_internal.cuh), so neither the tree's shape nor the
// visit order changes the answer; ties in t go to the smaller primitive id.
//
// Execution: one warp = 8 groups of 4 lanes; all state for 32 rays is in shared memory.
//  * A warp takes up to 32 consecutive rays ("slots": 32 per batch, or 4 to 16 where 32
//    would leave most warps idle, single_batch): origin, direction, reciprocal and
//    best-hit key per slot live in shared memory.
//  * Work items (slot, node) sit in a warp-local LIFO pool.  Each step every group
//    pops one item and each of its 4 lanes loads and slab-tests 2 of the node's 8
//    children: lane s takes children s and s + 4, so each of the two 256-bit loads of a
//    group reads one 128-byte line of the node (children 2s and 2s + 1 would spread each
//    load over two lines and double the L1 wavefronts: 15 % slower).  Hit inner children
//    are pushed back as items and hit leaf triangles are appended to a triangle queue,
//    at positions from ballots and popc, child-major (all lanes' first children, then
//    all second children: no position depends on the lane's previous child; the step
//    issues 16 % fewer ALU-pipe instructions than in lane order, and the half-rate ALU
//    pipe is what bounds it).  Roots of new rays are admitted whenever fewer than 8
//    items are left.  Unused child slots hold NaN boxes, which no plain slab test
//    passes.
//  * A batch whose rays are all regular (kind 0) takes the plain slab test (SlabRay) on
//    FP32 nodes, any other the test on bounds (AxisRay): rays with zero direction
//    components, mostly, and rays from far away.  Queries of up to some hundred rays per
//    warp and most cameras are one launch with both (pass 4, single_batch).  Larger
//    queries of ray buffers are two: a regular pass (1), which holds the plain test alone
//    and counts and skips the other batches, and a deferred pass (2) over those (it
//    returns at once when there are none).  Large images of few triangles (pass 0) start
//    each regular batch with a packet descent (packet_descent); counting runs are pass 0
//    as well.  A request server's serving launch (pass 3) takes its batches from device
//    queues that the host extends while it runs (claim_batch).
//  * When 32 triangles are queued, the 32 lanes test one each with the exact reference
//    test and fold (t, primitive id) into the slot's 64-bit key with a shared atomicMin;
//    with FP32 nodes the lane whose key the slot kept records its u, v (and a zero t's
//    sign) beside it, with compressed nodes the winner is tested again at the end.
//  * When the pool and the queue are empty the warp writes the 32 records in the
//    caller's HitReg<Tags...> layout to shared memory and stores them as 16-byte words.
//  * The pool holds at most 7 K (D - 1) + K items for K = 8 items per step and a tree of
//    depth D (each step's pushes leave at most 7 K items behind per level); it is sized
//    per launch as 7 K (D - 1) + 2 K; a push that would not fit, or a batch that takes
//    more steps than a tree can need, is reported as an error and ends the batch.
//
// Algorithmic bytes per ray: 24 (ray) + R (record) + node bytes visited + 48 per
// triangle tested; the counting variant (COUNT) measures the visits.
//
// Times in these comments are of the step they stand beside, both sides in turn on one GPU;
// the same workload differs by up to a tenth from one sitting to another, and later steps
// have shortened it since.
#include <algorithm>
#include <type_traits>
#include <mutex>

#include "../../include/prt_b200.h"
#include "prt_camera.cuh"
#include "prt_traverse.cuh"

namespace prt {

namespace {

constexpr int kWarpsPerBlock = 4;
// Lanes that test one node together (each takes 8 / kLanesPerNode children); a warp
// step visits 32 / kLanesPerNode nodes.
#ifndef PRT_TRAVERSE_LANES_PER_NODE
#define PRT_TRAVERSE_LANES_PER_NODE 4
#endif
constexpr int kLanesPerNode = PRT_TRAVERSE_LANES_PER_NODE;
constexpr int kItems = 32 / kLanesPerNode;       // items per step (K)
constexpr int kChildPerLane = 8 / kLanesPerNode;
constexpr int kMaxDepth = 32;
// Packet descent (packet_descent): rays that must share a node for the warp to test it for
// all of them at once; its stack (one entry per lane); the per-ray lists of nodes it leaves
// to item steps, and the length past which it stops descending.
constexpr uint32_t kPacketMin = 8;
constexpr uint32_t kPacketStack = 32;
constexpr uint32_t kListWords = 64;
constexpr uint32_t kListStop = kListWords - 8u - kPacketStack;
// Items that admission from the lists fills the pool up to.
constexpr uint32_t kAdmit = 24;

struct TravArgs {
	const SceneDesc *scenes; // scene table (n_segs > 0)
	const SegDesc *segs;     // segment table sorted by vbegin (n_segs > 0)
	uint32_t n_segs;         // 0: one run, described by seg0 / scene0
	uint32_t n_virtual;      // padded ray count
	SceneDesc scene0;
	SegDesc seg0;
	uint32_t n_nodes;        // largest node array (bounds the steps of a batch)
	uint32_t dead;           // index of a node of eight empty children in every scene's
	                         // node array (pads a step that has fewer than K items)
	uint32_t pool_cap;       // entries of the pool (>= 256, it also holds the staged records)
	uint32_t queue_cap;      // entries of the triangle queue
	uint32_t warp_bytes;     // shared memory per warp
	uint32_t max_leaf;       // most triangles in a leaf of any scene of the launch
	uint32_t max_batches;    // batches per warp before it exits (0 = no bound)
	uint32_t batch;          // rays a warp takes at a time: 32, or 4 to 16 where few rays
	                         // are to keep all warps busy (single_batch)
	uint32_t claims;         // PASS 4: rays per batch after a warp's first one (0: there are no
	                         // more batches than warps)
	uint32_t *counter;
	uint32_t *deferred;      // [0] batches the regular pass left to the general one,
	                         // [1] the deferred pass's batch counter
	uint32_t *err;
	unsigned long long *visits;
	uint32_t use_cam;        // 1: rays of the single run come from `cam`, not seg0.rays
	prt_b200_camera cam;
	const uint32_t *x_faces; // of the single run's scene (XFaces; null: none)
	ServeQueues serve;       // PASS 3 only
};

// Per-warp shared memory: fixed part, then the queue and the pool (sizes per launch).
// alignas(16): the queue follows this part and the pool after it doubles as the staging
// area of the output records, which is read with 16-byte vector loads.
struct alignas(16) WarpFixed {
	unsigned long long key[32]; // best (t, primitive id) per slot
	float4 ro[32];              // origin and kind (int bits) per slot
	float4 rf[32];              // reciprocals per slot
	float4 rd[32];              // direction per slot
	// rf[s].w and rd[s].w: u and v of slot s's winning hit (its key holds t exactly, up
	// to the sign of a zero, which bit s of negzero keeps); no array of their own, so
	// shared memory does not grow (a deep tree's pool already brings nine blocks close
	// to the SM's limit, and the L1 cache gets what shared memory leaves).
	SegDesc seg;                // the run the current 32 rays belong to
	uint32_t batches;           // batches this warp has taken (kept here, not in a register)
	// Serving launches: tickets past the published end per queue, and the queue whose
	// run `seg` holds (kept here, not in registers).
	uint32_t held[kServeQueues];
	uint32_t cached_q;
	uint32_t negzero; // bit s: slot s's winning t is -0 (read only when its key's t is 0)
	uint32_t pad_[(16 - (4 + 4 * kServeQueues + 4 + 4) % 16) % 16 / 4];
};
static_assert(sizeof(WarpFixed) % 16 == 0, "queue and pool must start 16-byte aligned");

__host__ __device__ inline uint32_t warp_smem_bytes(uint32_t pool_cap, uint32_t queue_cap) {
	return (uint32_t)sizeof(WarpFixed) + 4u * (queue_cap + pool_cap);
}

__device__ __forceinline__ uint32_t lanemask_lt() {
	uint32_t m;
	asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
	return m;
}

// One 32-byte read-only load (sm_100 and later; p 32-byte aligned): a whole child
// record, or a compressed node's header, in one instruction and one L1 sector.
__device__ __forceinline__ void ld_nc_256(const void *p, float4 &a, float4 &b) {
	asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
	    : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
	    : "l"(p));
}

// Three-input minimum and maximum (sm_100 and later; NaN operands ignored, as fminf and
// fmaxf ignore them).
__device__ __forceinline__ float max3f(float a, float b, float c) {
	float r;
	asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
	return r;
}
__device__ __forceinline__ float min3f(float a, float b, float c) {
	float r;
	asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
	return r;
}

// Packed FP32 pairs (sm_100 and later): one instruction for two lanes' worth of a
// component, each half rounded as the scalar operation rounds it.
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
	unsigned long long r;
	asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
	return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float &lo, float &hi) {
	asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
	unsigned long long r;
	asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
	return r;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
	unsigned long long r;
	asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
	return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b,
                                                   unsigned long long c) {
	unsigned long long r;
	asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
	return r;
}

// What the slab test on centres and half extents needs of a ray, x and y in pairs.
struct SlabRay {
	unsigned long long no, f, af, naf; // -origin, reciprocal, |reciprocal|, -|reciprocal|
	float oz, fz, afz;
};

__device__ __forceinline__ SlabRay slab_ray(const RayC &r) {
	SlabRay q;
	q.no = pack2(-r.ox, -r.oy);
	q.f = pack2(r.fx, r.fy);
	q.af = pack2(fabsf(r.fx), fabsf(r.fy));
	q.naf = pack2(-fabsf(r.fx), -fabsf(r.fy));
	q.oz = r.oz;
	q.fz = r.fz;
	q.afz = fabsf(r.fz);
	return q;
}

// Slab test of a regular ray (kind 0) on an inner box given as centre c and half extent e
// (encode_axis): per axis t = (c - o) * f, near = t - e |f|, far = t + e |f|.  Passes
// whenever the reference's slab test passes on some triangle box inside, so it prunes
// nothing the exact test would accept:
//  * with u = 2^-24, the computed near is at most its real value A plus 3.1 u |A| and far at
//    least B less 3.1 u |B|: the rounding of t is relative to |t| <= |A| + e |f|, and the
//    e |f| part is covered by the 8 u that encode_axis widens e by;
//  * the reference's own near and far of a box inside, (bound - o) * f, are off by at most
//    2.1 u of themselves;
//  * so for a triangle the reference passes (0 <= its tmax, its tmin <= its tmax), the
//    largest near (or 0) here is at most tmax (1 + 5.2 u) and the smallest far at least
//    tmax (1 - 5.2 u), up to underflow (a few 2^-149): the factor 1 + 16 u and the
//    2^-120 on the far side cover both, and the rounding of that product.
// 13 FP instructions and 3 on the half-rate ALU pipe for a box, against 12 and 9 for
// (bound - origin) * reciprocal on both bounds with its min / max per axis; x and y are
// packed, so 9 + 3 are issued.  (2,073,600 camera and 4,194,304 secondary rays on the
// 1,048,576-triangle heightfield: 1,514 -> 1,419 us under sustained load;
// 363 -> 323 M warp instructions for 1.5M of those rays, ALU-pipe 147 -> 118 M.)
__device__ __forceinline__ bool child_passes(const SlabRay &q, const float4 &a, const float4 &b) {
	const unsigned long long t = mul2(add2(pack2(a.x, a.y), q.no), q.f);
	const unsigned long long e = pack2(a.z, a.w);
	float nx, ny, fx, fy;
	unpack2(fma2(e, q.naf, t), nx, ny);
	unpack2(fma2(e, q.af, t), fx, fy);
	const float tz = (b.x - q.oz) * q.fz;
	const float nz = __fmaf_rn(-b.y, q.afz, tz), fz = __fmaf_rn(b.y, q.afz, tz);
	const float tmin = max3f(nx, ny, fmaxf(nz, 0.0f));
	const float tmax = min3f(fx, fy, fz);
	return tmin <= __fmaf_rn(tmax, 1.0f + 0x1p-20f, 0x1p-120f);
}

// The box test of any other ray (and of a regular one in a batch with such): on bounds, which
// a record's centre and half extent give rounded outwards, with the reference's own
// (bound - origin) * reciprocal.  That is monotone in the bound, infinities included, so it
// passes whatever the reference passes inside without a margin.
//
// An axis of infinite reciprocal (a zero component) takes +-1 in the reciprocal's place, so
// that its near and far tell by their signs, exactly, whether the origin lies before, inside
// or behind the box, and `g`, infinite there and 1 elsewhere, scales them to what the
// reference's slab test works with: two equal infinities outside, -inf and +inf inside, where
// a face's NaN removes y or z from its test.  The face's 0 * inf here is a NaN too, which
// max3f and min3f pass over (all axes may be: nothing constrains then).  On the x axis the
// reference's whole test passes at a lower face, so of kind 4 a box with the origin's x
// inside passes outright.
//
// Why: rays in a plane of two axes, a camera's middle row and column among them, are the
// longest chains of their launch.  Bounds stored as such and a branch per axis / decoded, with
// those branches / this, us: 2,400,000 rays in a z plane of the 1,048,576-triangle
// heightfield 679 / 721 / 578, 400,000 in an x plane that holds faces 12,734 / 13,513 / 12,121,
// 320 x 200 pixels on 65,536 triangles 118 / 117 / 108.  (The test on centre and half extent
// with the axes reduced the same way: 599 / 12,254 / 108, and 2 % slower for regular rays, by
// its registers; as a third instance of trace_batch 3 %.)
struct AxisRay {
	unsigned long long no, f, g; // x and y: -origin, reciprocal, scale
	float noz, fz, gz;
	bool inf_x, x_passes, all;
};

__device__ __forceinline__ AxisRay axis_ray(const RayC &r) {
	const bool ix = isinf(r.fx), iy = isinf(r.fy), iz = isinf(r.fz);
	AxisRay x;
	x.no = pack2(-r.ox, -r.oy);
	x.f = pack2(ix ? copysignf(1.0f, r.fx) : r.fx, iy ? copysignf(1.0f, r.fy) : r.fy);
	x.g = pack2(ix ? INFINITY : 1.0f, iy ? INFINITY : 1.0f);
	x.noz = -r.oz;
	x.fz = iz ? copysignf(1.0f, r.fz) : r.fz;
	x.gz = iz ? INFINITY : 1.0f;
	x.inf_x = ix;
	x.x_passes = r.kind == 4;
	x.all = r.kind == 2;
	return x;
}

// Bounds: lower x and y, upper x and y, lower and upper z; outside: known to be so on an x axis
// of infinite reciprocal.
__device__ __forceinline__ bool axis_passes(const AxisRay &x, unsigned long long l,
                                            unsigned long long h, unsigned long long z,
                                            bool outside) {
	float t1, t2, t3, t4, t5, t6, gx, gy;
	unpack2(mul2(add2(l, x.no), x.f), t1, t3);
	unpack2(mul2(add2(h, x.no), x.f), t2, t4);
	unpack2(mul2(add2(z, pack2(x.noz, x.noz)), pack2(x.fz, x.fz)), t5, t6);
	unpack2(x.g, gx, gy);
	float nx = fminf(t1, t2) * gx;
	const float fx = fmaxf(t1, t2) * gx;
	if (outside)
		nx = INFINITY; // (fx is +inf or a NaN if the bounds hold the origin)
	const bool outright = x.all || (x.x_passes && !(nx > 0.0f) && !(fx < 0.0f));
	const float tmin = max3f(nx, fminf(t3, t4) * gy, fmaxf(fminf(t5, t6) * x.gz, 0.0f));
	const float tmax = min3f(fx, fmaxf(t3, t4) * gy, fmaxf(t5, t6) * x.gz);
	return outright || !(tmin > tmax);
}

__device__ __forceinline__ bool child_passes(const AxisRay &x, const float4 &a, const float4 &b) {
	unsigned long long l, h;
	const unsigned long long c = pack2(a.x, a.y), e = pack2(a.z, a.w);
	asm("sub.rm.f32x2 %0, %1, %2;" : "=l"(l) : "l"(c), "l"(e)); // child_lo
	asm("add.rp.f32x2 %0, %1, %2;" : "=l"(h) : "l"(c), "l"(e)); // child_hi
	bool outside = false;
	if (x.inf_x) {
		float ox, oy;
		unpack2(x.no, ox, oy);
		// (Closer bounds: the widened extent of a box that ends near 0 reaches over it.)
		const uint32_t x16 = __float_as_uint(b.w);
		outside = -ox < __uint_as_float(x16 << 16) || -ox > __uint_as_float(x16 & 0xFFFF0000u);
	}
	return axis_passes(x, l, h, pack2(child_lo(b.x, b.y), child_hi(b.x, b.y)), outside);
}

__device__ __forceinline__ uint32_t byte_of(uint32_t w, int k) { return (w >> (8 * k)) & 0xFFu; }

// float(byte k of w), exactly: the byte placed in the mantissa of 2^23 (one byte
// permute), minus 2^23 -- full-rate instructions instead of an integer conversion.
__device__ __forceinline__ float byte_as_float(uint32_t w, int k) {
	return __fsub_rn(__uint_as_float(__byte_perm(w, 0x4B000000u, 0x7540u | (uint32_t)k)),
	                 8388608.0f);
}

// The byte alone in the mantissa of 2^23.
__device__ __forceinline__ float byte_biased(uint32_t w, int k) {
	return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7540u | (uint32_t)k));
}

// The bounds of child record ck of a compressed node with origin (oxy, oz) and scales (sxy,
// sz) as axis_passes takes them: the same decode (cdec_f), x and y and the two z in pairs.
__device__ __forceinline__ void compressed_bounds(const uint2 &ck, unsigned long long oxy, float oz,
                                                  unsigned long long sxy, float sz,
                                                  unsigned long long &l, unsigned long long &h,
                                                  unsigned long long &z) {
	const unsigned long long bias = pack2(-8388608.0f, -8388608.0f);
	l = fma2(add2(pack2(byte_biased(ck.x, 0), byte_biased(ck.x, 2)), bias), sxy, oxy);
	h = fma2(add2(pack2(byte_biased(ck.x, 1), byte_biased(ck.x, 3)), bias), sxy, oxy);
	z = fma2(add2(pack2(byte_biased(ck.y, 0), byte_biased(ck.y, 1)), bias), pack2(sz, sz),
	         pack2(oz, oz));
}

// regular_box on a child of a compressed node: the same decode and products, every operation
// rounded as the scalar one, in packed pairs: 12 FP instructions for 24 (a traversal of
// compressed nodes is bound by issue).  tmax >= 0 and tmin <= tmax as max(tmin, 0) <= tmax.
// 1,000,003 random rays on as many clustered triangles 934 -> 866 us, 2,097,152 rays on the
// 1,048,576-triangle heightfield 1,110 -> 1,053 (z scalar: 883, 1,077).
__device__ __forceinline__ bool compressed_passes(const SlabRay &q, const uint2 &ck,
                                                  unsigned long long oxy, float oz,
                                                  unsigned long long sxy, float sz) {
	unsigned long long l, h, z;
	compressed_bounds(ck, oxy, oz, sxy, sz, l, h, z);
	float t1, t2, t3, t4, t5, t6;
	unpack2(mul2(add2(l, q.no), q.f), t1, t3);
	unpack2(mul2(add2(h, q.no), q.f), t2, t4);
	unpack2(mul2(add2(z, pack2(-q.oz, -q.oz)), pack2(q.fz, q.fz)), t5, t6);
	const float tmin = max3f(fminf(t1, t2), fminf(t3, t4), fmaxf(fminf(t5, t6), 0.0f));
	const float tmax = min3f(fmaxf(t1, t2), fmaxf(t3, t4), fmaxf(t5, t6));
	return tmin <= tmax;
}

// The same of any other ray.
__device__ __forceinline__ bool compressed_passes(const AxisRay &x, const uint2 &ck,
                                                  unsigned long long oxy, float oz,
                                                  unsigned long long sxy, float sz) {
	unsigned long long l, h, z;
	compressed_bounds(ck, oxy, oz, sxy, sz, l, h, z);
	return axis_passes(x, l, h, z, false);
}

__device__ __forceinline__ RayC slot_ray(const WarpFixed &S, uint32_t s) {
	RayC r;
	// Two 16-byte shared loads for the slab test (the direction is dead there).
	const float4 o = S.ro[s], f = S.rf[s], d = S.rd[s];
	r.ox = o.x;
	r.oy = o.y;
	r.oz = o.z;
	r.dx = d.x;
	r.dy = d.y;
	r.dz = d.z;
	r.fx = f.x;
	r.fy = f.y;
	r.fz = f.z;
	r.kind = __float_as_int(o.w);
	return r;
}

// Tests queue entries [lo, lo + n) (n <= 32), one per lane.  KEEP: the lane whose hit a
// slot keeps also records its u, v (and the sign of a zero t) for the records.
template <bool COUNT, bool KEEP>
__device__ __forceinline__ void test_queued(const float4 *__restrict__ tri4, WarpFixed &S,
                                            const uint32_t *queue, uint32_t lo, uint32_t n,
                                            int lane, uint32_t &n_tests) {
	unsigned long long mykey = kNoHit;
	uint32_t my_slot = 0;
	float mt = 0.0f, mu = 0.0f, mv = 0.0f;
	if ((uint32_t)lane < n) {
		const uint32_t e = queue[lo + lane];
		const uint32_t slot = e >> kIndexBits;
		const RayC r = slot_ray(S, slot);
		const float4 *p = tri4 + 3 * (size_t)(e & kIndexMask);
		const float4 A = __ldg(p), B = __ldg(p + 1), C = __ldg(p + 2);
		float t, u, v;
		// Finite ray and triangle (nearly always): the box test with plain min/max.
		if (tri_test(r, A, B, C, t, u, v, r.kind <= 1 && tri_record_finite(B)) && t < INFINITY) {
			mykey = hit_key(t, __float_as_uint(A.w));
			atomicMin(&S.key[slot], mykey);
			my_slot = slot;
			mt = t;
			mu = u;
			mv = v;
		}
		if (COUNT)
			++n_tests;
	}
	// The lane whose key the slot kept (keys are unique: they hold the primitive id)
	// records its u and v, so the records need no second test of the winner.
	if (!KEEP)
		return;
	__syncwarp();
	if (mykey != kNoHit && S.key[my_slot] == mykey) {
		S.rf[my_slot].w = mu;
		S.rd[my_slot].w = mv;
		if (mt == 0.0f) { // the key holds +0 for both zeros
			if (signbit(mt))
				atomicOr(&S.negzero, 1u << my_slot);
			else
				atomicAnd(&S.negzero, ~(1u << my_slot));
		}
	}
}

// What the test of inner boxes takes: of a batch whose rays are all of kind 0, of any other.
template <bool REGULAR>
using NodeRay = std::conditional_t<REGULAR, SlabRay, AxisRay>;
template <bool REGULAR> __device__ __forceinline__ NodeRay<REGULAR> node_ray(const RayC &r) {
	if constexpr (REGULAR)
		return slab_ray(r);
	else
		return axis_ray(r);
}

// Child `k` of `node`: slab test and what it refers to.
template <int FMT, bool REGULAR>
__device__ __forceinline__ void test_child(const void *__restrict__ nodes,
                                           const NodeRay<REGULAR> &q, uint32_t node, int k,
                                           bool &hit, bool &inner, uint32_t &child,
                                           uint32_t &leaf_n) {
	hit = false;
	inner = false;
	child = 0;
	leaf_n = 0;
	if (FMT == PRT_NODES_FP32) {
		float4 a, b;
		ld_nc_256(&(static_cast<const Node8 *>(nodes) + node)->c[k], a, b);
		const uint32_t ref = __float_as_uint(b.z);
		// An unused slot has a NaN box, which a regular ray's test never passes; the
		// other test would, so only the general pass checks the reference.
		if (REGULAR || ref != kNone) {
			inner = !ref_is_leaf(ref);
			hit = child_passes(q, a, b);
			// A node index, or a leaf's first triangle: both below 2^27, under the
			// leaf flag and count bits.
			child = ref & kIndexMask;
			leaf_n = inner ? 0u : leaf_count(ref);
		}
	} else {
		const CNode8 *cn = static_cast<const CNode8 *>(nodes) + node;
		float4 h0, h1;
		ld_nc_256(cn, h0, h1); // the 32-byte header (96-byte nodes keep it 32-byte aligned)
		const uint4 w0 = make_uint4(__float_as_uint(h0.x), __float_as_uint(h0.y),
		                            __float_as_uint(h0.z), __float_as_uint(h0.w));
		const uint2 w1 = make_uint2(__float_as_uint(h1.x), __float_as_uint(h1.y));
		const uint2 ck = __ldg(reinterpret_cast<const uint2 *>(&cn->c[k]));
		const uint32_t imask = byte_of(w0.w, 3);
		const uint32_t m = byte_of(ck.y, 2);
		inner = (imask >> k) & 1u;
		if (inner || m) {
			const float sx = cscale((uint8_t)byte_of(w0.w, 0));
			const float sy = cscale((uint8_t)byte_of(w0.w, 1));
			const float sz = cscale((uint8_t)byte_of(w0.w, 2));
			const float ox = __uint_as_float(w0.x), oy = __uint_as_float(w0.y),
			            oz = __uint_as_float(w0.z);
			hit = compressed_passes(q, ck, pack2(ox, oy), oz, pack2(sx, sy), sz);
			if (inner) {
				child = w1.x + __popc(imask & ((1u << k) - 1u));
			} else {
				child = w1.y + byte_of(ck.y, 3);
				leaf_n = m;
			}
		}
	}
}

// What child `k` of `node` refers to, as a Node8 reference (kNone: an unused slot).
template <int FMT>
__device__ __forceinline__ uint32_t child_ref(const void *__restrict__ nodes, uint32_t node,
                                              int k) {
	if (FMT == PRT_NODES_FP32)
		return __ldg(&(static_cast<const Node8 *>(nodes) + node)->c[k].ref);
	const CNode8 *cn = static_cast<const CNode8 *>(nodes) + node;
	const uint4 w0 = __ldg(reinterpret_cast<const uint4 *>(cn));
	const uint2 w1 = __ldg(reinterpret_cast<const uint2 *>(cn) + 2);
	const uint32_t ck = __ldg(reinterpret_cast<const uint2 *>(&cn->c[k])).y;
	const uint32_t imask = byte_of(w0.w, 3), m = byte_of(ck, 2);
	if ((imask >> k) & 1u)
		return w1.x + __popc(imask & ((1u << k) - 1u));
	return m ? make_leaf(w1.y + byte_of(ck, 3), m) : kNone;
}

// Resident blocks per SM the register budget is set for, per node format (measured on
// the 1M-triangle heightfield: 9 blocks of 4 warps = 56 registers, with a few spilled
// words, is fastest for both formats).
#ifndef PRT_TRAVERSE_MIN_BLOCKS_FP32
#define PRT_TRAVERSE_MIN_BLOCKS_FP32 9
#endif
#ifndef PRT_TRAVERSE_MIN_BLOCKS_COMPRESSED
#define PRT_TRAVERSE_MIN_BLOCKS_COMPRESSED 9
#endif

// The packet descent of a batch: from the root, every node that at least kPacketMin of the
// warp's rays visit is tested for all of them at once, lane = slot, all lanes on the same
// child (its record is one broadcast load).  Inner children that fewer rays pass go to
// those rays' lists (`list`, local memory, `listed` entries), which the item steps then
// take up; leaf triangles are queued.  The same tests on the same rays as item steps
// make, so the same records.
//
// Why: a node that m rays of the warp visit costs m / 8 item steps of about 110 warp
// instructions and 2 L1 wavefronts per ray; here it costs the same few hundred instructions
// and 8 wavefronts for any m.  A camera's 32 neighbouring pixels share most of their nodes:
// 2048 x 2048 pixels on a closed mesh of 4,968 triangles, traversal and shading 404 ->
// 308 us (kPacketMin 8 / 12 / 16 / 20: 308 / 312 / 316 / 320).  Ray buffers keep the item
// steps: on the heightfield's camera and secondary rays the descent at 16 / 20 measured
// 1,644 / 1,618 us against 1,561 without, and incoherent rays share only the top levels.
// (Tiles of 8 x 4 pixels instead of 32 of a row: 4 % fewer instructions, but 365 us: the
// four rays of a tile with a zero x direction, which pass every box around x = 0, end up
// in one warp, and the last of those tiles is the launch's tail.)
//
// Bounds: a node with fewer than 8 free stack entries, or met when some list is past
// kListStop, is not opened but goes to its rays' lists; a list grows by at most 8 per
// opened node and one per unopened entry, so it stays under kListWords.
template <int FMT, bool LEAF1>
__device__ __forceinline__ void packet_descent(const TravArgs &a, const SceneDesc &sd,
                                               WarpFixed &S, uint32_t *queue, uint32_t nb,
                                               int lane, uint32_t lt, uint32_t step_limit,
                                               uint32_t *list, uint32_t &listed, uint32_t &q,
                                               bool &fault) {
	const float4 *__restrict__ tri4 = sd.tri4;
	const void *__restrict__ nodes = sd.nodes;
	// The stack: lane k holds entry k (a node and the slots that visit it).
	uint32_t st_node = sd.root, st_rays = 0xFFFFFFFFu >> (32u - nb), sp = 1, steps = 0;
	while (sp > 0u) {
		--sp;
		const uint32_t node = __shfl_sync(0xFFFFFFFFu, st_node, (int)sp);
		const uint32_t rays = __shfl_sync(0xFFFFFFFFu, st_rays, (int)sp);
		const bool mine = (rays >> lane) & 1u;
		if (++steps > step_limit) { // a malformed tree
			if (lane == 0)
				set_error_bits(a.err, kErrStack);
			fault = true;
			break;
		}
		if (__popc(rays) < (int)kPacketMin || sp + 8u > kPacketStack ||
		    __any_sync(0xFFFFFFFFu, listed > kListStop)) {
			if (mine)
				list[listed++] = node;
			continue;
		}
		const RayC r = slot_ray(S, (uint32_t)lane);
		const SlabRay sr = slab_ray(r);
		// Lane c: what child c refers to, and the rays that pass it.
		const uint32_t c_ref = child_ref<FMT>(nodes, node, lane & 7);
		uint32_t c_rays = 0;
#pragma unroll 4
		for (int c = 0; c < 8; ++c) {
			bool hit, inner;
			uint32_t child, leaf_n;
			test_child<FMT, true>(nodes, sr, node, c, hit, inner, child, leaf_n);
			const uint32_t b = __ballot_sync(0xFFFFFFFFu, hit && mine);
			if (lane == c)
				c_rays = b;
		}
		uint32_t todo = __ballot_sync(0xFFFFFFFFu, c_rays != 0u);
		while (todo) {
			const int c = __ffs(todo) - 1;
			todo &= todo - 1u;
			const uint32_t b = __shfl_sync(0xFFFFFFFFu, c_rays, c);
			const uint32_t ref = __shfl_sync(0xFFFFFFFFu, c_ref, c);
			const uint32_t n = __popc(b);
			const bool in = (b >> lane) & 1u;
			if (ref_is_leaf(ref)) {
				const uint32_t m = LEAF1 ? 1u : leaf_count(ref);
				for (uint32_t k = 0; k < m; ++k) {
					if (in)
						queue[q + __popc(b & lt)] =
						    ((uint32_t)lane << kIndexBits) | ((ref & kIndexMask) + k);
					q += n;
					__syncwarp();
					if (q >= 32u) {
						q -= 32u;
						uint32_t none = 0;
						test_queued<false, FMT == PRT_NODES_FP32>(tri4, S, queue, q, 32u, lane,
						                                          none);
						__syncwarp();
					}
				}
			} else if (n >= kPacketMin) {
				if (lane == (int)sp) {
					st_node = ref;
					st_rays = b;
				}
				++sp;
			} else if (in) {
				list[listed++] = ref;
			}
		}
	}
}

// (One-kernel launches hold both box tests: 64 registers, which 8 blocks allow, spill nothing.)
#ifndef PRT_TRAVERSE_MIN_BLOCKS_SMALL
#define PRT_TRAVERSE_MIN_BLOCKS_SMALL 8
#endif

// The traversal of one batch of up to 32 rays (slots 0..nb-1 of S) through scene sd.
// REGULAR: every ray of the batch is regular (kind 0), so inner boxes take the plain slab
// test only.  PACKET: it starts with a packet descent.
template <int FMT, bool COUNT, bool LEAF1, bool REGULAR, bool PACKET = false>
__device__ __forceinline__ void trace_batch(const TravArgs &a, WarpFixed &S, uint32_t *queue,
                                            uint32_t *pool, const SceneDesc &sd, uint32_t nb,
                                            int lane, int g, int s, uint32_t lt,
                                            uint32_t step_limit, uint32_t &n_visits,
                                            uint32_t &n_tests, bool &fault) {
	const float4 *__restrict__ tri4 = sd.tri4;
	const void *__restrict__ nodes = sd.nodes;
	uint32_t top = 0;  // items in the pool (warp-uniform)
	uint32_t q = 0;    // queued triangles (warp-uniform)
	uint32_t next = 0; // next slot whose root is not yet in the pool; after a packet
	                   // descent, the nodes left in this lane's list
	uint32_t steps = 0;
	uint32_t list[PACKET ? kListWords : 1u];
	bool listed = PACKET; // some list may hold a node
	if (PACKET)
		packet_descent<FMT, LEAF1>(a, sd, S, queue, nb, lane, lt, step_limit, list, next, q,
		                           fault);
	for (;;) {
		// Admit new work while fewer than K items are pending (a branch the common step
		// skips with one test).
		if (top < (uint32_t)kItems) {
			if (PACKET) {
				if (listed) {
					const uint32_t left = __ballot_sync(0xFFFFFFFFu, next > 0u);
					const uint32_t add = kAdmit - top, at = __popc(left & lt);
					if (next > 0u && at < add)
						pool[top + at] = ((uint32_t)lane << kIndexBits) | list[--next];
					top += min(add, (uint32_t)__popc(left));
					listed = left != 0u;
					__syncwarp();
				}
			} else if (next < nb) {
				const uint32_t add = min((uint32_t)kItems - top, nb - next);
				if ((uint32_t)lane < add)
					pool[top + lane] = ((next + lane) << kIndexBits) | sd.root;
				top += add;
				next += add;
				__syncwarp();
			}
			if (top == 0u)
				break;
			// Fewer than K items left: the empty node (slot 0's ray) fills the step, so
			// every step takes K items and no group needs a "has an item" test.  A
			// counting run keeps the test (it counts visits of real items only).
			if (!COUNT && top < (uint32_t)kItems) {
				if ((uint32_t)lane >= top && lane < kItems)
					pool[lane] = a.dead;
				top = kItems;
				__syncwarp();
			}
		}
		const uint32_t take = COUNT ? min(top, (uint32_t)kItems) : (uint32_t)kItems;
		top -= take;
		// (Counting runs: groups without an item repeat the first one and drop what they
		// find.)
		const bool work = !COUNT || (uint32_t)g < take;
		const uint32_t item = pool[top + (COUNT ? (work ? g : 0) : g)];
		__syncwarp(); // the pops above are read before the pushes below overwrite them
		const uint32_t slot = item >> kIndexBits, node = item & kIndexMask;
		const RayC r = slot_ray(S, slot);
		const NodeRay<REGULAR> sr = node_ray<REGULAR>(r);
		if (COUNT && work && s == 0)
			++n_visits;

		bool hit[kChildPerLane], inner[kChildPerLane];
		uint32_t child[kChildPerLane], leaf_n[kChildPerLane];
#pragma unroll
		for (int j = 0; j < kChildPerLane; ++j) {
			test_child<FMT, REGULAR>(nodes, sr, node, s + kLanesPerNode * j, hit[j], inner[j],
			                         child[j], leaf_n[j]);
			hit[j] = hit[j] && work;
		}
		// Every hit leaf of the step holds one triangle: always with single-triangle leaves
		// (predicates only on that path: the half-rate ALU pipe bounds the step).
		bool one_each = true;
		if (!LEAF1) {
			bool single = true;
#pragma unroll
			for (int j = 0; j < kChildPerLane; ++j)
				single = single && (!hit[j] || inner[j] || leaf_n[j] <= 1u);
			one_each = __all_sync(0xFFFFFFFFu, single);
		}

		// Positions, child-major: every lane's child j before any lane's child j + 1, so
		// no position waits on the lane's previous child.  Pushed inner children go to
		// the pool; with at most one triangle per hit leaf the queue positions come from
		// the same ballots.
		constexpr bool kOneArray = LEAF1 && FMT == PRT_NODES_FP32;
		uint32_t pp[kChildPerLane], pq[kChildPerLane];
		uint32_t ptop = top, qtop = q;
#pragma unroll
		for (int j = 0; j < kChildPerLane; ++j) {
			if (kOneArray) {
				// One place per hit child, in the pool or in the queue, which are one array:
				// one population count and one store instead of two of each (heightfield
				// 1,562 -> 1,521 us, 512-scene batch graph 10.42 -> 10.17 ms).
				const uint32_t bp = __ballot_sync(0xFFFFFFFFu, hit[j] && inner[j]);
				const uint32_t bl = __ballot_sync(0xFFFFFFFFu, hit[j] && !inner[j]);
				pp[j] = (inner[j] ? a.queue_cap + ptop : qtop) + __popc((inner[j] ? bp : bl) & lt);
				ptop += __popc(bp);
				qtop += __popc(bl);
				continue;
			}
			const uint32_t bp = __ballot_sync(0xFFFFFFFFu, hit[j] && inner[j]);
			pp[j] = ptop + __popc(bp & lt);
			ptop += __popc(bp);
			if (one_each) {
				const uint32_t bl = __ballot_sync(0xFFFFFFFFu, hit[j] && !inner[j]);
				pq[j] = qtop + __popc(bl & lt);
				qtop += __popc(bl);
			}
		}
		// The pool holds every push of a well-formed tree and a well-formed tree ends
		// within step_limit steps; anything else is reported and ends the batch.
		++steps;
		if (ptop > a.pool_cap || steps > step_limit) {
			if (lane == 0)
				set_error_bits(a.err, kErrStack);
			fault = true;
			break;
		}
		const uint32_t hi = slot << kIndexBits;
		if (kOneArray) {
#pragma unroll
			for (int j = 0; j < kChildPerLane; ++j)
				if (hit[j])
					queue[pp[j]] = hi | child[j];
		} else if (one_each) {
#pragma unroll
			for (int j = 0; j < kChildPerLane; ++j) {
				if (hit[j] && inner[j])
					pool[pp[j]] = hi | child[j];
				if (hit[j] && !inner[j])
					queue[pq[j]] = hi | child[j];
			}
		} else {
#pragma unroll
			for (int j = 0; j < kChildPerLane; ++j)
				if (hit[j] && inner[j])
					pool[pp[j]] = hi | child[j];
			// Leaves of several triangles: positions from a scan of the per-lane counts.
			uint32_t cnt[kChildPerLane], all_cnt = 0;
#pragma unroll
			for (int j = 0; j < kChildPerLane; ++j) {
				cnt[j] = (hit[j] && !inner[j]) ? leaf_n[j] : 0u;
				all_cnt += cnt[j];
			}
			uint32_t incl = all_cnt;
#pragma unroll
			for (int o = 1; o < 32; o <<= 1) {
				const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
				if (lane >= o)
					incl += y;
			}
			uint32_t pos = q + incl - all_cnt;
#pragma unroll
			for (int j = 0; j < kChildPerLane; ++j)
				for (uint32_t k = 0; k < cnt[j]; ++k)
					queue[pos++] = hi | (child[j] + k);
			qtop = q + __shfl_sync(0xFFFFFFFFu, incl, 31);
		}
		top = ptop;
		q = qtop;
		__syncwarp();
		while (q >= 32u) {
			q -= 32u;
			test_queued<COUNT, FMT == PRT_NODES_FP32>(tri4, S, queue, q, 32u, lane, n_tests);
			__syncwarp();
		}
	}
	while (q > 0u) {
		const uint32_t n = min(q, 32u);
		q -= n;
		test_queued<COUNT, FMT == PRT_NODES_FP32>(tri4, S, queue, q, n, lane, n_tests);
		__syncwarp();
	}
}

// A copy of a run descriptor that bypasses L1 (a serving launch reads descriptors that the
// host's copies write while it runs).
__device__ __forceinline__ SegDesc load_seg_cg(const SegDesc *p) {
	static_assert(sizeof(SegDesc) % 8 == 0, "descriptor copied as 8-byte words");
	SegDesc d;
	const unsigned long long *src = reinterpret_cast<const unsigned long long *>(p);
	unsigned long long *dst = reinterpret_cast<unsigned long long *>(&d);
#pragma unroll
	for (int k = 0; k < (int)(sizeof(SegDesc) / 8); ++k)
		dst[k] = __ldcg(src + k);
	return d;
}

// Serving launches (PASS 3): lane 0 takes the next batch, queues in priority order.  Batches
// are tickets drawn with atomicAdd on the queue's `next` (a compare-and-swap retried by
// thousands of warps on one word serialises them); a warp draws only when it saw a
// published batch, and a ticket that lands past the published end (another warp took
// the last one meanwhile) is kept in `held` until the host publishes that batch, while
// the warp serves the other queues.  The host stops a launch only when every published
// batch is finished, so tickets still held then are past all work.  Returns false when
// the warp should leave: stop set, or idle for idle_limit polls (an idle warp sleeps 0.25
// to 4 us between polls).  A warp that still holds a ticket after 16 x idle_limit polls
// without stop sets the error flag and leaves: every wait is bounded.
__device__ __forceinline__ bool claim_batch(const ServeQueues &q, uint32_t held[kServeQueues],
                                            uint32_t &qsel, uint32_t &batch) {
	uint32_t sleep_ns = 250;
	for (uint32_t idle = 0;; ++idle) {
		bool holding = false;
#pragma unroll
		for (uint32_t k = 0; k < (uint32_t)kServeQueues; ++k) {
			ServeQueueState *st = q.state[k];
			const uint32_t pub = *reinterpret_cast<volatile const uint32_t *>(&st->published);
			if (held[k] != kNone) {
				if (held[k] < pub) {
					qsel = k;
					batch = held[k];
					held[k] = kNone;
					return true;
				}
				holding = true;
				continue;
			}
			if (*reinterpret_cast<volatile const uint32_t *>(&st->next) < pub) {
				const uint32_t t = atomicAdd(&st->next, 1u);
				if (t < pub) {
					qsel = k;
					batch = t;
					return true;
				}
				held[k] = t; // past the end: served once published
				holding = true;
			}
		}
		if (*reinterpret_cast<volatile const uint32_t *>(q.stop))
			return false;
		if (idle >= (holding ? 16u * q.idle_limit : q.idle_limit)) {
			if (holding)
				*reinterpret_cast<volatile uint32_t *>(q.err_flag) = 1u;
			return false;
		}
		__nanosleep(sleep_ns);
		sleep_ns = min(sleep_ns * 2u, 4000u);
	}
}

// LEAF1: every leaf holds one triangle (leaf size 1), so a hit leaf queues exactly one.
// BOUNDED: a warp takes at most a.max_batches batches (a separate instantiation, so the
// unbounded kernels keep their register allocation).
// PASS: 0 = every batch with the general box test (the counting runs); 1 = batches whose
// rays are all regular, with the plain slab test only (no conservative code
// in the kernel at all: 8 % faster), the others counted in a.deferred and skipped; 2 =
// the skipped batches with the general test (returns at once when there are none); 3 =
// a serving launch: batches claimed from the serving queues (claim_batch), the plain or
// the general test chosen per batch, descriptors and rays read around L1; 4 = one kernel for
// a run of up to some hundred rays per warp, several runs of up to 16, and most cameras
// (single_batch): every
// batch, the test chosen per batch, a warp's first batch by its number and the next ones,
// if any, from the counter.
template <int FMT, bool COUNT, bool LEAF1, bool BOUNDED, int PASS>
__global__ void __launch_bounds__(32 * kWarpsPerBlock, PASS == 4 ? PRT_TRAVERSE_MIN_BLOCKS_SMALL
                                                       : FMT == PRT_NODES_FP32
                                                           ? PRT_TRAVERSE_MIN_BLOCKS_FP32
                                                           : PRT_TRAVERSE_MIN_BLOCKS_COMPRESSED)
    k_trace8(TravArgs a) {
	extern __shared__ __align__(16) unsigned char smem_raw[];
	unsigned char *wbase = smem_raw + (size_t)(threadIdx.x >> 5) * a.warp_bytes;
	WarpFixed &S = *reinterpret_cast<WarpFixed *>(wbase);
	uint32_t *queue = reinterpret_cast<uint32_t *>(wbase + sizeof(WarpFixed));
	uint32_t *pool = queue + a.queue_cap; // also the staging area of the output records
	const int lane = threadIdx.x & 31, g = lane / kLanesPerNode, s = lane % kLanesPerNode;
	const uint32_t lt = lanemask_lt();
	uint32_t n_visits = 0, n_tests = 0;
	// A tree is visited at most once per ray; more steps than this means a malformed
	// tree, which is reported instead of looping.
	const uint32_t step_limit = (uint32_t)min(32ull * a.n_nodes + 64ull, 0xFFFFFFFFull);
	if (PASS == 2 && *(volatile const uint32_t *)a.deferred == 0u)
		return; // the regular pass took every batch (it ran before, on the same stream)

	uint32_t dealt = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * a.batch; // PASS 4
	if (BOUNDED && lane == 0)
		S.batches = 0;
	if (PASS == 3 && lane == 0) {
		for (int k = 0; k < kServeQueues; ++k)
			S.held[k] = kNone;
		S.cached_q = kNone;
	}
	__syncwarp();
	for (;;) {
		if (BOUNDED) {
			if (S.batches == a.max_batches)
				break;
			__syncwarp();
			if (lane == 0)
				++S.batches;
		}
		// Batches are taken in order from a counter (the deferred pass has its own, so
		// the few batches it works on spread over all warps); a one-kernel launch (4)
		// deals out the first ones by warp; a serving launch claims them from its queues.
		uint32_t base = 0, take = PASS == 3 ? 32u : a.batch;
		const SegDesc *segs = a.segs;
		if (PASS == 3) {
			uint32_t qsel = 0, batch = 0;
			const bool got = lane == 0 ? claim_batch(a.serve, S.held, qsel, batch) : false;
			if (!__shfl_sync(0xFFFFFFFFu, got, 0))
				break;
			qsel = __shfl_sync(0xFFFFFFFFu, qsel, 0);
			base = 32u * __shfl_sync(0xFFFFFFFFu, batch, 0);
			segs = a.serve.segs[qsel];
			// The run of this batch: the warp's last one when it still covers it (a large
			// request's batches mostly go to the same warps in turn), else a binary search
			// of the table (around L1: the host writes it while the launch runs).
			if (lane == 0 && !(S.cached_q == qsel && base >= (uint32_t)S.seg.vbegin &&
			                   base - (uint32_t)S.seg.vbegin < S.seg.n_rays)) {
				// Published after the table: covers every claimed batch.
				const uint32_t n_segs = *reinterpret_cast<volatile const uint32_t *>(
				    &a.serve.state[qsel]->n_segs);
				uint32_t lo_s = 0, hi_s = n_segs;
				while (hi_s - lo_s > 1) {
					const uint32_t mid = (lo_s + hi_s) >> 1;
					if (__ldcg(&segs[mid].vbegin) <= base)
						lo_s = mid;
					else
						hi_s = mid;
				}
				S.seg = load_seg_cg(segs + lo_s);
				S.cached_q = qsel;
			}
		} else {
			if (PASS == 4) {
				base = dealt; // the warp's first batch
				dealt = kNone;
				if (base == kNone) { // the next one that no warp has
					if (!a.claims)
						break;
					take = a.claims;
					if (lane == 0)
						base = atomicAdd(a.counter, a.claims) +
						       gridDim.x * (blockDim.x >> 5) * a.batch;
					base = __shfl_sync(0xFFFFFFFFu, base, 0);
				}
			} else {
				if (lane == 0)
					base = atomicAdd(PASS == 2 ? a.deferred + 1 : a.counter, a.batch);
				base = __shfl_sync(0xFFFFFFFFu, base, 0);
			}
			if (base >= a.n_virtual)
				break;
			// The run these rays belong to (runs are padded to whole warps of 32, and
			// a batch of fewer rays never straddles one).
			uint32_t si = 0;
			if (a.n_segs) {
				if (lane == 0) {
					uint32_t lo_s = 0, hi_s = a.n_segs;
					while (hi_s - lo_s > 1) {
						const uint32_t mid = (lo_s + hi_s) >> 1;
						if (a.segs[mid].vbegin <= base)
							lo_s = mid;
						else
							hi_s = mid;
					}
					si = lo_s;
				}
				si = __shfl_sync(0xFFFFFFFFu, si, 0);
			}
			if (lane == 0)
				S.seg = a.n_segs ? a.segs[si] : a.seg0;
		}
		__syncwarp();
		const uint32_t local = base - (uint32_t)S.seg.vbegin;
		const uint32_t run_rays = S.seg.n_rays;
		if (local >= run_rays)
			continue; // padding of the run
		const uint32_t nb = min(take, run_rays - local);
		const SceneDesc sd = (PASS == 3 || a.n_segs) ? a.scenes[S.seg.scene] : a.scene0;
		const float4 *__restrict__ tri4 = sd.tri4;
		float4 far = make_float4(0.0f, 0.0f, 0.0f, INFINITY);
		if (FMT == PRT_NODES_FP32)
			far = __ldg(reinterpret_cast<const float4 *>(static_cast<const Node8 *>(sd.nodes) + a.dead +
			                                             1u) + sd.root);

		if ((uint32_t)lane < nb) {
			RayC r;
			if (a.use_cam) {
				float o[3], d[3];
				camera_ray(a.cam, local + lane, o, d);
				r = make_ray(o[0], o[1], o[2], d[0], d[1], d[2]);
			} else {
				const float2 *rp =
				    reinterpret_cast<const float2 *>(S.seg.rays + 6 * (size_t)(local + lane));
				float2 p0, p1, p2;
				if (PASS == 3) {
					p0 = __ldcg(rp);
					p1 = __ldcg(rp + 1);
					p2 = __ldcg(rp + 2);
				} else {
					p0 = __ldcs(rp);
					p1 = __ldcs(rp + 1);
					p2 = __ldcs(rp + 2);
				}
				r = make_ray(p0.x, p0.y, p1.x, p1.y, p2.x, p2.y);
			}
			if (FMT == PRT_NODES_FP32 && r.kind == 0 &&
			    max3f(fabsf(r.ox - far.x), fabsf(r.oy - far.y), fabsf(r.oz - far.z)) > far.w)
				r.kind = 1;
			if ((PASS == 0 || PASS == 2 || PASS == 4) && r.kind == 4 && a.x_faces &&
			    x_face_free(a.x_faces, r.ox))
				--r.kind;
			S.ro[lane] = make_float4(r.ox, r.oy, r.oz, __int_as_float(r.kind));
			S.rf[lane] = make_float4(r.fx, r.fy, r.fz, 0.0f);
			S.rd[lane] = make_float4(r.dx, r.dy, r.dz, 0.0f);
		}
		S.key[lane] = kNoHit;
		__syncwarp();

		bool fault = false; // the batch's traversal reported an error (warp-uniform)
		if (sd.n_tris) {
			// Nearly every batch has only regular rays.
			const bool regular =
			    __all_sync(0xFFFFFFFFu, (uint32_t)lane >= nb || __float_as_int(S.ro[lane].w) == 0);
			if (PASS == 1 && !regular) {
				if (lane == 0)
					atomicAdd(a.deferred, 1u);
				continue; // left to the deferred pass
			}
			if (PASS == 2 && regular)
				continue; // done by the regular pass
			constexpr bool kPacket = PASS == 0 && !COUNT;
			if ((PASS == 3 || PASS == 4 || kPacket) && regular)
				trace_batch<FMT, COUNT, LEAF1, true, kPacket>(a, S, queue, pool, sd, nb, lane, g, s, lt,
				                                     step_limit, n_visits, n_tests, fault);
			else
				trace_batch<FMT, COUNT, LEAF1, PASS == 1>(a, S, queue, pool, sd, nb, lane, g, s,
				                                          lt, step_limit, n_visits, n_tests, fault);
		} else if (PASS == 2) {
			continue; // the regular pass wrote this empty scene's misses
		}
		__syncwarp();

		// Finalise: stage each slot's record (its winner's t, u, v as its test found them)
		// in the run's HitReg<Tags...> layout.
		uint32_t *stage = pool;
		const uint32_t rec = S.seg.rec_size, fmask = S.seg.mask;
		const uint32_t rw = rec >> 2;
		// 32 records of rw words: rw * 8 16-byte words (record sizes are multiples of 4).
		for (uint32_t k = lane; k < rw * 8u; k += 32u)
			reinterpret_cast<uint4 *>(stage)[k] = make_uint4(0u, 0u, 0u, 0u);
		__syncwarp();
		if ((uint32_t)lane < nb) {
			const RayC r = slot_ray(S, lane);
			Best best;
			best_init(best);
			const unsigned long long key = S.key[lane];
			if (key != kNoHit && FMT == PRT_NODES_FP32) {
				const float tk = ord2f((uint32_t)(key >> 32));
				best.t = tk != 0.0f ? tk : (((S.negzero >> lane) & 1u) ? -0.0f : 0.0f);
				best.u = S.rf[lane].w;
				best.v = S.rd[lane].w;
				best.pid = (uint32_t)key;
			} else if (key != kNoHit) {
				// Compressed nodes (measured 1 % faster this way): the winner's test again.
				const uint32_t pid = (uint32_t)key;
				const float4 *p = tri4 + 3 * (size_t)__ldg(&sd.inv[pid]);
				const float4 A = __ldg(p), B = __ldg(p + 1), C = __ldg(p + 2);
				float t, u, v;
				if (tri_test(r, A, B, C, t, u, v, r.kind <= 1 && tri_record_finite(B))) {
					best.t = t;
					best.u = u;
					best.v = v;
					best.pid = pid;
				}
			}
			const uint8_t *off = S.seg.off;
			uint8_t *rb = reinterpret_cast<uint8_t *>(stage) + lane * rec;
			if (fmask & PRT_FIELD_UV) {
				*reinterpret_cast<float *>(rb + off[PRT_OFF_U]) = best.u;
				*reinterpret_cast<float *>(rb + off[PRT_OFF_V]) = best.v;
			}
			if (fmask & PRT_FIELD_T)
				*reinterpret_cast<float *>(rb + off[PRT_OFF_T]) = best.t;
			if (fmask & PRT_FIELD_PRIMITIVE_ID)
				*reinterpret_cast<uint32_t *>(rb + off[PRT_OFF_PID]) = best.pid;
			if (fmask & PRT_FIELD_VALID)
				rb[off[PRT_OFF_VALID]] = best.t < INFINITY ? 1 : 0;
			if (fmask & PRT_FIELD_P) {
				// bvh.hpp:261-263: p = origin + t * direction, per component.
				*reinterpret_cast<float *>(rb + off[PRT_OFF_PX]) =
				    __fadd_rn(r.ox, __fmul_rn(best.t, r.dx));
				*reinterpret_cast<float *>(rb + off[PRT_OFF_PY]) =
				    __fadd_rn(r.oy, __fmul_rn(best.t, r.dy));
				*reinterpret_cast<float *>(rb + off[PRT_OFF_PZ]) =
				    __fadd_rn(r.oz, __fmul_rn(best.t, r.dz));
			}
		}
		__syncwarp();
		uint8_t *dst = S.seg.out + (size_t)local * rec;
		const uint32_t bytes = nb * rec;
		const uint32_t mode = S.seg.store_mode;
		if (mode == 0 && (bytes & 15u) == 0u) { // local is a multiple of 4: 16-byte aligned
			uint4 *d4 = reinterpret_cast<uint4 *>(dst);
			const uint4 *s4 = reinterpret_cast<const uint4 *>(stage);
			for (uint32_t k = lane; k < bytes / 16u; k += 32u)
				__stcs(d4 + k, s4[k]);
		} else if (mode <= 1) {
			uint32_t *d1 = reinterpret_cast<uint32_t *>(dst);
			for (uint32_t k = lane; k < bytes / 4u; k += 32u)
				d1[k] = stage[k];
		} else {
			const uint8_t *sb = reinterpret_cast<const uint8_t *>(stage);
			for (uint32_t k = lane; k < bytes; k += 32u)
				dst[k] = sb[k];
		}
		if (S.seg.done_ctr) {
			// The run's completion count (SegDesc): every lane's record stores are made
			// visible system-wide before lane 0 counts the batch; the batch that finishes
			// the run raises the host flag after another system fence.
			__threadfence_system();
			__syncwarp();
			if (lane == 0 && !fault) {
				const uint32_t before = atomicAdd(S.seg.done_ctr, nb);
				if (before + nb == run_rays) {
					__threadfence_system();
					*reinterpret_cast<volatile uint32_t *>(S.seg.done_flag) = 1u;
				}
			}
		}
		if (PASS == 3 && fault && lane == 0) {
			// The host learns of the fault at once (the run will never complete).
			__threadfence_system();
			*reinterpret_cast<volatile uint32_t *>(a.serve.err_flag) = 1u;
		}
		__syncwarp();
	}
	if (COUNT) {
		unsigned long long a0 = n_visits, a1 = n_tests;
		for (int o = 16; o > 0; o >>= 1) {
			a0 += __shfl_xor_sync(0xFFFFFFFFu, a0, o);
			a1 += __shfl_xor_sync(0xFFFFFFFFu, a1, o);
		}
		if (lane == 0) {
			atomicAdd(&a.visits[0], a0);
			atomicAdd(&a.visits[1], a1);
		}
	}
}

// Resident blocks per SM for `warps` warps of `warp_bytes` shared memory each, on the
// current device.  The kernel's dynamic shared-memory limit is a per-device attribute
// that only grows (under a lock), so a launch that another thread sized earlier still
// fits when this one needs less.
constexpr int kCachedDevices = 16;
template <int FMT, bool COUNT, bool LEAF1, bool BOUNDED, int PASS>
int blocks_per_sm(int warps, uint32_t warp_bytes) {
	struct Cache {
		int warps = -1;
		uint32_t bytes = 0;
		int blocks = 1;
		size_t limit = 0;
	};
	static std::mutex mu;
	static Cache cache[kCachedDevices];
	int dev = 0;
	cudaGetDevice(&dev);
	const size_t smem = (size_t)warp_bytes * warps;
	std::lock_guard<std::mutex> lk(mu);
	Cache uncached;
	Cache &c = (dev >= 0 && dev < kCachedDevices) ? cache[dev] : uncached;
	if (smem > c.limit &&
	    cudaFuncSetAttribute(k_trace8<FMT, COUNT, LEAF1, BOUNDED, PASS>,
	                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess)
		c.limit = smem;
	if (c.warps != warps || c.bytes != warp_bytes) {
		int b = 0;
		cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_trace8<FMT, COUNT, LEAF1, BOUNDED, PASS>,
		                                              32 * warps, smem);
		c.blocks = b > 0 ? b : 1;
		c.warps = warps;
		c.bytes = warp_bytes;
	}
	return c.blocks;
}

template <int FMT, bool COUNT, bool LEAF1, bool BOUNDED, int PASS>
void launch_t(const TravArgs &a, int warps, int sm_count, cudaStream_t st) {
	const int bps = blocks_per_sm<FMT, COUNT, LEAF1, BOUNDED, PASS>(warps, a.warp_bytes);
	const uint64_t batches = (a.n_virtual + a.batch - 1ull) / a.batch;
	// Unbounded warps: at most one block per resident slot (persistent).  Bounded: enough
	// blocks that every batch has a warp even if each warp takes its maximum.
	const uint64_t per_block = (uint64_t)warps * (BOUNDED ? a.max_batches : 1u);
	const uint64_t need = (batches + per_block - 1) / per_block;
	const uint64_t grid = BOUNDED ? need : std::min<uint64_t>((uint64_t)sm_count * bps, need);
	k_trace8<FMT, COUNT, LEAF1, BOUNDED, PASS>
	    <<<(unsigned)grid, 32 * warps, (size_t)a.warp_bytes * warps, st>>>(a);
}

int warps_for(const TravConfig &cfg) {
	return (cfg.block >= 32 && cfg.block <= 32 * kWarpsPerBlock && cfg.block % 32 == 0)
	           ? cfg.block / 32
	           : kWarpsPerBlock;
}

// Rays per batch of a one-kernel launch (PASS 4), by the rays per resident warp (4,864 warps on
// 152 SMs); 0: too many, the two passes or the camera's packets take it.  The two passes
// cost a second launch, their batches of 32 make long serial chains, and a batch deferred for
// one zero direction component starts when all others are done; but with the plain test alone
// they need fewer registers, which pays in the end.
//
// Ray buffers.  One round of batches while 8 rays a warp suffice; when that leaves a quarter
// of the rays or less, they are claimed by fours, so that the second round is short (39,000
// to 50,000 rays 4 to 8 % faster, at most 20 %; with eights some were up to 9 % slower than as
// two passes); else batches claimed from the counter.  Speed against a regular and a
// deferred pass (mean over eight scenes, least of them; FP32 nodes, one triangle per leaf), of
// regular rays alone and with a zero x component in every 977th:
//                        regular                               with zeros
//     batches of   8          12         16         32         8          16         32
//     20,000       1.17 1.10  1.08 0.96  1.01 0.81  0.78 0.52  1.44 1.09  1.21 0.98  0.95 0.59
//     100,000      1.09 1.01  1.10 0.99  1.07 0.91  1.04 0.85  1.41 1.20  1.32 1.02  1.17 0.85
//     250,000      1.03 0.88  1.06 1.00  1.07 1.00  1.05 0.95  1.41 1.25  1.44 1.23  1.31 1.09
//     600,000      0.95 0.73  1.00 0.88  1.04 0.98  1.03 0.96  1.38 1.09  1.49 1.19  1.37 1.10
//     1,300,000    0.87 0.72  0.93 0.81  0.98 0.94  1.00 0.95  1.17 1.04  1.26 1.08  1.25 1.05
//     2,000,000    0.83 0.66  0.89 0.75  0.95 0.89  0.99 0.95  1.07 0.91  1.18 1.04  1.19 1.02
// So from 600,000 on a query without any such ray may lose up to 5 % against two passes, and
// one with a few gains 19 to 49 % (any camera of even width has them).  With compressed nodes or
// larger leaves the loss would be up to 10 % from 900,000 on, so two passes take those.
// Batches of rays that mostly miss are short, and eights cost them 11 % at 250,000 to 310,000
// rays: twelves there.  With FP32 nodes and one triangle per leaf a small scene's batch is
// short as well (us; two passes / 8 / 16 / 32):
//     64 triangles       60,000  20 / 15 / 11 / 12    320,000  41 / 43 / 35 / 31
//                     1,300,000  103 / 154 / 119 / 98
//     2,500 triangles    60,000  52 / 28 / 37 / 51    320,000  75 / 76 / 70 / 72
//                     1,300,000  288 / 272 / 233 / 218
// (Nine blocks per SM, 56 registers: 4 % slower for regular rays, 2 to 4 % for others.)
//
// Several runs (padded to whole warps of 32).  One round of batches of 4, 8 or 16.  Batch
// graphs, us: 20 scenes of up to 6,836 triangles and 5,762 rays 324 -> 273, 48 of 18,789 and
// 4,847 418 -> 362, 7 of 31,983 and 4,384 419 -> 306.  (A server's waves are bounded and keep
// batches of 32: each batch ends with a system fence, and small ones cost up to 6 %.)
//
// Cameras.  The packet descent (batches of 32) pays where a triangle covers many pixels and
// there are enough batches.  Batches of 8 / 16 / 32 / packets, us:
//     triangles  900 x 600                1600 x 900               2048 x 2048
//     256        75 / 60 / 59 / 61        166 / 119 / 103 / 96     440 / 299 / 239 / 210
//     4,968      105 / 110 / 140 / 148    207 / 171 / 183 / 183    515 / 383 / 332 / 311
//     65,536     202 / 218 / 277 / 287    284 / 274 / 288 / 294    638 / 514 / 464 / 472
// (12 triangles, 900 x 600: batches of 16 / 32 47 / 40.)
uint32_t single_batch(const TravArgs &a, const TravConfig &cfg, uint64_t slots) {
	const uint64_t n = a.n_virtual, per = (n + slots - 1) / slots;
	if (a.n_segs)
		return per <= 4u ? 4u : per <= 8u ? 8u : per <= 16u ? 16u : 0u;
	if (per <= 8u)
		return ((uint32_t)per + 3u) & ~3u;
	if (a.use_cam) {
		const bool wide = n >= 640ull * a.scene0.n_tris;
		if (wide && per > 120u)
			return 0u;
		if (wide)
			return per <= 32u ? 8u : per > 64u && a.scene0.n_tris <= 64u ? 32u : 16u;
		return per <= 120u ? 8u : per <= 450u ? 16u : 32u;
	}
	if (cfg.format != PRT_NODES_FP32 || a.max_leaf > 1u) {
		const bool tiny = a.scene0.n_tris <= 256u; // (as the small scenes below)
		return per <= (tiny ? 32u : 36u) ? 8u
		       : per <= 64u              ? (tiny ? 16u : 12u)
		       : per <= 130u             ? (tiny ? 32u : 16u)
		                                 : 0u;
	}
	const bool small = a.scene0.n_tris <= 4096u;
	if (per <= (small ? 16u : 36u))
		return 8u;
	if (per <= 64u)
		return small ? 16u : 12u;
	return per <= 300u && !small ? 16u : per <= 420u ? 32u : 0u;
}

template <int FMT, bool LEAF1>
bool launch_single(TravArgs a, const TravConfig &cfg, int warps, int sm_count, cudaStream_t st) {
	const uint64_t slots = (uint64_t)sm_count * warps *
	                       blocks_per_sm<FMT, false, LEAF1, false, 4>(warps, a.warp_bytes);
	a.batch = single_batch(a, cfg, slots);
	if (!a.batch)
		return false;
	const uint64_t dealt = (uint64_t)a.batch * slots;
	a.claims = dealt >= a.n_virtual ? 0u : 4u * dealt >= 3u * (uint64_t)a.n_virtual ? 4u : a.batch;
	if (a.claims && cudaMemsetAsync(a.counter, 0, 4, st) != cudaSuccess)
		return true; // (dispatch reports the error)
	launch_t<FMT, false, LEAF1, false, 4>(a, warps, sm_count, st);
	return true;
}

// Whether one kernel took the launch: not counting, not bounded.
bool try_single(const TravArgs &a, const TravConfig &cfg, int warps, int sm_count,
                cudaStream_t st) {
	if (cfg.count || (a.max_batches && !a.use_cam))
		return false;
	if (cfg.format == PRT_NODES_COMPRESSED)
		return a.max_leaf <= 1u
		           ? launch_single<PRT_NODES_COMPRESSED, true>(a, cfg, warps, sm_count, st)
		           : launch_single<PRT_NODES_COMPRESSED, false>(a, cfg, warps, sm_count, st);
	return a.max_leaf <= 1u ? launch_single<PRT_NODES_FP32, true>(a, cfg, warps, sm_count, st)
	                        : launch_single<PRT_NODES_FP32, false>(a, cfg, warps, sm_count, st);
}

template <int FMT, bool LEAF1>
void launch_passes(const TravArgs &a, int warps, int sm_count, cudaStream_t st) {
	if (a.max_batches > 0)
		launch_t<FMT, false, LEAF1, true, 1>(a, warps, sm_count, st);
	else
		launch_t<FMT, false, LEAF1, false, 1>(a, warps, sm_count, st);
	launch_t<FMT, false, LEAF1, false, 2>(a, warps, sm_count, st);
}

template <int FMT, bool COUNT>
void launch(const TravArgs &a, int warps, int sm_count, cudaStream_t st) {
	// A counting run is one general pass over all the work (no bounded warps).  So are
	// cameras that take packets: the examples' cameras put a zero direction component in one batch of
	// every row, and finding those batches again costs the deferred pass a recomputation
	// of every ray.
	if (COUNT || a.use_cam) {
		if (a.max_leaf <= 1u)
			launch_t<FMT, COUNT, true, false, 0>(a, warps, sm_count, st);
		else
			launch_t<FMT, COUNT, false, false, 0>(a, warps, sm_count, st);
	} else if (a.max_leaf <= 1u) {
		launch_passes<FMT, true>(a, warps, sm_count, st);
	} else {
		launch_passes<FMT, false>(a, warps, sm_count, st);
	}
}

void size_smem(TravArgs &a, uint32_t depth, int leaf_size) {
	depth = std::max<uint32_t>(depth, 1u);
	a.pool_cap = std::max<uint32_t>(256u, 7u * kItems * (depth - 1u) + kItems +
	                                          (a.use_cam ? kAdmit : (uint32_t)kItems));
	a.queue_cap = 32u + (uint32_t)kItems * 8u * (uint32_t)std::max(leaf_size, 1);
	a.max_leaf = (uint32_t)std::max(leaf_size, 1);
	a.max_batches = 0;
	a.warp_bytes = (warp_smem_bytes(a.pool_cap, a.queue_cap) + 15u) & ~15u;
}

// Rays per batch of a run of m rays that is not one kernel: 32, but for counting runs of few
// rays, where 8 or 16 keep more warps busy (bounded waves keep 32: their batch count per warp
// is the caller's).
uint32_t batch_rays(uint64_t m, int sm_count, uint32_t max_batches) {
	const uint64_t wave = (uint64_t)std::max(sm_count, 1) * 36u * 32u;
	if (max_batches > 0 || m >= 2 * wave)
		return 32;
	return m >= wave ? 16 : 8;
}

cudaError_t dispatch(const TravArgs &a, const TravConfig &cfg, int sm_count, cudaStream_t st) {
	const int warps = warps_for(cfg);
	if (try_single(a, cfg, warps, sm_count, st))
		return cudaGetLastError();
	// The counter and the two deferred words, in one go unless the word between them is the
	// launch's error word, which stays set until the host reads it.
	const bool between = a.err == a.counter + 1;
	cudaError_t e = cudaMemsetAsync(a.counter, 0, between ? 4 : 16, st);
	if (e == cudaSuccess && between)
		e = cudaMemsetAsync(a.deferred, 0, 8, st);
	if (e != cudaSuccess)
		return e;
	if (cfg.format == PRT_NODES_COMPRESSED) {
		if (cfg.count)
			launch<PRT_NODES_COMPRESSED, true>(a, warps, sm_count, st);
		else
			launch<PRT_NODES_COMPRESSED, false>(a, warps, sm_count, st);
	} else {
		if (cfg.count)
			launch<PRT_NODES_FP32, true>(a, warps, sm_count, st);
		else
			launch<PRT_NODES_FP32, false>(a, warps, sm_count, st);
	}
	return cudaGetLastError();
}

} // namespace

int traversal_stack_depth() { return kMaxDepth; }

cudaError_t launch_nearest_hits(const SceneGPU &sc, const float *d_rays, uint64_t n,
                                const OutLayout &lay, void *d_out, const TravConfig &cfg,
                                uint32_t *d_work, unsigned long long *d_visits, uint32_t *d_err,
                                cudaStream_t st, int sm_count, const prt_b200_camera *cam) {
	if (cfg.count)
		cudaMemsetAsync(d_visits, 0, 2 * sizeof(unsigned long long), st);
	const uint64_t chunk = 1ull << 31;
	if (cam && n > chunk)
		return cudaErrorInvalidValue; // camera rays are numbered within one launch
	for (uint64_t s = 0; s < n; s += chunk) {
		const uint64_t m = std::min(chunk, n - s);
		TravArgs a;
		a.use_cam = cam ? 1u : 0u;
		if (cam)
			a.cam = *cam;
		a.scenes = nullptr;
		a.segs = nullptr;
		a.n_segs = 0;
		a.n_virtual = (uint32_t)m;
		a.scene0.tri4 = sc.tri4.as<float4>();
		a.scene0.inv = sc.inv.as<uint32_t>();
		a.scene0.nodes = cfg.format == PRT_NODES_COMPRESSED ? sc.cnodes.p : sc.nodes.p;
		a.scene0.root = 0;
		a.scene0.n_tris = (uint32_t)sc.n_tris;
		a.x_faces = sc.x_log ? sc.x_faces.as<uint32_t>() : nullptr;
		a.seg0.vbegin = 0;
		a.seg0.rays = cam ? nullptr : d_rays + 6 * s;
		a.seg0.out = static_cast<uint8_t *>(d_out) + s * lay.rec_size;
		a.seg0.n_rays = (uint32_t)m;
		a.seg0.scene = 0;
		a.seg0.mask = lay.mask;
		a.seg0.rec_size = lay.rec_size;
		for (int k = 0; k < 8; ++k)
			a.seg0.off[k] = lay.off[k];
		a.seg0.store_mode = store_mode_for(a.seg0.out);
		a.seg0.pad = 0;
		a.n_nodes = sc.n_nodes;
		a.dead = sc.dead;
		size_smem(a, cfg.pool_depth ? (uint32_t)cfg.pool_depth : sc.depth, sc.leaf_size);
		a.max_batches = cfg.max_batches;
		a.batch = batch_rays(m, sm_count, cfg.max_batches);
		a.counter = d_work;
		a.deferred = d_work + 2;
		a.err = d_err;
		a.visits = d_visits;
		cudaError_t e = dispatch(a, cfg, sm_count, st);
		if (e != cudaSuccess)
			return e;
	}
	return cudaSuccess;
}

cudaError_t launch_nearest_hits_segments(const SceneDesc *d_scenes, const SegDesc *d_segs,
                                         uint32_t n_segs, unsigned long long n_virtual,
                                         uint32_t depth, int leaf_size, uint32_t n_nodes,
                                         uint32_t dead, const TravConfig &cfg,
                                         uint32_t *d_work, unsigned long long *d_visits,
                                         uint32_t *d_err, cudaStream_t st, int sm_count) {
	if (cfg.count)
		cudaMemsetAsync(d_visits, 0, 2 * sizeof(unsigned long long), st);
	if (n_segs == 0 || n_virtual == 0)
		return cudaSuccess;
	if (n_virtual > (1ull << 31))
		return cudaErrorInvalidValue;
	TravArgs a;
	memset(&a, 0, sizeof a);
	a.scenes = d_scenes;
	a.segs = d_segs;
	a.n_segs = n_segs;
	a.n_virtual = (uint32_t)n_virtual;
	a.n_nodes = n_nodes;
	a.dead = dead;
	size_smem(a, cfg.pool_depth ? (uint32_t)cfg.pool_depth : depth, leaf_size);
	a.max_batches = cfg.max_batches;
	a.batch = 32; // runs are padded to whole warps of 32
	a.counter = d_work;
	a.deferred = d_work + 2;
	a.err = d_err;
	a.visits = d_visits;
	return dispatch(a, cfg, sm_count, st);
}

namespace {

template <int FMT, bool LEAF1>
void launch_serving_t(const TravArgs &a, int sm_count, cudaStream_t st) {
	const int bps = blocks_per_sm<FMT, false, LEAF1, false, 3>(kWarpsPerBlock, a.warp_bytes);
	k_trace8<FMT, false, LEAF1, false, 3>
	    <<<(unsigned)(sm_count * bps), 32 * kWarpsPerBlock, (size_t)a.warp_bytes * kWarpsPerBlock,
	       st>>>(a);
}

} // namespace

cudaError_t launch_serving(const SceneDesc *d_scenes, const ServeQueues &q, uint32_t depth,
                           int leaf_size, uint32_t n_nodes, uint32_t dead, int format,
                           uint32_t *d_err, cudaStream_t st, int sm_count) {
	TravArgs a;
	memset(&a, 0, sizeof a);
	a.scenes = d_scenes;
	a.serve = q;
	a.n_nodes = n_nodes;
	a.dead = dead;
	size_smem(a, depth, leaf_size);
	a.batch = 32; // one ticket = 32 rays
	a.err = d_err;
	// Every resident slot: the warps poll for work, none waits for another, so the
	// launch needs no co-residency (blocks that do not fit start as others leave).
	if (format == PRT_NODES_COMPRESSED) {
		if (a.max_leaf <= 1u)
			launch_serving_t<PRT_NODES_COMPRESSED, true>(a, sm_count, st);
		else
			launch_serving_t<PRT_NODES_COMPRESSED, false>(a, sm_count, st);
	} else {
		if (a.max_leaf <= 1u)
			launch_serving_t<PRT_NODES_FP32, true>(a, sm_count, st);
		else
			launch_serving_t<PRT_NODES_FP32, false>(a, sm_count, st);
	}
	return cudaGetLastError();
}

} // namespace prt
