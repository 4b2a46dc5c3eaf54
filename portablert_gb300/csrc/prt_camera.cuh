// prt_camera.cuh - the examples' pinhole sensor camera as a device function (shared by
// the fused camera traversal, the ray writer and the shading kernel).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "../../include/prt_b200.h"

namespace prt {

// sensor_size * (float(k) / extent - 0.5): the float quotient widened to double by the
// 0.5 literal, the product rounded to float (examples/bunny/main.cpp:103-104).
__device__ __forceinline__ float sensor_coord_f64(float size, float q) {
	return __double2float_rn(__dmul_rn((double)size, __dsub_rn((double)q, 0.5)));
}

// The same bits without the FP64 pipe (about 2 lanes per clock and SM), which took eight
// operations per ray in the traversal and again in the shading: traversal and shading of
// 2048 x 2048 pixels 305.5 -> 302.4 us, of 1919 x 1081 176.7 -> 170.7.
//
// q is 0 or in [2^-31, 1], so q - 0.5 is exact in double, and here it is hi + lo exactly
// (Dekker's sum).  Where lo is 0, always for a power-of-two extent, double holds the product
// size * hi exactly and one rounding to float remains: the float product.  Otherwise the
// exact product is p + (e + size * lo), with e the rounding error of p; r is the second
// term to 2^-24 of itself.  Widened to either side by 2^-20 of r, which also covers the
// rounding to double (2^-53 of the product: below 2^-21 of r, unless r is so small that p
// is the answer), both ends rounding to the same float is proof that double's two roundings
// give it too.  The rest (ends that differ, about one product in a million; e inexact near
// the denormals; overflow) takes the double path.
__device__ __forceinline__ float sensor_coord(float size, uint32_t k, uint32_t extent) {
	const float q = __fdiv_rn((float)k, (float)extent);
	const float hi = __fsub_rn(q, 0.5f);
	const float lo = __fsub_rn(q, __fadd_rn(hi, 0.5f));
	const float p = __fmul_rn(size, hi);
	if (lo == 0.0f)
		return p;
	const float r = __fmaf_rn(size, lo, __fmaf_rn(size, hi, -p));
	const float m = __fmul_rn(fabsf(r), 0x1p-20f);
	const float a = __fadd_rn(p, __fsub_rn(r, m)), b = __fadd_rn(p, __fadd_rn(r, m));
	if (a == b && fabsf(p) >= 0x1p-100f && fabsf(p) <= 0x1p126f)
		return a;
	return sensor_coord_f64(size, q);
}

// Ray i of the camera (examples/bunny/main.cpp:101-124, validation/main.cpp:170-198,
// sponza/main.cpp:193-218), FP32 operation for operation, no contraction.
__device__ __forceinline__ void camera_ray(const prt_b200_camera &c, uint32_t i, float o[3],
                                           float d[3]) {
	const uint32_t x = i % c.width;
	const uint32_t y = c.height - 1u - i / c.width;
	const float sx = sensor_coord(c.sensor_size, x, c.width);
	const float sy = sensor_coord(c.sensor_size, y, c.height);
	float sp[3];
	if (c.form == PRT_CAMERA_ROTATED) {
		const float dx = __fadd_rn(__fmul_rn(c.cos_a, sx), __fmul_rn(c.sin_a, c.sensor_dist));
		const float dz = __fadd_rn(__fmul_rn(-c.sin_a, sx), __fmul_rn(c.cos_a, c.sensor_dist));
		sp[0] = __fadd_rn(c.pos[0], dx);
		sp[1] = __fadd_rn(c.pos[1], sy);
		sp[2] = __fadd_rn(c.pos[2], dz);
	} else {
		sp[0] = sx;
		sp[1] = sy;
		sp[2] = c.sensor_z;
	}
	for (int k = 0; k < 3; ++k) {
		o[k] = c.pos[k];
		d[k] = __fsub_rn(sp[k], c.pos[k]);
	}
	const float *l = c.form == PRT_CAMERA_PLANE_SENSOR_NORM ? sp : d;
	const float len = __fsqrt_rn(
	    __fadd_rn(__fadd_rn(__fmul_rn(l[0], l[0]), __fmul_rn(l[1], l[1])), __fmul_rn(l[2], l[2])));
	for (int k = 0; k < 3; ++k)
		d[k] = __fdiv_rn(d[k], len);
}

// Validates a camera (non-empty, at most 2^31 rays, a known form).
bool camera_ok(const prt_b200_camera *c, std::string &why);

} // namespace prt
