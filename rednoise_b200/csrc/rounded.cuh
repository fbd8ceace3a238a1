// Correctly rounded reciprocal and square root without branches, for arguments known to lie
// in a stated range: the surrounding work is scheduled around the operation's latency, which a
// lone warp would otherwise wait out each time. tests/rounded_check.cu compares the results
// with CUDA's correctly rounded operations on every float.
#pragma once

#include <cuda_runtime.h>

namespace rnb {

#ifdef __CUDACC__

// 1 / x for 2^-126 <= |x| < 2^126: the hardware's approximation and one Newton step with
// fused residual and update (Markstein 1990).
__device__ __forceinline__ float rcp_bounded(float x) {
	float y;
	asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
	return __fmaf_rn(y, __fmaf_rn(-x, y, 1.0f), y);
}

// sqrt(x) for 2^-100 <= x: from the approximate reciprocal square root y, s = x y and its
// fused residual times y / 2 (the same paper).
__device__ __forceinline__ float sqrt_bounded(float x) {
	float y;
	asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
	const float s = __fmul_rn(x, y);
	return __fmaf_rn(__fmaf_rn(-s, s, x), __fmul_rn(0.5f, y), s);
}

__device__ __forceinline__ bool sqrt_in_range(float x) { return x >= 0x1p-100f && x < 0x1p126f; }

// sqrt(x) and 1 / sqrt(x), each operation correctly rounded, for any x: the forms above where
// they hold (lengths of vectors always are), CUDA's elsewhere.
__device__ __forceinline__ float sqrt_exact(float x) {
	float s = sqrt_bounded(x);
	if (!sqrt_in_range(x))
		s = __fsqrt_rn(x);
	return s;
}
__device__ __forceinline__ float inv_sqrt_exact(float x) {
	float r = rcp_bounded(sqrt_bounded(x));
	if (!sqrt_in_range(x))
		r = __fdiv_rn(1.0f, __fsqrt_rn(x));
	return r;
}

#endif

} // namespace rnb
