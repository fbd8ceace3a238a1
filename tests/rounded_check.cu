// rounded.cuh and make_ray's reciprocals on every float, against CUDA's correctly rounded
// operations. Prints the number of floats on which any result has other bits.
#include <cstdio>

#include "traverse.cuh"

using namespace rnb;

namespace {

__device__ bool differ(float a, float b) {
	return __float_as_uint(a) != __float_as_uint(b) && !(a != a && b != b); // any NaN is a NaN
}

// wrong[0]: rcp_bounded, [1]: sqrt_bounded, [2]: sqrt_exact, [3]: inv_sqrt_exact, [4]: make_ray
__global__ void k_check(unsigned long long *wrong, unsigned long long *tried) {
	unsigned long long w[5] = {}, n[2] = {};
	for (unsigned long long i = blockIdx.x * 256ull + threadIdx.x; i < 1ull << 32; i += gridDim.x * 256ull) {
		const float x = __uint_as_float(static_cast<unsigned>(i));
		const float rcp = __fdiv_rn(1.0f, x), root = __fsqrt_rn(x);
		if (fabsf(x) >= 0x1p-126f && fabsf(x) < 0x1p126f) {
			n[0]++;
			w[0] += differ(rcp_bounded(x), rcp);
		}
		if (sqrt_in_range(x)) {
			n[1]++;
			w[1] += differ(sqrt_bounded(x), root);
		}
		w[2] += differ(sqrt_exact(x), root);
		w[3] += differ(inv_sqrt_exact(x), __fdiv_rn(1.0f, root));
		// in each place among ordinary components
		const float a = 0.3f, b = -7.0f, ra = __fdiv_rn(1.0f, a), rb = __fdiv_rn(1.0f, b);
		const RayPre p = make_ray(0, 0, 0, x, a, b), q = make_ray(0, 0, 0, b, x, a), r = make_ray(0, 0, 0, a, b, x);
		w[4] += differ(p.ix, rcp) | differ(p.iy, ra) | differ(p.iz, rb) | differ(q.ix, rb) | differ(q.iy, rcp) |
		        differ(q.iz, ra) | differ(r.ix, ra) | differ(r.iy, rb) | differ(r.iz, rcp);
	}
	for (int k = 0; k < 5; k++)
		atomicAdd(wrong + k, w[k]);
	atomicAdd(tried, n[0]);
	atomicAdd(tried + 1, n[1]);
}

} // namespace

int main() {
	unsigned long long *d, h[7];
	if (cudaMalloc(&d, sizeof(h)) != cudaSuccess || cudaMemset(d, 0, sizeof(h)) != cudaSuccess)
		return 2;
	k_check<<<148 * 8, 256>>>(d, d + 5);
	if (cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess)
		return 2;
	std::printf("wrong %llu %llu %llu %llu %llu tried %llu %llu\n", h[0], h[1], h[2], h[3], h[4], h[5], h[6]);
	// 252 binades of both signs, 226 of one
	return h[0] | h[1] | h[2] | h[3] | h[4] || h[5] != 2ull * 252 << 23 || h[6] != 226ull << 23;
}
