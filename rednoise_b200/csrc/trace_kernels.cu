// Batched ray queries: one thread per ray over the flattened reference BVH.
#include "scene_impl.hpp"

namespace rnb {

template <int kOrder>
__global__ void __launch_bounds__(128) k_trace_closest(SceneView s, int n, const float *__restrict__ o,
                                                       const float *__restrict__ d, const int *__restrict__ ignore,
                                                       int *__restrict__ tri, float *__restrict__ t,
                                                       float *__restrict__ u, float *__restrict__ v, int *err) {
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n)
		return;
	const RayPre r = make_ray(o[3 * i], o[3 * i + 1], o[3 * i + 2], d[3 * i], d[3 * i + 1], d[3 * i + 2]);
	int e = 0;
	const HitRec h = trace_closest_best<kOrder>(s, r, ignore ? ignore[i] : -1, e);
	if (e)
		atomicOr(err, 1);
	tri[i] = h.idx;
	if (t)
		t[i] = h.t;
	if (u)
		u[i] = h.u;
	if (v)
		v[i] = h.v;
}

__global__ void __launch_bounds__(128) k_trace_any(SceneView s, int n, const float *__restrict__ o,
                                                   const float *__restrict__ d, const float *__restrict__ tmax,
                                                   const int *__restrict__ ignore, int *__restrict__ occ, int *err) {
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n)
		return;
	const RayPre r = make_ray(o[3 * i], o[3 * i + 1], o[3 * i + 2], d[3 * i], d[3 * i + 1], d[3 * i + 2]);
	int e = 0;
	const bool hit = trace_any_best(s, r, tmax[i], ignore ? ignore[i] : -1, e);
	if (e)
		atomicOr(err, 1);
	occ[i] = hit ? 1 : 0;
}

// Many rays: a persistent grid whose lanes take the next ray when theirs is done.
constexpr int kStreamBlocks = 7;                                    // per SM: 72 registers, what measured best
constexpr size_t kStreamSmem = 128 * 8 * sizeof(unsigned long long); // the stacks' tops
__global__ void __launch_bounds__(128, kStreamBlocks)
    k_trace_closest_stream(SceneView s, int n, const float *__restrict__ o, const float *__restrict__ d,
                           const int *__restrict__ ignore, int *__restrict__ tri, float *__restrict__ t,
                           float *__restrict__ u, float *__restrict__ v, int *err) {
	extern __shared__ unsigned long long closest_top[];
	SharedShortStack<unsigned long long, 8> st(closest_top + threadIdx.x, blockDim.x);
	StreamTurns turns(static_cast<unsigned>(n));
	int e = 0;
	unsigned i = 0;
	trace_closest_stream(
	    s, st, e,
	    [&](bool want, unsigned idle, RayPre &r, int &ig) {
		    unsigned k;
		    if (!turns.next(want, idle, k))
			    return false;
		    i = k;
		    const size_t a = 3 * static_cast<size_t>(i);
		    r = make_ray(o[a], o[a + 1], o[a + 2], d[a], d[a + 1], d[a + 2]);
		    ig = ignore ? ignore[i] : -1;
		    return true;
	    },
	    [&](const HitRec &h) {
		    tri[i] = h.idx;
		    if (t)
			    t[i] = h.t;
		    if (u)
			    u[i] = h.u;
		    if (v)
			    v[i] = h.v;
	    });
	if (e)
		atomicOr(err, 1);
}

// Few rays over a small scene: kGroup lanes per ray (trace_closest_group).
constexpr int kGroup = 8;
__global__ void __launch_bounds__(128) k_trace_closest_group(SceneView s, int n, const float *__restrict__ o,
                                                             const float *__restrict__ d,
                                                             const int *__restrict__ ignore, int *__restrict__ tri,
                                                             float *__restrict__ t, float *__restrict__ u,
                                                             float *__restrict__ v, int *err) {
	__shared__ TriList list;
	list.load(s);
	__syncthreads();
	const int ray = static_cast<int>((blockIdx.x * blockDim.x + threadIdx.x) / kGroup);
	const int i = min(ray, n - 1); // the last block's spare groups repeat the last ray
	const RayPre r = make_ray(o[3 * i], o[3 * i + 1], o[3 * i + 2], d[3 * i], d[3 * i + 1], d[3 * i + 2]);
	int e = 0;
	const HitRec h = trace_closest_group<kGroup>(s, list, r, ignore ? ignore[i] : -1, e);
	if (e)
		atomicOr(err, 1);
	if (ray != i || threadIdx.x % kGroup != 0)
		return;
	tri[i] = h.idx;
	if (t)
		t[i] = h.t;
	if (u)
		u[i] = h.u;
	if (v)
		v[i] = h.v;
}

__global__ void __launch_bounds__(128) k_trace_any_group(SceneView s, int n, const float *__restrict__ o,
                                                         const float *__restrict__ d, const float *__restrict__ tmax,
                                                         const int *__restrict__ ignore, int *__restrict__ occ,
                                                         int *err) {
	__shared__ TriList list;
	list.load(s);
	__syncthreads();
	const int ray = static_cast<int>((blockIdx.x * blockDim.x + threadIdx.x) / kGroup);
	const int i = min(ray, n - 1);
	const RayPre r = make_ray(o[3 * i], o[3 * i + 1], o[3 * i + 2], d[3 * i], d[3 * i + 1], d[3 * i + 2]);
	int e = 0;
	const bool hit = trace_any_group<kGroup>(s, list, r, tmax[i], ignore ? ignore[i] : -1, e);
	if (e)
		atomicOr(err, 1);
	if (ray == i && threadIdx.x % kGroup == 0)
		occ[i] = hit ? 1 : 0;
}

// kGroup lanes per ray up to this many rays, a thread per ray beyond: closest and any hits of
// the 36-triangle box take 6 us of device time for 4 096 rays (39 with a thread per ray), 12
// (40) for 16 384, 31 (45) for 65 536 and 62 (56) for 131 072. At the list's end, 128
// triangles, 65 536 rays take 41 and 37 us where a thread per ray over 129 takes 43 and 34.
constexpr int kGroupRays = 1 << 16;
// Closest hits of this many rays and more, over scenes of this many triangles and more, take the
// persistent kernel. Below, too few warps have a ray to go on with, or the rays are too alike in
// length to repay the exchange. Time with a thread per ray over time with it:
//   rays                       131 072  262 144  2M
//   128 random + 1 triangles   0.95     0.90     0.83
//   512                        0.92     1.00     0.97
//   1 000                      0.92     1.00     1.01
//   5 000                      0.95     1.11     1.20
//   1 300-triangle sphere      0.85     1.03     1.10
//   20 500                     0.98     1.07     1.26
//   1.31M                      0.99     1.02     1.38 (1.12 -> 0.82 ms)
constexpr int kStreamRays = 1 << 18, kStreamTris = 768;

cudaError_t launch_trace_closest(const SceneView &v, int n, const float *o, const float *d, const int *ignore,
                                 int order, int *tri, float *t, float *u, float *vv, int *err, cudaStream_t st) {
	if (n <= 0)
		return cudaSuccess;
	const int bs = 128;
	if (order == kOrderReference && v.list && n <= kGroupRays)
		k_trace_closest_group<<<ceil_div(static_cast<long>(n) * kGroup, bs), bs, 0, st>>>(v, n, o, d, ignore, tri, t, u,
		                                                                                  vv, err);
	else if (order == kOrderNearest)
		k_trace_closest<kOrderNearest><<<ceil_div(n, bs), bs, 0, st>>>(v, n, o, d, ignore, tri, t, u, vv, err);
	else if (v.nodes4 && v.n_tris >= kStreamTris && n >= kStreamRays)
		k_trace_closest_stream<<<148 * kStreamBlocks, bs, kStreamSmem, st>>>(v, n, o, d, ignore, tri, t, u, vv, err);
	else
		k_trace_closest<kOrderReference><<<ceil_div(n, bs), bs, 0, st>>>(v, n, o, d, ignore, tri, t, u, vv, err);
	return cudaGetLastError();
}

cudaError_t launch_trace_any(const SceneView &v, int n, const float *o, const float *d, const float *tmax,
                             const int *ignore, int *occ, int *err, cudaStream_t st) {
	if (n <= 0)
		return cudaSuccess;
	const int bs = 128;
	if (v.list && n <= kGroupRays)
		k_trace_any_group<<<ceil_div(static_cast<long>(n) * kGroup, bs), bs, 0, st>>>(v, n, o, d, tmax, ignore, occ, err);
	else
		k_trace_any<<<ceil_div(n, bs), bs, 0, st>>>(v, n, o, d, tmax, ignore, occ, err);
	return cudaGetLastError();
}

} // namespace rnb
