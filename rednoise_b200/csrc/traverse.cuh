// Ray traversal of the flattened reference BVH on sm_100a.
//
// Arithmetic contract: every operation on the closest-hit/any-hit path is an
// explicitly rounded IEEE single-precision op (__fadd_rn/__fsub_rn/__fmul_rn/
// __fdiv_rn never contract into FMA), evaluated in the order of the reference:
//   * slab test             src/BVH.cpp:66-75
//   * ray/triangle test     src/Geometry.cpp:11-25, which solves
//                           inverse(mat3(-d, e0, e1)) * (o - v0) with glm's
//                           determinant / inverse / mat3*vec3 expression order
//                           (third_party/glm/detail/func_matrix.inl:253-344,
//                            detail/type_mat3x3.inl:468-474)
// so t, u, v and the accept/reject decision are bit-identical to the reference.
//
// Two closest-hit traversal orders share that arithmetic:
//   * kOrderReference: the reference's depth-first order (push left, push right,
//     pop right first) with its strict `tenter < closest` pruning, so the hit is
//     the reference's hit by construction (src/BVH.cpp:77-111).
//   * kOrderNearest: nearer child first, `tenter <= closest` pruning and ties on
//     t broken by the triangle's rank in the reference's static order, which
//     returns the same (t, rank)-minimal hit whenever the float slab test is
//     conservative for the hit triangle.
// Any-hit (src/BVH.cpp:113-139) is order independent on a fixed tree: the set of
// reachable leaves depends only on the slab tests against the fixed maxDistance.
#pragma once

#include "common.cuh"
#include "rounded.cuh"

#include <cuda_runtime.h>
#include <stdint.h>

namespace rnb {

constexpr int kStack = 64; // same bound as the reference's int stack[64]

struct SceneView {
	const float4 *__restrict__ nodes;  // 4 float4 per internal node (2-wide)
	const float4 *__restrict__ nodes4; // 8 float4 per node (4-wide collapse), may be null
	const float4 *__restrict__ tris;   // 3 float4 per triangle position
	float root_lo[3];
	float root_hi[3];
	int root_ref;
	int root4_ref;
	int n_tris;
	int n_nodes;  // internal nodes of the 2-wide layout
	int n_nodes4; // nodes of the 4-wide layout (0 when absent)
	// Scenes of at most kListTris triangles: the triangles in the reference's static
	// traversal order, 5 float4 each: (v0, index), (e0, leaf lo.x), (e1, leaf lo.y),
	// (leaf lo.z, leaf hi), the cofactors of (e0, e1). Null for larger scenes.
	const float4 *__restrict__ list;
	// |det| <= 6 max|d| max|e|^2 in the triangle test: directions with components below
	// max_dir keep it under 2^126
	float max_dir;
};

struct RayPre {
	float ox, oy, oz;
	float dx, dy, dz;
	float ix, iy, iz;    // 1 / d, IEEE division (glm: 1.0f / direction)
};

enum TraversalOrder : int { kOrderReference = 0, kOrderNearest = 1 };

struct HitRec {
	int idx;  // original triangle index, -1 on a miss
	int rank; // rank in the reference's static traversal order
	float t, u, v;
};

#ifdef __CUDACC__
// Paired single-precision arithmetic of sm_100 (PTX sub/mul .rn.f32x2): two independently,
// correctly rounded IEEE operations per instruction, so products keep the reference's
// bits at half the instruction count. A product may only feed scalar sums: ptxas
// contracts mul.rn.f32x2 into a following packed sum in spite of .rn (measured), while the
// slab's order, differences first, leaves it nothing to contract.
__device__ __forceinline__ unsigned long long pair2(float lo, float hi) {
	unsigned long long r;
	asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
	return r;
}
__device__ __forceinline__ void unpair2(unsigned long long v, float &lo, float &hi) {
	asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ unsigned long long sub2(unsigned long long a, unsigned long long b) {
	unsigned long long r;
	asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
	return r;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
	unsigned long long r;
	asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
	return r;
}

__device__ __forceinline__ RayPre make_ray(float ox, float oy, float oz, float dx, float dy, float dz) {
	RayPre r;
	r.ox = ox;
	r.oy = oy;
	r.oz = oz;
	r.dx = dx;
	r.dy = dy;
	r.dz = dz;
	r.ix = rcp_bounded(dx);
	r.iy = rcp_bounded(dy);
	r.iz = rcp_bounded(dz);
	const float ax = fabsf(dx), ay = fabsf(dy), az = fabsf(dz);
	if (!(fminf(ax, fminf(ay, az)) >= 0x1p-126f && fmaxf(ax, fmaxf(ay, az)) < 0x1p126f)) { // a zero, say
		r.ix = __fdiv_rn(1.0f, dx);
		r.iy = __fdiv_rn(1.0f, dy);
		r.iz = __fdiv_rn(1.0f, dz);
	}
	return r;
}

// Slab test split into its tMax-independent part (returned) and tenter, so the
// `tenter < tMax` half can be applied when the node is popped, exactly where
// the reference applies it. Min/max keep glm's and std::min/max({...})'s
// comparison order (NaN and signed-zero behaviour included).
__device__ __forceinline__ bool slab(float lox, float hix, float loy, float hiy, float loz, float hiz,
                                     const RayPre &r, float &tenter) {
	const float t0x = __fmul_rn(__fsub_rn(lox, r.ox), r.ix);
	const float t1x = __fmul_rn(__fsub_rn(hix, r.ox), r.ix);
	const float t0y = __fmul_rn(__fsub_rn(loy, r.oy), r.iy);
	const float t1y = __fmul_rn(__fsub_rn(hiy, r.oy), r.iy);
	const float t0z = __fmul_rn(__fsub_rn(loz, r.oz), r.iz);
	const float t1z = __fmul_rn(__fsub_rn(hiz, r.oz), r.iz);
	const float sx = (t1x < t0x) ? t1x : t0x;
	const float sy = (t1y < t0y) ? t1y : t0y;
	const float sz = (t1z < t0z) ? t1z : t0z;
	const float bx = (t0x < t1x) ? t1x : t0x;
	const float by = (t0y < t1y) ? t1y : t0y;
	const float bz = (t0z < t1z) ? t1z : t0z;
	float te = sx;
	if (te < sy)
		te = sy;
	if (te < sz)
		te = sz;
	float tx = bx;
	if (by < tx)
		tx = by;
	if (bz < tx)
		tx = bz;
	const float m0 = (te < 0.0f) ? 0.0f : te;
	tenter = te;
	return tx >= m0;
}

// Reference ray/triangle test on a stored record of (v0, e0 = v1 - v0, e1 = v2 - v0):
// a = (v0, index), b = (e1.x, e0.x, e1.y, e0.y), c = (e1.z, e0.z, e0.y * e1.z - e1.y * e0.z,
// rank). e0, e1 and the cofactor were computed on the host with the IEEE operations the
// reference performs at test time, so they carry the same bits. kBounded: the ray is a
// bounded_ray of the scene, whose determinants stay in rcp_bounded's range (those below
// 1e-8 are rejected whatever their reciprocal).
// u needs the cofactors of e1, v those of e0, in the same expressions: the record holds the
// edges side by side and their products are formed in pairs. (Expressions are the
// reference's with signs moved, which changes no bit: -(x * y) and (-x) * y are the same, and so
// are (-x) - (-y) and y - x.)
// A ray takes 11 to 14 of these tests, with 16 to 18 of a warp's lanes in step, and a warp
// rarely leaves at an early exit of its lanes: between the determinant and t there is one,
// behind u and v together, and the 4-wide traversals load the whole record before they look
// at the index to ignore. Against the reference's order of tests and unpaired products: the
// 1.31M-triangle 1080p x 32 spp frame 47.9 -> 45.5 ms, the room at 720p x 64 spp 25.2 ->
// 24.4, the drop-in's 320 x 240 x 16 frame 3.42 -> 3.06, four adjoint views of the room
// 24.6 -> 22.8. kStraight has no exit at all: for rays that share nothing but the warp (2M
// unordered ones 0.83 -> 0.78 ms), while the room's frames lose 2 % with it.
template <bool kBounded = false, bool kStraight = false>
__device__ __forceinline__ bool tri_test(const float4 a, const float4 b, const float4 c, const RayPre &r, float &t,
                                         float &u, float &v) {
	const float spx = __fsub_rn(r.ox, a.x);
	const float spy = __fsub_rn(r.oy, a.y);
	const float spz = __fsub_rn(r.oz, a.z);
	const unsigned long long X = pair2(b.x, b.y), Y = pair2(b.z, b.w), Z = pair2(c.x, c.y);
	const unsigned long long dx = pair2(r.dx, r.dx), dy = pair2(r.dy, r.dy), dz = pair2(r.dz, r.dz);
	// mat3(m0 = -d, m1 = e0, m2 = e1): A = m01*m22 - m21*m02, B = m01*m12 - m11*m02
	float p0, p1, q0, q1;
	unpair2(mul2(Y, dz), p0, p1);
	unpair2(mul2(dy, Z), q0, q1);
	const float A = __fsub_rn(p0, q0), B = __fsub_rn(p1, q1);
	const float det = __fadd_rn(__fsub_rn(__fmul_rn(-r.dx, c.z), __fmul_rn(b.y, A)), __fmul_rn(b.x, B));
	if (!kStraight && fabsf(det) < 1e-8f)
		return false;
	const float k = kBounded ? rcp_bounded(det) : __fdiv_rn(1.0f, det);
	// Rows 1 and 2 of the inverse give u and v.
	const unsigned long long kk = pair2(k, k);
	unpair2(mul2(X, dz), p0, p1);
	unpair2(mul2(dx, Z), q0, q1);
	const float P = __fsub_rn(p0, q0), Q = __fsub_rn(p1, q1);
	unpair2(mul2(X, dy), p0, p1);
	unpair2(mul2(dx, Y), q0, q1);
	const float S = __fsub_rn(p0, q0), T = __fsub_rn(p1, q1);
	float u0, u1, u2, v0, v1, v2;
	unpair2(mul2(mul2(pair2(A, B), kk), pair2(spx, spx)), u0, v0);
	unpair2(mul2(mul2(pair2(P, Q), kk), pair2(spy, spy)), u1, v1);
	unpair2(mul2(mul2(pair2(S, T), kk), pair2(spz, spz)), u2, v2);
	u = __fsub_rn(__fsub_rn(u1, u0), u2);
	v = __fadd_rn(__fsub_rn(v0, v1), v2);
	if (!kStraight && !((u >= 0.0f) & (v >= 0.0f) & (__fadd_rn(u, v) <= 1.0f)))
		return false;
	const float i00 = __fmul_rn(c.z, k);
	const float i10 = __fmul_rn(-__fsub_rn(__fmul_rn(b.y, c.x), __fmul_rn(b.x, c.y)), k);
	const float i20 = __fmul_rn(__fsub_rn(__fmul_rn(b.y, b.z), __fmul_rn(b.x, b.w)), k);
	t = __fadd_rn(__fadd_rn(__fmul_rn(i00, spx), __fmul_rn(i10, spy)), __fmul_rn(i20, spz));
	if (!kStraight)
		return t > 1e-5f;
	return !(fabsf(det) < 1e-8f) & (u >= 0.0f) & (v >= 0.0f) & (__fadd_rn(u, v) <= 1.0f) & (t > 1e-5f);
}

__device__ __forceinline__ int leaf_start(int ref) { return (~ref) >> 3; }
__device__ __forceinline__ int leaf_count(int ref) { return (~ref) & 7; }

// Debug-build checks of tree references (compiled away unless RN_BOUNDS_CHECK).
__device__ __forceinline__ bool bad_node(const SceneView &s, int ref, bool four) {
	return kBoundsCheck && ref >= (four ? s.n_nodes4 : s.n_nodes);
}
__device__ __forceinline__ bool bad_leaf(const SceneView &s, int start, int count) {
	return kBoundsCheck && (start < 0 || count < 0 || start + count > s.n_tris);
}

// Closest hit. `ignore` is an original triangle index to skip (-1 = none).
// `err` is set to 1 if the stack bound would be exceeded (the host rejects
// trees deeper than the bound, so this only reports corrupted input).
template <int kOrder, bool kStraight = false>
__device__ __forceinline__ HitRec trace_closest(const SceneView &s, const RayPre &r, int ignore, int &err) {
	HitRec h;
	h.idx = -1;
	h.rank = 0x7fffffff;
	h.t = __int_as_float(0x7f800000);
	h.u = 0.0f;
	h.v = 0.0f;
	int st_ref[kStack];
	float st_t[kStack];
	int sp = 0;
	float te;
	if (s.n_tris > 0 && slab(s.root_lo[0], s.root_hi[0], s.root_lo[1], s.root_hi[1], s.root_lo[2], s.root_hi[2], r, te)) {
		st_ref[0] = s.root_ref;
		st_t[0] = te;
		sp = 1;
	}
	while (sp > 0) {
		--sp;
		int ref = st_ref[sp];
		const float tent = st_t[sp];
		if (kOrder == kOrderReference) {
			if (!(tent < h.t))
				continue;
		} else {
			if (tent > h.t)
				continue;
		}
		// Descend through internal nodes until a leaf is reached.
		while (ref >= 0) {
			if (bad_node(s, ref, false)) {
				err = 1;
				return h;
			}
			const float4 *nd = s.nodes + 4 * static_cast<size_t>(ref);
			const float4 n0 = __ldg(nd + 0);
			const float4 n1 = __ldg(nd + 1);
			const float4 n2 = __ldg(nd + 2);
			const float4 n3 = __ldg(nd + 3);
			float tl, tr;
			const bool hl = slab(n0.x, n0.y, n0.z, n0.w, n2.x, n2.y, r, tl);
			const bool hr = slab(n1.x, n1.y, n1.z, n1.w, n2.z, n2.w, r, tr);
			const int cl = __float_as_int(n3.x);
			const int cr = __float_as_int(n3.y);
			int next = -1;
			bool have_next = false;
			if (kOrder == kOrderReference) {
				// Reference: push left, push right; the right child is popped next and
				// tested against the (unchanged) closest distance.
				if (hl) {
					if (sp >= kStack) {
						err = 1;
						return h;
					}
					st_ref[sp] = cl;
					st_t[sp] = tl;
					++sp;
				}
				if (hr && tr < h.t) {
					next = cr;
					have_next = true;
				}
			} else {
				const bool vl = hl && !(tl > h.t);
				const bool vr = hr && !(tr > h.t);
				if (vl && vr) {
					// Nearer first; on equal entry distance keep the reference's right-first order.
					const bool left_first = tl < tr;
					if (sp >= kStack) {
						err = 1;
						return h;
					}
					st_ref[sp] = left_first ? cr : cl;
					st_t[sp] = left_first ? tr : tl;
					++sp;
					next = left_first ? cl : cr;
					have_next = true;
				} else if (vl) {
					next = cl;
					have_next = true;
				} else if (vr) {
					next = cr;
					have_next = true;
				}
			}
			if (!have_next) {
				ref = 0x7fffffff; // sentinel: nothing to descend into
				break;
			}
			ref = next;
		}
		if (ref == 0x7fffffff)
			continue;
		// Leaf: test its triangles in ascending order.
		const int start = leaf_start(ref);
		const int count = leaf_count(ref);
		if (bad_leaf(s, start, count)) {
			err = 1;
			return h;
		}
		for (int p = start; p < start + count; p++) {
			const float4 *tp = s.tris + 3 * static_cast<size_t>(p);
			const float4 a = __ldg(tp + 0);
			const int ti = __float_as_int(a.w);
			if (ti == ignore)
				continue;
			const float4 b = __ldg(tp + 1);
			const float4 c = __ldg(tp + 2);
			float t, u, v;
			if (!tri_test<false, kStraight>(a, b, c, r, t, u, v))
				continue;
			if (kOrder == kOrderReference) {
				if (t < h.t) {
					h.idx = ti;
					h.t = t;
					h.u = u;
					h.v = v;
					h.rank = __float_as_int(c.w);
				}
			} else {
				const int rk = __float_as_int(c.w);
				if (t < h.t || (t == h.t && rk < h.rank)) {
					h.idx = ti;
					h.t = t;
					h.u = u;
					h.v = v;
					h.rank = rk;
				}
			}
		}
	}
	return h;
}

// Any hit strictly before tmax (the reference's occluded()).
__device__ __forceinline__ bool trace_any(const SceneView &s, const RayPre &r, float tmax, int ignore, int &err) {
	int st[kStack];
	int sp = 0;
	float te;
	if (s.n_tris > 0 && slab(s.root_lo[0], s.root_hi[0], s.root_lo[1], s.root_hi[1], s.root_lo[2], s.root_hi[2], r, te) &&
	    te < tmax) {
		st[0] = s.root_ref;
		sp = 1;
	}
	while (sp > 0) {
		int ref = st[--sp];
		while (ref >= 0) {
			if (bad_node(s, ref, false)) {
				err = 1;
				return false;
			}
			const float4 *nd = s.nodes + 4 * static_cast<size_t>(ref);
			const float4 n0 = __ldg(nd + 0);
			const float4 n1 = __ldg(nd + 1);
			const float4 n2 = __ldg(nd + 2);
			const float4 n3 = __ldg(nd + 3);
			float tl, tr;
			const bool hl = slab(n0.x, n0.y, n0.z, n0.w, n2.x, n2.y, r, tl) && tl < tmax;
			const bool hr = slab(n1.x, n1.y, n1.z, n1.w, n2.z, n2.w, r, tr) && tr < tmax;
			const int cl = __float_as_int(n3.x);
			const int cr = __float_as_int(n3.y);
			if (hl && hr) {
				if (sp >= kStack) {
					err = 1;
					return false;
				}
				const bool left_first = tl < tr;
				st[sp++] = left_first ? cr : cl;
				ref = left_first ? cl : cr;
			} else if (hl) {
				ref = cl;
			} else if (hr) {
				ref = cr;
			} else {
				ref = 0x7fffffff;
				break;
			}
		}
		if (ref == 0x7fffffff)
			continue;
		const int start = leaf_start(ref);
		const int count = leaf_count(ref);
		if (bad_leaf(s, start, count)) {
			err = 1;
			return false;
		}
		for (int p = start; p < start + count; p++) {
			const float4 *tp = s.tris + 3 * static_cast<size_t>(p);
			const float4 a = __ldg(tp + 0);
			if (__float_as_int(a.w) == ignore)
				continue;
			const float4 b = __ldg(tp + 1);
			const float4 c = __ldg(tp + 2);
			float t, u, v;
			if (tri_test(a, b, c, r, t, u, v) && t < tmax)
				return true;
		}
	}
	return false;
}

// ---- 4-wide traversal in the reference's order ---------------------------------
// The tree is the host's own over the reference tree's leaves (split_by_area), which it meets in
// the reference's order. Entries of a node are stored in that order; entries 1..count-1 are
// pushed (last first) and entry 0 is descended into at once, which is the reference's
// push-then-pop. The reference reaches a leaf whose own box the ray enters before the best
// distance of that moment, for then it passed every box above it too (boxes that contain
// the leaf's are entered no later: the slab arithmetic rounds monotonically); so do these
// traversals, whatever boxes stand above the leaves. Rays with an infinite 1/d component (a
// zero or subnormal direction component, where a slab product can be NaN) take the 2-wide
// path instead.

// Three-input min / max of sm_100 (PTX min.f32 / max.f32 with three sources).
__device__ __forceinline__ float max3(float a, float b, float c) {
	float r;
	asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
	return r;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
	float r;
	asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
	return r;
}

// The ray's origin and inverse direction duplicated into pairs, and per axis the byte
// offset in a 4-wide node of the row that holds the planes the ray meets first (lo for a
// positive inverse direction, hi for a negative one); the other row is 16 bytes away.
struct RayPair {
	unsigned long long ox, oy, oz, ix, iy, iz;
	unsigned nx, ny, nz;
};
__device__ __forceinline__ RayPair make_pair_ray(const RayPre &r) {
	return {pair2(r.ox, r.ox),
	        pair2(r.oy, r.oy),
	        pair2(r.oz, r.oz),
	        pair2(r.ix, r.ix),
	        pair2(r.iy, r.iy),
	        pair2(r.iz, r.iz),
	        r.ix < 0.0f ? 16u : 0u,
	        r.iy < 0.0f ? 48u : 32u,
	        r.iz < 0.0f ? 80u : 64u};
}

__device__ __forceinline__ void plane4(const char *row, unsigned long long o, unsigned long long i, float t[4]) {
	const ulonglong2 q = __ldg(reinterpret_cast<const ulonglong2 *>(row));
	unpair2(mul2(sub2(q.x, o), i), t[0], t[1]);
	unpair2(mul2(sub2(q.y, o), i), t[2], t[3]);
}

// The reference slab test on a 4-wide node's four boxes: te[k] = tenter, hit[k] = the
// tMax-independent part of the verdict; refs = the entries' node or leaf refs. Valid for
// rays whose inverse direction is finite: then (lo - o) * i and (hi - o) * i round
// monotonically, so the row the direction's sign picks holds the smaller product and the
// reference's min / max of the two is known without computing it (a +0/-0 difference in
// tenter changes no comparison the traversal makes). Absent entries have lo = +inf and
// hi = -inf, which no ray passes.
// The traversal issues close to what the SMs can and spends most of it here. Taking
// the nearer plane by address instead of by six min / max operations a box, and the
// absent entries by their boxes instead of by a count word, leaves 24 packed
// subtractions and products and 16 three-input min / max and compares a node
// (on the 1.31M-triangle scene: 2M unordered rays 2.02 -> 1.92 ms for closest hits and
// 1.08 -> 0.95 ms for any hits, the 1080p x 32 spp frame's closest-hit stage 49.9 -> 47.9
// ms; the box's per-path adjoint of 4 x 384 x 384 x 16 spp 21.4 -> 15.2 ms).
__device__ __forceinline__ void node4_test(const SceneView &s, int node, const RayPair &r, float te[4], bool hit[4],
                                           int4 &refs) {
	const char *nd = reinterpret_cast<const char *>(s.nodes4) + 128 * static_cast<size_t>(node);
	float nx[4], ny[4], nz[4], fx[4], fy[4], fz[4];
	plane4(nd + r.nx, r.ox, r.ix, nx);
	plane4(nd + r.ny, r.oy, r.iy, ny);
	plane4(nd + r.nz, r.oz, r.iz, nz);
	plane4(nd + (r.nx ^ 16u), r.ox, r.ix, fx);
	plane4(nd + (r.ny ^ 16u), r.oy, r.iy, fy);
	plane4(nd + (r.nz ^ 16u), r.oz, r.iz, fz);
	refs = __ldg(reinterpret_cast<const int4 *>(nd + 96));
#pragma unroll
	for (int k = 0; k < 4; k++) {
		te[k] = max3(nx[k], ny[k], nz[k]);
		hit[k] = min3(fx[k], fy[k], fz[k]) >= fmaxf(te[k], 0.0f);
	}
}

__device__ __forceinline__ unsigned long long pack_entry(int ref, float tenter) {
	return (static_cast<unsigned long long>(static_cast<unsigned>(__float_as_int(tenter))) << 32) |
	       static_cast<unsigned>(ref);
}

__device__ __forceinline__ bool finite_inverse(const RayPre &r) {
	const float inf = __int_as_float(0x7f800000);
	return (fabsf(r.ix) < inf) & (fabsf(r.iy) < inf) & (fabsf(r.iz) < inf);
}
// Rays for the 4-wide tree and the triangle list: a finite inverse direction, and a direction
// short enough that no determinant leaves rcp_bounded's range (SceneView::max_dir).
__device__ __forceinline__ bool bounded_ray(const SceneView &s, const RayPre &r) {
	return finite_inverse(r) & (fmaxf(fabsf(r.dx), fmaxf(fabsf(r.dy), fabsf(r.dz))) < s.max_dir);
}

// Traversal stack storage. LocalStack keeps the whole stack in the thread's
// local memory. SharedShortStack keeps the top kN entries in this thread's column
// of a shared-memory array (entry i of thread t at base[i * stride + t]) and
// deeper entries in local memory: the frequent shallow pushes and pops then cost
// one shared-memory access instead of a scattered local-memory access.
template <typename T> struct LocalStack {
	T st[kStack];
	__device__ __forceinline__ void put(int i, T v) { st[i] = v; }
	__device__ __forceinline__ T get(int i) const { return st[i]; }
};
template <typename T, int kN> struct SharedShortStack {
	T *col;
	int stride;
	T spill[kStack - kN];
	__device__ __forceinline__ SharedShortStack(T *column, int stride_) : col(column), stride(stride_) {}
	__device__ __forceinline__ void put(int i, T v) {
		if (i < kN)
			col[i * stride] = v;
		else
			spill[i - kN] = v;
	}
	__device__ __forceinline__ T get(int i) const { return i < kN ? col[i * stride] : spill[i - kN]; }
};

// Closest hit in the reference's order with postponed leaves (speculative traversal,
// Aila & Laine 2009): a lane whose descent reaches a leaf keeps the leaf aside and goes on descending
// until every active lane of the warp holds a leaf, then the warp tests leaves
// together, so more lanes run the triangle tests converged. The result is the
// reference's, bit for bit:
//   * leaves are tested in the reference's order (the waiting leaf precedes the one
//     the descent stops at), with the reference's strict `<`;
//   * interior nodes popped while a leaf waits are pruned against a distance that is
//     at least the reference's at that point (the waiting leaf's hits are not in it
//     yet), so every leaf the reference reaches is reached;
//   * each leaf is tested only if its entry distance is below the best distance
//     when its turn comes -- the reference's pop-time test with the same best, since
//     both have tested the same leaves before it. A leaf the reference never reaches
//     lies under a node the reference pruned, and its entry distance is at least that
//     node's (a child's box lies inside its parent's and the slab arithmetic rounds
//     monotonically), so the same test rejects it.
constexpr int kNoRef = static_cast<int>(0x80000000u); // no leaf ref can take this value

template <class Stack>
__device__ __forceinline__ HitRec trace_closest4_spec(const SceneView &s, const RayPre &r, int ignore, int &err,
                                                      Stack &st) {
	const RayPair r2 = make_pair_ray(r);
	HitRec h;
	h.idx = -1;
	h.rank = 0x7fffffff;
	h.t = __int_as_float(0x7f800000);
	h.u = 0.0f;
	h.v = 0.0f;
	int sp = 0;
	int cur = kNoRef, leaf = kNoRef;
	float cur_te = 0.0f, leaf_te = 0.0f;
	{
		float te;
		if (s.n_tris > 0 &&
		    slab(s.root_lo[0], s.root_hi[0], s.root_lo[1], s.root_hi[1], s.root_lo[2], s.root_hi[2], r, te)) {
			cur = s.root4_ref;
			cur_te = te;
		}
	}
	// next entry of the stack that survives the reference's pop-time test
	auto pop = [&]() {
		while (sp > 0) {
			const unsigned long long e = st.get(--sp);
			const float te = __int_as_float(static_cast<int>(e >> 32));
			if (te < h.t) {
				cur = static_cast<int>(static_cast<unsigned>(e));
				cur_te = te;
				return;
			}
		}
		cur = kNoRef;
	};
	for (;;) {
		// Interior nodes. A leaf reached while another waits ends the loop; so does
		// every active lane holding a leaf.
		while (cur >= 0) {
			if (bad_node(s, cur, true)) {
				err = 1;
				return h;
			}
			float t[4];
			bool b[4];
			int4 rf;
			node4_test(s, cur, r2, t, b, rf);
			if (sp + 3 > kStack) {
				err = 1;
				return h;
			}
			if (b[3])
				st.put(sp++, pack_entry(rf.w, t[3]));
			if (b[2])
				st.put(sp++, pack_entry(rf.z, t[2]));
			if (b[1])
				st.put(sp++, pack_entry(rf.y, t[1]));
			if (b[0] && t[0] < h.t) {
				cur = rf.x;
				cur_te = t[0];
			} else {
				pop();
			}
			if (cur < 0 && cur != kNoRef && leaf == kNoRef) { // keep the leaf aside, descend on
				leaf = cur;
				leaf_te = cur_te;
				pop();
			}
			if (__all_sync(__activemask(), leaf != kNoRef))
				break;
		}
		// Leaves, in the reference's order: the waiting leaf, then the one the descent
		// stopped at (if any).
		if (leaf == kNoRef && cur < 0 && cur != kNoRef) {
			leaf = cur;
			leaf_te = cur_te;
			pop();
		}
		while (leaf != kNoRef) {
			if (leaf_te < h.t) { // the reference's pop-time test, with the current best
				const int start = leaf_start(leaf);
				const int count = leaf_count(leaf);
				if (bad_leaf(s, start, count)) {
					err = 1;
					return h;
				}
				for (int p = start; p < start + count; p++) {
					const float4 *tp = s.tris + 3 * static_cast<size_t>(p);
					const float4 a = __ldg(tp + 0);
					const int ti = __float_as_int(a.w);
					const float4 b = __ldg(tp + 1);
					const float4 c = __ldg(tp + 2);
					float t, u, v;
					if (tri_test<true>(a, b, c, r, t, u, v) && t < h.t && ti != ignore) {
						h.idx = ti;
						h.t = t;
						h.u = u;
						h.v = v;
						h.rank = __float_as_int(c.w);
					}
				}
			}
			leaf = kNoRef;
			if (cur < 0 && cur != kNoRef) {
				leaf = cur;
				leaf_te = cur_te;
				pop();
			}
		}
		if (cur == kNoRef)
			break;
	}
	return h;
}

// Closest hit in the reference's order for lanes with little company (the row streams of the
// bidirectional renderer, where one candidate start in eight is taken): nothing is postponed, and a
// leaf's triangles, up to four at a time, are loaded together and tested as independent
// straight-line work, then merged in leaf order. 120 x 480 x 4 samples over 20 000 random
// triangles: 99.5 -> 73 ms, over a 20 000-triangle sphere 18.4 -> 16.8.
template <class Stack>
__device__ __forceinline__ HitRec trace_closest4_flat(const SceneView &s, const RayPre &r, int ignore, int &err,
                                                      Stack &st) {
	const RayPair r2 = make_pair_ray(r);
	HitRec h;
	h.idx = -1;
	h.rank = 0x7fffffff;
	h.t = __int_as_float(0x7f800000);
	h.u = 0.0f;
	h.v = 0.0f;
	int sp = 0;
	float te;
	if (s.n_tris > 0 && slab(s.root_lo[0], s.root_hi[0], s.root_lo[1], s.root_hi[1], s.root_lo[2], s.root_hi[2], r, te)) {
		st.put(0, pack_entry(s.root4_ref, te));
		sp = 1;
	}
	while (sp > 0) {
		const unsigned long long e = st.get(--sp);
		int ref = static_cast<int>(static_cast<unsigned>(e));
		if (!(__int_as_float(static_cast<int>(e >> 32)) < h.t))
			continue;
		while (ref >= 0) {
			if (bad_node(s, ref, true) || sp + 3 > kStack) {
				err = 1;
				return h;
			}
			float t[4];
			bool b[4];
			int4 rf;
			node4_test(s, ref, r2, t, b, rf);
			if (b[3])
				st.put(sp++, pack_entry(rf.w, t[3]));
			if (b[2])
				st.put(sp++, pack_entry(rf.z, t[2]));
			if (b[1])
				st.put(sp++, pack_entry(rf.y, t[1]));
			ref = b[0] && t[0] < h.t ? rf.x : kNoRef;
		}
		if (ref == kNoRef)
			continue;
		const int start = leaf_start(ref), count = leaf_count(ref);
		if (bad_leaf(s, start, count)) {
			err = 1;
			return h;
		}
		for (int at = 0; at < count; at += 4) {
			float4 ta[4], tb[4], tc[4];
#pragma unroll
			for (int q = 0; q < 4; q++) {
				const float4 *tp = s.tris + 3 * static_cast<size_t>(start + min(at + q, count - 1));
				ta[q] = __ldg(tp + 0);
				tb[q] = __ldg(tp + 1);
				tc[q] = __ldg(tp + 2);
			}
#pragma unroll
			for (int q = 0; q < 4; q++) {
				float t, u, v;
				const bool hit = tri_test<true, true>(ta[q], tb[q], tc[q], r, t, u, v);
				const bool ok = hit & (at + q < count) & (__float_as_int(ta[q].w) != ignore) & (t < h.t);
				h.idx = ok ? __float_as_int(ta[q].w) : h.idx;
				h.t = ok ? t : h.t;
				h.u = ok ? u : h.u;
				h.v = ok ? v : h.v;
				h.rank = ok ? __float_as_int(tc[q].w) : h.rank;
			}
		}
	}
	return h;
}

// ---- one ray by a group of lanes, for scenes of few triangles ----
// A lone ray's traversal is a chain of dependent loads and tests: 5 000 to 20 000 cycles in
// a scene of 36 triangles. Where rays are few, or come one after another, a group of
// kGroup lanes takes each: every lane tests each kGroup-th triangle of the scene's list,
// without a branch, and the group reduces to the hit.
// The result is the reference's: a leaf's ancestors admit every ray that its own box admits
// (rays with a finite inverse direction), so the triangles the reference may test are those
// whose leaf's slab test passes. Of these the smallest t, the earliest in the order among
// equals, is the hit: nothing later can replace it, and its leaf is skipped only if an
// earlier hit lies at or before the leaf's entry distance. That distance is at most t but
// for rounding (a wall's box is as flat as the wall); where another hit falls into the gap,
// the exact traversal decides.
template <int kGroup> __device__ __forceinline__ unsigned group_lanes() {
	return kGroup == 32 ? 0xffffffffu : (1u << (kGroup % 32)) - 1u;
}
constexpr int kListTris = 128; // most triangles of a list (the host's kMaxListTris)

// The list in shared memory, row by row, so that a group's loads are contiguous.
struct TriList {
	float4 row[5][kListTris];
	__device__ __forceinline__ void load(const SceneView &s) {
		for (int i = threadIdx.x; i < 5 * s.n_tris; i += blockDim.x)
			row[i % 5][i / 5] = __ldg(s.list + i);
	}
	// Whether the leaf of triangle j is entered (te) and the triangle hit (t, u, v), with the
	// operations of slab and tri_test and no early exit.
	__device__ __forceinline__ bool test(int j, const RayPre &r, int ignore, float &te, float &t, float &u,
	                                     float &v) const {
		const float4 a = row[0][j], b = row[1][j], c = row[2][j], x = row[3][j], n = row[4][j];
		const float t0x = __fmul_rn(__fsub_rn(b.w, r.ox), r.ix), t1x = __fmul_rn(__fsub_rn(x.y, r.ox), r.ix);
		const float t0y = __fmul_rn(__fsub_rn(c.w, r.oy), r.iy), t1y = __fmul_rn(__fsub_rn(x.z, r.oy), r.iy);
		const float t0z = __fmul_rn(__fsub_rn(x.x, r.oz), r.iz), t1z = __fmul_rn(__fsub_rn(x.w, r.oz), r.iz);
		te = max3(fminf(t0x, t1x), fminf(t0y, t1y), fminf(t0z, t1z));
		const bool in = min3(fmaxf(t0x, t1x), fmaxf(t0y, t1y), fmaxf(t0z, t1z)) >= fmaxf(te, 0.0f);
		const float spx = __fsub_rn(r.ox, a.x), spy = __fsub_rn(r.oy, a.y), spz = __fsub_rn(r.oz, a.z);
		const float A = __fsub_rn(__fmul_rn(-r.dy, c.z), __fmul_rn(c.y, -r.dz));
		const float B = __fsub_rn(__fmul_rn(-r.dy, b.z), __fmul_rn(b.y, -r.dz));
		const float det = __fadd_rn(__fsub_rn(__fmul_rn(-r.dx, n.x), __fmul_rn(b.x, A)), __fmul_rn(c.x, B));
		const float k = rcp_bounded(det);
		const float i01 = __fmul_rn(-A, k), i02 = __fmul_rn(B, k);
		const float i11 = __fmul_rn(__fsub_rn(__fmul_rn(-r.dx, c.z), __fmul_rn(c.x, -r.dz)), k);
		const float i21 = __fmul_rn(-__fsub_rn(__fmul_rn(-r.dx, c.y), __fmul_rn(c.x, -r.dy)), k);
		const float i12 = __fmul_rn(-__fsub_rn(__fmul_rn(-r.dx, b.z), __fmul_rn(b.x, -r.dz)), k);
		const float i22 = __fmul_rn(__fsub_rn(__fmul_rn(-r.dx, b.y), __fmul_rn(b.x, -r.dy)), k);
		u = __fadd_rn(__fadd_rn(__fmul_rn(i01, spx), __fmul_rn(i11, spy)), __fmul_rn(i21, spz));
		v = __fadd_rn(__fadd_rn(__fmul_rn(i02, spx), __fmul_rn(i12, spy)), __fmul_rn(i22, spz));
		t = __fadd_rn(__fadd_rn(__fmul_rn(__fmul_rn(n.x, k), spx), __fmul_rn(__fmul_rn(n.y, k), spy)),
		              __fmul_rn(__fmul_rn(n.z, k), spz));
		// all of them, without a branch
		return in & !(fabsf(det) < 1e-8f) & (u >= 0.0f) & (v >= 0.0f) & (__fadd_rn(u, v) <= 1.0f) & (t > 1e-5f) &
		       (__float_as_int(a.w) != ignore);
	}
};

// Closest hit of each group's ray (the same in all its lanes, which all return the hit).
// Every lane of the warp must call it.
template <int kGroup>
__device__ __forceinline__ HitRec trace_closest_group(const SceneView &s, const TriList &list, const RayPre &r,
                                                      int ignore, int &err) {
	const int lane = threadIdx.x & 31, g = lane % kGroup, base = lane - g;
	unsigned best_t = 0x7f800000u, best_j = 0xffffffffu; // t > 0, so its bits order as it does
	unsigned next_t = 0x7f800000u;                       // this lane's second smallest
	float bte = 0.0f, bu = 0.0f, bv = 0.0f;
	for (int at = 0; at < s.n_tris; at += kGroup) { // the same number of turns in every lane
		const int j = min(at + g, s.n_tris - 1);
		float te, t, u, v;
		const bool ok = list.test(j, r, ignore, te, t, u, v) & (j == at + g);
		const unsigned bits = ok ? static_cast<unsigned>(__float_as_int(t)) : 0x7f800000u;
		const bool better = bits < best_t;
		next_t = min(next_t, better ? best_t : bits);
		best_t = better ? bits : best_t;
		best_j = better ? static_cast<unsigned>(j) : best_j;
		bte = better ? te : bte;
		bu = better ? u : bu;
		bv = better ? v : bv;
	}
	unsigned win_t = best_t, win_j = best_j;
	if constexpr (kGroup == 32) {
		win_t = __reduce_min_sync(0xffffffffu, best_t);
		win_j = __reduce_min_sync(0xffffffffu, best_t == win_t ? best_j : 0xffffffffu);
	} else {
#pragma unroll
		for (int o = kGroup / 2; o > 0; o >>= 1) {
			const unsigned ot = __shfl_xor_sync(0xffffffffu, win_t, o), oj = __shfl_xor_sync(0xffffffffu, win_j, o);
			if (ot < win_t || (ot == win_t && oj < win_j)) {
				win_t = ot;
				win_j = oj;
			}
		}
	}
	const bool hit = win_t != 0x7f800000u;
	const int from = base + static_cast<int>(win_j % kGroup);
	const float entry = __shfl_sync(0xffffffffu, bte, from);
	HitRec h;
	h.t = __int_as_float(static_cast<int>(win_t));
	h.u = __shfl_sync(0xffffffffu, bu, from);
	h.v = __shfl_sync(0xffffffffu, bv, from);
	h.idx = hit ? __float_as_int(list.row[0][win_j % kListTris].w) : -1;
	h.rank = hit ? static_cast<int>(win_j) : 0x7fffffff;
	if (!hit)
		h.u = h.v = 0.0f;
	// another hit, perhaps an earlier one, in the gap before the entry?
	const unsigned other = lane == from ? next_t : best_t;
	const bool gap = hit & (entry > h.t) & (other != 0x7f800000u) & (__int_as_float(static_cast<int>(other)) <= entry);
	const unsigned exact = __ballot_sync(0xffffffffu, gap | !bounded_ray(s, r));
	if (exact & (group_lanes<kGroup>() << base))
		h = trace_closest<kOrderReference>(s, r, ignore, err);
	return h;
}

// Occlusion of each group's ray before tmax (the order does not matter). Every lane of the
// warp must call it.
template <int kGroup>
__device__ __forceinline__ bool trace_any_group(const SceneView &s, const TriList &list, const RayPre &r, float tmax,
                                                int ignore, int &err) {
	const int lane = threadIdx.x & 31, g = lane % kGroup;
	bool any = false;
	if (!bounded_ray(s, r)) {
		any = trace_any(s, r, tmax, ignore, err);
	} else {
		for (int j = g; j < s.n_tris; j += kGroup) {
			float te, t, u, v;
			const bool hit = list.test(j, r, ignore, te, t, u, v);
			any |= hit & (te < tmax) & (t < tmax);
		}
	}
	return (__ballot_sync(0xffffffffu, any) & (group_lanes<kGroup>() << (lane - g))) != 0;
}

// Any hit with postponed leaves (the closest-hit version's scheme): occlusion does not
// depend on the order in which a fixed tree's reachable leaves are tested.
template <class Stack>
__device__ __forceinline__ bool trace_any4_spec(const SceneView &s, const RayPre &r, float tmax, int ignore,
                                                int &err, Stack &st) {
	const RayPair r2 = make_pair_ray(r);
	int sp = 0;
	int cur = kNoRef, leaf = kNoRef;
	float te;
	if (s.n_tris > 0 && slab(s.root_lo[0], s.root_hi[0], s.root_lo[1], s.root_hi[1], s.root_lo[2], s.root_hi[2], r, te) &&
	    te < tmax)
		cur = s.root4_ref;
	auto pop = [&]() { cur = sp > 0 ? st.get(--sp) : kNoRef; };
	for (;;) {
		while (cur >= 0) {
			if (bad_node(s, cur, true)) {
				err = 1;
				return false;
			}
			float t[4];
			bool b[4];
			int4 rf;
			node4_test(s, cur, r2, t, b, rf);
			const bool b0 = b[0] && t[0] < tmax;
			const bool b1 = b[1] && t[1] < tmax;
			const bool b2 = b[2] && t[2] < tmax;
			const bool b3 = b[3] && t[3] < tmax;
			if (sp + 3 > kStack) {
				err = 1;
				return false;
			}
			if (b3)
				st.put(sp++, rf.w);
			if (b2)
				st.put(sp++, rf.z);
			if (b1)
				st.put(sp++, rf.y);
			if (b0)
				cur = rf.x;
			else
				pop();
			if (cur < 0 && cur != kNoRef && leaf == kNoRef) {
				leaf = cur;
				pop();
			}
			if (__all_sync(__activemask(), leaf != kNoRef))
				break;
		}
		if (leaf == kNoRef && cur < 0 && cur != kNoRef) {
			leaf = cur;
			pop();
		}
		while (leaf != kNoRef) {
			const int start = leaf_start(leaf);
			const int count = leaf_count(leaf);
			if (bad_leaf(s, start, count)) {
				err = 1;
				return false;
			}
			for (int p = start; p < start + count; p++) {
				const float4 *tp = s.tris + 3 * static_cast<size_t>(p);
				const float4 a = __ldg(tp + 0);
				const float4 b = __ldg(tp + 1);
				const float4 c = __ldg(tp + 2);
				float t, u, v;
				if (tri_test<true>(a, b, c, r, t, u, v) && t < tmax && __float_as_int(a.w) != ignore)
					return true;
			}
			leaf = kNoRef;
			if (cur < 0 && cur != kNoRef) {
				leaf = cur;
				pop();
			}
		}
		if (cur == kNoRef)
			return false;
	}
}

// ---- streams of rays: a warp whose idle lanes take new rays ----
// The rays of one warp differ in length: with a ray per lane until the warp's last is done,
// 6.7 (unordered rays) and 9.1 (binned rays) of 32 lanes worked per instruction on the
// 1.31M-triangle scene. Here the warp goes round by round (a descent and the leaves it
// gathered, as in the functions above) and, once kStreamRefill lanes are idle, gives each of
// them the next ray; a round's descent ends when fewer than kStreamActive lanes are left in
// it (while there are rays to refill from). The order of a ray's own steps is unchanged.
// 2M unordered closest hits: 1.09 -> 0.88 ms (12.3 lanes), 0.78 with tri_test's straight form;
// without the second rule 0.98, and 0.90 to 0.93 with other numbers of lanes (8 and 12, 8 and
// 20, 12 and 24). Where neighbours already take the same way the exchange costs more than it
// gives: any hits towards one light 0.49 -> 0.48 ms, the wavefront's binned rays 24.7 -> 33 ms
// a frame, a scene of 36 triangles 0.34 -> 0.41 ms.
// source(want, idle, ...) gives every lane with want set its next ray, false if there is none
// (it is called by all lanes; idle is the mask of those that want one); sink takes a finished
// ray's result. Every lane of the warp must call this function; rays that are not
// bounded_ray take the 2-wide tree at once.
constexpr int kStreamRefill = 4, kStreamActive = 16;

// The indices of n entries for a warp's lanes: chunks of kStreamChunk go round the grid's warps in
// turn, so a launch shares no counter with others and neighbours stay in one warp.
constexpr unsigned kStreamChunk = 32;
struct StreamTurns {
	unsigned n, turn, stride;
	unsigned at = 0, end = 0; // what is left of the current chunk
	__device__ __forceinline__ explicit StreamTurns(unsigned n_)
	    : n(n_), turn((blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * kStreamChunk),
	      stride(gridDim.x * (blockDim.x >> 5) * kStreamChunk) {}
	__device__ __forceinline__ bool next(bool want, unsigned idle, unsigned &i) {
		const unsigned lane = threadIdx.x & 31, need = static_cast<unsigned>(__popc(idle)), left = end - at;
		const unsigned k = static_cast<unsigned>(__popc(idle & ((1u << lane) - 1u)));
		i = at + k;
		at += need;
		if (need > left) { // the rest from the next chunk (need is at most a chunk)
			if (k >= left)
				i = turn + (k - left);
			at = min(turn + (need - left), n);
			end = min(turn + kStreamChunk, n);
			turn = min(turn + stride, n);
		}
		return want && i < n;
	}
};

template <class Stack, class Source, class Sink>
__device__ __forceinline__ void trace_closest_stream(const SceneView &s, Stack &st, int &err, Source &&source,
                                                     Sink &&sink) {
	RayPre r;
	RayPair r2;
	HitRec h;
	int ignore = -1, sp = 0, cur = kNoRef, leaf = kNoRef;
	float cur_te = 0.0f, leaf_te = 0.0f;
	bool busy = false, more = true;
	auto pop = [&]() {
		while (sp > 0) {
			const unsigned long long e = st.get(--sp);
			const float te = __int_as_float(static_cast<int>(e >> 32));
			if (te < h.t) {
				cur = static_cast<int>(static_cast<unsigned>(e));
				cur_te = te;
				return;
			}
		}
		cur = kNoRef;
	};
	for (;;) {
		const unsigned idle = __ballot_sync(0xffffffffu, !busy);
		if (more && __popc(idle) >= kStreamRefill) {
			const bool got = source(!busy, idle, r, ignore); // false for lanes that want none
			more = __ballot_sync(0xffffffffu, got) == idle;
			if (got) {
				h.idx = -1;
				h.rank = 0x7fffffff;
				h.t = __int_as_float(0x7f800000);
				h.u = 0.0f;
				h.v = 0.0f;
				sp = 0;
				cur = leaf = kNoRef;
				float te;
				if (!bounded_ray(s, r)) {
					sink(trace_closest<kOrderReference, true>(s, r, ignore, err));
				} else if (slab(s.root_lo[0], s.root_hi[0], s.root_lo[1], s.root_hi[1], s.root_lo[2], s.root_hi[2], r,
				                te)) {
					r2 = make_pair_ray(r);
					cur = s.root4_ref;
					cur_te = te;
					busy = true;
				} else {
					sink(h);
				}
			}
		}
		if (!__any_sync(0xffffffffu, busy)) {
			if (more)
				continue;
			return;
		}
		if (!busy)
			continue;
		while (cur >= 0) {
			if (bad_node(s, cur, true) || sp + 3 > kStack) {
				err = 1;
				cur = leaf = kNoRef;
				sp = 0;
				break;
			}
			float t[4];
			bool b[4];
			int4 rf;
			node4_test(s, cur, r2, t, b, rf);
			if (b[3])
				st.put(sp++, pack_entry(rf.w, t[3]));
			if (b[2])
				st.put(sp++, pack_entry(rf.z, t[2]));
			if (b[1])
				st.put(sp++, pack_entry(rf.y, t[1]));
			if (b[0] && t[0] < h.t) {
				cur = rf.x;
				cur_te = t[0];
			} else {
				pop();
			}
			if (cur < 0 && cur != kNoRef && leaf == kNoRef) {
				leaf = cur;
				leaf_te = cur_te;
				pop();
			}
			const unsigned act = __activemask();
			if (__all_sync(act, leaf != kNoRef) || (more && __popc(act) < kStreamActive))
				break;
		}
		if (leaf == kNoRef && cur < 0 && cur != kNoRef) {
			leaf = cur;
			leaf_te = cur_te;
			pop();
		}
		while (leaf != kNoRef) {
			if (leaf_te < h.t) {
				const int start = leaf_start(leaf);
				const int count = leaf_count(leaf);
				if (bad_leaf(s, start, count)) {
					err = 1;
					cur = kNoRef;
					sp = 0;
					break;
				}
				for (int p = start; p < start + count; p++) {
					const float4 *tp = s.tris + 3 * static_cast<size_t>(p);
					const float4 a = __ldg(tp + 0);
					const int ti = __float_as_int(a.w);
					const float4 b = __ldg(tp + 1);
					const float4 c = __ldg(tp + 2);
					float t, u, v;
					if (tri_test<true, true>(a, b, c, r, t, u, v) && t < h.t && ti != ignore) {
						h.idx = ti;
						h.t = t;
						h.u = u;
						h.v = v;
						h.rank = __float_as_int(c.w);
					}
				}
			}
			leaf = kNoRef;
			if (cur < 0 && cur != kNoRef) {
				leaf = cur;
				leaf_te = cur_te;
				pop();
			}
		}
		if (cur == kNoRef) {
			sink(h);
			busy = false;
		}
	}
}

// ---- resumable 4-wide traversal for persistent kernels that replace finished rays ----
// The reference's visit order and tests, cut into steps
// (one pop, a descent through internal nodes, one leaf) so that a warp can hand
// a new ray to every lane whose ray has finished between steps.
constexpr int kPopRef = static_cast<int>(0x80000000u); // no leaf ref can take this value

struct TravState {
	RayPre r;
	RayPair r2;
	HitRec h;
	float tmax; // any-hit bound (closest hit: unused)
	int ignore;
	int cur;    // node (>= 0), leaf (< 0), or kPopRef
	int sp;
	bool hit_any;
	unsigned long long st[kStack];
};

// Start a ray with the root box test.
template <bool kAny>
__device__ __forceinline__ void trav_begin(TravState &ts, const SceneView &s, const RayPre &r, float tmax, int ignore) {
	ts.r = r;
	ts.r2 = make_pair_ray(r);
	ts.h.idx = -1;
	ts.h.rank = 0x7fffffff;
	ts.h.t = __int_as_float(0x7f800000);
	ts.h.u = ts.h.v = 0.0f;
	ts.tmax = tmax;
	ts.ignore = ignore;
	ts.hit_any = false;
	ts.sp = 0;
	ts.cur = kPopRef;
	float te;
	if (s.n_tris > 0 && slab(s.root_lo[0], s.root_hi[0], s.root_lo[1], s.root_hi[1], s.root_lo[2], s.root_hi[2], r, te) &&
	    (!kAny || te < tmax)) {
		ts.st[0] = pack_entry(s.root4_ref, te);
		ts.sp = 1;
	}
}

// One step; returns false once the ray is finished.
template <bool kAny>
__device__ __forceinline__ bool trav_step(TravState &ts, const SceneView &s, int &err) {
	const float bound = kAny ? ts.tmax : ts.h.t;
	if (ts.cur == kPopRef) {
		if (ts.sp == 0)
			return false;
		const unsigned long long e = ts.st[--ts.sp];
		if (!kAny && !(__int_as_float(static_cast<int>(e >> 32)) < bound))
			return true;
		ts.cur = static_cast<int>(static_cast<unsigned>(e));
	}
	while (ts.cur >= 0) {
		if (bad_node(s, ts.cur, true)) {
			err = 1;
			return false;
		}
		float t[4];
		bool b[4];
		int4 rf;
		node4_test(s, ts.cur, ts.r2, t, b, rf);
		const float bd = kAny ? ts.tmax : ts.h.t;
		const bool b0 = b[0] && t[0] < bd;
		const bool b1 = b[1] && (!kAny || t[1] < bd);
		const bool b2 = b[2] && (!kAny || t[2] < bd);
		const bool b3 = b[3] && (!kAny || t[3] < bd);
		if (ts.sp + 3 > kStack) {
			err = 1;
			return false;
		}
		if (b3)
			ts.st[ts.sp++] = pack_entry(rf.w, t[3]);
		if (b2)
			ts.st[ts.sp++] = pack_entry(rf.z, t[2]);
		if (b1)
			ts.st[ts.sp++] = pack_entry(rf.y, t[1]);
		if (!b0) {
			ts.cur = kPopRef;
			return true;
		}
		ts.cur = rf.x;
	}
	// Leaf.
	const int start = leaf_start(ts.cur);
	const int count = leaf_count(ts.cur);
	if (bad_leaf(s, start, count)) {
		err = 1;
		return false;
	}
	ts.cur = kPopRef;
	for (int p = start; p < start + count; p++) {
		const float4 *tp = s.tris + 3 * static_cast<size_t>(p);
		const float4 a = __ldg(tp + 0);
		const int ti = __float_as_int(a.w);
		if (ti == ts.ignore)
			continue;
		const float4 bb = __ldg(tp + 1);
		const float4 c = __ldg(tp + 2);
		float t, u, v;
		if (!tri_test<true>(a, bb, c, ts.r, t, u, v))
			continue;
		if (kAny) {
			if (t < ts.tmax) {
				ts.hit_any = true;
				return false;
			}
		} else if (t < ts.h.t) {
			ts.h.idx = ti;
			ts.h.t = t;
			ts.h.u = u;
			ts.h.v = v;
			ts.h.rank = __float_as_int(c.w);
		}
	}
	return true;
}

// Closest hit / occlusion with the fastest form that keeps the reference result: the
// 4-wide speculative traversals (postponed leaves) for rays with a finite inverse
// direction, else the 2-wide reference traversal. Measured on the 1.31M-triangle
// 1080p frame, postponing leaves took the closest-hit stage from 118.2 to 105.2 ms
// and the any-hit stage from 40.3 to 36.6 ms, images unchanged.
template <int kOrder>
__device__ __forceinline__ HitRec trace_closest_best(const SceneView &s, const RayPre &r, int ignore, int &err) {
	if (kOrder == kOrderReference && s.nodes4 && bounded_ray(s, r)) {
		LocalStack<unsigned long long> st;
		return trace_closest4_spec(s, r, ignore, err, st);
	}
	return trace_closest<kOrder>(s, r, ignore, err);
}

__device__ __forceinline__ bool trace_any_best(const SceneView &s, const RayPre &r, float tmax, int ignore, int &err) {
	if (s.nodes4 && bounded_ray(s, r)) {
		LocalStack<int> st;
		return trace_any4_spec(s, r, tmax, ignore, err, st);
	}
	return trace_any(s, r, tmax, ignore, err);
}

// The same with caller-provided stack storage for the 4-wide traversals.
template <int kOrder, class Stack>
__device__ __forceinline__ HitRec trace_closest_best(const SceneView &s, const RayPre &r, int ignore, int &err,
                                                     Stack &st) {
	if (kOrder == kOrderReference && s.nodes4 && bounded_ray(s, r))
		return trace_closest4_spec(s, r, ignore, err, st);
	return trace_closest<kOrder>(s, r, ignore, err);
}
template <class Stack>
__device__ __forceinline__ bool trace_any_best(const SceneView &s, const RayPre &r, float tmax, int ignore, int &err,
                                               Stack &st) {
	if (s.nodes4 && bounded_ray(s, r))
		return trace_any4_spec(s, r, tmax, ignore, err, st);
	return trace_any(s, r, tmax, ignore, err);
}

// Instrumented emulation of the reference traversal (src/BVH.cpp:77-139) for
// the algorithmic-bytes counters: both children are pushed and each node's box
// test is counted when it is popped, exactly as the reference does it, so
// `boxes` and `tris` are the reference's test counts for this ray. Closest-hit
// mode (kAny = false) returns the reference's hit in `h`; any-hit mode returns
// the occlusion flag.
template <bool kAny>
__device__ bool count_reference_query(const SceneView &s, const RayPre &r, int ignore, float tmax, HitRec &h,
                                      unsigned long long &boxes, unsigned long long &tris, int &err) {
	int st_ref[kStack];
	float st_te[kStack];
	int sp = 0;
	float best = kAny ? tmax : __int_as_float(0x7f800000);
	h.idx = -1;
	h.rank = 0;
	h.t = best;
	h.u = h.v = 0.0f;
	if (s.n_tris <= 0)
		return false;
	float te;
	const bool ok = slab(s.root_lo[0], s.root_hi[0], s.root_lo[1], s.root_hi[1], s.root_lo[2], s.root_hi[2], r, te);
	st_ref[0] = s.root_ref;
	st_te[0] = ok ? te : __int_as_float(0x7fc00000); // NaN never passes te < best
	sp = 1;
	while (sp > 0) {
		--sp;
		const int ref = st_ref[sp];
		const float tent = st_te[sp];
		boxes++;
		if (!(tent < best))
			continue;
		if (ref < 0) {
			const int start = leaf_start(ref);
			const int count = leaf_count(ref);
			if (bad_leaf(s, start, count)) {
				err = 1;
				return false;
			}
			for (int p = start; p < start + count; p++) {
				const float4 *tp = s.tris + 3 * static_cast<size_t>(p);
				const float4 a = __ldg(tp + 0);
				const int ti = __float_as_int(a.w);
				if (ti == ignore)
					continue;
				tris++;
				const float4 b = __ldg(tp + 1);
				const float4 c = __ldg(tp + 2);
				float t, u, v;
				if (tri_test(a, b, c, r, t, u, v) && t < best) {
					if (kAny)
						return true;
					best = t;
					h.idx = ti;
					h.t = t;
					h.u = u;
					h.v = v;
					h.rank = __float_as_int(c.w);
				}
			}
			continue;
		}
		if (sp + 2 > kStack) {
			err = 1;
			return false;
		}
		if (bad_node(s, ref, false)) {
			err = 1;
			return false;
		}
		const float4 *nd = s.nodes + 4 * static_cast<size_t>(ref);
		const float4 n0 = __ldg(nd + 0), n1 = __ldg(nd + 1), n2 = __ldg(nd + 2), n3 = __ldg(nd + 3);
		float tl, tr;
		const bool hl = slab(n0.x, n0.y, n0.z, n0.w, n2.x, n2.y, r, tl);
		const bool hr = slab(n1.x, n1.y, n1.z, n1.w, n2.z, n2.w, r, tr);
		st_ref[sp] = __float_as_int(n3.x);
		st_te[sp] = hl ? tl : __int_as_float(0x7fc00000);
		st_ref[sp + 1] = __float_as_int(n3.y);
		st_te[sp + 1] = hr ? tr : __int_as_float(0x7fc00000);
		sp += 2;
	}
	return false;
}

#endif // __CUDACC__

} // namespace rnb
