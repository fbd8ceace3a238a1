// Host-side scene representation, reference-identical BVH build and the
// flattening of that BVH into the device layout read by the CUDA kernels.
#pragma once

#include <cstdint>
#include <future>
#include <string>
#include <system_error>
#include <type_traits>
#include <utility>
#include <vector>

namespace rnb {

// Surface responses of the reference renderer, same order as its Material enum
// (framework/ModelTriangle.h:12-24).
enum RefMaterial : int {
	kRefDiffuse = 0,
	kRefMirror = 1,
	kRefGlass = 2,
	kRefProcedural = 3,
	kRefBump = 4,
	kRefParallax = 5,
	kRefMetal = 6,
	kRefDispersive = 7,
	kRefSubsurface = 8,
	kRefNormalMap = 9,
	kRefEmissive = 10,
};

// Physical-mode BSDFs (the additive path-tracing API).
enum PhysMaterial : int { kLambert = 0, kGGX = 1, kDielectric = 2 };

struct Vec3 {
	float x, y, z;
};

// Triangle list in structure-of-arrays form. `v` holds 9 floats per triangle.
// The reference fields (rgb/material/roughness/normal) drive the drop-in
// reference-mode renderer; the physical fields drive the additive API.
struct TriangleSet {
	std::vector<float> v;           // 9 per triangle: v0, v1, v2
	std::vector<int> rgb;           // 3 per triangle, reference Colour 0..255
	std::vector<int> ref_material;  // reference Material code
	std::vector<float> roughness;   // reference Metal roughness (default 0.2)
	std::vector<float> normal;      // 3 per triangle, face normal as the loader computes it
	std::vector<float> vnormal;     // 9 per triangle, vertex normals (ModelTriangle::vertexNormals)
	std::vector<float> albedo;      // 3 per triangle (physical mode)
	std::vector<float> emission;    // 3 per triangle (physical mode, Le)
	std::vector<int> phys_material; // PhysMaterial
	std::vector<float> phys_param;  // GGX alpha or dielectric IOR
	size_t size() const { return v.size() / 9; }
};

// Reference BVH node (src/BVH.h:22-26): box, children or a leaf range in `order`.
struct BvhNode {
	Vec3 bmin, bmax;
	int left = -1, right = -1;
	int start = 0, count = 0;
};

struct Bvh2 {
	std::vector<int> order;
	std::vector<BvhNode> nodes;
	int root = -1;
	int depth = 0; // maximum root-to-leaf depth (root = 1)
};

// Median-split build with leaves of <= 4 triangles, identical node order and
// triangle order to the reference (src/BVH.cpp:6-63).
void build_reference_bvh(const float *v9, int n, Bvh2 &out);

// Face normal as the reference OBJ loader computes it (src/ObjLoader.cpp:170-176).
Vec3 loader_face_normal(const float *v9);

// Unit geometric normal cross(v1 - v0, v2 - v0) (computed in double, rounded
// once), (0, 0, 0) for a degenerate triangle; and the triangle's area.
Vec3 geometric_normal(const float *v9);
double triangle_area(const float *v9);

// Wavefront OBJ/MTL loader with the reference loader's semantics
// (src/ObjLoader.cpp:23-214): `v` scaled by `scale`, first three face tokens,
// `usemtl` name -> Material mapping and Kd colour as int(Kd*255).
bool load_obj(const std::string &path, float scale, TriangleSet &out, std::string &err);

// Device layout of a flattened reference BVH.
//  nodes: 4 float4 per internal node ("child pair" node):
//     n0 = (L.lo.x, L.hi.x, L.lo.y, L.hi.y)
//     n1 = (R.lo.x, R.hi.x, R.lo.y, R.hi.y)
//     n2 = (L.lo.z, L.hi.z, R.lo.z, R.hi.z)
//     n3 = (ref L, ref R, -, -) as int bits
//  child ref >= 0: dense internal node index; ref < 0: leaf ~((start << 3) | count)
//  tris: 3 float4 per triangle position in leaf order:
//     (v0.xyz, original index), (e1.x, e0.x, e1.y, e0.y),
//     (e1.z, e0.z, e0.y * e1.z - e1.y * e0.z, rank), e0 = v1 - v0, e1 = v2 - v0
//  rank = position of the triangle in the reference's static traversal order
//  (leaves visited right child first, triangles ascending within a leaf).
struct F4 {
	float x, y, z, w;
};
struct DeviceLayout {
	std::vector<F4> nodes;
	std::vector<F4> tris;
	float root_lo[3], root_hi[3];
	int root_ref = 0;
	int internal_count = 0;
	int depth = 0;
};
void flatten_bvh(const TriangleSet &ts, const Bvh2 &bvh, DeviceLayout &out);

// Four-wide collapse of a binary tree for the fast traversal. A node holds two to four entries,
// a frontier of descendants of one binary node, in the order the reference pops them; which
// descendants is chosen bottom-up by an area-weighted fetch cost. refs are int bits (>= 0
// node, < 0 leaf as in the 2-wide layout).
// Because float subtraction and multiplication round monotonically, a descendant's slab
// interval lies inside its ancestor's, so skipping an ancestor's test never admits a leaf the
// reference would prune (rays with an infinite 1/d component excepted: those
// use the 2-wide layout).
// Node rows: [2a] = lo_a[4], [2a+1] = hi_a[4] for axis a = x, y, z (an absent entry's
// box is empty: lo = +inf, hi = -inf); [6] = refs[4]; [7] = (count, 0, 0, 0).
struct DeviceLayout4 {
	std::vector<F4> nodes;
	int root_ref = 0; // node index, or a leaf ref when the reference root is a leaf
};
void flatten_bvh4(const Bvh2 &bvh, DeviceLayout4 &out);
// Most entries the 4-wide traversals' stack holds at once on this layout.
int stack_need4(const DeviceLayout4 &layout);

// Another tree over the reference tree's leaves, in the same order (a leaf met before another
// in the reference's traversal is met before it here): every range of the leaf sequence
// splits where the surface area heuristic is least. The traversals test a leaf by its own
// box when its turn comes and their boxes above it only skip leaves it would fail, so closest
// hits and occlusion are the reference's on any such tree.
// The reference splits at the median centroid, so a few triangles much larger than the rest
// (a room's walls around a mesh) inflate every box above their leaves, down to the finest;
// here they leave the ranges around them early. On the 1.31M-triangle sphere in its room, with
// the collapse below: 2M unordered rays 1.72 -> 1.09 ms for closest hits and 0.97 -> 0.49 for
// any hits, the 1080p x 32 spp frame 84.6 -> 47.9 ms, the drop-in's 1080p frame 19.2 -> 10.6.
// It costs 1.5 to 3 times the collapse of the reference's own shape (5 000 triangles 0.1 -> 0.3 ms
// of one core, 1.31M 78 -> 160), from 2 000 triangles on beside the reference layout's arrays;
// with the reference tree built on more threads than before, preparing takes 1.8 -> 1.5 ms (5 000
// triangles), 4.5 -> 2.7 (15 000), 27 -> 23 (150 000) and 251 -> 218 (1.31M).
// bvh must be the reference tree; out keeps its triangle order.
void split_by_area(const Bvh2 &bvh, Bvh2 &out);

// The triangles of a small scene in the static traversal order, each with its leaf's box and
// the cofactors of its edges, rounded as the triangle test rounds them: (v0, index),
// (e0, lo.x), (e1, lo.y), (lo.z, hi.x, hi.y, hi.z), (e0.y e1.z - e1.y e0.z,
// -(e0.x e1.z - e1.x e0.z), e0.x e1.y - e1.x e0.y, 0). Empty above kMaxListTris.
constexpr int kMaxListTris = 128;
void list_triangles(const TriangleSet &ts, const Bvh2 &bvh, std::vector<F4> &out);

// f() on a thread of its own if `beside` is set and the system gives one, else when the future is
// asked for its result.
template <class F> std::future<std::invoke_result_t<F>> run_beside(bool beside, F f) {
	if (beside) {
		try {
			return std::async(std::launch::async, f);
		} catch (const std::system_error &) {
		}
	}
	return std::async(std::launch::deferred, std::move(f));
}

} // namespace rnb
