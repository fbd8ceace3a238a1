// The tree over the reference's leaves (split_by_area) and its 4-wide collapse, on scenes of
// even, mixed and exponentially growing triangles: the leaves and their order are the
// reference's, every box contains the boxes below it, and a walk of the 4-wide layout that
// enters every box never holds more than stack_need4 entries.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include "host_scene.hpp"

using namespace rnb;

static int g_fail = 0;
#define CHECK(c)                                                                                                       \
	do {                                                                                                               \
		if (!(c)) {                                                                                                    \
			std::printf("check failed: %s (line %d)\n", #c, __LINE__);                                                 \
			g_fail = 1;                                                                                                \
		}                                                                                                              \
	} while (0)

static std::vector<int> leaf_order(const Bvh2 &b) {
	std::vector<int> out, st{b.root};
	while (!st.empty()) {
		const BvhNode &n = b.nodes[static_cast<size_t>(st.back())];
		st.pop_back();
		if (n.count > 0) {
			out.push_back((n.start << 3) | n.count);
		} else {
			st.push_back(n.left);
			st.push_back(n.right);
			for (int c : {n.left, n.right}) {
				const BvhNode &k = b.nodes[static_cast<size_t>(c)];
				CHECK(k.bmin.x >= n.bmin.x && k.bmin.y >= n.bmin.y && k.bmin.z >= n.bmin.z);
				CHECK(k.bmax.x <= n.bmax.x && k.bmax.y <= n.bmax.y && k.bmax.z <= n.bmax.z);
			}
		}
	}
	return out;
}

static void check(const std::vector<float> &v) {
	Bvh2 ref, tree;
	build_reference_bvh(v.data(), static_cast<int>(v.size() / 9), ref);
	split_by_area(ref, tree);
	const std::vector<int> want = leaf_order(ref);
	CHECK(leaf_order(tree) == want);
	DeviceLayout4 l4;
	flatten_bvh4(tree, l4);
	const int need = stack_need4(l4);
	std::vector<int> got, st{l4.root_ref};
	size_t most = 1;
	while (!st.empty()) {
		const int r = st.back();
		st.pop_back();
		if (r < 0) {
			got.push_back(~r);
			continue;
		}
		const F4 *o = &l4.nodes[8 * static_cast<size_t>(r)];
		int refs[4], cnt;
		std::memcpy(refs, &o[6], sizeof(refs));
		std::memcpy(&cnt, &o[7].x, sizeof(cnt));
		CHECK(cnt >= 2 && cnt <= 4);
		CHECK(static_cast<int>(st.size()) + 3 <= need); // the traversals' check before they push
		for (int k = cnt; k-- > 0;)
			st.push_back(refs[k]);
		most = std::max(most, st.size() - 1); // the first entry is descended into at once
	}
	CHECK(got == want);
	CHECK(static_cast<int>(most) <= need);
}

int main() {
	std::mt19937 rng(7);
	std::uniform_real_distribution<float> u(-1.0f, 1.0f);
	for (int n : {1, 4, 5, 9, 64, 1000, 20000})
		for (int kind = 0; kind < 4; kind++) {
			std::vector<float> v(9 * static_cast<size_t>(n));
			for (int i = 0; i < n; i++) {
				// even sizes; a few triangles as large as the scene; sizes and places that grow by
				// halves (chains); all in one place
				const float at = kind == 2 ? std::pow(1.5f, static_cast<float>(i % 150)) : 1.0f;
				const float size = kind == 1 && i % 37 == 0 ? 3.0f : kind == 2 ? at : 0.02f;
				const float c[3] = {u(rng) * at, u(rng) * at, u(rng) * at};
				for (int k = 0; k < 9; k++)
					v[9 * static_cast<size_t>(i) + static_cast<size_t>(k)] = kind == 3 ? 0.25f * static_cast<float>(k % 4)
					                                                                  : c[k % 3] + size * u(rng);
			}
			check(v);
		}
	if (g_fail == 0)
		std::printf("tree checks passed\n");
	return g_fail;
}
