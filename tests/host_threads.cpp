// The host's tree builds where the system gives few threads or none: pthread_create, as these
// functions see it, fails from the n-th call on. The trees are those of a system that gives all
// it is asked for.
#include <dlfcn.h>
#include <pthread.h>

#include <atomic>
#include <cerrno>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include "host_scene.hpp"

using namespace rnb;

static std::atomic<int> g_left{1 << 30}, g_refused{0};

extern "C" int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*f)(void *), void *arg) {
	using Fn = int (*)(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *);
	if (g_left.fetch_sub(1) <= 0) {
		g_refused++;
		return EAGAIN;
	}
	return reinterpret_cast<Fn>(dlsym(RTLD_NEXT, "pthread_create"))(t, a, f, arg);
}

static bool same(const Bvh2 &a, const Bvh2 &b) {
	return a.root == b.root && a.depth == b.depth && a.order == b.order && a.nodes.size() == b.nodes.size() &&
	       std::memcmp(a.nodes.data(), b.nodes.data(), a.nodes.size() * sizeof(BvhNode)) == 0;
}

int main() {
	constexpr int kTris = 300000; // enough for threads in both builds
	std::mt19937 rng(3);
	std::uniform_real_distribution<float> u(-1.0f, 1.0f);
	std::vector<float> v(9 * static_cast<size_t>(kTris));
	for (int i = 0; i < kTris; i++) {
		const float c[3] = {u(rng), u(rng), u(rng)};
		for (size_t k = 0; k < 9; k++)
			v[9 * static_cast<size_t>(i) + k] = c[k % 3] + 0.02f * u(rng);
	}
	Bvh2 want, want_area;
	build_reference_bvh(v.data(), kTris, want);
	split_by_area(want, want_area);
	for (int allowed : {0, 1, 2, 5}) {
		g_left = allowed;
		g_refused = 0;
		Bvh2 ref, area;
		build_reference_bvh(v.data(), kTris, ref);
		g_left = allowed;
		split_by_area(want, area);
		auto beside = run_beside(true, [] { return 7; });
		if (!same(ref, want) || !same(area, want_area) || beside.get() != 7 || g_refused == 0) {
			std::printf("failed with %d threads\n", allowed);
			return 1;
		}
	}
	std::printf("thread checks passed\n");
	return 0;
}
