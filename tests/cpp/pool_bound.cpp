// pool_bound.cpp - whatever frees buffers of the device's pool leaves at most 1 GiB unused in it: a batch that is
// destroyed, a build that fails, scratch that grows, a context that goes while another stays.
#include <cstdio>
#include <vector>

#include "../../include/mrt_cuda.h"
#include "fake_cuda.h"

static int bad = 0;
#define CHECK(cond, ...) do { if (!(cond)) { ++bad; printf(__VA_ARGS__); printf("  [%s]\n", #cond); } } while (0)
constexpr uint64_t kKeep = 1ull << 30;

static uint64_t unused() { return fake::pool_reserved - fake::pool_used(); }

int main() {
    MrtContext *ctx = nullptr;
    if (mrt_context_create(0, &ctx) != MRT_OK) return printf("no context\n"), 1;

    // four pipelines of 9 buffers, the largest of them 250 MB each
    MrtBatchOpts bo{};
    bo.max_wave_roots = bo.wave_roots = 150000;
    bo.pipelines = 4;
    MrtBatch *b = nullptr;
    CHECK(mrt_batch_create(ctx, &bo, &b) == MRT_OK, "batch");
    CHECK(fake::pool_used() > kKeep + (kKeep >> 2), "the batch takes %llu bytes", (unsigned long long)fake::pool_used());
    mrt_batch_destroy(b);
    CHECK(unused() <= kKeep, "after a batch: %llu", (unsigned long long)unused());

    // a build that runs out of memory in its last allocation
    const uint32_t n = 7900000;
    std::vector<float> t(9ull * n, 1.0f);
    MrtSceneDesc d{};
    d.n_triangles = n;
    d.tri_abc = t.data();
    MrtScene *s = nullptr;
    CHECK(mrt_scene_create(ctx, &d, &s) == MRT_OK, "scene");
    const MrtAccelOpts fast{MRT_ACCEL_BVH, MRT_BVH_FAST};
    fake::reset();
    mrt_scene_build(s, &fast);   // (fails: kernels do nothing here)
    CHECK(unused() <= kKeep, "after a failed build: %llu", (unsigned long long)unused());
    mrt_scene_destroy(s);
    CHECK(unused() <= kKeep, "after a scene: %llu", (unsigned long long)unused());

    // contexts with 300 MB of scratch each
    const uint32_t n_rays = 6000000;
    std::vector<MrtRay> rays(n_rays);
    std::vector<MrtHit> hits(n_rays);
    MrtContext *others[4];
    for (MrtContext *&c : others) {
        CHECK(mrt_context_create(0, &c) == MRT_OK, "context");
        MrtSceneDesc none{};
        const MrtAccelOpts naive{MRT_ACCEL_NAIVE};
        CHECK(mrt_scene_create(c, &none, &s) == MRT_OK && mrt_scene_build(s, &naive) == MRT_OK, "empty scene");
        for (uint32_t k : {n_rays / 2, n_rays})
            CHECK(mrt_trace_closest(s, rays.data(), k, hits.data(), MRT_MEM_HOST) == MRT_OK, "rays");
        CHECK(unused() <= kKeep, "scratch that grows: %llu", (unsigned long long)unused());
        mrt_scene_destroy(s);
    }
    for (MrtContext *c : others) {
        mrt_context_destroy(c);
        CHECK(unused() <= kKeep, "after a context: %llu", (unsigned long long)unused());
    }
    mrt_context_destroy(ctx);
    CHECK(fake::pool_reserved == 0, "after the last context: %llu", (unsigned long long)fake::pool_reserved);
    if (!bad) printf("ok\n");
    return bad != 0;
}
