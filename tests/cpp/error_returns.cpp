// error_returns.cpp - scene creation and builds made to fail at every allocation and at every queued operation
// in turn: the call reports the failure, frees nothing that queued work uses, and the scene's buffers are all
// gone once it is destroyed.  Prints one line per failure of the test.
#include <cstdio>
#include <cstring>
#include <vector>

#include "../../include/mrt_cuda.h"
#include "fake_cuda.h"

static int bad = 0;
#define CHECK(cond, ...) do { if (!(cond)) { ++bad; printf(__VA_ARGS__); printf("  [%s]\n", #cond); } } while (0)

static std::vector<float> tris(uint32_t n) {
    std::vector<float> t(9ull * n);
    for (size_t i = 0; i < t.size(); ++i) t[i] = (float)((i * 7919u) % 1000u) * 1e-3f;
    return t;
}

// collapse counters that never run out: the build meets its limit of tree levels with launches in flight
static void endless_levels(void *dst, size_t bytes) {
    if (bytes != 292) return;
    for (int k = 4; k < 73; ++k) static_cast<uint32_t *>(dst)[k] = 1;
}

int main() {
    MrtContext *ctx = nullptr;
    if (mrt_context_create(0, &ctx) != MRT_OK) return printf("no context\n"), 1;
    const uint32_t n = 500;
    const std::vector<float> t = tris(n);
    const std::vector<int32_t> m(n, 0);
    MrtMaterial mat{};
    MrtLightDesc lights[2]{};
    lights[1].kind = MRT_LIGHT_AREA;
    const float sphere[4] = {0, 0, 0, 1}, plane[6] = {0, 0, 0, 0, 1, 0};
    MrtSceneDesc d{};
    d.n_triangles = n;
    d.tri_abc = d.tri_normals = d.tri_colors = t.data();
    d.tri_material = m.data();
    d.n_spheres = d.n_planes = d.n_materials = 1;
    d.sphere_center_radius = sphere;
    d.plane_point_normal = plane;
    d.materials = &mat;
    d.n_lights = 2;
    d.lights = lights;
    const size_t held = fake::live_buffers();

    // an unknown light kind is refused before anything is queued
    fake::reset();
    lights[1].kind = 7;
    MrtScene *s = nullptr;
    CHECK(mrt_scene_create(ctx, &d, &s) == MRT_ERR_ARG, "light kind");
    CHECK(fake::operations == 0 && fake::violations == 0 && fake::live_buffers() == held, "light kind");
    CHECK(strstr(mrt_context_error(ctx), "light kind"), "light kind: %s", mrt_context_error(ctx));
    lights[1].kind = MRT_LIGHT_AREA;

    const struct { const char *name; MrtAccelOpts o; } builds[] = {
        {"fast", {MRT_ACCEL_BVH, MRT_BVH_FAST}},
        {"reference", {MRT_ACCEL_BVH, MRT_BVH_REFERENCE}},
        {"grid", {MRT_ACCEL_REGULAR_GRID, 0, 12}},
        {"naive", {MRT_ACCEL_NAIVE}},
    };
    for (const auto &b : builds)
        for (int rebuild = 0; rebuild < 2; ++rebuild)
            for (int what = 0; what < 2; ++what)
                for (uint64_t k = 0;; ++k) {
                    fake::reset();
                    if (!rebuild) (what ? fake::fail_operations_from : fake::fail_allocations_from) = k;
                    int st = mrt_scene_create(ctx, &d, &s);
                    if (st == MRT_OK && rebuild) {
                        mrt_scene_build(s, &b.o);
                        CHECK(fake::violations == 0, "%s first build", b.name);
                        fake::allocations = fake::operations = 0;
                        (what ? fake::fail_operations_from : fake::fail_allocations_from) = k;
                    }
                    const bool created = st == MRT_OK;
                    if (created) st = mrt_scene_build(s, &b.o);
                    const bool failed = fake::failed != 0;
                    CHECK(fake::violations == 0, "%s %d %d %llu", b.name, rebuild, what, (unsigned long long)k);
                    CHECK(!failed || st != MRT_OK, "%s %d %d %llu: failure not reported", b.name, rebuild, what, (unsigned long long)k);
                    fake::fail_allocations_from = fake::fail_operations_from = ~0ull;
                    if (created) mrt_scene_destroy(s);
                    CHECK(fake::violations == 0, "%s %d %d %llu destroy", b.name, rebuild, what, (unsigned long long)k);
                    CHECK(fake::live_buffers() == held, "%s %d %d %llu: buffers left", b.name, rebuild, what, (unsigned long long)k);
                    if (!failed) break;
                }

    fake::reset();
    CHECK(mrt_scene_create(ctx, &d, &s) == MRT_OK, "create");
    fake::on_copy_out = endless_levels;
    CHECK(mrt_scene_build(s, &builds[0].o) == MRT_ERR_LIMIT, "level limit");
    CHECK(fake::violations == 0, "level limit");
    mrt_scene_destroy(s);
    mrt_context_destroy(ctx);
    CHECK(fake::violations == 0 && fake::live_buffers() == 0, "context");
    if (!bad) printf("ok\n");
    return bad != 0;
}
