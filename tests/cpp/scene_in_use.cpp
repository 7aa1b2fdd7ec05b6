// scene_in_use.cpp - a scene destroyed or rebuilt while a batch's waves read it, and batches that fail to be
// created: no buffer is freed under queued work.
#include <cstdio>
#include <vector>

#include "../../include/mrt_cuda.h"
#include "fake_cuda.h"

static int bad = 0;
#define CHECK(cond, ...) do { if (!(cond)) { ++bad; printf(__VA_ARGS__); printf("  [%s]\n", #cond); } } while (0)

constexpr uint32_t n_tri = 3;
// the collapse counters of a whole tree of one node
static void whole_tree(void *dst, size_t bytes) {
    if (bytes == 292) static_cast<uint32_t *>(dst)[2] = n_tri;
}

int main() {
    MrtContext *ctx = nullptr;
    if (mrt_context_create(0, &ctx) != MRT_OK) return printf("no context\n"), 1;
    float t[9 * n_tri];
    for (int k = 0; k < 9 * (int)n_tri; ++k) t[k] = (float)(k * 7 % 11);
    MrtSceneDesc d{};
    d.n_triangles = n_tri;
    d.tri_abc = t;
    const MrtAccelOpts fast{MRT_ACCEL_BVH, MRT_BVH_FAST};
    MrtBatchOpts bo{};
    bo.wave_roots = bo.max_wave_roots = 1024;
    bo.block_threads = 128;
    bo.blocks_per_sm = 8;
    bo.pipelines = 2;
    bo.no_graph = 1;
    bo.kernel = MRT_BATCH_KERNEL_WAVEFRONT;
    std::vector<uint32_t> image(64 * 64);
    for (int rebuild = 0; rebuild < 2; ++rebuild)
        for (uint32_t waves = 1; waves <= 4; ++waves) {   // the job takes four
            fake::reset();
            fake::on_copy_out = whole_tree;
            MrtScene *s = nullptr;
            MrtBatch *b = nullptr;
            CHECK(mrt_scene_create(ctx, &d, &s) == MRT_OK && mrt_scene_build(s, &fast) == MRT_OK, "scene");
            CHECK(mrt_batch_create(ctx, &bo, &b) == MRT_OK, "batch");
            MrtBatchJob job{};
            job.scene = s;
            job.camera = MrtCamera{MRT_CAMERA_PERSPECTIVE, {0, 0, -3}, {0, 0, 0}, {0, 1, 0}, 45, 45};
            job.opts.shader = MRT_SHADER_PATHTRACER;
            job.opts.width = job.opts.height = 64;
            job.opts.spp = job.opts.spl = 1;
            job.opts.depth_max = 1;
            job.bitmap = image.data();
            job.stride_bytes = 4 * 64;
            uint64_t id = 0;
            uint32_t launched = 0;
            CHECK(mrt_batch_submit(b, &job, &id) == MRT_OK, "submit: %s", mrt_context_error(ctx));
            CHECK(mrt_batch_step(b, waves, &launched) == MRT_OK && launched == waves, "step: %s", mrt_context_error(ctx));
            if (rebuild) CHECK(mrt_scene_build(s, &fast) == MRT_OK, "rebuild");
            CHECK(fake::violations == 0, "rebuild %d after %u waves", rebuild, waves);
            mrt_scene_destroy(s);
            CHECK(fake::violations == 0, "destroy %d after %u waves", rebuild, waves);
            mrt_batch_destroy(b);
            CHECK(fake::violations == 0, "batch destroy %d after %u waves", rebuild, waves);
        }
    for (int what = 0; what < 2; ++what)
        for (uint64_t k = 0;; ++k) {
            fake::reset();
            (what ? fake::fail_operations_from : fake::fail_allocations_from) = k;
            MrtBatch *b = nullptr;
            const int st = mrt_batch_create(ctx, &bo, &b);
            const bool failed = fake::failed != 0;
            CHECK(failed == (st != MRT_OK), "batch create %d %llu", what, (unsigned long long)k);
            if (st == MRT_OK) mrt_batch_destroy(b);
            CHECK(fake::violations == 0, "batch create %d %llu", what, (unsigned long long)k);
            if (!failed) break;
        }
    mrt_context_destroy(ctx);
    CHECK(fake::live_buffers() == 0, "buffers left");
    if (!bad) printf("ok\n");
    return bad != 0;
}
