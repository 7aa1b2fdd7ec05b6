"""Queues of the wavefront's shade kernel (places per block, continuation rays ordered by octant): levels of
a few rays up to many blocks, several children and light samples per ray, against mrt_render's
whole-path launch, which has no queues (the last sizes on both sides of the path count from which PathTracer
frames of few triangles take more blocks): the same words (GPU)."""
import ctypes

import pytest

from mobileraytracer_b200 import Batch, Scene, capi, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shader", [capi.MRT_SHADER_WHITTED, capi.MRT_SHADER_PATHTRACER])
@pytest.mark.parametrize("w,h,spp,spl", [(16, 16, 1, 1), (16, 16, 7, 4), (48, 32, 1, 3), (112, 48, 2, 2), (352, 368, 1, 1), (368, 368, 1, 2)])
def test_queued_levels_equal_whole_paths(ctx, shader, w, h, spp, spl):
    torch = pytest.importorskip("torch")
    sc = scenes.glass_room()
    g = Scene(ctx, sc).build(capi.MRT_ACCEL_BVH)
    opts = capi.render_opts(shader=shader, width=w, height=h, spp=spp, spl=spl, seed=11, depth_min=2, depth_max=6)
    out = []
    for queued in (False, True):
        bm = torch.zeros(w * h, dtype=torch.int32, device="cuda")
        acc = torch.zeros(w * h * 4, dtype=torch.float32, device="cuda")
        if queued:
            st = capi.MrtRenderStats()
            torch.cuda.synchronize()
            assert g.lib.mrt_render_noalloc(g.h, ctypes.byref(sc.camera), ctypes.byref(opts), ctypes.c_void_p(bm.data_ptr()),
                                            w * 4, ctypes.c_void_p(acc.data_ptr()), ctypes.byref(st)) == capi.MRT_OK
        else:
            st = g.render(sc.camera, opts, bitmap=bm, accum=acc)[2]
        out.append((bm, acc, st.rays_closest, st.rays_shadow))
    assert out[0][2:] == out[1][2:]
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])


@pytest.mark.parametrize("jobs,soup", [(2, False), (3, False), (3, True)])
def test_batches_of_small_scenes_equal_frames(ctx, jobs, soup):
    """Waves below and above the path count of the small-scene launch, and one with a larger scene among them."""
    torch = pytest.importorskip("torch")
    batch, want = Batch(ctx, max_depth=6, max_spl=2), []
    for i in range(jobs):
        sc = scenes.triangle_soup(500, 3, 256, 256) if soup and i == 1 else scenes.glass_room()
        g = Scene(ctx, sc).build(capi.MRT_ACCEL_BVH)
        opts = capi.render_opts(shader=capi.MRT_SHADER_PATHTRACER, width=256, height=256, spp=1, spl=2, seed=i, depth_min=2, depth_max=6)
        got, frame = (torch.zeros(256, 256, dtype=torch.int32, device="cuda") for _ in range(2))
        g.render(sc.camera, opts, bitmap=frame)
        batch.submit(g, sc.camera, opts, got)
        want.append((g, got, frame))
    batch.run()
    batch.completed()
    torch.cuda.synchronize()
    assert all(torch.equal(got, frame) for _, got, frame in want)
