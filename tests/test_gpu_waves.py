"""PathTracer wavefronts that run as two waves at once (from 2^19 paths), whose waves split pixels' samples
(7 samples, waves of 2^21 paths), and just below the limit, against mrt_render_noalloc's sequence of
4,096-path waves: the same words (GPU)."""
import ctypes

import pytest

from mobileraytracer_b200 import Scene, capi, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("accel", [capi.MRT_ACCEL_BVH, capi.MRT_ACCEL_REGULAR_GRID])
@pytest.mark.parametrize("w,h,spp", [(256, 256, 7), (256, 256, 8), (272, 256, 9), (1024, 640, 7)])
def test_paired_waves_equal_small_waves(ctx, accel, w, h, spp):
    torch = pytest.importorskip("torch")
    sc = scenes.glass_room()
    g = Scene(ctx, sc).build(accel)
    opts = capi.render_opts(shader=capi.MRT_SHADER_PATHTRACER, width=w, height=h, spp=spp, spl=1, seed=3, depth_min=2, depth_max=4)
    out = []
    for noalloc in (False, True):
        bm = torch.zeros(w * h, dtype=torch.int32, device="cuda")
        acc = torch.zeros(w * h * 4, dtype=torch.float32, device="cuda")
        if noalloc:
            st = capi.MrtRenderStats()
            torch.cuda.synchronize()
            assert g.lib.mrt_render_noalloc(g.h, ctypes.byref(sc.camera), ctypes.byref(opts), ctypes.c_void_p(bm.data_ptr()),
                                            w * 4, ctypes.c_void_p(acc.data_ptr()), ctypes.byref(st)) == capi.MRT_OK
        else:
            st = g.render(sc.camera, opts, bitmap=bm, accum=acc)[2]
        out.append((bm, acc, st.rays_closest, st.rays_shadow))
    assert out[0][2:] == out[1][2:]
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
