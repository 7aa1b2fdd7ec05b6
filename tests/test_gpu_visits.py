"""Frames whose block schedule renders pixels more than once a pass (sizes that are no multiple of 16), with
several samples, through the direct shaders' one-launch form: the folding order is the reference's
(sample by sample, within a sample in block order), against the oracle (GPU).  250x250 at 80 samples is
more than one hit buffer holds; 17x16 and 31x31 are the smallest such schedules."""
import numpy as np
import pytest

import orc as O
from mobileraytracer_b200 import Scene, capi, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("accel,oacc", [(capi.MRT_ACCEL_BVH, 3), (capi.MRT_ACCEL_REGULAR_GRID, 1)])
@pytest.mark.parametrize("w,h,spp,shader", [(17, 16, 3, capi.MRT_SHADER_NOSHADOWS), (31, 31, 1, capi.MRT_SHADER_DEPTHMAP),
                                            (100, 50, 5, capi.MRT_SHADER_NOSHADOWS), (230, 101, 2, capi.MRT_SHADER_DIFFUSE),
                                            (250, 250, 80, capi.MRT_SHADER_NOSHADOWS)])
def test_revisited_pixels(ctx, accel, oacc, w, h, spp, shader):
    sc = scenes.glass_room()
    opts = capi.render_opts(shader=shader, width=w, height=h, spp=spp, spl=2, seed=9)
    before = np.full((h, w), 0x11223344, np.uint32)
    g = Scene(ctx, sc).build(accel)
    bm_g, acc_g, st = g.render(sc.camera, opts, bitmap=before.copy(), accum=np.zeros((h, w, 4), np.float32))
    bm_o, acc_o, _ = O.OrcScene(sc, oacc).render(sc.camera, opts, bitmap=before.copy())
    assert np.array_equal(bm_g, bm_o)
    assert np.array_equal(acc_g[..., :3], acc_o[..., :3])
    assert g.progress() == spp
