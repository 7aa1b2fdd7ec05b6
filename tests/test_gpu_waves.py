"""PathTracer wavefronts that run as two waves at once (from 2^19 paths), whose waves split pixels' samples
(7 samples, waves of 2^21 paths), and just below the limit, against mrt_render_noalloc's sequence of
4,096-path waves: the same words.  Views whose rays branch more in one half of the frame than the half's
queues hold, though not more than the frame's, against whole-path launches (GPU)."""
import ctypes
import os
import subprocess
import sys
import tempfile

import numpy as np
import pytest

from mobileraytracer_b200 import MrtError, Scene, capi, scenes

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


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


# camera height, depth_min, depth_max: 6.2 rays a path over the frame and 7.6 in its upper half, of 7 a path that
# the queues hold; 9.8 and 11.2 of 11
UNEVEN = [(0.1, 3, 4), (0.2, 4, 8)]


def _inside(ctx, y, depth_min, depth_max, w, h, spp):
    sc = scenes.glass_room()
    sc.camera = scenes.camera((0.1, y, 0.1), (0.1, y, 1.1))
    return sc, Scene(ctx, sc).build(), capi.render_opts(shader=capi.MRT_SHADER_PATHTRACER, width=w, height=h, spp=spp,
                                                         spl=1, seed=3, depth_min=depth_min, depth_max=depth_max)


# two waves dealt in turn, also of an irregular schedule; samples too many to deal: split by rows, done again
@pytest.mark.parametrize("y,depth_min,depth_max", UNEVEN)
@pytest.mark.parametrize("w,h,spp", [(512, 512, 4), (500, 1200, 1), (32, 32, 700)])
def test_uneven_frames_fit_their_queues(ctx, y, depth_min, depth_max, w, h, spp):
    torch = pytest.importorskip("torch")
    sc, g, opts = _inside(ctx, y, depth_min, depth_max, w, h, spp)
    bm = torch.full((w * h,), 5, dtype=torch.int32, device="cuda")
    acc = torch.full((w * h * 4,), 0.25, dtype=torch.float32, device="cuda")
    want_bm, want_acc = bm.clone(), acc.clone()
    st = g.render(sc.camera, opts, bitmap=bm, accum=acc)[2]
    rays = 0
    if spp > 1:   # one sample at a time, below 2^19 paths: whole paths, no queues
        for k in range(spp):
            opts.spp, opts.spp_offset = 1, k
            rays += g.render(sc.camera, opts, bitmap=want_bm, accum=want_acc)[2].rays_closest
        assert st.rays_closest == rays
        assert torch.equal(bm, want_bm) and torch.equal(acc, want_acc)
    else:
        want = _whole_paths(y, depth_min, depth_max, w, h)
        assert st.rays_closest == int(want["rays"])
        assert (bm.cpu().numpy() == want["bm"]).all() and (acc.cpu().numpy() == want["acc"]).all()


def _whole_paths(y, depth_min, depth_max, w, h):
    """The frame in whole-path launches (no queues) of a process of their own, from the same pixels."""
    code = f"""
import sys, torch, numpy as np
sys.path[:0] = {[os.path.dirname(HERE), HERE]!r}
import test_gpu_waves as t
from mobileraytracer_b200 import Context
sc, g, opts = t._inside(Context(0), {y}, {depth_min}, {depth_max}, {w}, {h}, 1)
bm = torch.full(({w * h},), 5, dtype=torch.int32, device="cuda")
acc = torch.full(({w * h * 4},), 0.25, dtype=torch.float32, device="cuda")
st = g.render(sc.camera, opts, bitmap=bm, accum=acc)[2]
np.savez(sys.argv[1], bm=bm.cpu().numpy(), acc=acc.cpu().numpy(), rays=st.rays_closest)
"""
    with tempfile.TemporaryDirectory() as d:
        out = os.path.join(d, "whole.npz")
        subprocess.run([sys.executable, "-c", code, out], check=True, env={**os.environ, "MRT_PATHS_MAX": str(1 << 30)})
        return dict(np.load(out))


def test_waves_of_a_long_list_get_smaller(ctx):
    """2,190,000 paths of an irregular schedule at 7.04 rays a path: more than one wave of 2^21 holds."""
    torch = pytest.importorskip("torch")
    w, h = 1500, 1460
    sc, g, opts = _inside(ctx, 0.2, 3, 4, w, h, 1)
    bm = torch.full((w * h,), 5, dtype=torch.int32, device="cuda")
    acc = torch.full((w * h * 4,), 0.25, dtype=torch.float32, device="cuda")
    st = g.render(sc.camera, opts, bitmap=bm, accum=acc)[2]
    want = _whole_paths(0.2, 3, 4, w, h)
    assert st.rays_closest == int(want["rays"]) > 7 * st.paths
    assert (bm.cpu().numpy() == want["bm"]).all() and (acc.cpu().numpy() == want["acc"]).all()


def test_frames_beyond_their_queues_are_refused(ctx):
    """9.8 rays a path of 9: refused, as by one wave with all of the queues."""
    torch = pytest.importorskip("torch")
    sc, g, opts = _inside(ctx, 0.1, 6, 6, 512, 512, 4)
    bm = torch.zeros(512 * 512, dtype=torch.int32, device="cuda")
    with pytest.raises(MrtError) as e:
        g.render(sc.camera, opts, bitmap=bm)
    assert e.value.status == capi.MRT_ERR_LIMIT
