"""Scenes opened, rendered and closed by several threads, each on a context of its own, over the device's
shared buffer pool: every frame is the one a single thread renders, and the pool's memory goes back when
the contexts are gone (GPU)."""
import threading

import numpy as np
import pytest

from mobileraytracer_b200 import Context, Scene, capi, scenes

pytestmark = pytest.mark.gpu


def _frames(device, sizes, out, slot):
    ctx = Context(device)
    got = []
    for n in sizes:
        sc = scenes.triangle_soup(n, n, 64, 48)
        for accel in (capi.MRT_ACCEL_BVH, capi.MRT_ACCEL_REGULAR_GRID):
            s = Scene(ctx, sc).build(accel)
            got.append(s.render(sc.camera, capi.render_opts(width=64, height=48, spp=2, seed=n))[0])
            s.close()
    ctx.close()
    out[slot] = got


@pytest.mark.parametrize("threads", [1, 4])
def test_scenes_of_several_threads(threads):
    torch = pytest.importorskip("torch")
    sizes = [1, 2, 3, 700, 20_000, 5, 90_001]
    want = {}
    _frames(0, sizes, want, 0)
    out = {}
    work = [threading.Thread(target=_frames, args=(0, sizes, out, k)) for k in range(threads)]
    for t in work:
        t.start()
    for t in work:
        t.join()
    assert len(out) == threads
    for k in out:
        assert all(np.array_equal(a, b) for a, b in zip(out[k], want[0]))
    assert torch.cuda.mem_get_info(0)[0] > 0
