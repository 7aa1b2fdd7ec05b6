"""The warp-wide covering of small triangles in the raster preview, bit for bit against the oracle's serial
restatement (GPU): triangles from below a pixel to beyond 64 pixels a side (boxes around the 64-pixel
limit, long thin boxes one pixel wide or high, corners just within and beyond the 32-bit range), cut by
every side of frames of one pixel, one row, one column and ordinary sizes, in scenes of fewer triangles
than a warp, a block and a ragged number of blocks."""
import numpy as np
import pytest

import orc as O
from mobileraytracer_b200 import Scene, scenes

pytestmark = pytest.mark.gpu


def _triangles(n, w, h, seed):
    """n triangles facing a film of w x h pixels (1 unit = 1 pixel), sides around the limits"""
    rng = np.random.default_rng(seed)
    c = rng.uniform([-0.6 * w - 1, -0.6 * h - 1, 1.0], [0.6 * w + 1, 0.6 * h + 1, 5.0], (n, 3))
    side = rng.choice([0.3, 1.0, 2.0, 7.9, 8.1, 16.0, 63.9, 64.1, 90.0], (n, 1, 1))
    flat = rng.choice([1.0, 1.0, 0.02], (n, 1, 1)) * np.array([1.0, 0.0, 0.0]) + np.array([0.0, 1.0, 0.0])
    flat = np.where(rng.random((n, 1, 1)) < 0.5, flat, flat[..., [1, 0, 2]])
    v = rng.uniform(-0.5, 0.5, (n, 3, 3)) * side * flat
    v[:, :, 2] = rng.uniform(-0.2, 0.2, (n, 3))
    t = c[:, None, :] + v
    snap = rng.random(n) < 0.3
    t[snap, :, :2] = np.round(t[snap, :, :2])      # corners and edges on pixel centres and borders
    return t.reshape(n, 9).astype(np.float32)


@pytest.mark.parametrize("w,h", [(1, 1), (1, 70), (70, 1), (33, 17), (256, 256), (300, 200)])
@pytest.mark.parametrize("n", [1, 31, 257, 4000])
def test_small_triangles(ctx, w, h, n):
    sc = scenes.Scene()
    sc.tri_abc = _triangles(n, w, h, 7 * n + w)
    sc.tri_material = np.full(n, -1, np.int32)
    sc.tri_colors = np.repeat(np.random.default_rng(n).random((n, 1, 3)), 3, 1).reshape(n, 9).astype(np.float32)
    # the film's half sizes are a quarter of the sizes given: 1 unit = 1 pixel
    cam = scenes.orthographic((0.0, 0.0, 0.0), (0.0, 0.0, 1.0), (0.0, 1.0, 0.0), 2.0 * w, 2.0 * h)
    g = Scene(ctx, sc)
    bm, st = g.raster_preview(cam, w, h)
    want, drawn, frags = O.raster_preview(sc, cam, w, h)
    assert (st.drawn, st.fragments) == (drawn, frags)
    assert np.array_equal(bm, want)
    g.close()
