"""The RegularGrid's persistent walks against the oracle's restatement of the reference walk (GPU), where
their short cuts could go wrong: long empty runs (records that skip ahead), cells that share references
(skip bits), both addressing modes at sizes that are and are not powers of two, the smallest grids, rays
that start outside, run along axes or cell borders or have no direction, and distances that are not
numbers (coordinates near the ends of the float range).  Grids of triangles with coordinates that are not
numbers or infinite, whose bounds depend on the order of the triangles."""
import numpy as np
import pytest

import orc as O
from helpers import random_rays
from mobileraytracer_b200 import Scene, capi, scenes

pytestmark = pytest.mark.gpu


def _same(a, b):
    """ids equal and distances equal bit for bit (not-a-number: on both sides)"""
    ta, tb = a["t"], b["t"]
    return (a["id"] == b["id"]) & ((ta.view(np.uint32) == tb.view(np.uint32)) | (np.isnan(ta) & np.isnan(tb)))


def _rays(scale):
    r = random_rays(6000, seed=21, lo=-1.6, hi=1.6)      # some start outside the grid
    r["direction"][::5, 0] = 0.0
    r["direction"][1::5, 1] = 0.0
    r["direction"][2::25] = (0.0, 0.0, 1.0)
    r["direction"][3::25] = (-1.0, 0.0, 0.0)
    r["direction"][4::50] = 0.0
    r["origin"][::7] = np.round(r["origin"][::7] * 4) / 4     # on cell borders of the even sizes
    r["origin"] *= np.float32(scale)
    r["exclude"][::3] = capi.hit_id(capi.MRT_PRIM_TRIANGLE, 5)
    return r


def _scene(kind, scale):
    sc = scenes.triangle_soup(200 if kind == "sparse" else 1500, 13, 64, 64)
    t = sc.tri_abc.reshape(-1, 3, 3)
    c = t.mean(axis=1, keepdims=True)
    if kind == "large":      # triangles over many cells
        t = c + (t - c) * 60.0
    if kind == "mesh":       # shared edges: equal distances
        sc = scenes.heightfield(20)
        t = sc.tri_abc.reshape(-1, 3, 3)
    sc.tri_abc = (t * scale).reshape(-1, 9).astype(np.float32)
    sc.camera = scenes.camera((0.0, 0.0, -3.4 * scale), (0.0, 0.0, 1.0))
    return sc


@pytest.mark.parametrize("kind,scale", [("sparse", 1.0), ("small", 1.0), ("large", 1.0), ("mesh", 1.0), ("large", 3e18)])
@pytest.mark.parametrize("size,index", [(0, 0), (2, 0), (3, 0), (16, 0), (50, 0), (50, 1), (64, 1), (97, 1)])
def test_walks_equal_the_reference_walk(ctx, kind, scale, size, index):
    sc, rays = _scene(kind, scale), _rays(scale)
    g = Scene(ctx, sc).build(capi.MRT_ACCEL_REGULAR_GRID, grid_size=size, grid_index=index)
    o = O.OrcScene(sc, 1, grid_size=size, grid_index=index)
    same = _same(g.trace_closest(rays), o.trace_closest(rays))
    assert same.all(), f"{(~same).sum()} of {len(rays)} rays differ"
    for d in (0.3, 4.0):
        dist = np.full(len(rays), d * scale, np.float32)
        assert (g.trace_any(rays, dist) == o.trace_any(rays, dist)).all()


def test_walks_with_planes_and_spheres(ctx):
    sc, rays = scenes.glass_room(), _rays(1.0)
    g = Scene(ctx, sc).build(capi.MRT_ACCEL_REGULAR_GRID)
    o = O.OrcScene(sc, 1)
    assert _same(g.trace_closest(rays), o.trace_closest(rays)).all()
    dist = np.full(len(rays), 1.2, np.float32)
    assert (g.trace_any(rays, dist) == o.trace_any(rays, dist)).all()


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("at", [0, 700, 1499, None])
def test_bounds_with_coordinates_that_are_not_finite(ctx, value, at):
    sc, rays = _scene("small", 1.0), _rays(1.0)
    if at is None:
        sc.tri_abc[::10, 4] = value
    else:
        sc.tri_abc[at, 0:3] = value
    g = Scene(ctx, sc).build(capi.MRT_ACCEL_REGULAR_GRID)
    o = O.OrcScene(sc, 1)
    assert _same(g.trace_closest(rays), o.trace_closest(rays)).all()
    dist = np.full(len(rays), 1.2, np.float32)
    assert (g.trace_any(rays, dist) == o.trace_any(rays, dist)).all()
