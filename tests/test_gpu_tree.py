"""The FAST tree at the sizes and shapes its build can go wrong at, against the oracle's exact closest hit and
occlusion (GPU): one to a few triangles (root leaves of 1 to 3, a node that is not full), counts around a
sort tile, triangles that coincide (no area to choose by, equal Morton codes), scenes along a line and in a
plane (one or two axes without extent), far from the origin and of very different extents.  A triangle far away costs the others' tree little."""
import numpy as np
import pytest

import orc as O
from helpers import hits_equal, near_tie_mask, random_rays
from mobileraytracer_b200 import Scene, capi, scenes

pytestmark = pytest.mark.gpu


def _scene(kind, n):
    sc = scenes.triangle_soup(n, n, 64, 64)
    t = sc.tri_abc.reshape(-1, 3, 3).astype(np.float64)
    c = t.mean(axis=1, keepdims=True)
    t = c + (t - c) * 20.0
    if kind == "coincident":
        t[:] = t[0]
    elif kind == "line":
        t = (t - c) + c * np.array([1.0, 0.0, 0.0])
    elif kind == "flat":
        t = t * np.array([1.0, 0.0, 1.0])
    elif kind == "thin":
        t = t * np.array([1.0, 1e-4, 0.3])
    elif kind == "far":
        t = t + 50.0
    sc.tri_abc = t.reshape(-1, 9).astype(np.float32)
    return sc


@pytest.mark.parametrize("n", [1, 2, 3, 4, 8, 9, 33, 2047, 2049])
@pytest.mark.parametrize("kind", ["random", "coincident", "line", "flat", "thin", "far"])
def test_tree_equals_every_triangle(ctx, kind, n):
    sc = _scene(kind, n)
    rays = random_rays(3000, seed=n)
    if kind == "far":
        rays["origin"] += np.float32(50.0)
    if kind == "flat":      # towards the plane, not along it
        rays["origin"][:, 1] += np.float32(0.01)
    g = Scene(ctx, sc).build(capi.MRT_ACCEL_BVH, capi.MRT_BVH_FAST)
    o = O.OrcScene(sc, 0)
    got, want = g.trace_closest(rays), o.trace_closest(rays)
    assert (hits_equal(got, want) | near_tie_mask(rays, got, want)).all()
    dist = np.full(len(rays), 0.7, np.float32)
    assert (g.trace_any(rays, dist) == o.trace_any(rays, dist)).all()
    assert 1 <= g.accel_info()["nodes"] <= max(1, n)
    g.close()


def _nodes(ctx, sc, rays):
    g = Scene(ctx, sc).build(capi.MRT_ACCEL_BVH, capi.MRT_BVH_FAST)
    nodes = g.trace_counts(rays)[0].mean()
    g.close()
    return nodes


# nodes a ray against the same scene without the far triangle (30.2): 30.6, 31.0, 31.1, 31.5 and 59.1 (92.7 with ten
# bits of the code an axis in turn)
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("far,most", [(4.0, 1.1), (30.0, 1.1), (200.0, 1.1), (1000.0, 1.2), (1e4, 2.5)])
def test_a_far_triangle_costs_little(ctx, axis, far, most):
    sc = scenes.triangle_soup(100_000, 5, 64, 64)
    rays = random_rays(20_000, seed=9)
    alone = _nodes(ctx, sc, rays)
    away = sc.tri_abc[:1].copy().reshape(3, 3)
    away[:, axis] += np.float32(far)
    sc.tri_abc = np.concatenate([sc.tri_abc, away.reshape(1, 9)])
    sc.tri_material = np.concatenate([sc.tri_material, sc.tri_material[:1]])
    assert _nodes(ctx, sc, rays) <= most * alone + 1.0
