"""Timed cases of the render path: what a program that uses this framework has it do.

Each case is one pass through the public entry points of mobileraytracer_b200 (Scene.render,
Scene.trace_closest / trace_any, Scene.raster_preview, Batch, Scene creation and build), on procedural
scenes of the kinds the benchmark and the tests use.  Every output (bitmaps, fp32 sums, hit distances
and ids, occlusion flags) is a deterministic function of the inputs, so results are compared exactly.
"""
import math

import numpy as np
import torch

from mobileraytracer_b200 import Batch, Context, Scene, capi, scenes

SHADERS = {"noshadows": capi.MRT_SHADER_NOSHADOWS, "whitted": capi.MRT_SHADER_WHITTED,
           "path": capi.MRT_SHADER_PATHTRACER, "depth": capi.MRT_SHADER_DEPTHMAP,
           "diffuse": capi.MRT_SHADER_DIFFUSE}
SAMPLERS = {"constant": capi.MRT_SAMPLER_CONSTANT, "stratified": capi.MRT_SAMPLER_STRATIFIED,
            "halton": capi.MRT_SAMPLER_HALTON, "random": capi.MRT_SAMPLER_RANDOM}


def _frame(name, scene, n, accel, shader, width, height, spp, spl=1, sampler="constant", depth=8, roulette=4,
           memory="device", sums=True):
    """One render of a resident scene: `memory` is where the caller's bitmap (and fp32 sums) live."""
    return {"name": name, "kind": "frame", "scene": scene, "n": n, "accel": accel, "shader": shader, "width": width,
            "height": height, "spp": spp, "spl": spl, "sampler": sampler, "depth": depth, "roulette": roulette,
            "memory": memory, "sums": sums}


def _rays(name, scene, n, accel, query, rays):
    """Closest-hit or any-hit queries for rays the caller holds on the device."""
    return {"name": name, "kind": "rays", "scene": scene, "n": n, "accel": accel, "query": query, "rays": rays}


def listed():
    return [
        # the reference application's first scene at its default size: a frame of 65,536 short paths,
        # where launches, synchronisation and the latency of one path count
        _frame("whitted_cornell_256", "cornell", 34, "fast", "whitted", 256, 256, 1),
        # the benchmark's headline: a full-HD frame of a million-triangle model, one sample per pixel
        _frame("frame_soup_1080p", "soup", 1_000_000, "fast", "noshadows", 1920, 1080, 1, sums=False),
        # the same on the reference's other accelerator, the regular grid sized by its rule
        _frame("frame_soup_grid_1080p", "soup", 1_000_000, "grid", "noshadows", 1920, 1080, 1, sums=False),
        # a window of an ordinary size that is no multiple of 16 (an irregular block schedule), jittered
        # samples, the bitmap in plain host memory as the C API's callers have it
        _frame("frame_host_1366x770", "terrain", 65_522, "fast", "noshadows", 1366, 770, 4, sampler="stratified",
               memory="host", sums=False),
        # path tracing of a large terrain, the longest kind of frame (six bounces, roulette beyond three)
        _frame("path_terrain_1024", "terrain", 524_288, "fast", "path", 1024, 1024, 16, sampler="halton", depth=6,
               roulette=3),
        # path tracing with mirrors, glass, planes and spheres, two light samples per hit: shading rather
        # than traversal
        _frame("path_glass_room_512", "glass", 3, "fast", "path", 512, 512, 4, spl=2, sampler="random"),
        # opening a model: upload, accelerator build and the first frame into host memory
        {"name": "open_soup_200k", "kind": "open", "scene": "soup", "n": 200_003, "accel": "fast", "width": 640,
         "height": 480},
        # incoherent queries from a program's own rays (an odd number of them), the library as a ray caster
        _rays("closest_terrain_1m", "terrain", 301_088, "fast", "closest", 1_000_003),
        # visibility queries on the regular grid
        _rays("any_soup_grid_300k", "soup", 100_003, "grid", "any", 300_007),
        # a handful of queries (picking, a probe): the latency of one call
        _rays("closest_cornell_1021", "cornell", 34, "fast", "closest", 1021),
        # the raster preview that the application shows while the first frame renders
        {"name": "preview_soup_1080p", "kind": "preview", "scene": "soup", "n": 1_000_000, "width": 1920,
         "height": 1080},
        # many renders of different scenes and sizes as one batch (the served form's engine)
        {"name": "batch_12_soups", "kind": "batch", "jobs": 12, "n_min": 1000, "n_max": 200_000, "side_min": 128,
         "side_max": 512, "spp": 4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["direct", "direct", "path", "path", "open", "rays", "rays", "preview", "batch"])
    if kind == "batch":
        n_min = _log(rng, 500, 5000)
        side_min = 16 * rng.randint(4, 12)
        return {"kind": "batch", "jobs": rng.randint(2, 16), "n_min": n_min, "n_max": n_min * rng.randint(4, 40),
                "side_min": side_min, "side_max": side_min * rng.randint(1, 3), "spp": rng.choice([1, 2, 4])}
    scene = rng.choice(["soup", "terrain"])
    n = _log(rng, 1000, 1_000_000 if scene == "soup" else 524_288)
    if kind == "open":
        return {"kind": "open", "scene": scene, "n": min(n, 500_000), "accel": "fast", "width": rng.randint(64, 1280),
                "height": rng.randint(64, 720)}
    if kind == "preview":
        return {"kind": "preview", "scene": scene, "n": n, "width": rng.randint(64, 1920), "height": rng.randint(64, 1080)}
    accel = rng.choice(["fast", "fast", "grid"])
    if kind == "rays":
        if rng.random() < 0.2:
            scene, n, accel = "cornell", 34, "fast"
        c = _rays("", scene, n, accel, rng.choice(["closest", "any"]), _log(rng, 100, 1_000_000))
    elif kind == "direct":
        w, h = _log(rng, 64, 1920), _log(rng, 64, 1080)
        spp = max(1, min(rng.choice([1, 1, 2, 3, 4, 8]), 2_100_000 // (w * h)))
        c = _frame("", scene, n, accel, rng.choice(["noshadows", "noshadows", "depth", "diffuse"]), w, h, spp,
                   spl=rng.choice([1, 1, 2]), sampler="constant" if spp == 1 else rng.choice(["stratified", "halton", "random"]),
                   memory=rng.choice(["device", "host"]), sums=rng.random() < 0.5)
    else:
        scene = rng.choice(["terrain", "soup_lit", "cornell", "glass"])
        n = {"cornell": 34, "glass": 3}.get(scene, min(n, 500_000))
        w, h = _log(rng, 64, 1024), _log(rng, 64, 1024)
        spp = max(1, min(rng.choice([1, 2, 4, 9]), (300_000 if accel == "grid" else 2_500_000) // (w * h)))
        c = _frame("", scene, n, accel, rng.choice(["path", "path", "whitted"]), w, h, spp, spl=rng.choice([1, 1, 2, 4]),
                   sampler=rng.choice(["halton", "random", "stratified"]), depth=rng.randint(3, 8), roulette=rng.randint(2, 4),
                   memory=rng.choice(["device", "host"]), sums=rng.random() < 0.5)
    del c["name"]
    return c


def _host_scene(case, seed):
    w, h = case.get("width", 1024), case.get("height", 1024)
    if case["scene"] == "soup":
        return scenes.triangle_soup(case["n"], seed, w, h)
    if case["scene"] == "soup_lit":
        s = scenes.Job(0, case["n"], 256, 1, seed).scene()
        s.camera = scenes.cli_camera(w, h)
        return s
    if case["scene"] == "terrain":
        return scenes.heightfield(max(2, int(round(math.sqrt(case["n"] / 2)))), seed, width=w, height=h)
    # the fixed rooms: the viewer stands somewhere else for every seed
    s = scenes.cornell_box() if case["scene"] == "cornell" else scenes.glass_room()
    u = scenes.uniform(seed, 3, stream=31) - 0.5
    at = list(s.camera.position)
    s.camera = scenes.camera((at[0] + 0.2 * u[0], at[1] + 0.2 * u[1], at[2] + 0.1 * u[2]), (0.0, 0.0, 1.0))
    return s


def _build(scene, case):
    if case.get("accel") == "grid":
        return scene.build(capi.MRT_ACCEL_REGULAR_GRID)
    return scene.build(capi.MRT_ACCEL_BVH, capi.MRT_BVH_FAST)


def _opts(case, seed):
    s = SAMPLERS[case.get("sampler", "constant")]
    random_one = capi.MRT_SAMPLER_RANDOM if s == capi.MRT_SAMPLER_CONSTANT else s
    return capi.render_opts(shader=SHADERS[case.get("shader", "noshadows")], width=case["width"], height=case["height"],
                            spp=case.get("spp", 1), spl=case.get("spl", 1), pixel_sampler=s, light_sampler=random_one,
                            rr_sampler=random_one, depth_min=case.get("roulette", 4), depth_max=case.get("depth", 8),
                            seed=seed)


def _query_rays(case, seed):
    """Origins through the scene's volume, directions uniform over the sphere, on the device."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = case["rays"]
    lo, hi = (0.49, 0.49) if case["scene"] == "cornell" else (1.0, 1.0)
    o = torch.rand((n, 3), generator=g, device="cuda") * (lo + hi) - lo
    d = torch.randn((n, 3), generator=g, device="cuda")
    d = d / d.norm(dim=1, keepdim=True)
    rays = torch.empty((n, 8), dtype=torch.float32, device="cuda")
    rays[:, 0:3], rays[:, 3:6] = o, d
    rays.view(torch.int32)[:, 6] = 1
    rays.view(torch.int32)[:, 7] = -1   # no excluded primitive
    dist = torch.rand(n, generator=g, device="cuda") * 1.5 + 0.05
    return rays, dist


def prepare(case, seed):
    ctx = Context(0)
    st = {"case": case, "ctx": ctx}
    if case["kind"] == "batch":
        st["batch"] = Batch(ctx, max_depth=6, max_spl=1)
        st["jobs"] = []
        for i in range(case["jobs"]):
            u = scenes.uniform(i, 2, stream=11)   # the sizes are the case's, the models the seed's
            n = int(round(case["n_min"] * (case["n_max"] / case["n_min"]) ** u[0]))
            side = int(case["side_min"] * (case["side_max"] / case["side_min"]) ** u[1]) // 16 * 16
            spp = case["spp"]
            job = scenes.Job(i, n, side, spp, seed * 64 + i)
            host = job.scene()
            o = capi.render_opts(shader=capi.MRT_SHADER_PATHTRACER, width=side, height=side, spp=spp,
                                 light_sampler=capi.MRT_SAMPLER_HALTON, rr_sampler=capi.MRT_SAMPLER_HALTON, depth_min=3,
                                 depth_max=6, seed=seed + i)
            bitmap = torch.zeros((side, side), dtype=torch.int32, device="cuda")
            st["jobs"].append((Scene(ctx, host).build(), host.camera, o, bitmap))
        return st
    host = _host_scene(case, seed)
    st["host"] = host
    if case["kind"] == "open":
        st["opts"] = _opts(case, seed)
        return st
    st["scene"] = _build(Scene(ctx, host), case)
    if case["kind"] == "rays":
        st["rays"], st["dist"] = _query_rays(case, seed)
    elif case["kind"] == "preview":
        st["bitmap"] = torch.zeros((case["height"], case["width"]), dtype=torch.int32, device="cuda")
    else:
        st["opts"] = _opts(case, seed)
        w, h = case["width"], case["height"]
        if case["memory"] == "host":
            st["bitmap"] = np.zeros((h, w), np.uint32)
            st["sums"] = np.zeros((h, w, 4), np.float32) if case["sums"] else None
        else:
            st["bitmap"] = torch.zeros((h, w), dtype=torch.int32, device="cuda")
            st["sums"] = torch.zeros((h, w, 4), dtype=torch.float32, device="cuda") if case["sums"] else None
    return st


def run(st):
    case = st["case"]
    if case["kind"] == "frame":
        bitmap, sums = st["bitmap"], st["sums"]
        if case["memory"] == "host":
            bitmap.fill(0)   # an irregular schedule leaves some pixels as they are and renders others again
            if sums is not None:
                sums.fill(0)
        else:
            bitmap.zero_()
            if sums is not None:
                sums.zero_()
        st["scene"].render(st["host"].camera, st["opts"], bitmap, sums)
        out = {"bitmap": bitmap}
        if sums is not None:
            out["sums"] = sums
        return out
    if case["kind"] == "rays":
        if case["query"] == "any":
            return st["scene"].trace_any(st["rays"], st["dist"])
        hits = st["scene"].trace_closest(st["rays"])
        return {"t": hits[:, 0].view(torch.float32), "id": hits[:, 1]}
    if case["kind"] == "preview":
        return st["scene"].raster_preview(st["host"].camera, case["width"], case["height"], st["bitmap"])[0]
    if case["kind"] == "open":
        scene = _build(Scene(st["ctx"], st["host"]), case)
        bitmap = scene.render(st["host"].camera, st["opts"])[0]
        scene.close()
        return bitmap
    for scene, camera, opts, bitmap in st["jobs"]:
        st["batch"].submit(scene, camera, opts, bitmap)
    st["batch"].run()
    st["batch"].completed()
    return [job[3] for job in st["jobs"]]


def _ray_flops(n):
    """One ray's least work: a path of 8-wide boxes (12 operations each) down to one triangle (40)."""
    return 96.0 * max(1.0, math.ceil(math.log(max(n, 2)) / math.log(8))) + 40.0


def work(case):
    """Geometry (36 bytes a triangle) read once, what the caller hands over and gets back moved once."""
    if case["kind"] == "batch":
        mean_n = (case["n_max"] - case["n_min"]) / max(1e-9, math.log(case["n_max"] / case["n_min"]))
        a, b = case["side_min"], case["side_max"]
        pixels = a * a if a == b else (b * b - a * a) / (2.0 * math.log(b / a))   # log-uniform sides
        return {"bytes": case["jobs"] * (36.0 * mean_n + 4.0 * pixels),
                "flops": case["jobs"] * pixels * case["spp"] * _ray_flops(mean_n)}
    n = case["n"]
    if case["kind"] == "rays":
        out = 8 if case["query"] == "closest" else 5
        return {"bytes": 36.0 * n + (32.0 + out) * case["rays"], "flops": case["rays"] * _ray_flops(n)}
    pixels = case["width"] * case["height"]
    if case["kind"] == "preview":
        return {"bytes": 36.0 * n + 4.0 * pixels, "flops": 80.0 * n}
    paths = pixels * case.get("spp", 1)
    per_path = 1.0 if case.get("shader", "noshadows") in ("noshadows", "depth", "diffuse") else 2.0
    return {"bytes": 36.0 * n + pixels * (4.0 + (32.0 if case.get("sums") else 0.0)), "flops": per_path * paths * _ray_flops(n)}


def tolerance(case):
    """Every random draw is a function of the seed, and a closest hit is the least distance with ties to
    the lower index: two correct implementations give the same words."""
    return "exact"


def _closest64(host, o, d):
    """Distances and ids of the closest hits in 64 bits, every primitive tested."""
    best = torch.full((len(o),), 1e30, dtype=torch.float64, device=o.device)
    ids = torch.full((len(o),), -1, dtype=torch.int64, device=o.device)

    def keep(t, hit, kind, first):
        t = torch.where(hit, t, torch.inf)
        v, i = t.min(dim=1)
        closer = v < best
        best[closer] = v[closer]
        ids[closer] = (kind << 30) | (i[closer] + first)

    def triangles(abc, kind):
        step = max(1, 20_000_000 // max(1, len(o)))
        for k in range(0, len(abc), step):
            a = torch.as_tensor(abc[k:k + step].astype(np.float64), device=o.device).reshape(-1, 3, 3)
            p0, e1, e2 = a[:, 0], a[:, 1] - a[:, 0], a[:, 2] - a[:, 0]
            p = torch.linalg.cross(d[:, None], e2[None], dim=-1)
            det = (p * e1).sum(-1)
            s = o[:, None] - p0[None]
            q = torch.linalg.cross(s, e1[None].expand_as(s), dim=-1)
            u, v, t = (s * p).sum(-1) / det, (q * d[:, None]).sum(-1) / det, (q * e2).sum(-1) / det
            keep(t, (det.abs() >= 1e-6) & (u >= 0) & (v >= 0) & (u + v <= 1) & (t >= 1e-6), kind, k)

    if len(host.spheres):
        s = torch.as_tensor(host.spheres.astype(np.float64), device=o.device)
        oc = s[None, :, :3] - o[:, None]
        b = (oc * d[:, None]).sum(-1)
        disc = b * b - (oc * oc).sum(-1) + s[None, :, 3] ** 2
        t = b - disc.clamp(min=0).sqrt()
        keep(t, (disc >= 0) & (t >= 1e-5), capi.MRT_PRIM_SPHERE, 0)
    triangles(host.tri_abc, capi.MRT_PRIM_TRIANGLE)
    areas = [list(light.p0) + list(light.p1) + list(light.p2) for light in host.lights if light.kind == capi.MRT_LIGHT_AREA]
    if areas:
        triangles(np.asarray(areas), capi.MRT_PRIM_LIGHT)
    return best, ids


def exact(case, seed):
    """Closest-hit distances in 64 bits, and the sums of an unjittered NoShadows frame of a soup (one
    point light, one diffuse material), where testing every triangle is quick; else None."""
    if case["kind"] == "rays" and case["query"] == "closest" and case["rays"] * case["n"] <= 2e9:
        rays, _ = _query_rays(case, seed)
        t, _ = _closest64(_host_scene(case, seed), rays[:, 0:3].double(), rays[:, 3:6].double())
        return {"t": t, "id": None}
    if case["kind"] != "frame" or case["scene"] != "soup" or case["shader"] != "noshadows" or case["spp"] != 1 or \
            not case["sums"] or case["width"] % 16 or case["height"] % 16 or case["width"] * case["height"] * case["n"] > 2e9:
        return None
    host = _host_scene(case, seed)
    w, h = case["width"], case["height"]
    y, x = torch.meshgrid(torch.arange(h, device="cuda").double(), torch.arange(w, device="cuda").double(), indexing="ij")

    def arctan(v):   # the camera's polynomial
        return 0.785398163397448309616 * v - v * (v.abs() - 1) * (0.2447 + 0.0663 * v.abs())

    o = torch.tensor(list(host.camera.position), dtype=torch.float64, device="cuda")
    rf = arctan(math.radians(host.camera.fov_h_deg) * (x / w - 0.5)).reshape(-1, 1)
    uf = arctan(math.radians(host.camera.fov_v_deg) * (0.5 - y / h)).reshape(-1, 1)
    axes = torch.eye(3, dtype=torch.float64, device="cuda")   # the default camera looks along +z, x to the right
    d = axes[2] + axes[0] * rf + axes[1] * uf
    d = d / d.norm(dim=1, keepdim=True)
    o = o.expand_as(d)
    t, ids = _closest64(host, o, d)
    hit = ids >= 0
    tri = torch.as_tensor(host.tri_abc.astype(np.float64), device="cuda").reshape(-1, 3, 3)[(ids & 0x3FFFFFFF)[hit]]
    normal = torch.linalg.cross(tri[:, 2] - tri[:, 0], tri[:, 1] - tri[:, 0], dim=-1)
    normal = normal / normal.norm(dim=1, keepdim=True)
    light = torch.tensor(list(host.lights[0].p0), dtype=torch.float64, device="cuda")
    to = light - (o + d * t[:, None])[hit]
    cos = ((normal * to).sum(-1) / to.norm(dim=1)).clamp(min=0)
    sums = torch.zeros((w * h, 4), dtype=torch.float64, device="cuda")
    sums[hit, :3] = (0.8 * (0.9 * cos + 0.1))[:, None].expand(-1, 3)
    sums[:, 3] = 1
    return {"bitmap": None, "sums": sums.reshape(h, w, 4)}
