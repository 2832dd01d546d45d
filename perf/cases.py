"""Timed workloads of the rendering core, each through its public Python entry points.

Every case is a dict of plain values. `kind` says which call a program makes:

* trace      Scene.trace_closest on device rays (closest hits with the reference's exact ids, or
             the fast mode of the renderer's extension rays)
* any        Scene.trace_any / trace_any_bits: shadow rays from surface points to lights
* load       a mesh is loaded, committed and probed with host rays: what an editor or a
             simulation does each time its geometry changes
* render     Scene.render, one frame
* views      Scene.render_batch, several seeded views of one scene in one call
* hybrid     Scene.render in hybrid photon + path mode with subsurface gathers
* photons    Scene.trace_photons, PhotonMap.build and a density estimate: a photon pass
* knn        PhotonMap.knn on a built map
* guide      Guide.sample and Guide.pdf: network inference on a batch of shading points
* train      Guide.train_step: forward, backward and weight gradient of one batch

Scenes are the repository's own (scenes.py), with the random parts drawn from the seed.
"""
from __future__ import annotations

import functools
import importlib
import math

import numpy as np
import torch

PKG = "2023_render_engine_b200"
N = importlib.import_module(PKG + "._native")
core = importlib.import_module(PKG + ".core")
scenes = importlib.import_module(PKG + ".scenes")
configs = importlib.import_module(PKG + ".configs")


def listed():
    return [
        # a handful of rays into a 12-triangle box with two spheres: picking, autofocus, a light
        # probe; an odd count. Latency and launches are all there is.
        dict(name="probe_rays", kind="trace", scene="cornell", detail=0, rays=997, mode="exact"),
        # the ray-set benchmark: 2^24 incoherent rays through a 1.3M-triangle mesh
        dict(name="stress_rays", kind="trace", scene="stress", detail=8, rays=1 << 24, mode="exact"),
        # visibility between surface points and a light, as a bit mask (a lightmap or an
        # ambient-occlusion pass), a ragged count of rays over an 82k-triangle mesh
        dict(name="visibility", kind="any", scene="stress", detail=6, rays=2_000_003, mode="exact", bits=True),
        # geometry changes: a 328k-triangle mesh is loaded, built and probed from host arrays
        dict(name="load_and_probe", kind="load", scene="stress", detail=7, rays=262_147, mode="fast"),
        # the smallest frame of the benchmark: the Cornell box at 256x256, 16 spp, depth 8
        dict(name="cornell_frame", kind="render", scene="cornell", detail=0, width=256, height=256, spp=16, depth=8),
        # the headline frame: 1.3M GGX triangles at 1920x1080, 64 spp, depth 12
        dict(name="stress_frame", kind="render", scene="stress", detail=8, width=1920, height=1080, spp=64, depth=12),
        # a batch of small seeded views (data generation, turntables) of the 200k-triangle room
        dict(name="room_views", kind="views", scene="room", detail=200_000, views=8),
        # photon mapping + subsurface: hybrid frame over a displaced terrain with glass spheres
        dict(name="terrain_hybrid", kind="hybrid", scene="terrain", detail=500, width=960, height=540, spp=2, depth=16,
             photons=2_000_000, k=50),
        # the photon pass alone: emission, tree build and one density estimate per query point
        dict(name="photon_pass", kind="photons", scene="terrain", detail=500, photons=1_000_000, queries=50_021, k=100),
        # nearest photons with ids and distances for a point set (irradiance caching, analysis)
        dict(name="neighbours", kind="knn", points=500_000, queries=200_003, k=50),
        # guide inference on the hits of a wave: sampled directions and mixture densities
        dict(name="guide_query", kind="guide", rows=1_000_003),
        # one gradient evaluation of the guide at the configured batch size
        dict(name="guide_gradient", kind="train", rows=37_888),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["trace", "trace", "any", "load", "render", "render", "views", "hybrid", "photons", "knn", "guide",
                       "train"])
    if kind in ("trace", "any", "load"):
        scene = rng.choice(["stress", "stress", "cornell", "room"])
        detail = {"cornell": 0, "room": _log(rng, 20_000, 200_000), "stress": rng.randint(4, 8)}[scene]
        if kind == "load" and scene == "cornell":
            scene, detail = "stress", rng.randint(4, 7)
        rays = _log(rng, 1000, 1 << 24 if kind == "trace" else 1 << 22)
        c = dict(kind=kind, scene=scene, detail=detail, rays=rays, mode=rng.choice(["exact", "exact", "fast"]))
        if kind == "any":
            c["bits"] = rng.random() < 0.5
        if kind == "load":
            c["rays"] = min(rays, 1 << 20)
        return c
    if kind == "render":
        scene = rng.choice(["stress", "cornell", "room"])
        detail = {"cornell": 0, "room": _log(rng, 20_000, 200_000), "stress": rng.randint(5, 8)}[scene]
        w = _log(rng, 100, 1920)
        h = max(1, int(w * rng.uniform(0.5, 1.0)))
        spp = min(_log(rng, 1, 64), max(1, (40 * 1920 * 1080) // (w * h)))
        return dict(kind=kind, scene=scene, detail=detail, width=w, height=h, spp=spp, depth=rng.randint(3, 16))
    if kind == "views":
        return dict(kind=kind, scene="room", detail=_log(rng, 20_000, 200_000), views=rng.randint(2, 8))
    if kind == "hybrid":
        w = _log(rng, 100, 960)
        return dict(kind=kind, scene="terrain", detail=_log(rng, 50, 500), width=w, height=max(1, int(w * rng.uniform(0.5, 1.0))),
                    spp=rng.randint(1, 2), depth=rng.randint(4, 16), photons=_log(rng, 100_000, 2_000_000),
                    k=rng.randint(10, 128))
    if kind == "photons":
        return dict(kind=kind, scene="terrain", detail=_log(rng, 50, 500), photons=_log(rng, 10_000, 1_000_000),
                    queries=_log(rng, 1000, 100_000), k=rng.randint(10, 128))
    if kind == "knn":
        return dict(kind=kind, points=_log(rng, 1000, 500_000), queries=_log(rng, 1000, 200_003), k=rng.randint(1, 128))
    if kind == "guide":
        return dict(kind=kind, rows=_log(rng, 500, 2_000_000))
    return dict(kind=kind, rows=_log(rng, 500, 262_144))


# ------------------------------------------------------------------ scenes and inputs


@functools.lru_cache(maxsize=None)
def _context():
    """One context on a torch stream of its own, as a program that mixes both sets it up."""
    torch.cuda.set_device(0)
    ctx = core.Context(0)
    stream = torch.cuda.Stream()
    torch.cuda.set_stream(stream)
    ctx.set_stream(stream.cuda_stream)
    return ctx, stream


@functools.lru_cache(maxsize=3)
def _sphere(subdiv):
    v, f = scenes.icosphere(subdiv)
    return torch.from_numpy(v.astype(np.float32)), np.ascontiguousarray(f.astype(np.uint32))


def _bumpy_sphere(subdiv, seed):
    """Icosphere of radius 0.55 displaced radially by three octaves of trilinear lattice noise
    (amplitude 0.05): (vertices, faces)."""
    v, f = _sphere(subdiv)
    p = v.cuda()
    g = torch.Generator(device="cuda").manual_seed(seed)
    noise = torch.zeros(p.shape[0], device="cuda")
    for o in range(3):
        m = 8 * 2 ** o
        lattice = torch.rand(1, 1, m, m, m, generator=g, device="cuda") * 2 - 1
        at = torch.nn.functional.grid_sample(lattice, p.view(1, 1, 1, -1, 3), align_corners=True)
        noise += at.view(-1) * 0.5 ** o
    p = p * (0.55 * (1 + 0.05 * noise / 1.75))[:, None]
    return np.ascontiguousarray(p.cpu().numpy()), f


def _scene(case, seed, materials):
    """(scene, camera maker) of the case's scene, committed; materials only where rendered."""
    ctx, _ = _context()
    rng = np.random.default_rng(seed)
    name = case["scene"]
    sc = core.Scene(ctx)
    if name == "cornell" or name == "stress":
        extra, bumpy = [], None
        if name == "stress":
            bumpy = _bumpy_sphere(case["detail"], seed)
            if materials:  # GGX roughness per block of 64 triangles
                rough = rng.uniform(0.05, 0.5, (bumpy[1].shape[0] + 63) // 64)
                extra = [core.material(N.RT_MAT_TROWBRIDGE, color=(1, 1, 1), eta=(1.5, 1.5, 1.5), k=(0, 0, 0),
                                       roughness=(float(r), float(r))) for r in rough]
        if materials:
            sc.set_materials(configs.cornell_materials(extra))
        for i, ((v, f), m) in enumerate(scenes.cornell_walls().values()):
            sc.add_mesh(v, f, material=m, shape_id=i)
        if bumpy is not None:
            t0 = sc.add_mesh(*bumpy, material=scenes.MAT_GGX, shape_id=50)
            if materials:
                ids = len(configs.CORNELL_MATERIALS) + np.arange(bumpy[1].shape[0]) // 64
                sc.set_triangle_materials(t0, ids.astype(np.uint32))
        else:
            for j, s in enumerate(scenes.cornell_box()["spheres"]):
                c = np.asarray(s["center"]) + rng.uniform(-0.05, 0.05, 3) * (1, 0, 1)
                o2w, w2o = scenes.sphere_matrices(c, s["radius"])
                sc.add_sphere(o2w, w2o, s["radius"], material=s["material"], shape_id=100 + j)
        eye = rng.uniform(-0.1, 0.1, 3) + (0, 0, 3.5)

        def camera(w, h):
            return core.look_at_camera(tuple(eye), (0, 0, 0), (0, 1, 0), 40.0, w, h)
    elif name == "room":
        meshes, mats = scenes.guiding_room(seed=seed % 100_003, target_triangles=case["detail"])
        if materials:
            table = []
            for m in mats:
                if m["kind"] == "lambert":
                    table.append(core.material(N.RT_MAT_LAMBERTIAN, color=m["albedo"]))
                elif m["kind"] == "ggx":
                    table.append(core.material(N.RT_MAT_TROWBRIDGE, color=(1, 1, 1), eta=(1.5, 1.5, 1.5), k=(0, 0, 0),
                                               roughness=(m["roughness"], m["roughness"])))
                else:
                    table.append(core.material(N.RT_MAT_LIGHT, color=m["emission"], intensity=1.0))
            sc.set_materials(table)
        for i, (v, f, mi) in enumerate(meshes):
            sc.add_mesh(v, f, material=mi, shape_id=i)

        def camera(w, h):
            return core.look_at_camera((0.25, 1.3, 0.75), (-0.8, 0.5, -1.6), (0, 1, 0), 65.0, w, h)
    else:  # the photon scene: terrain, a subsurface slab, 16 glass spheres, two point lights
        (tv, tf), (sv, sf), balls = scenes.photon_terrain(seed=seed % 100_003, n=case["detail"])
        sc.set_materials([
            core.material(N.RT_MAT_LAMBERTIAN, color=(0.6, 0.55, 0.45)),
            core.material(N.RT_MAT_DIELECTRIC, color=(1, 1, 1), ior=1.5, transparent=True),
            core.subsurface_material(kd=(0.9, 0.9, 0.9), ks=(0.04, 0.04, 0.04), ns=40.0, eta=1.3,
                                     sigma_s=(1.0, 0.8, 0.6), sigma_a=(0.01, 0.02, 0.05), g=0.0)])
        sc.add_mesh(tv, tf, material=0, shape_id=0)
        sc.add_mesh(sv, sf, material=2, shape_id=1)
        for j, (c, r) in enumerate(balls):
            o2w, w2o = scenes.sphere_matrices(c, r)
            sc.add_sphere(o2w, w2o, r, material=1, shape_id=100 + j, transparent=True)
        sc.add_point_light((-1.6, 2.6, 1.4), (1.0, 1.0, 1.0), 50.0)
        sc.add_point_light((1.8, 3.2, -1.2), (1.0, 1.0, 1.0), 50.0)

        def camera(w, h):
            return core.look_at_camera((0.0, 2.4, 5.6), (0.0, -0.1, 0.0), (0, 1, 0), 45.0, w, h)
        sc.terrain = tv
    sc.commit()
    return sc, camera


def _bounds(case):
    return ((-1.9, 0.0, -1.9), (1.9, 2.4, 1.9)) if case["scene"] == "room" else ((-1, -1, -1), (1, 1, 1))


def _views(n, seed):
    """Seeded poses in the room. The images' sizes, samples and depths go by n alone: resolution
    log-uniform in [128^2, 1024^2] pixels, aspect 0.5 to 2, 4 to 64 samples, depth 8 to 16."""
    shape, pose = np.random.default_rng(n), np.random.default_rng(seed)
    views = []
    for _ in range(n):
        area, aspect = math.exp(shape.uniform(math.log(128 * 128), math.log(1024 * 1024))), shape.uniform(0.5, 2)
        eye, target = pose.uniform((-1.7, 0.4, -1.7), (1.7, 2.2, 0.8)), pose.uniform((-1.9, 0.0, -1.9), (1.9, 1.5, 0.5))
        cam = core.look_at_camera(tuple(eye), tuple(target), (0, 1, 0), float(pose.uniform(35, 70)),
                                  round(math.sqrt(area * aspect)), round(math.sqrt(area / aspect)))
        views.append(dict(camera=cam, spp=int(shape.choice([4, 8, 16, 32, 64])), max_depth=int(shape.integers(8, 17)),
                          rr_depth=3, seed=int(pose.integers(0, 2 ** 31))))
    return views


def _unit(n, g):
    d = torch.randn(n, 3, generator=g, device="cuda")
    return d / d.norm(dim=1, keepdim=True)


def _uniform(n, lo, hi, g):
    lo, hi = (torch.tensor(x, dtype=torch.float32, device="cuda") for x in (lo, hi))
    return lo + (hi - lo) * torch.rand(n, 3, generator=g, device="cuda")


def _rays(case, seed):
    """(n, 8) device rays. Closest hits: origins uniform in the scene, directions uniform on the
    sphere. Shadow rays: towards points of a ceiling light, as far as the light."""
    n = case["rays"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    lo, hi = _bounds(case)
    o = _uniform(n, lo, hi, g)
    rays = torch.zeros(n, 8, device="cuda")
    rays[:, :3] = o
    if case["kind"] == "any":
        light = _uniform(n, (0.35, 1.0, 1.8), (0.65, 1.3, 1.8), g) if case["scene"] == "room" else \
            _uniform(n, (-0.25, 0.98, -0.25), (0.25, 0.98, 0.25), g)
        d = light - o
        dist = d.norm(dim=1, keepdim=True)
        rays[:, 3:4] = dist
        rays[:, 4:7] = d / dist
    else:
        rays[:, 3] = math.inf
        rays[:, 4:7] = _unit(n, g)
    return rays


GUIDE_LO, GUIDE_HI = (-2.0, 0.0, -2.0), (2.0, 2.5, 2.0)
LAYERS = (144, 64, 64, 64, 64, 48)


def _guide_inputs(case, seed):
    """A guide with seeded weights and a batch of shading points of the room."""
    n = case["rows"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    q = torch.cat([_uniform(n, GUIDE_LO, GUIDE_HI, g), _unit(n, g), _unit(n, g)], 1).contiguous()
    u = torch.rand(n, 3, generator=g, device="cuda")
    wi = _unit(n, g)
    pdf = 0.05 + 0.95 * torch.rand(n, generator=g, device="cuda")
    w = torch.randn(n, generator=g, device="cuda").exp()
    return q, u, wi, pdf, w


def _guide_params(seed):
    """He-uniform hidden layers, a Glorot-uniform output layer, small biases."""
    rng = np.random.default_rng(seed)
    parts = []
    for i, (a, b) in enumerate(zip(LAYERS[:-1], LAYERS[1:])):
        s = math.sqrt(6 / (a + b)) if i == 4 else math.sqrt(6 / a)
        parts += [rng.uniform(-s, s, a * b), rng.uniform(-0.05, 0.05, b)]
    return np.concatenate(parts).astype(np.float32)


def prepare(case, seed):
    ctx, _ = _context()
    kind = case["kind"]
    s = dict(case=case)
    if kind in ("trace", "any"):
        s["scene"], _ = _scene(case, seed, materials=False)
        s["rays"] = _rays(case, seed)
        n = case["rays"]
        if kind == "trace":
            s["hits"] = torch.empty(n, 4, device="cuda")
        elif case["bits"]:
            s["out"] = torch.empty((n + 31) // 32, dtype=torch.int32, device="cuda")
        else:
            s["out"] = torch.empty(n, dtype=torch.uint8, device="cuda")
    elif kind == "load":
        if case["scene"] == "stress":
            s["meshes"] = [(v, f) for (v, f), _ in scenes.cornell_walls().values()] + [_bumpy_sphere(case["detail"], seed)]
        else:
            s["meshes"] = [(v, f) for v, f, _ in scenes.guiding_room(seed % 100_003, case["detail"])[0]]
        r = _rays(case, seed).cpu().numpy()
        s["rays"] = core.make_rays(r[:, :3], r[:, 4:7])
    elif kind in ("render", "views", "hybrid"):
        s["scene"], camera = _scene(case, seed, materials=True)
        s["seed"] = seed % (1 << 31)
        if kind == "views":
            s["views"] = _views(case["views"], seed)
        else:
            s["camera"] = camera(case["width"], case["height"])
        if kind == "hybrid":
            s["map"], _ = s["scene"].trace_photons(case["photons"], max_depth=16, rr_depth=3, seed=s["seed"])
            s["map"].build()
            s["scene"].set_photon_map(s["map"], k=case["k"], radius=100.0)
    elif kind == "photons":
        s["scene"], _ = _scene(case, seed, materials=True)
        s["seed"] = seed % (1 << 31)
        g = torch.Generator(device="cuda").manual_seed(seed)
        tv = torch.from_numpy(s["scene"].terrain).cuda()
        nq = case["queries"]
        s["points"] = tv[torch.randint(0, tv.shape[0], (nq,), generator=g, device="cuda")].contiguous()
        s["normals"] = torch.tensor([0.0, 1.0, 0.0], device="cuda").expand(nq, 3).contiguous()
        d = _unit(nq, g)
        d[:, 1] = d[:, 1].abs() + 0.1
        s["wo"] = (d / d.norm(dim=1, keepdim=True)).contiguous()
        s["material"] = core.material(N.RT_MAT_LAMBERTIAN, color=(0.6, 0.55, 0.45))
    elif kind == "knn":
        g = torch.Generator(device="cuda").manual_seed(seed)
        pts = _uniform(case["points"], (-4, -0.4, -4), (4, 0.4, 4), g)
        s["map"] = core.PhotonMap.from_points(ctx, pts).build()
        s["queries"] = _uniform(case["queries"], (-4, -0.4, -4), (4, 0.4, 4), g)
    else:
        s["guide"] = core.Guide(ctx, GUIDE_LO, GUIDE_HI, learning_rate=1e-3, seed=1)
        s["guide"].set_params(_guide_params(seed))
        s["q"], s["u"], s["wi"], s["pdf"], s["w"] = _guide_inputs(case, seed)
    torch.cuda.synchronize()
    return s


# ------------------------------------------------------------------ the timed calls


def _hits(h):
    return dict(t=h[:, 0], prim=h.view(torch.int32)[:, 1], b=h[:, 2:])


def run(state):
    s, c = state, state["case"]
    kind = c["kind"]
    if kind == "trace":
        s["scene"].trace_closest(s["rays"], s["hits"], c["rays"], flags=N.RT_TRACE_FAST if c["mode"] == "fast" else 0)
        return _hits(s["hits"])
    if kind == "any":
        call = s["scene"].trace_any_bits if c["bits"] else s["scene"].trace_any
        call(s["rays"], s["out"], c["rays"], flags=N.RT_TRACE_FAST if c["mode"] == "fast" else 0)
        return s["out"]
    if kind == "load":
        sc = core.Scene(_context()[0])
        for i, (v, f) in enumerate(s["meshes"]):
            sc.add_mesh(v, f, shape_id=i)
        sc.commit()
        h = sc.trace_closest_host(s["rays"], flags=N.RT_TRACE_FAST if c["mode"] == "fast" else 0)
        sc.close()
        return dict(t=h["t"], prim=h["prim"], b1=h["b1"], b2=h["b2"])
    if kind == "render":
        film, _ = s["scene"].render(s["camera"], spp=c["spp"], max_depth=c["depth"], rr_depth=3, seed=s["seed"],
                                    flags=N.RT_RENDER_NEE_AREA)
        return film
    if kind == "views":
        film, _, _ = s["scene"].render_batch(s["views"], flags=N.RT_RENDER_NEE_AREA)
        return film
    if kind == "hybrid":
        film, _ = s["scene"].render(s["camera"], spp=c["spp"], max_depth=c["depth"], rr_depth=3, seed=s["seed"],
                                    flags=configs.CONFIG4_FLAGS)
        return film
    if kind == "photons":
        pmap, st = s["scene"].trace_photons(c["photons"], max_depth=16, rr_depth=3, seed=s["seed"])
        pmap.build()
        rgb = pmap.density(s["material"], s["points"], s["normals"], s["wo"], c["k"], 100.0)
        pmap.close()
        return dict(stored=int(st["stored"]), rays=int(st["rays"]), rgb=rgb)
    if kind == "knn":
        idx, dist, count = s["map"].knn(s["queries"], c["k"], 100.0)
        return dict(idx=idx, dist=dist, count=count)
    if kind == "guide":
        dirs, density = s["guide"].sample(s["q"], s["u"])
        return dict(dirs=dirs, density=density, pdf=s["guide"].pdf(s["q"], s["wi"], s["pdf"]))
    loss, grad = s["guide"].train_step(s["q"], s["wi"], s["pdf"], s["w"], apply=False, want_grad=True)
    return dict(loss=loss, grad=grad)


# ------------------------------------------------------------------ the work of one pass


def _triangles(case):
    return {"cornell": 12, "stress": 12 + 20 * 4 ** case["detail"], "room": case["detail"],
            "terrain": 2 * case["detail"] ** 2 + 12}[case["scene"]]


def work(case):
    """Each input read and each output written once. A ray is 32 bytes and a hit 16; a scene is 36
    bytes a triangle. Arithmetic: for a ray one 8-wide node per factor of 8 in triangles (8 boxes
    of 12 operations) and two triangle tests of 60."""
    kind = case["kind"]
    tri = _triangles(case) if "scene" in case else 0
    ray = 96 * max(1.0, math.log(max(tri, 8), 8)) + 120
    if kind == "trace":
        return dict(bytes=48 * case["rays"] + 36 * tri, flops=case["rays"] * ray)
    if kind == "any":
        return dict(bytes=32 * case["rays"] + case["rays"] // (8 if case["bits"] else 1) + 36 * tri,
                    flops=case["rays"] * ray)
    if kind == "load":
        return dict(bytes=48 * case["rays"] + 24 * tri, flops=case["rays"] * ray + 200 * tri)
    if kind == "views":
        views = _views(case["views"], 0)
        pixels = [v["camera"].width * v["camera"].height for v in views]
        samples = sum(p * v["spp"] for p, v in zip(pixels, views))
        return dict(bytes=36 * tri + 16 * sum(pixels), flops=samples * 3 * 2 * (ray + 100))
    if kind in ("render", "hybrid"):
        pixels = case["width"] * case["height"]
        bounces = min(case["depth"], 3)
        flops = pixels * case["spp"] * bounces * 2 * (ray + 100)
        size = 36 * tri + 16 * pixels
        if kind == "hybrid":  # an estimate per bounce: k photons of 40 bytes and 40 operations
            flops += pixels * case["spp"] * case["k"] * 40
            size += 0.2 * case["photons"] * 40
        return dict(bytes=size, flops=flops)
    if kind == "photons":
        stored = 0.25 * case["photons"]
        return dict(bytes=36 * tri + 64 * stored + 48 * case["queries"],
                    flops=case["photons"] * 1.3 * (ray + 200) + stored * 100 + case["queries"] * case["k"] * 40)
    if kind == "knn":
        return dict(bytes=12 * case["points"] + (16 + 8 * case["k"]) * case["queries"],
                    flops=case["queries"] * case["k"] * 10)
    weights = sum(a * b for a, b in zip(LAYERS[:-1], LAYERS[1:]))
    if kind == "guide":
        return dict(bytes=case["rows"] * (36 + 12 + 16 + 36 + 16 + 4) + 8 * weights, flops=2 * 2 * weights * case["rows"])
    return dict(bytes=case["rows"] * 56 + 8 * weights, flops=3 * 2 * weights * case["rows"])


# ------------------------------------------------------------------ the same in 64 bits


def _exact_trace(case, seed):
    """Distances to the walls and spheres of the Cornell box by testing each ray with each."""
    rng = np.random.default_rng(seed)
    r = _rays(case, seed).double()
    o, d = r[:, :3], r[:, 4:7]
    best = torch.full((r.shape[0],), math.inf, dtype=torch.float64, device="cuda")
    for (v, f), _ in scenes.cornell_walls().values():
        for tri in torch.from_numpy(v[f.astype(np.int64)]).double().cuda():
            e1, e2 = tri[1] - tri[0], tri[2] - tri[0]
            p = torch.linalg.cross(d, e2.expand_as(d))
            det = (p * e1).sum(1)
            t0 = o - tri[0]
            a = (t0 * p).sum(1) / det
            q = torch.linalg.cross(t0, e1.expand_as(t0))
            b = (d * q).sum(1) / det
            t = (q * e2).sum(1) / det
            ok = (a >= 0) & (b >= 0) & (a + b <= 1) & (t > 0) & (t < best)
            best = torch.where(ok, t, best)
    for s in scenes.cornell_box()["spheres"]:
        c = np.asarray(s["center"]) + rng.uniform(-0.05, 0.05, 3) * (1, 0, 1)
        oc = o - torch.tensor(c.astype(np.float32), device="cuda").double()
        a, b, k = (d * d).sum(1), 2 * (d * oc).sum(1), (oc * oc).sum(1) - float(np.float32(s["radius"])) ** 2
        root = (b * b - 4 * a * k).clamp_min(0).sqrt()
        near, far = (-b - root) / (2 * a), (-b + root) / (2 * a)
        t = torch.where(near > 0, near, far)
        ok = (b * b - 4 * a * k >= 0) & (t > 0) & (t < best)
        best = torch.where(ok, t, best)
    return dict(t=best, prim=None, b=None)


def _encode(q):
    lo, hi = (torch.tensor(x, dtype=torch.float64, device="cuda") for x in (GUIDE_LO, GUIDE_HI))
    u = ((q[:, :3] - lo) / (hi - lo)).clamp(0, 1)
    x = math.pi * u[:, :, None] * 2.0 ** (torch.arange(12, device="cuda", dtype=torch.float64) / 2)
    bands = torch.stack([x.sin(), x.cos()], -1).reshape(-1, 72)
    th = q[:, 8].clamp(-1, 1).acos() / math.pi
    ph = torch.atan2(q[:, 7], q[:, 6]) / (2 * math.pi) + 0.5
    bins = torch.arange(32, device="cuda", dtype=torch.float64) + 0.5
    blobs = [torch.exp(-0.5 * (a[:, None] * 32 - bins) ** 2) for a in (th, ph)]
    return torch.cat([bands, *blobs, q[:, 3:6], torch.zeros_like(q[:, :5])], 1)


def _network(p, q):
    x, at = _encode(q), 0
    for i, (a, b) in enumerate(zip(LAYERS[:-1], LAYERS[1:])):
        x = x @ p[at:at + a * b].view(a, b) + p[at + a * b:at + a * b + b]
        at += a * b + b
        x = x.relu() if i < 4 else x
    return x


def _mixture(o, w):
    """(log density of the vMF mixture at w, guide probability alpha) of raw outputs o."""
    lobe = o[:, :32].view(-1, 8, 4)
    th, ph = math.pi * lobe[..., 0].sigmoid(), 2 * math.pi * lobe[..., 1].sigmoid()
    lk = -4 + 12 * lobe[..., 2].sigmoid()
    k = lk.exp()
    mu = torch.stack([th.sin() * ph.cos(), th.sin() * ph.sin(), th.cos()], -1)
    cos = (mu * w[:, None, :]).sum(-1)
    each = lobe[..., 3].log_softmax(1) + lk - math.log(2 * math.pi) - torch.log(-torch.expm1(-2 * k)) + k * (cos - 1)
    return each.logsumexp(1), 0.05 + 0.9 * o[:, 32].sigmoid()


def exact(case, seed):
    kind = case["kind"]
    _context()
    if kind == "trace" and case["scene"] == "cornell" and case["rays"] <= 1 << 20:
        return _exact_trace(case, seed)
    if kind == "knn" and case["points"] * case["queries"] <= 4e9 and case["points"] >= case["k"]:
        g = torch.Generator(device="cuda").manual_seed(seed)
        pts = _uniform(case["points"], (-4, -0.4, -4), (4, 0.4, 4), g).double()
        q = _uniform(case["queries"], (-4, -0.4, -4), (4, 0.4, 4), g).double()
        dist = [(a[:, None, :] - pts).square().sum(-1).topk(case["k"], largest=False).values.sqrt()
                for a in q.split(max(1, 200_000_000 // case["points"]))]
        return dict(idx=None, dist=torch.cat(dist), count=None)
    if kind in ("guide", "train"):
        p = torch.from_numpy(_guide_params(seed)).double().cuda()
        q, _, wi, pdf, w = (x.double() for x in _guide_inputs(case, seed))
        if kind == "guide":
            out = []
            for a, b, c in zip(q.split(1 << 18), wi.split(1 << 18), pdf.split(1 << 18)):
                logv, alpha = _mixture(_network(p, a), b)
                out.append(alpha * logv.exp() + (1 - alpha) * c)
            return dict(dirs=None, density=None, pdf=torch.cat(out))
        p.requires_grad_(True)
        wt = (w / w.mean()).clamp_max(32)
        logv, alpha = _mixture(_network(p, q), wi)
        density = alpha * logv.exp().detach() + (1 - alpha) * pdf
        loss = (-wt * logv + wt * wt * density.detach() / density).mean()
        loss.backward()
        return dict(loss=loss.item(), grad=p.grad)
    return None
