"""Scenes of a few nodes, whose calls run in one kernel of their own (closest hits on one node, occlusion on
up to four), against the reference's closest hits: from no triangle to just beyond those sizes, with up to
one shape more than that kernel takes, at ragged counts of rays."""
import importlib

import numpy as np
import pytest

import cases
from test_trace_gpu import S, distances_around, make_scene, occlusion_gpu, trace_gpu

N = importlib.import_module("2023_render_engine_b200._native")
scenes = importlib.import_module("2023_render_engine_b200.scenes")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spheres", [0, 1, 4, 5])
@pytest.mark.parametrize("ntri", [0, 1, 2, 3, 12, 24, 40, 100])
def test_tiny_scenes(core, gpu_ctx, restated, ntri, spheres):
    v, f = cases.soup(max(ntri, 1), 5 + ntri, size=0.5)
    f = f[:ntri]
    tr = (np.arange(ntri) % 3 == 2).astype(np.uint8)
    balls = []
    for j in range(spheres):
        o2w, w2o = scenes.sphere_matrices((0.5 * j - 1.0, 0.2 * j, 0.1), 0.3)
        balls.append(dict(o2w=o2w, w2o=w2o, radius=0.3, glass=j % 2 == 1))
    # the shapes' own answer, in a scene without triangles and with one shape at a time
    rng = np.random.default_rng(ntri)
    o, d = S.random_rays(4099, seed=ntri + spheres, lo=-1.5, hi=1.5)
    d[::16] = np.eye(3, dtype=np.float32)[rng.integers(0, 3, d[::16].shape[0])]  # axis-parallel too
    sc = make_scene(core, gpu_ctx, v, f, transparent=tr if ntri else None, spheres=balls)
    for shadow in (False, True):
        flags = N.RT_TRACE_SHADOW if shadow else 0
        if ntri:
            prim, t = restated.bvh(v, f, tr).intersect(o, d, shadow=shadow)
            prim, t = prim.astype(np.int64), np.where(prim >= 0, t, np.inf).astype(np.float32)
        else:
            prim, t = np.full(len(o), -1, np.int64), np.full(len(o), np.inf, np.float32)
        for j, b in enumerate(balls):
            if shadow and b["glass"]:
                continue
            _, ts, hs = trace_gpu(make_scene(core, gpu_ctx, np.zeros((0, 3), np.float32), np.zeros((0, 3), np.uint32),
                                             spheres=[dict(b, glass=False)]), o, d)
            nearer = (hs["prim"] >= 0) & (ts < t)
            prim, t = np.where(nearer, N.RT_PRIM_SHAPE | j, prim), np.where(nearer, ts, t)
        for n in (1, 31, 33, 4099):
            ids, tt, _ = trace_gpu(sc, o[:n], d[:n], flags=flags)
            assert np.array_equal(ids, prim[:n])
            assert np.array_equal(tt[ids >= 0], t[:n][ids >= 0])
        hit = prim >= 0
        dist = distances_around(t, hit, rng)
        assert np.array_equal(occlusion_gpu(sc, o, d, dist, flags), hit & (t <= dist))
        # fast mode: the same away from the reference's offset quirk and the boundary
        ids, tt, _ = trace_gpu(sc, o, d, flags=flags | N.RT_TRACE_FAST)
        assert (ids == prim).mean() > 0.999
        away = ~hit | (np.abs(dist - t) > 1e-5 * np.maximum(t, 1))
        fast = occlusion_gpu(sc, o, d, dist, flags | N.RT_TRACE_FAST)
        assert (fast[away] == (hit & (t <= dist))[away]).mean() > 0.999
