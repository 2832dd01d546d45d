"""rt_trace_any / rt_trace_any_bits from origins far outside the scene: the decision of the closest
hit along the unbounded ray (Scene::isVisible, Scene.cu:238-276), whatever the distance. An entry
distance of a node is rounded by about 1e-7 of the origin's distance, which there is more than the
margin of its box."""
import numpy as np
import pytest

import cases
from test_trace_gpu import distances_around, make_scene, occlusion_gpu, trace_gpu

pytestmark = pytest.mark.gpu


def scene(name):
    if name == "floor":
        v = np.array([[-1, 0, -1], [1, 0, -1], [1, 0, 1], [-1, 0, 1]], np.float32)
        return v, np.array([[0, 1, 2], [0, 2, 3]], np.uint32)
    if name == "wall":
        v, f = scene("floor")
        return np.ascontiguousarray(v[:, [1, 0, 2]]), f
    return cases.soup(2000, 11)


@pytest.mark.parametrize("away", [1.0, 100.0, 1000.0, 10000.0])
@pytest.mark.parametrize("name", ["floor", "wall", "soup"])
def test_trace_any_from_afar(core, gpu_ctx, name, away):
    v, f = scene(name)
    sc = make_scene(core, gpu_ctx, v, f)
    rng = np.random.default_rng(int(away) + len(name))
    n = 20_011
    lo, hi = v.min(0), v.max(0)
    target = rng.uniform(lo - 0.05, hi + 0.05, (n, 3))
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    o = (target - d * away * np.abs(v).max() * rng.uniform(1.0, 3.0, (n, 1))).astype(np.float32)
    d = d.astype(np.float32)
    ids, t, _ = trace_gpu(sc, o, d)
    hit = ids >= 0
    assert hit.mean() > 0.1
    dist = distances_around(t, hit, rng)
    for flags in (0, core.N.RT_TRACE_SHADOW):
        assert np.array_equal(occlusion_gpu(sc, o, d, dist, flags), hit & (t <= dist))
