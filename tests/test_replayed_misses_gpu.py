"""Rays that the reference's offset quirk (Triangle.cu:569-593) makes miss although a triangle is hit: the walk
finds the triangle, the replay of the reference's traversal decides, and the hit keeps the walk's barycentrics
whichever kernel ends it."""
import importlib

import numpy as np
import pytest

import cases
from test_trace_gpu import make_scene, trace_gpu

N = importlib.import_module("2023_render_engine_b200._native")

pytestmark = pytest.mark.gpu


def quads(n, z):
    """n quads at height z, side by side along x, and one below them all."""
    v, f = [], []
    for i in range(n):
        a = 4 * i
        x0, x1 = 2.0 * i - n, 2.0 * i - n + 2.0
        v += [[x0, -1, z], [x1, -1, z], [x1, 1, z], [x0, 1, z]]
        f += [[a, a + 1, a + 2], [a, a + 2, a + 3]]
    a = len(v)
    v += [[-n, -1, z - 1], [n, -1, z - 1], [n, 1, z - 1], [-n, 1, z - 1]]
    f += [[a, a + 1, a + 2], [a, a + 2, a + 3]]
    return np.array(v, np.float32), np.array(f, np.uint32)


@pytest.mark.parametrize("copies", [1, 400])  # a short queue, and one of several rays per lane
@pytest.mark.parametrize("n", [1, 40])  # a scene of one node, and of several
def test_barycentrics_of_replayed_misses(core, gpu_ctx, n, copies):
    v, f = quads(n, np.float32(0.7))
    sc = make_scene(core, gpu_ctx, v, f)
    rng = np.random.default_rng(n)
    m = 600
    o = np.empty((m, 3), np.float32)
    o[:, 0] = rng.uniform(-n, n, m)
    o[:, 1] = rng.uniform(-0.9, 0.9, m)
    o[:, 2] = np.float32(0.7) + rng.choice([1e-7, 2e-7, 1e-6, 1e-3], m).astype(np.float32)  # within its error bound
    d = rng.normal(size=(m, 3)).astype(np.float32)
    d[:, 2] = -np.abs(d[:, 2]) - 0.2
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    o, d = np.tile(o, (copies, 1)), np.tile(d.astype(np.float32), (copies, 1))
    ids, _, exact = trace_gpu(sc, o, d)
    fast_ids, _, fast = trace_gpu(sc, o, d, flags=N.RT_TRACE_FAST)
    missed = (ids < 0) & (fast_ids >= 0)
    assert missed.sum() >= 10 * copies
    for b in ("b1", "b2"):
        assert np.array_equal(exact[b][missed], fast[b][missed])
