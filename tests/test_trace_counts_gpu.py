"""rt_trace_counts over whole warps against one ray per call, where the warp's steps test more triangles
than it has lanes (several rounds of pairs): a ray's counts do not depend on the rays beside it."""
import importlib

import numpy as np
import pytest

import cases
from test_trace_gpu import S, make_scene, trace_counts

N = importlib.import_module("2023_render_engine_b200._native")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags", [0, N.RT_TRACE_COUNT_ANY, N.RT_TRACE_COUNT_ANY | N.RT_TRACE_SHADOW])
def test_trace_counts_do_not_depend_on_the_warp(core, gpu_ctx, flags):
    v, f = cases.soup(3000, 5, spread=0.5, size=0.4)  # a ray meets dozens of leaves
    transparent = np.zeros(f.shape[0], np.uint8)
    transparent[-1000:] = 1  # a mesh of its own
    sc = make_scene(core, gpu_ctx, v, f, transparent=transparent)
    o, d = S.random_rays(320, seed=3, lo=-1.5, hi=1.5)
    nodes, tris = trace_counts(sc, o, d, flags=flags)
    alone = [trace_counts(sc, o[i:i + 1], d[i:i + 1], flags=flags) for i in range(o.shape[0])]
    assert np.array_equal(nodes, [a[0][0] for a in alone])
    assert np.array_equal(tris, [a[1][0] for a in alone])
    if not flags:
        assert np.mean(tris / nodes) > 1  # 32 lanes offer more than 32 pairs a step
