"""Meshes whose boxes have no finite area (an infinite vertex, or one so far out that squares of the boxes'
margin overflow): the clustering finds no neighbours, and the commit is refused."""
import importlib

import numpy as np
import pytest

import cases
from test_trace_gpu import S, make_scene, trace_gpu

N = importlib.import_module("2023_render_engine_b200._native")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [np.inf, 3e38, 1e25])
@pytest.mark.parametrize("n", [2, 100, 4096, 5000])  # clustered in one block, and in rounds before that
def test_commit_is_refused(core, gpu_ctx, n, value):
    v, f = cases.soup(n, 3)
    good = make_scene(core, gpu_ctx, v, f)
    o, d = S.random_rays(500, seed=1, lo=-1.0, hi=1.0)
    want = trace_gpu(good, o, d)[0]
    v[len(v) // 2] = value
    sc = core.Scene(gpu_ctx)
    sc.add_mesh(v, f)
    with pytest.raises(N.RtError):
        sc.commit()
    sc.close()
    assert np.array_equal(trace_gpu(good, o, d)[0], want)
    assert np.array_equal(trace_gpu(make_scene(core, gpu_ctx, *cases.soup(n, 3)), o, d)[0], want)
