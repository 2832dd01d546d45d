"""Frames whose depth limit lies well above where their paths end, on either side of the limit up to which
the waves are launched without a loop."""
import importlib
import time

import numpy as np
import pytest

N = importlib.import_module("2023_render_engine_b200._native")
configs = importlib.import_module("2023_render_engine_b200.configs")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("depth", [1, 3, 4, 5, 8, 9, 16, 31, 32, 33, 64])
@pytest.mark.parametrize("view", ["box", "away"])
def test_waves_and_film_are_the_host_loops(core, gpu_ctx, view, depth):
    """Same waves, rays and samples as with the host's look after every group (RT_RENDER_HOST_LOOP); sums
    agree to the order of their additions."""
    sc, cam, _ = configs.build_config0(gpu_ctx, 48, 40)
    if view == "away":  # no path survives its first wave
        cam = core.look_at_camera((0, 0, 3.5), (0, 0, 9.0), (0, 1, 0), 40.0, 48, 40)
    args = dict(spp=3, max_depth=depth, rr_depth=2, seed=7, fp64=True)
    a, sa = sc.render(cam, **args)
    b, sb = sc.render(cam, flags=N.RT_RENDER_HOST_LOOP, **args)
    for k in ("waves", "extension_rays", "shadow_rays", "camera_rays"):
        assert sa[k] == sb[k], k
    ia, ib = core.film_mean(a), core.film_mean(b)
    assert np.allclose(ia, ib, rtol=1e-5, atol=1e-7)


@pytest.mark.parametrize("shape", [(64, 64, 1), (1920, 1080, 1), (1920, 1080, 8)])
def test_a_deep_limit_costs_little_where_paths_end_early(core, gpu_ctx, shape):
    w, h, spp = shape
    sc, _, _ = configs.build_config0(gpu_ctx, w, h)
    cam = core.look_at_camera((0, 0, 3.5), (0, 0, 9.0), (0, 1, 0), 40.0, w, h)

    def best(depth):
        t = []
        for _ in range(9):
            t0 = time.perf_counter()
            sc.render(cam, spp=spp, max_depth=depth, rr_depth=2, seed=7)
            t.append(time.perf_counter() - t0)
        return min(t)

    best(8)
    assert best(32) < 1.5 * best(8)  # two groups of waves, whatever the limit; eight took 2 to 4 times as long
    assert best(64) < 2.5 * best(8)
