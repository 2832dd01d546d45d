"""Short ray queues, traced in one launch, against the same rays in a long queue (two launches)."""
import importlib

import numpy as np
import pytest
import torch

import cases

pytestmark = pytest.mark.gpu

N = importlib.import_module("2023_render_engine_b200._native")
S = importlib.import_module("2023_render_engine_b200.scenes")

LONG = 400_000  # above 32 rays per warp of the device
SIZES = [1, 2, 15, 16, 17, 31, 33, 997, 5000, 20_001, 150_000, 170_495, 170_496, 170_497, LONG - 1]


@pytest.fixture(scope="module", params=["box with spheres", "stacked grids"])
def traced(request, core, gpu_ctx):
    sc = core.Scene(gpu_ctx)
    if request.param == "stacked grids":  # equal offsets, replays of the reference's traversal
        sc.add_mesh(*cases.stacked_grids())
    else:
        box = S.cornell_box()
        v, f, _ = S.flatten(box)
        sc.add_mesh(v, f)
        for j, s in enumerate(box["spheres"]):
            o2w, w2o = S.sphere_matrices(s["center"], s["radius"])
            sc.add_sphere(o2w, w2o, s["radius"], material=0, shape_id=j, transparent=j == 0)
    sc.commit()
    o, d = S.random_rays(LONG, seed=3, lo=-1.2, hi=1.2)
    eo, ed = cases.edge_rays(4)
    o[: len(eo)], d[: len(ed)] = eo, ed
    tmax = np.full(LONG, np.inf, np.float32)
    tmax[5::7] = 0.7
    rays = torch.from_numpy(core.make_rays(o, d, tmax).view(np.float32).reshape(-1)).cuda()
    yield sc, rays
    sc.close()


@pytest.mark.parametrize("flags", [0, N.RT_TRACE_SHADOW, N.RT_TRACE_FAST, N.RT_TRACE_FAST | N.RT_TRACE_SHADOW])
def test_short_queues_give_the_long_queues_hits(traced, flags):
    sc, rays = traced
    want = torch.empty(LONG * 4, dtype=torch.float32, device="cuda")
    sc.trace_closest(rays, want, LONG, flags=flags)
    want = want.view(torch.int32).view(LONG, 4)
    replays = []
    for n in SIZES:
        got = torch.full((n * 4 + 4,), -7.0, dtype=torch.float32, device="cuda")
        sc.trace_closest(rays, got, n, flags=flags)
        assert torch.equal(got[: 4 * n].view(torch.int32).view(n, 4), want[:n]), n
        assert (got[4 * n:] == -7.0).all()
        replays.append(sc.trace_stats()["exact_fallback_rays"])
        assert sc.trace_stats()["rays"] == n
    assert replays == sorted(replays)  # the counters start from zero in every call
